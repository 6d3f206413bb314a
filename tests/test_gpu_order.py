"""The native visiting order: a permutation, longest first."""

import pytest
import torch

from menodax_b200 import autotune

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 2048, 2049, 70001])
@pytest.mark.parametrize("high", [1, 200, 256, 5000, 2**31 - 1])
def test_longest_first_is_a_sorted_permutation(n, high):
    gen = torch.Generator(device="cuda").manual_seed(n + high)
    steps = torch.randint(0, high, (n,), generator=gen, device="cuda", dtype=torch.int64).to(torch.int32)
    steps[-1] = high - 1
    order = autotune.longest_first(steps).long()
    assert torch.equal(order.sort().values, torch.arange(n, device="cuda"))
    seen = steps[order].double()
    # Nothing later is longer by more than a bucket: exact below 256, one part in 128 above.
    longest_after = seen.flip(0).cummax(0).values.flip(0)
    slack = torch.where(seen < 256, torch.zeros_like(seen), seen / 128)
    assert bool((longest_after <= seen + slack).all())
