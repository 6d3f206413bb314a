"""The kernels' scalar arithmetic, compiled for the host: division by a kept
reciprocal, the controller's roots and its accept test, against IEEE results."""

import ctypes
import subprocess

import numpy as np
import pytest

from menodax_b200._native import KERNEL_DIR

from test_lu_host import PRELUDE, _p

SOURCE = """
#include "mdx_dense_lu.cuh"
#define DIV(T) extern "C" void div_##T(const T* a, const T* d, T* q, int n) { \\
  for (int i = 0; i < n; ++i) { const T r = (T)(1.0 / (double)d[i]); q[i] = mdx::div_by<T>(a[i], r == 0 ? (T)0 : d[i], r); } }
DIV(double) DIV(float)
extern "C" void root(const double* x, double* y, int n, int order) {
  for (int i = 0; i < n; ++i) y[i] = order == 5 ? mdx::inverse_root<10>(x[i]) : mdx::inverse_root<12>(x[i]);
}
template <int ORDER> void controller(const double* sums, double n_err, double* factor, int* accept, int n) {
  for (int i = 0; i < n; ++i) {
    bool ok; double safe;
    factor[i] = mdx::controller_factor<ORDER>(sums[i], n_err, 1.0, 1.0, -1.0 / ORDER, 0.0, 0.0, false, false, ok, safe);
    accept[i] = ok;
  }
}
extern "C" void controller5(const double* s, double n_err, double* f, int* ok, int n) { controller<5>(s, n_err, f, ok, n); }
extern "C" void controller6(const double* s, double n_err, double* f, int* ok, int n) { controller<6>(s, n_err, f, ok, n); }
#define SOLVE(T, N) extern "C" void solve_##T##N(const T* a, const T* b, T* x, int t, int recip) { \\
  T lu[N * N + N]; int piv[N]; T r[N]; for (int i = 0; i < N * N; ++i) lu[i] = a[i]; for (int i = 0; i < N; ++i) r[i] = b[i]; \\
  if (recip) { mdx::dense_factorize<N, T, true>(lu, piv); \\
    if (t) mdx::dense_solve_t<N, T, true>(lu, piv, r); else mdx::dense_solve<N, T, true>(lu, piv, r); } \\
  else { mdx::dense_factorize<N, T>(lu, piv); \\
    if (t) mdx::dense_solve_t<N, T>(lu, piv, r); else mdx::dense_solve<N, T>(lu, piv, r); } \\
  for (int i = 0; i < N; ++i) x[i] = r[i]; }
SOLVE(double, 2) SOLVE(double, 3) SOLVE(double, 20) SOLVE(float, 3) SOLVE(float, 20)
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    path = tmp_path_factory.mktemp("scalar")
    (path / "s.cpp").write_text(PRELUDE + SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-w", f"-I{KERNEL_DIR}",
                    str(path / "s.cpp"), "-o", str(path / "s.so")], check=True)
    return ctypes.CDLL(str(path / "s.so"))


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_division_by_a_kept_reciprocal_rounds_like_a_division(lib, dtype):
    rng = np.random.default_rng(1)
    n = 200_000
    low, high = (-200, 200) if dtype is np.float64 else (-25, 25)
    a = (rng.choice([-1.0, 1.0], n) * np.exp2(rng.uniform(low, high, n))).astype(dtype)
    d = (rng.choice([-1.0, 1.0], n) * np.exp2(rng.uniform(low, high, n))).astype(dtype)
    a[:4], d[:4] = [0.0, 1.0, np.nan, 3.0], [2.0, np.inf, 1.0, 3.0]
    q = np.empty_like(a)
    getattr(lib, "div_double" if dtype is np.float64 else "div_float")(_p(a), _p(d), _p(q), n)
    np.testing.assert_array_equal(q, a / d)


@pytest.mark.parametrize("order", [5, 6])
def test_controller_root_and_accept(lib, order):
    rng = np.random.default_rng(2)
    x = np.exp2(rng.uniform(np.log2(1e-36), np.log2(1e36), 100_000))
    y = np.empty_like(x)
    lib.root(_p(x), _p(y), len(x), order)
    exact = np.power(x.astype(np.longdouble), -1 / np.longdouble(2 * order))
    assert np.max(np.abs(y / exact - 1)) < 6 * 2.0 ** -53   # the last Newton step's four roundings
    for n_err in (1.0, 3.0, 8.0):
        near = n_err * (1.0 + np.arange(-8, 9) * 2.0 ** -53)
        sums = np.concatenate([near, [0.0, 1e-40, 1e40, np.inf, np.nan], np.exp2(rng.uniform(-60, 60, 1000))])
        factor, ok = np.empty_like(sums), np.empty(len(sums), dtype=np.int32)
        getattr(lib, f"controller{order}")(_p(sums), ctypes.c_double(n_err), _p(factor), _p(ok), len(sums))
        norm = np.sqrt(sums / n_err)
        np.testing.assert_array_equal(ok != 0, norm <= 1.0)
        safe = np.where(np.isnan(norm) | (norm > 1e18), 1e18, np.where(norm == 0.0, 1e-18, norm))
        limit = np.clip(0.9 * safe ** (-1.0 / order), 0.2, 10.0)
        np.testing.assert_allclose(np.clip(factor, 0.2, 10.0), limit, rtol=1e-14)


@pytest.mark.parametrize("t,n", [("double", 2), ("double", 3), ("double", 20), ("float", 3), ("float", 20)])
def test_kept_pivots_solve_to_the_same_bits(lib, t, n):
    dtype = np.float64 if t == "double" else np.float32
    rng = np.random.default_rng(n)
    run = getattr(lib, f"solve_{t}{n}")
    for _ in range(50):
        a, b = rng.normal(size=(n, n)).astype(dtype), rng.normal(size=n).astype(dtype)
        for transposed in (0, 1):
            x, y = np.empty_like(b), np.empty_like(b)
            run(_p(a), _p(b), _p(x), transposed, 1)
            run(_p(a), _p(b), _p(y), transposed, 0)
            np.testing.assert_array_equal(x, y)


CLOSED = """
#include "mdx_dense_lu.cuh"
#define CLOSED(N) extern "C" void closed##N(const double* a, const double* b, double* x, double* xt) { \\
  double m[N * N], r[N], rt[N]; for (int i = 0; i < N * N; ++i) m[i] = a[i]; for (int i = 0; i < N; ++i) r[i] = rt[i] = b[i]; \\
  mdx::closed_inverse<N>(m); mdx::inverse_solve<N, false>(m, r); mdx::inverse_solve<N, true>(m, rt); \\
  for (int i = 0; i < N; ++i) { x[i] = r[i]; xt[i] = rt[i]; } }
CLOSED(1) CLOSED(2) CLOSED(3)
"""


@pytest.mark.parametrize("n", [1, 2, 3])
def test_closed_inverse(tmp_path, n):
    """Row-scaled random matrices against NumPy: an entry is a few products over the
    determinant, so the inverse is off by at most about 8 n roundings times the condition number;
    a determinant past the range of a double gives NaN, not the zero that would pass an error
    test."""
    (tmp_path / "c.cpp").write_text(PRELUDE + CLOSED)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-w", f"-I{KERNEL_DIR}", str(tmp_path / "c.cpp"),
                    "-o", str(tmp_path / "c.so")], check=True)
    run = getattr(ctypes.CDLL(str(tmp_path / "c.so")), f"closed{n}")
    rng = np.random.default_rng(n)
    x, xt = np.empty(n), np.empty(n)
    for _ in range(300):
        a = rng.normal(size=(n, n)) * np.exp(rng.uniform(-12, 12, (n, 1)))
        b = rng.normal(size=n)
        run(_p(a), _p(b), _p(x), _p(xt))
        inv = np.linalg.inv(a)
        bound = 16 * n * 2.0 ** -53 * np.linalg.cond(a) * np.linalg.norm(inv) * np.linalg.norm(b)
        assert np.linalg.norm(x - np.linalg.solve(a, b)) <= bound
        assert np.linalg.norm(xt - np.linalg.solve(a.T, b)) <= bound
    run(_p(np.eye(n) * 1e200 if n > 1 else np.array([[np.inf]])), _p(np.ones(n)), _p(x), _p(xt))
    assert np.isnan(x).all()


@pytest.mark.parametrize("modes", [1, 2])
def test_closed_inverse_of_fast_modes_is_as_accurate_as_an_lu(tmp_path, lib, modes):
    """M = I + s u v^T (one fast reaction that couples all three states, and a second at
    sqrt(s)), in states of very different sizes: an LU loses eps s of a solve, cofactors of the
    whole matrix eps s^2.  The two orders of elimination round differently, by less than a
    factor of four in the median of 50."""
    from fractions import Fraction

    (tmp_path / "c.cpp").write_text(PRELUDE + CLOSED)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-w", f"-I{KERNEL_DIR}",
                    str(tmp_path / "c.cpp"), "-o", str(tmp_path / "c.so")], check=True)
    run = ctypes.CDLL(str(tmp_path / "c.so")).closed3
    rng = np.random.default_rng(modes)

    def exact(m, b):  # Cramer's rule in rational numbers
        m = [[Fraction(v) for v in row] for row in m]
        det = lambda a: (a[0][0] * (a[1][1] * a[2][2] - a[1][2] * a[2][1])  # noqa: E731
                         - a[0][1] * (a[1][0] * a[2][2] - a[1][2] * a[2][0])
                         + a[0][2] * (a[1][0] * a[2][1] - a[1][1] * a[2][0]))
        whole = det(m)
        return np.array([float(det([[Fraction(b[i]) if k == j else m[i][k] for k in range(3)] for i in range(3)]) / whole)
                         for j in range(3)])

    for s in 10.0 ** np.arange(0, 11):
        errors = []
        for _ in range(50):
            m = np.eye(3)
            for size in (s, np.sqrt(s))[:modes]:
                u, v = rng.normal(size=(2, 3))
                m += size * np.outer(u, v if u @ v > 0 else -v)
            scale = np.exp(rng.uniform(-10, 10, 3))
            m *= scale[None, :] / scale[:, None]
            b, x, xt, y, yt = rng.normal(size=3), *np.empty((4, 3))
            run(_p(m), _p(b), _p(x), _p(xt))
            lib.solve_double3(_p(m), _p(b), _p(y), 0, 0)
            lib.solve_double3(_p(m), _p(b), _p(yt), 1, 0)
            right, right_t = exact(m, b), exact(m.T, b)
            errors.append([np.linalg.norm(got - ref) / np.linalg.norm(ref)
                           for got, ref in ((x, right), (y, right), (xt, right_t), (yt, right_t))])
        closed, lu, closed_t, lu_t = np.median(errors, axis=0)
        assert closed <= 4 * max(lu, 2.0 ** -53) and closed_t <= 4 * max(lu_t, 2.0 ** -53), s
