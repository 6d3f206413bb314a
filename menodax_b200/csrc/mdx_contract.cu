// The backward of a forward-sensitivity solve: out[i, k] = sum over saves s and
// states r of cotangent[i, s, r] * S[i, s, r, k], S read from the joint history where
// the solve wrote it (state, then one block of n_vars per direction).
//
// One thread per trajectory and direction; the threads of a trajectory read one
// contiguous stretch of its row per save, so the pass is one read of the history.  What
// bounds it is the latency of a thread's loads over the saves: 57% of the card's copy
// rate.  The general contraction first transposed and copied the sensitivities,
// then ran two batched products: for 65,536 trajectories of a two-state system with
// 20 saves on a B200 about 400 us, against 28 us here (105 MB at 3.7 TB/s); with a wait
// for the save times gone too, the gradient call 3.13 -> 2.53 ms.
#include "../../include/menodax.h"
#include "mdx_internal.h"

#include <cuda_runtime.h>

namespace {

constexpr int THREADS = 256;

__global__ void __launch_bounds__(THREADS) contract(const double* __restrict__ joint, const double* __restrict__ cotangent,
                                                    long long total, int n_save, int n_vars, int n_sens, int n_first,
                                                    double* __restrict__ first, double* __restrict__ rest) {
  const long long at = (long long)blockIdx.x * THREADS + threadIdx.x;
  if (at >= total) return;
  const long long i = at / n_sens;
  const int k = (int)(at - i * n_sens);
  const int width = n_vars * (1 + n_sens);
  const double* s = joint + (size_t)i * n_save * width + (size_t)n_vars * (1 + k);
  const double* g = cotangent + (size_t)i * n_save * n_vars;
  double acc = 0.0;
  for (int save = 0; save < n_save; ++save, s += width, g += n_vars)
    for (int r = 0; r < n_vars; ++r) acc += __ldg(g + r) * __ldg(s + r);
  if (k < n_first) first[(size_t)i * n_first + k] = acc;
  else rest[(size_t)i * (n_sens - n_first) + (k - n_first)] = acc;
}

}  // namespace

extern "C" int mdx_sens_contract(const double* joint, const double* cotangent, int n_traj, int n_save, int n_vars,
                                 int n_sens, int n_first, double* first, double* rest, void* stream) {
  if (n_traj < 0 || n_save < 1 || n_vars < 1 || n_sens < 1 || n_first < 0 || n_first > n_sens)
    return mdx_internal::fail_message(MDX_E_INVALID, "mdx_sens_contract: bad sizes");
  if (n_traj == 0) return MDX_OK;
  if (!joint || !cotangent || (n_first > 0 && !first) || (n_first < n_sens && !rest))
    return mdx_internal::fail_message(MDX_E_INVALID, "mdx_sens_contract: a required buffer is NULL");
  const long long total = (long long)n_traj * n_sens;
  const long long blocks = (total + THREADS - 1) / THREADS;
  if (blocks > 0x7fffffffLL)
    return mdx_internal::fail_message(MDX_E_INVALID, "mdx_sens_contract: too many trajectories and directions");
  contract<<<(unsigned)blocks, THREADS, 0, (cudaStream_t)stream>>>(joint, cotangent, total, n_save, n_vars, n_sens,
                                                                  n_first, first, rest);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return mdx_internal::fail_message(MDX_E_CUDA, cudaGetErrorString(e));
  return MDX_OK;
}
