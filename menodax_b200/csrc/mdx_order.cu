// The visiting order of a persistent launch: trajectories by descending step count.
//
// A counting sort over buckets of step counts, exact up to 256 steps and within
// one part in 128 above, in no particular order inside a bucket: what the order is
// for -- long integrations first, warps of about equal length -- needs no more, and
// no result depends on it.  Every persistent solve pays for it, and launches bound
// it: two and a memset here, against a general stable sort's thirteen kernels, copies
// and memsets.  Whole calls on a B200: Robertson, 65,536 trajectories, 576 -> 524
// us; Lorenz, 250,007, 957 -> 901.
#include "../../include/menodax.h"
#include "mdx_internal.h"

#include <cuda_runtime.h>

namespace {

constexpr int EXACT = 256;                        // counts below have a bucket each
constexpr int BUCKETS = EXACT + (31 - 8) * 128;   // then 128 per power of two
constexpr int THREADS = 256;
constexpr int PER_BLOCK = 2048;                   // trajectories a block takes

__device__ __forceinline__ int bucket_of(int steps) {
  if (steps < EXACT) return steps < 0 ? 0 : steps;
  const int e = 31 - __clz(steps);
  return EXACT + (e - 8) * 128 + ((steps >> (e - 7)) - 128);
}

__global__ void __launch_bounds__(THREADS) count_steps(const int* steps, int n, int* counts) {
  __shared__ int mine[BUCKETS];
  for (int b = threadIdx.x; b < BUCKETS; b += THREADS) mine[b] = 0;
  __syncthreads();
  const int first = blockIdx.x * PER_BLOCK;
  const int end = min(n, first + PER_BLOCK);
  for (int i = first + threadIdx.x; i < end; i += THREADS) atomicAdd(&mine[bucket_of(steps[i])], 1);
  __syncthreads();
  for (int b = threadIdx.x; b < BUCKETS; b += THREADS)
    if (mine[b]) atomicAdd(&counts[b], mine[b]);
}

// Each block finds where every bucket starts (the trajectories of longer ones come
// before it), takes room in each for its own, and places them.
__global__ void __launch_bounds__(THREADS) place(const int* steps, int n, const int* counts, int* taken, int* order) {
  __shared__ int mine[BUCKETS];
  __shared__ int at[BUCKETS];
  __shared__ int sums[THREADS];
  constexpr int EACH = (BUCKETS + THREADS - 1) / THREADS;
  for (int b = threadIdx.x; b < BUCKETS; b += THREADS) mine[b] = 0;
  // Thread k sums a run of buckets from the longest down, then scans the sums.
  int sum = 0;
  for (int j = 0; j < EACH; ++j) {
    const int b = BUCKETS - 1 - ((int)threadIdx.x * EACH + j);
    if (b >= 0) sum += counts[b];
  }
  sums[threadIdx.x] = sum;
  __syncthreads();
  for (int d = 1; d < THREADS; d *= 2) {
    const int before = (int)threadIdx.x >= d ? sums[threadIdx.x - d] : 0;
    __syncthreads();
    sums[threadIdx.x] += before;
    __syncthreads();
  }
  int start = sums[threadIdx.x] - sum;
  for (int j = 0; j < EACH; ++j) {
    const int b = BUCKETS - 1 - ((int)threadIdx.x * EACH + j);
    if (b >= 0) {
      at[b] = start;
      start += counts[b];
    }
  }
  const int first = blockIdx.x * PER_BLOCK;
  const int end = min(n, first + PER_BLOCK);
  for (int i = first + threadIdx.x; i < end; i += THREADS) atomicAdd(&mine[bucket_of(steps[i])], 1);
  __syncthreads();
  for (int b = threadIdx.x; b < BUCKETS; b += THREADS)
    if (mine[b]) at[b] += atomicAdd(&taken[b], mine[b]);
  __syncthreads();
  for (int i = first + threadIdx.x; i < end; i += THREADS) order[atomicAdd(&at[bucket_of(steps[i])], 1)] = i;
}

}  // namespace

extern "C" {

int mdx_order_workspace_size(size_t* bytes) {
  if (!bytes) return mdx_internal::fail_message(MDX_E_INVALID, "mdx_order_workspace_size: null argument");
  *bytes = 2 * BUCKETS * sizeof(int);
  return MDX_OK;
}

int mdx_order_longest_first(const int* steps, int n, int* order, void* workspace, size_t workspace_bytes, void* stream) {
  if (n < 0) return mdx_internal::fail_message(MDX_E_INVALID, "mdx_order_longest_first: n must be non-negative");
  if (n == 0) return MDX_OK;
  if (!steps || !order || !workspace)
    return mdx_internal::fail_message(MDX_E_INVALID, "mdx_order_longest_first: a required buffer is NULL");
  if (workspace_bytes < 2 * BUCKETS * sizeof(int))
    return mdx_internal::fail_message(MDX_E_INVALID, "mdx_order_longest_first: the workspace is too small");
  cudaStream_t s = (cudaStream_t)stream;
  int* counts = (int*)workspace;
  const int blocks = (n - 1) / PER_BLOCK + 1;
  cudaError_t e = cudaMemsetAsync(counts, 0, 2 * BUCKETS * sizeof(int), s);
  if (e == cudaSuccess) {
    count_steps<<<blocks, THREADS, 0, s>>>(steps, n, counts);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) {
    place<<<blocks, THREADS, 0, s>>>(steps, n, counts, counts + BUCKETS, order);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) return mdx_internal::fail_message(MDX_E_CUDA, cudaGetErrorString(e));
  return MDX_OK;
}

}  // extern "C"
