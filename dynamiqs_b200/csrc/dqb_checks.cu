// Hermiticity defect ||rho - rho^+||_F / ||rho||_F of saved states, in FP64.
//
// Bound: HBM, every state read once (the FP64 conversions, 16 per SM and cycle, come next).
// A block takes the tile pair (ti, tj), (tj, ti) of 32 x 32 tiles, ti <= tj, reads both row
// by row and meets the mirror through shared memory, so that no transposed or converted copy
// of the states is made: the chain of array operations this replaces converted to
// complex128, transposed, subtracted and took two norms, nine times the bytes.  States are
// split over as many blocks as fill the chip (few large states), each block adding up its
// pairs, and a second kernel adds the blocks' sums in order (deterministic).
//
// Measured (one B200), with the launches: 6 states of n = 4096: 2.21 -> 0.16 ms; 11264 of
// n = 64: 1.00 -> 0.10 ms; 101 of n = 16: eight launches -> two.
#include <cuda_runtime.h>

#include <algorithm>

#include "dqb_common.cuh"

namespace dqb {
namespace {

constexpr int kCT = 32;

// blockIdx.x = state * blocks + part; partial[blockIdx.x] = (sum |rho - rho^+|^2, sum |rho|^2)
// over the part's tile pairs.
__global__ void __launch_bounds__(256) herm_partial_kernel(const float2* __restrict__ states, int n, int blocks,
                                                           double2* __restrict__ partial) {
  __shared__ float2 sh[kCT][kCT + 1];
  __shared__ double red[72];
  const long long s = blockIdx.x / blocks;
  const float2* __restrict__ M = states + s * n * n;
  const int T = (n + kCT - 1) / kCT, pairs = T * (T + 1) / 2;
  const int lx = threadIdx.x & 31, ly = threadIdx.x >> 5;
  double num = 0.0, den = 0.0;
  int p = (int)(blockIdx.x % blocks), ti = 0, at = 0;  // row ti of the pairs starts at `at`
  for (; p < pairs; p += blocks) {
    while (p - at >= T - ti) at += T - ti, ++ti;
    const int tj = ti + p - at;
    __syncthreads();  // the previous pair's tile has been read
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = tj * kCT + ly + 8 * q, c = ti * kCT + lx;
      sh[ly + 8 * q][lx] = (r < n && c < n) ? M[(long long)r * n + c] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    const double w = ti == tj ? 1.0 : 2.0;  // both triangles have the same differences
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = ti * kCT + ly + 8 * q, c = tj * kCT + lx;
      if (r < n && c < n) {
        const float2 a = M[(long long)r * n + c], b = sh[lx][ly + 8 * q];
        const double ax = a.x, ay = a.y, bx = b.x, by = b.y;
        const double dx = ax - bx, dy = ay + by;
        num += w * (dx * dx + dy * dy);
        den += ax * ax + ay * ay;
        if (ti != tj) den += bx * bx + by * by;
      }
    }
  }
  const double2 v = block_sum2(num, den, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = v;
}

// One thread per state.
__global__ void herm_ratio_kernel(const double2* __restrict__ partial, long long count, int blocks,
                                  double* __restrict__ out) {
  const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (s >= count) return;
  double num = 0.0, den = 0.0;
  for (int b = 0; b < blocks; ++b) {
    const double2 v = partial[s * blocks + b];
    num += v.x;
    den += v.y;
  }
  den = sqrt(den);
  out[s] = sqrt(num) / (den < 1e-300 ? 1e-300 : den);
}

// Blocks per state: eight per SM over all states, at most one per tile pair.
int blocks_per_state(int n, long long count) {
  const long long T = (n + kCT - 1) / kCT, want = std::max<long long>(1, 1184 / std::max<long long>(count, 1));
  return (int)std::min(want, T * (T + 1) / 2);
}

}  // namespace
}  // namespace dqb

extern "C" size_t dqb_state_hermiticity_workspace_size(int32_t n, int64_t count) {
  if (n < 1 || count < 1) return 0;
  return (size_t)count * dqb::blocks_per_state(n, count) * sizeof(double2);
}

extern "C" int dqb_state_hermiticity(const void* states, int32_t n, int64_t count, double* out, void* workspace,
                                     size_t workspace_bytes, void* stream) {
  if (n < 1 || count < 0) return DQB_ERR_INVALID_ARGUMENT;
  if (count == 0) return DQB_OK;
  if (!states || !out) return DQB_ERR_INVALID_ARGUMENT;
  const int blocks = dqb::blocks_per_state(n, count);
  if (count > (int64_t)0x7fffffff / blocks) return DQB_ERR_UNSUPPORTED;
  if (!workspace || workspace_bytes < dqb_state_hermiticity_workspace_size(n, count))
    return DQB_ERR_WORKSPACE_TOO_SMALL;
  cudaStream_t s = (cudaStream_t)stream;
  double2* partial = (double2*)workspace;
  dqb::herm_partial_kernel<<<(unsigned)(count * blocks), 256, 0, s>>>((const float2*)states, n, blocks, partial);
  dqb::herm_ratio_kernel<<<(unsigned)((count + 127) / 128), 128, 0, s>>>(partial, count, blocks, out);
  return cudaGetLastError() == cudaSuccess ? DQB_OK : DQB_ERR_CUDA;
}
