// Hermiticity defect ||rho - rho^+||_F / ||rho||_F and trace of saved states, in FP64.
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

struct Partial {
  double num, den;     // sum |rho - rho^+|^2, sum |rho|^2
  double tr_re, tr_im;  // sum rho_ii
};

// blockIdx.x = state * blocks + part; partial[blockIdx.x]: the sums over the part's tile pairs.
__global__ void __launch_bounds__(256) checks_partial_kernel(const float2* __restrict__ states, int n, int blocks,
                                                             Partial* __restrict__ partial) {
  __shared__ float2 sh[kCT][kCT + 1];
  __shared__ double red[72];
  const long long s = blockIdx.x / blocks;
  const float2* __restrict__ M = states + s * n * n;
  const int T = (n + kCT - 1) / kCT, pairs = T * (T + 1) / 2;
  const int lx = threadIdx.x & 31, ly = threadIdx.x >> 5;
  double num = 0.0, den = 0.0, tr = 0.0, ti_sum = 0.0;
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
        if (r == c) tr += ax, ti_sum += ay;
      }
    }
  }
  const double2 v = block_sum2(num, den, red), t = block_sum2(tr, ti_sum, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = Partial{v.x, v.y, t.x, t.y};
}

// One thread per state.
__global__ void checks_sum_kernel(const Partial* __restrict__ partial, long long count, int blocks,
                                  double* __restrict__ herm, double2* __restrict__ trace) {
  const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (s >= count) return;
  Partial v{0.0, 0.0, 0.0, 0.0};
  for (int b = 0; b < blocks; ++b) {
    const Partial p = partial[s * blocks + b];
    v.num += p.num;
    v.den += p.den;
    v.tr_re += p.tr_re;
    v.tr_im += p.tr_im;
  }
  const double den = sqrt(v.den);
  herm[s] = sqrt(v.num) / (den < 1e-300 ? 1e-300 : den);
  trace[s] = make_double2(v.tr_re, v.tr_im);
}

// Blocks per state: eight per SM over all states, at most one per tile pair.
int blocks_per_state(int n, long long count) {
  const long long T = (n + kCT - 1) / kCT, want = std::max<long long>(1, 1184 / std::max<long long>(count, 1));
  return (int)std::min(want, T * (T + 1) / 2);
}

}  // namespace
}  // namespace dqb

extern "C" size_t dqb_state_checks_workspace_size(int32_t n, int64_t count) {
  if (n < 1 || count < 1) return 0;
  return (size_t)count * dqb::blocks_per_state(n, count) * sizeof(dqb::Partial);
}

extern "C" int dqb_state_checks(const void* states, int32_t n, int64_t count, double* hermiticity, void* trace,
                                void* workspace, size_t workspace_bytes, void* stream) {
  if (n < 1 || count < 0) return DQB_ERR_INVALID_ARGUMENT;
  if (count == 0) return DQB_OK;
  if (!states || !hermiticity || !trace) return DQB_ERR_INVALID_ARGUMENT;
  const int blocks = dqb::blocks_per_state(n, count);
  if (count > (int64_t)0x7fffffff / blocks) return DQB_ERR_UNSUPPORTED;
  if (!workspace || workspace_bytes < dqb_state_checks_workspace_size(n, count)) return DQB_ERR_WORKSPACE_TOO_SMALL;
  cudaStream_t s = (cudaStream_t)stream;
  dqb::Partial* partial = (dqb::Partial*)workspace;
  dqb::checks_partial_kernel<<<(unsigned)(count * blocks), 256, 0, s>>>((const float2*)states, n, blocks, partial);
  dqb::checks_sum_kernel<<<(unsigned)((count + 127) / 128), 128, 0, s>>>(partial, count, blocks, hermiticity,
                                                                        (double2*)trace);
  return cudaGetLastError() == cudaSuccess ? DQB_OK : DQB_ERR_CUDA;
}
