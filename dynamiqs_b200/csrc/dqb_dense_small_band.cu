// Persistent batched mesolve kernel for n <= 64 when an instance's dense operators are
// banded: few nonzero diagonals in Hnh = -iH - 1/2 sum L^+L and in the jump operators, as
// for every bosonic ladder, number and drive operator.  Products with the zeros of such a
// matrix contribute nothing, so the right-hand side is the stencil of the sparse-DIA path
//   f(X)[i][j] = sum_d Hnh[i][i+d] X[i+d][j] + sum_d conj(Hnh[j][j+d]) X[i][j+d]
//              + sum_(p,s) L[i][i+p] conj(L[j][j+s]) X[i+p][j+s]
// (dynamiqs/qarrays/sparsedia_primitives.py:199-261; diffrax_integrator.py:312-323), a few
// multiply-adds per element against n (1 + 2K) of the full products.
//
// The kernel reads each instance's operators, lists their nonzero diagonals and solves the
// instance if there are at most kMaxH and kMaxL of them; any other instance (full matrices,
// a rho0 that is not hermitian to rounding, more jumps than the tables hold) is marked in
// `pend` and left to the product kernel, which runs next on the stream and takes the marked
// instances only.  The host decides on the thread layout alone, by the size of the batch, and
// no result depends on it (block_sums).
//
// What bounds it: with the products gone a step is short, and the 27 reads of y and the
// stages that the combinations of a step make would dominate from L2 (where the product
// kernel keeps them).  In the hermitian form only the elements on and above the diagonal
// are independent, so the Runge-Kutta state stays on the SM: the matrix is cut into T x T
// tiles, thread (ty, tx) owns element (ty, tx) of each of the R (R + 1) / 2 upper tiles and
// keeps k_2..k_7 of them in registers (120 of a thread's 255 at n = 64) and y and k_1 in
// shared memory, where the rest of the registers is wanted for the right-hand side (with
// all of them in registers the spills went to L2: 20.0 against 17.1 ms then).  Shared
// memory also holds the stage input X, whole (the stencil reads both triangles; the owner of
// (i, j) also writes conj(X) at (j, i)), in two buffers, so that a right-hand side costs one
// barrier.  A row (column) coefficient is read once per tile row (column) and used on all
// its tiles; a version that took the tile rows one after another, with fewer accumulators,
// waited on shared memory (31.9 ms).  All threads compute the controller's few FP64 values
// alike, which needs no barrier.  Two warps per scheduler issue in 40% of the cycles; the
// rest are fixed latencies, shared-memory waits and instruction fetch.
//
// Measured (one B200): driven Kerr, n = 64, two jumps, 1024 instances, t = 1.6: 16.1 ms
// against 153.4 ms for the product kernel; n = 21, one jump, 1000 instances: 1.5 against
// 5.31 ms; n = 8, 2000 instances: 0.42 against 2.28 ms; one n = 16 oscillator with 101 saves:
// 0.25 against 0.72 ms (0.38 with one diagonal per pass and registers for four CTAs per SM).
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "dqb_small_band.cuh"

namespace dqb {
namespace band {

// What the packed offsets (offset_of) and the tables hold; at eight the kernel is still 1.6
// (n = 32) to 3.3 (n = 8) times as fast as the products, eight jump operators 5 to 7 times.
constexpr int kMaxH = 8;   // nonzero diagonals of Hnh
constexpr int kMaxK = 8;   // jump operators
constexpr int kMaxL = 8;   // nonzero diagonals of all jump operators together
constexpr int kMaxM = DQB_TD_MAX_TERMS;
constexpr int kMaxDevices = 64;
constexpr int kMid = 63;   // bit of offset 0 in a diagonal mask

// T x T threads, R x R tiles.  Row stride of X: odd for T = 16 (a half-warp reads one row's
// 16 values: any stride is free of conflicts, and odd frees the mirrored column writes);
// 8 mod 16 for T = 8 (a half-warp reads two rows' 8 values, which then fall on disjoint
// banks).
template <int T, int R>
struct Geo {
  static constexpr int NP = T * R, NT = T * T, Q = R * (R + 1) / 2;
  static constexpr int LD = T == 16 ? NP + 1 : (NP % 16 == 8 ? NP : NP + 8);
  static constexpr int XM = NP * LD;
  static constexpr int NW = NT / 32;
  // whether tile (r, c) lies in a 16 x 16 block of the diagonal
  static __host__ __device__ constexpr bool diag_block(int r, int c) { return T * r / 16 == T * c / 16; }
};

// Offset of diagonal d from the packed list (one signed byte each, d < 8): no memory access
// before the accesses that it displaces.
__device__ __forceinline__ int offset_of(unsigned long long packed, int d) {
  return (int)(signed char)(packed >> (8 * d));
}

// 0.5 a x, rounded as the product kernel rounds a one-term sum and its half.
__device__ __forceinline__ float2 half_cmul(float2 a, float2 x) {
  const float2 u = cfma(a, x, make_float2(0.f, 0.f));
  return make_float2(0.5f * u.x, 0.5f * u.y);
}

struct Lists {
  unsigned mask[1 + kMaxK + kMaxM][4];  // nonzero diagonals: H, the jumps, the terms of H(t)
  int ok, flag;
  int given;       // rho0's triangles differ in rounding: save points at t0 take rho0 itself
  int nh, nk, nl;  // diagonals of Hnh (ascending), jump operators, their diagonals (ascending)
  unsigned long long hpack, lpack;  // their offsets, packed (offset_of)
  int hoff[kMaxH];
  int loff[kMaxL], lstart[kMaxK + 1];
};

template <int T, int R>
struct Shared {
  using G = Geo<T, R>;
  Lists ls;
  double a21[21];             // a[s][j], j < s, row by row
  double red[2][4 * (T == 16 ? 128 : 2)];  // two sets, used in turn (block_sums)
  float cf[G::NW][24];        // each warp's copy of the stage coefficients h a[s][j]
  double inv_nn, t1;
  long long inst;
  InstView v;  // (here and not in registers: the Runge-Kutta state needs those)
};

// Dynamic shared memory, in complex values: two X buffers, the owned elements of y and k_1, Hnh's diagonals (two sets and
// the constant part when H depends on time, and the terms' diagonals), the jumps'.
template <int T, int R>
__host__ __device__ constexpr int dyn_values(bool td) {
  return 2 * Geo<T, R>::XM + 2 * Geo<T, R>::Q * Geo<T, R>::NT + (td ? 3 + kMaxM : 1) * kMaxH * Geo<T, R>::NP + kMaxL * Geo<T, R>::NP;
}

// Sets the bits of M's nonzero diagonals (bit j - i + kMid).
template <int NT>
__device__ __forceinline__ void scan_diagonals(const float2* __restrict__ M, int n, unsigned* mask) {
  constexpr int U = 4;  // values in flight per thread
  for (int e0 = threadIdx.x; e0 < n * n; e0 += U * NT) {
    float2 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = e0 + u * NT < n * n ? __ldg(M + e0 + u * NT) : make_float2(0.f, 0.f);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (v[u].x != 0.f || v[u].y != 0.f) {
        const int e = e0 + u * NT, i = e / n, b = e - i * n - i + kMid;
        const unsigned bit = 1u << (b & 31);
        if (!(*(volatile unsigned*)&mask[b >> 5] & bit)) atomicOr(&mask[b >> 5], bit);
      }
  }
}

// One thread: the lists of diagonals and pairs; ls.ok = 0 when the tables do not hold them.
__device__ inline void build_lists(Lists& ls, int n, int K, int M) {
  unsigned hm[4];
  ls.ok = 0;
  for (int w = 0; w < 4; ++w) {
    hm[w] = ls.mask[0][w];
    for (int m = 0; m < M; ++m) hm[w] |= ls.mask[1 + kMaxK + m][w];
  }
  int nl = 0;
  for (int k = 0; k < K; ++k) {
    ls.lstart[k] = nl;
    for (int w = 0; w < 4; ++w)
      for (unsigned x = ls.mask[1 + k][w]; x; x &= x - 1) {
        if (nl == kMaxL) return;
        ls.loff[nl++] = 32 * w + __ffs((int)x) - 1 - kMid;
      }
    for (int p = ls.lstart[k]; p < nl; ++p)
      for (int s = ls.lstart[k]; s < nl; ++s) {
        const int d = ls.loff[s] - ls.loff[p];  // a diagonal of L^+L
        if (d > -n && d < n) hm[(d + kMid) >> 5] |= 1u << ((d + kMid) & 31);
      }
  }
  ls.lstart[K] = ls.nl = nl;
  ls.nk = K;
  int nh = 0;
  for (int w = 0; w < 4; ++w)
    for (unsigned x = hm[w]; x; x &= x - 1) {
      if (nh == kMaxH) return;
      ls.hoff[nh++] = 32 * w + __ffs((int)x) - 1 - kMid;
    }
  ls.nh = nh;
  ls.hpack = ls.lpack = 0;
  for (int d = 0; d < nh; ++d) ls.hpack |= (unsigned long long)(ls.hoff[d] & 0xff) << (8 * d);
  for (int p = 0; p < nl; ++p) ls.lpack |= (unsigned long long)(ls.loff[p] & 0xff) << (8 * p);
  ls.ok = 1;
}

// Block sums over the elements.  Their order is the same in both thread layouts, so that a
// result does not depend on the layout, which the size of the batch chooses: elements of one
// place in the 16 x 16 blocks, tile by tile; the place's four images in the 8 x 8 blocks; then
// the 8 x 8 places, as a tree over rows 0-3 and one over rows 4-7.  With T = 8 a thread is an
// 8 x 8 place (the parity of its tile's row and column gives the image) and the trees are
// shuffles before the barrier; with T = 16 it is one image, and they follow the barrier that the
// exchange of images needs.  (An order that suits T = 16 better, the rows last, cost T = 8 up
// to 9% of a solve.)

// Before the barrier: N quantities to red, where add(e, r, c) adds the thread's element of tile
// (r, c) to e, for the tiles r <= c (or, not kUpper, all).
template <int T, int R, int N, bool kUpper, class Add>
__device__ __forceinline__ void sums_begin(double* red, Add add) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // the sums over the tiles (r, c) of parity (a, b), or over all
  auto tiles = [&](double (&e)[N], int a, int b) {
    constexpr int kStep = T == 16 ? 1 : 2;
#pragma unroll
    for (int i = 0; i < N; ++i) e[i] = 0.0;
#pragma unroll
    for (int r = a; r < R; r += kStep)
#pragma unroll
      for (int c = b; c < R; c += kStep)
        if (!kUpper || r <= c) add(e, r, c);
  };
  double e[N];
  tiles(e, 0, 0);
  if constexpr (T == 16) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      e[i] += __shfl_xor_sync(0xffffffffu, e[i], 8);  // the images in a block's two halves of a row
      if ((lane & 8) == 0) red[i * 128 + (threadIdx.x >> 4) * 8 + (lane & 7)] = e[i];
    }
  } else {
    double f[N], g[N];
    tiles(f, 0, 1);
#pragma unroll
    for (int i = 0; i < N; ++i) g[i] = e[i] + f[i];
    tiles(e, 1, 0);
    tiles(f, 1, 1);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const double x = warp_sum(g[i] + (e[i] + f[i]));
      if (lane == 0) red[i * 2 + warp] = x;
    }
  }
}

// After it: quantity i (to every thread of the calling warps).
template <int T>
__device__ __forceinline__ double sums_end(const double* red, int i) {
  if (T == 8) return red[i * 2] + red[i * 2 + 1];
  const double* p = red + i * 128 + (threadIdx.x & 31);
  return warp_sum(p[0] + p[64]) + warp_sum(p[32] + p[96]);
}

// Sums to every thread.  One barrier: `par` selects the set of partial sums, used in turn, so a
// set is rewritten only after a barrier that every reader of it has passed.
template <int T, int R, int N, class Add>
__device__ __forceinline__ void block_sums(double (&v)[N], Shared<T, R>& sh, int& par, Add add) {
  double* red = sh.red[par];
  par ^= 1;
  sums_begin<T, R, N, true>(red, add);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = sums_end<T>(red, i);
}

// Expectation values `m` on of save point `sidx`, up to two: add(e, E, r, c) adds the thread's
// element of tile (r, c) to the value of operator E.  One barrier.
template <int T, int R, bool kUpper, class Add>
__device__ __forceinline__ void expect_sums(const InstView& a, Shared<T, R>& sh, int& par, int m, int sidx, Add add) {
  double* red = sh.red[par];
  par ^= 1;
  const int ops = min(a.nE - m, 2);
#pragma unroll 1
  for (int k = 0; k < ops; ++k) {
    const float2* E = a.E + (long long)(m + k) * a.n * a.n;
    sums_begin<T, R, 2, kUpper>(red + k * (T == 16 ? 256 : 4), [&](double (&e)[2], int r, int c) { add(e, E, r, c); });
  }
  __syncthreads();
  const int i = T == 16 ? threadIdx.x >> 5 : threadIdx.x;  // a warp, or a thread, per part
  if (i >= 2 * ops) return;
  const double x = sums_end<T>(red, i);
  if (T == 8 || (threadIdx.x & 31) == 0)
    reinterpret_cast<float*>(a.expects + (long long)(m + (i >> 1)) * a.ntsave + sidx)[i & 1] = (float)x;
}

// The first `saved` save points that lie at t0, and the final state where only that is kept
// and no step was taken (`at_start`), from rho0 as given: the solve has gone by its upper
// triangle.  A call at the end of a solve, so that its registers cost the solve none.
template <int T, int R>
__device__ __noinline__ void save_given(const InstView& a, Shared<T, R>& sh, int saved, bool at_start) {
  const int n = a.n;
  int par = 0;
  __syncthreads();  // the states have been written, the sums read
  if (!a.save_states && at_start)
    for (int e = threadIdx.x; e < n * n; e += T * T) a.states[e] = a.rho0[e];
  for (int s = 0; s < saved && a.tsave[s] <= a.t0; ++s) {
    if (a.save_states)
      for (int e = threadIdx.x; e < n * n; e += T * T) a.states[(long long)s * n * n + e] = a.rho0[e];
    for (int m = 0; m < a.nE; m += 2)
      expect_sums<T, R, false>(a, sh, par, m, s, [&](double (&e)[2], const float2* E, int r, int c) {
        const int i = threadIdx.x / T + T * r, j = threadIdx.x % T + T * c;
        if (i >= n || j >= n) return;
        const float2 u = a.rho0[i * n + j], eji = __ldg(E + j * n + i);
        e[0] += (double)eji.x * u.x - (double)eji.y * u.y;
        e[1] += (double)eji.x * u.y + (double)eji.y * u.x;
      });
  }
}

// One instance.  Returns false (to every thread) when the instance is not banded or its
// rho0 not hermitian to rounding: nothing has been written then.  FEAT as in
// mesolve_small_kernel: 1 = time-dependent H, 2 = gradient tape (rows of tape_np values).
template <int T, int R, int FEAT>
__device__ bool solve(const CtrlOpts& o, const TdArgs* td, Shared<T, R>& sh, float2* dyn, int tape_np) {
  using G = Geo<T, R>;
  constexpr int NP = G::NP, LD = G::LD, NT = G::NT, Q = G::Q;
  constexpr bool kTd = FEAT == 1, kTape = FEAT == 2;
  constexpr int kStep = Q <= 3 && !kTd ? 4 : 1;
  // Diagonals of a jump operator from which the right-hand side multiplies it in two steps (V
  // below) and not term by term, and diagonals per pass there.  Measured at n = 8 and 16, one
  // instance, four diagonals: 63 and 72 us in two steps, 99 and 118 term by term, 70 and 92
  // with the products of full matrices; n = 32: 107, 144 and 176.  With T = 8 two steps pay
  // later (their transposed reads of V conflict on banks): n = 4 with full jumps, 2000
  // instances, 275 against 823 us, but three diagonals the same either way.
  constexpr int kFactor = T == 16 ? (R == 1 ? 2 : 3) : 4, kGroup = T == 16 && R == 1 && !kTd ? 4 : 1;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = tid % T, ty = tid / T;
  const InstView& a = sh.v;
  const int n = a.n, M = kTd ? td->M : 0;
  Lists& ls = sh.ls;
  float2* const Xb[2] = {dyn, dyn + G::XM};
  float2* const y = dyn + 2 * G::XM + tid;             // element of tile q at q * NT
  float2* const k1 = y + Q * NT;                       // the same of the first stage
  float2* hd = dyn + 2 * G::XM + 2 * Q * NT;           // [kMaxH][NP] (two sets when kTd)
  float2* h0d = hd + 2 * kMaxH * NP;                   // kTd: the constant part
  float2* opd = h0d + kMaxH * NP;                      // kTd: [kMaxM][kMaxH][NP]
  float2* ld = kTd ? opd + kMaxM * kMaxH * NP : hd + kMaxH * NP;  // [kMaxL][NP]

  // ---- operators: nonzero diagonals, lists, tables -------------------------------------
  const int K = a.K;
  if (K > kMaxK) return false;
  for (int e = tid; e < (1 + kMaxK + kMaxM) * 4; e += NT) (&ls.mask[0][0])[e] = 0u;
  // Full matrices are told by their first and last rows: the nonzeros of the two lie on
  // different diagonals but for the main one, which both may have.  (A middle row alone tells
  // them only beyond 8 columns, and one instance of n = 8 spent 11 us on its lists.)
  unsigned ends = 0;  // bit m: a nonzero of operator m (H, the jumps) at the thread's place
  if (tid < 2 * n) {
    const long long at = tid < n ? tid : (long long)n * n - 2 * n + tid;
    float2 e = __ldg(a.H + at);
    ends = e.x != 0.f || e.y != 0.f;
#pragma unroll 1
    for (int k = 0; k < K; ++k) {
      e = __ldg(a.L + (long long)k * n * n + at);
      if (e.x != 0.f || e.y != 0.f) ends |= 2u << k;
    }
  }
  if (__syncthreads_count(ends & 1u) > kMaxH + 1) return false;
  int jumps = 0;
  for (int k = 0; k < K; ++k) jumps += __syncthreads_count(ends >> (k + 1) & 1u);
  if (jumps > kMaxL + K) return false;
  scan_diagonals<NT>(a.H, n, ls.mask[0]);
  for (int k = 0; k < K; ++k) scan_diagonals<NT>(a.L + (long long)k * n * n, n, ls.mask[1 + k]);
  for (int m = 0; m < M; ++m) scan_diagonals<NT>(td->ops + (long long)m * n * n, n, ls.mask[1 + kMaxK + m]);
  __syncthreads();
  if (tid == 0) build_lists(ls, n, K, M);
  __syncthreads();
  if (!ls.ok) return false;
  for (int k = 0; k < K; ++k)
    for (int p = ls.lstart[k]; p < ls.lstart[k + 1]; ++p)
      for (int i = tid; i < NP; i += NT) {  // L[i][i + p]
        const int j = i + ls.loff[p];
        ld[p * NP + i] = (i < n && j >= 0 && j < n) ? a.L[((long long)k * n + i) * n + j] : make_float2(0.f, 0.f);
      }
  __syncthreads();
  for (int e = tid; e < kMaxH * NP; e += NT) {  // Hnh[i][i + d]; zeros beyond the last diagonal
    const int q = e / NP, i = e - q * NP, j = q < ls.nh ? i + ls.hoff[q] : -1;
    float2 v = make_float2(0.f, 0.f);
    const bool in = i < n && j >= 0 && j < n;
    if (in) {
      // (sum L^+L)[i][j] = sum_m conj(L[m][i]) L[m][j], by ascending m
      float2 s = make_float2(0.f, 0.f);
      for (int jk = 0; jk < K; ++jk)
        for (int pa = ls.lstart[jk + 1] - 1; pa >= ls.lstart[jk]; --pa)
          for (int pb = ls.lstart[jk]; pb < ls.lstart[jk + 1]; ++pb) {
            const int m = i - ls.loff[pa];
            if (ls.loff[pb] - ls.loff[pa] == ls.hoff[q] && m >= 0 && m < n)
              cmac(s, cconj(ld[pa * NP + m]), ld[pb * NP + m]);
          }
      const float2 h = a.H[i * n + j];
      v = make_float2(h.y - 0.5f * s.x, -h.x - 0.5f * s.y);  // -i h - s / 2
    }
    if constexpr (kTd) {
      h0d[e] = v;
      for (int m = 0; m < M; ++m)
        opd[m * kMaxH * NP + e] = in ? td->ops[((long long)m * n + i) * n + j] : make_float2(0.f, 0.f);
    } else {
      hd[e] = v;
    }
  }
  // entries beyond n x n stay zero: the stencil reads them with zero coefficients
  for (int e = tid; e < 2 * G::XM; e += NT) dyn[e] = make_float2(0.f, 0.f);

  // ---- initial state: upper elements, hermiticity (rtol = atol = 1e-5) -----------------
  // own: bit q = the thread's element of tile q is an element of the upper triangle;
  // strict: it is strictly above the diagonal
  unsigned own = 0, strict = 0;
  float2 k[7][Q];  // (k[0], the first stage, is k1)
  float big = 0.f, asym = 0.f;
  int bad = 0;
  {
    int q = 0;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = r; c < R; ++c, ++q) {
        const int i = ty + T * r, j = tx + T * c;
        const bool in = i < n && j < n && i <= j;
        if (in) own |= 1u << q;
        if (in && i < j) strict |= 1u << q;
        float2 v = make_float2(0.f, 0.f);
        if (in && a.is_ket) {
          v = cmul(a.rho0[i], cconj(a.rho0[j]));
          if (i == j) v.y = 0.f;
        } else if (in) {
          v = a.rho0[i * n + j];
          const float2 u = cconj(a.rho0[j * n + i]);
          const float d = cabsf(make_float2(v.x - u.x, v.y - u.y));
          const float av = cabsf(v), au = cabsf(u);
          if (!(d <= 1e-5f + 1e-5f * au) || !(d <= 1e-5f + 1e-5f * av)) bad = 1;
          big = fmaxf(big, fmaxf(au, av));
          asym = fmaxf(asym, d);
          if (!(d < INFINITY)) asym = INFINITY;
          if (i == j) v.y = 0.f;
        }
        y[q * NT] = v;
      }
  }
  if (__syncthreads_or(bad && o.check_hermitian)) {
    if (tid == 0) {
      a.infos[0] = a.infos[1] = a.infos[2] = 0;
      __threadfence_system();  // status last: a caller may poll it from the host
      a.status[0] = DQB_INST_NOT_HERMITIAN;
    }
    __syncthreads();
    return true;
  }
  if (!a.is_ket) {
    // the upper triangle stands for the matrix only when the two agree to rounding
    big = warp_max(big);
    asym = warp_max(asym);
    if (lane == 0) sh.red[0][2 * warp] = big, sh.red[0][2 * warp + 1] = asym;
    __syncthreads();
    for (int w = 0; w < G::NW; ++w) {
      big = fmaxf(big, (float)sh.red[0][2 * w]);
      asym = fmaxf(asym, (float)sh.red[0][2 * w + 1]);
    }
    __syncthreads();
    if (!(asym <= 4.8e-7f * big)) return false;
  }
  if (tid == 0) ls.given = !a.is_ket && asym != 0.f;
  for (int e = tid; e < 21; e += NT) {
    int s = 1;
    while (e >= s * (s + 1) / 2) ++s;
    sh.a21[e] = c_tab[o.method].a[s][e - s * (s - 1) / 2];
  }
  if (tid == 0) {
    sh.inv_nn = 1.0 / ((double)n * (double)n);
    sh.t1 = a.tsave[a.ntsave - 1];
  }
  __syncthreads();
  double t = a.t0, tnext = t, h = 0.0, dt_prop = 0.0;
  auto tile_of = [](int r, int c) { return r * R - r * (r - 1) / 2 + c - r; };  // of the upper tiles, row by row
  int made_jump = 0, xb = 0, par = 0, sidx = 0, status = DQB_INST_OK;
  long long nsteps = 0, nacc = 0;
  const int nh = ls.nh, nk = ls.nk;
  const unsigned long long hoffs = ls.hpack, loffs = ls.lpack;
  float* const cfw = sh.cf[warp];
  float2 v[Q];

  // X <- v (and its mirror) in the next buffer; returns it.  The caller's barrier follows.
  auto stage = [&](const float2 (&u)[Q]) {
    xb ^= 1;
    float2* X = Xb[xb];
    int q = 0;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = r; c < R; ++c, ++q) {
        const int i = ty + T * r, j = tx + T * c;
        if ((own >> q) & 1u) X[i * LD + j] = u[q];
        if ((strict >> q) & 1u) X[j * LD + i] = cconj(u[q]);
      }
    return X;
  };
  // stage coefficients of the step (every warp its own copy)
  auto set_coefs = [&] {
    __syncwarp();
    if (lane < 21) cfw[lane] = (float)(h * sh.a21[lane]);
    __syncwarp();
  };
  // X (n x n) -> dst, rows of ldo values
  auto copy_out = [&](const float2* X, float2* dst, int ldo) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = 0; c < R; ++c) {
        const int i = ty + T * r, j = tx + T * c;
        if (i < n && j < n) dst[i * ldo + j] = X[i * LD + j];
      }
  };
  // one save point: the state u (its upper elements) and tr(E u), FP64 sums
  auto save = [&](const float2 (&u)[Q]) {
    if (a.save_states) {
      const float2* X = stage(u);
      __syncthreads();
      copy_out(X, a.states + (long long)sidx * n * n, n);
    }
#pragma unroll 1
    for (int m = 0; m < a.nE; m += 2)
      expect_sums<T, R, true>(a, sh, par, m, sidx, [&](double (&e)[2], const float2* E, int r, int c) {
        const int q = tile_of(r, c), i = ty + T * r, j = tx + T * c;
        if (!((own >> q) & 1u)) return;
        const float2 eji = __ldg(E + j * n + i);
        e[0] += (double)eji.x * u[q].x - (double)eji.y * u[q].y;
        e[1] += (double)eji.x * u[q].y + (double)eji.y * u[q].x;
        if ((strict >> q) & 1u) {
          const float2 eij = __ldg(E + i * n + j);
          e[0] += (double)eij.x * u[q].x + (double)eij.y * u[q].y;
          e[1] += (double)eij.y * u[q].x - (double)eij.x * u[q].y;
        }
      });
    ++sidx;
  };

  // v <- f(ts, v) on the owned elements; returns the buffer that holds the stage input
  auto rhs = [&](double ts) {
    const float2* X = stage(v);
    const float2* hq = hd;
    if constexpr (kTd) {  // Hnh(t) = Hnh0 - i sum_m c_m(t) H_m, in the set that goes with the X buffer
      float2* w = hd + xb * kMaxH * NP;
      float2 cm[kMaxM];
#pragma unroll
      for (int m = 0; m < kMaxM; ++m)
        if (m < M) {
          const double2 c = td_coef(td->term[m], a.inst, ts);
          cm[m] = make_float2((float)c.x, (float)c.y);
        }
      for (int e = tid; e < (nh + kStep - 1) / kStep * kStep * NP; e += NT) {
        float2 acc = make_float2(0.f, 0.f);
#pragma unroll
        for (int m = 0; m < kMaxM; ++m)
          if (m < M) cmac(acc, cm[m], opd[m * kMaxH * NP + e]);
        const float2 c = h0d[e];
        w[e] = make_float2(c.x + acc.y, c.y - acc.x);
      }
      hq = w;
    }
    __syncthreads();
    // On element (i, j) of an upper tile: A = (Hnh X)[i][j], B = conj((Hnh X)[j][i]) and S
    // half the dissipator.  Every sum runs over the same nonzero products in the same
    // order, with the same roundings, as the product kernel's (which adds the zeros in
    // between): Hnh X by ascending column of Hnh; S onto A and B of a 16 x 16 diagonal
    // block, and twice onto B of the others (the block below the diagonal, whose mirror this
    // is).  With X hermitian to the last bit the two kernels' right-hand sides agree to the last
    // bit; the FP64 norms, which decide on steps, are added up in another order (block_sums).
    float2 A[Q], B[Q], S[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) A[q] = B[q] = S[q] = make_float2(0.f, 0.f);
    // positions in X of the thread's rows (plus its column) and columns (plus its row)
    // displaced by `off`; beyond the matrix any entry will do, the coefficient is zero
    int xr[R], xc[R];
    auto displaced = [&](int off_r, int off_c) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        xr[r] = min(max(ty + T * r + off_r, 0), NP - 1) * LD;
        xc[r] = min(max(tx + T * r + off_c, 0), NP - 1);
      }
    };
    float2 cr[R], cc[R];
    auto coefs = [&](const float2* dr, const float2* dc) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        cr[r] = dr[ty + T * r];
        cc[r] = cconj(dc[tx + T * r]);
      }
    };
    // kStep diagonals per pass: with few elements per thread the reads of several hide one
    // another's latency (the rows of the table beyond nh are zero; a time-dependent H has no
    // registers left for it)
#pragma unroll 1
    for (int d0 = 0; d0 < nh; d0 += kStep) {
#pragma unroll
      for (int dd = 0; dd < kStep; ++dd) {
        const int d = d0 + dd, off = offset_of(hoffs, d);
        coefs(hq + d * NP, hq + d * NP);
        displaced(off, off);
        int q = 0;
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int c = r; c < R; ++c, ++q) {
            A[q] = cfma(cr[r], X[xr[r] + tx + T * c], A[q]);
            B[q] = cfma(cc[c], X[xc[c] + (ty + T * r) * LD], B[q]);
          }
      }
    }
#pragma unroll 1
    for (int jk = 0; jk < nk; ++jk) {
      const int p0 = ls.lstart[jk], p1 = ls.lstart[jk + 1];
      if (p1 == p0 + 1) {  // one diagonal: L[i][i + p] X[i + p][j + p] conj(L[j][j + p])
        const int off = offset_of(loffs, p0);
        coefs(ld + p0 * NP, ld + p0 * NP);
        displaced(off, off);
        int q = 0;
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int c = r; c < R; ++c, ++q) {
            const float2 x = X[xr[r] + xc[c]];
            const float2 u = half_cmul(cc[c], x);
            if (G::diag_block(r, c)) {
              A[q] = cfma(half_cmul(cr[r], x), cc[c], A[q]);
              B[q] = cfma(u, cr[r], B[q]);
            } else {
              S[q] = cfma(u, cr[r], S[q]);
            }
          }
        continue;
      }
      if (p1 - p0 >= kFactor) {
        // Many diagonals: V = X L^+ first, whole, in the buffer that the previous right-hand side
        // has left, so that each of the two sums below runs over the diagonals once.  By X's
        // hermiticity V[i + p][j] = conj((L X)[j][i + p]) and conj(V[j + t][i]) = (L X)[i][j + t].
        float2* V = Xb[xb ^ 1];
#pragma unroll 1
        for (int r = 0; r < R; ++r) {
          float2 u[R];
#pragma unroll
          for (int c = 0; c < R; ++c) u[c] = make_float2(0.f, 0.f);
          const int i = ty + T * r;
#pragma unroll 1
          for (int t0 = p0; t0 < p1; t0 += kGroup) {
#pragma unroll
            for (int tt = 0; tt < kGroup; ++tt) {
              const int t = min(t0 + tt, kMaxL - 1), off = offset_of(loffs, t);
#pragma unroll
              for (int c = 0; c < R; ++c) {
                const int j = tx + T * c;
                float2 w = cconj(ld[t * NP + j]);
                if (tt > 0 && t0 + tt >= p1) w = make_float2(0.f, 0.f);
                u[c] = cfma(w, X[i * LD + min(max(j + off, 0), NP - 1)], u[c]);
              }
            }
          }
#pragma unroll
          for (int c = 0; c < R; ++c) V[i * LD + tx + T * c] = make_float2(0.5f * u[c].x, 0.5f * u[c].y);
        }
        __syncthreads();
#pragma unroll 1
        for (int t0 = p0; t0 < p1; t0 += kGroup) {
#pragma unroll
          for (int tt = 0; tt < kGroup; ++tt) {
            const int t = min(t0 + tt, kMaxL - 1), off = offset_of(loffs, t);
            coefs(ld + t * NP, ld + t * NP);
            displaced(off, off);
            const bool in = tt == 0 || t0 + tt < p1;
            int q = 0;
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
              for (int c = r; c < R; ++c, ++q) {
                float2& dst = G::diag_block(r, c) ? B[q] : S[q];
                const float2 none = make_float2(0.f, 0.f);
                dst = cfma(V[xr[r] + tx + T * c], in ? cr[r] : none, dst);
                if (G::diag_block(r, c)) A[q] = cfma(cconj(V[xc[c] * LD + ty + T * r]), in ? cc[c] : none, A[q]);
              }
          }
        }
        __syncthreads();  // V has been read
        continue;
      }
#pragma unroll 1
      for (int p = p0; p < p1; ++p) {  // conj((L X)[j][i + p]) / 2 times L[i][i + p]
        float2 u[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) u[q] = make_float2(0.f, 0.f);
#pragma unroll 1
        for (int t = p0; t < p1; ++t) {
          coefs(ld + p * NP, ld + t * NP);
          displaced(offset_of(loffs, p), offset_of(loffs, t));
          int q = 0;
#pragma unroll
          for (int r = 0; r < R; ++r)
#pragma unroll
            for (int c = r; c < R; ++c, ++q) u[q] = cfma(cc[c], X[xr[r] + xc[c]], u[q]);
        }
        int q = 0;
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int c = r; c < R; ++c, ++q) {
            float2& dst = G::diag_block(r, c) ? B[q] : S[q];
            dst = cfma(make_float2(0.5f * u[q].x, 0.5f * u[q].y), cr[r], dst);
          }
      }
#pragma unroll 1
      for (int t = p0; t < p1; ++t) {  // diagonal blocks: (L X)[i][j + t] / 2 times conj(L[j][j + t])
        float2 u[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) u[q] = make_float2(0.f, 0.f);
#pragma unroll 1
        for (int p = p0; p < p1; ++p) {
          coefs(ld + p * NP, ld + t * NP);
          displaced(offset_of(loffs, p), offset_of(loffs, t));
          int q = 0;
#pragma unroll
          for (int r = 0; r < R; ++r)
#pragma unroll
            for (int c = r; c < R; ++c, ++q)
              if (G::diag_block(r, c)) u[q] = cfma(cr[r], X[xr[r] + xc[c]], u[q]);
        }
        int q = 0;
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int c = r; c < R; ++c, ++q)
            if (G::diag_block(r, c)) A[q] = cfma(make_float2(0.5f * u[q].x, 0.5f * u[q].y), cc[c], A[q]);
      }
    }
    int q = 0;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = r; c < R; ++c, ++q) {
        if (!G::diag_block(r, c)) B[q] = caxpy(2.f, S[q], B[q]);
        v[q] = cadd(A[q], B[q]);
        // a hermitian matrix's diagonal is real; elements that no thread owns stay zero
        if (!((own >> q) & 1u)) v[q] = make_float2(0.f, 0.f);
        if (!((strict >> q) & 1u)) v[q].y = 0.f;
      }
    return X;
  };
  auto copy = [](float2 (&d)[Q], const float2 (&u)[Q]) {
#pragma unroll
    for (int q = 0; q < Q; ++q) d[q] = u[q];
  };
  auto store_k1 = [&](const float2 (&u)[Q]) {
#pragma unroll
    for (int q = 0; q < Q; ++q) k1[q * NT] = u[q];
  };
  // k_(j + 1) on the thread's element of tile q
  auto kval = [&](int j, int q) { return j == 0 ? k1[q * NT] : k[j][q]; };
  auto load_y = [&] {
#pragma unroll
    for (int q = 0; q < Q; ++q) v[q] = y[q * NT];
  };

  // ---- starting step (Hairer-Norsett-Wanner, RMS norm) ---------------------------------
  load_y();
  rhs(t);
  store_k1(v);
  {
    double sm[2], s2[1];
    block_sums(sm, sh, par, [&](double (&e)[2], int r, int c) {
      const int q = tile_of(r, c);
      if (!((own >> q) & 1u)) return;
      const double sc = o.atol + o.rtol * (double)cabsf(y[q * NT]), w = (strict >> q) & 1u ? 2.0 : 1.0;
      e[0] += w * (double)cabs2f(y[q * NT]) / (sc * sc);
      e[1] += w * (double)cabs2f(v[q]) / (sc * sc);
    });
    const double d0 = sqrt(sm[0] * sh.inv_nn), d1 = sqrt(sm[1] * sh.inv_nn);
    const double h0 = (d0 < 1e-5 || d1 < 1e-5) ? 1e-6 : 0.01 * d0 / d1;
    const float c0 = (float)h0;
#pragma unroll
    for (int q = 0; q < Q; ++q) v[q] = caxpy(c0, k1[q * NT], y[q * NT]);
    rhs(t + h0);
    block_sums(s2, sh, par, [&](double (&e)[1], int r, int c) {
      const int q = tile_of(r, c);
      if (!((own >> q) & 1u)) return;
      const double sc = o.atol + o.rtol * (double)cabsf(y[q * NT]), w = (strict >> q) & 1u ? 2.0 : 1.0;
      const float2 f0 = k1[q * NT];
      const double dx = (double)v[q].x - (double)f0.x, dy = (double)v[q].y - (double)f0.y;
      e[0] += w * fma(dx, dx, dy * dy) / (sc * sc);
    });
    const double d2 = sqrt(s2[0] * sh.inv_nn) / h0;
    const double md = d1 > d2 ? d1 : d2;
    const double hh = md <= 1e-15 ? fmax(1e-6, h0 * 1e-3) : pow(0.01 / md, 0.25);
    dt_prop = fmin(100.0 * h0, hh);
    if constexpr (kTd) {
      tnext = next_trial(a.jump_ts, a.n_jump, t, dt_prop, sh.t1, true, made_jump);
    } else {
      double tn = t + dt_prop;
      if (tn > sh.t1 - 1e-10) tn = sh.t1;
      tnext = tn < sh.t1 ? tn : sh.t1;
    }
  }

  // ---- main loop -----------------------------------------------------------------------
  while (t < sh.t1) {
    if (nsteps >= o.max_steps) {
      status = DQB_INST_MAX_STEPS;
      break;
    }
    if (a.cancel != nullptr && (nsteps & 15) == 0) {  // a caller's stop request
      __syncthreads();
      if (tid == 0) ls.flag = *a.cancel;
      __syncthreads();
      if (ls.flag != 0) {
        status = DQB_INST_CANCELLED;
        break;
      }
    }
    h = tnext - t;
    set_coefs();
    const float2* X = nullptr;
#pragma unroll
    for (int s = 1; s < 7; ++s) {  // stages 2..7; the input of the last is y1 (FSAL)
      load_y();
#pragma unroll
      for (int j = 0; j < 6; ++j)
        if (j < s) {
          const float cj = cfw[s * (s - 1) / 2 + j];
#pragma unroll
          for (int q = 0; q < Q; ++q) v[q] = caxpy(cj, kval(j, q), v[q]);
        }
      X = rhs(s == 6 ? tnext : t + c_tab[o.method].c[s] * h);
      copy(k[s], v);
    }
    // ---- embedded error, FP64 ----
    double sm[1];
    {
      const Tableau& tab = c_tab[o.method];
      double cb[7];
#pragma unroll
      for (int j = 0; j < 7; ++j) cb[j] = h * tab.btilde[j];
      block_sums(sm, sh, par, [&](double (&e)[1], int r, int c) {
        const int q = tile_of(r, c);
        if (!((own >> q) & 1u)) return;
        const float2 y1 = X[(ty + T * r) * LD + tx + T * c];
        double ex = 0.0, ey = 0.0;
#pragma unroll
        for (int j = 0; j < 7; ++j) {
          const float2 kv = kval(j, q);
          ex = fma(cb[j], (double)kv.x, ex);
          ey = fma(cb[j], (double)kv.y, ey);
        }
        const float ya = cabsf(y[q * NT]), yb = cabsf(y1);
        const double sc = o.atol + o.rtol * (double)(ya > yb ? ya : yb);
        e[0] += ((strict >> q) & 1u ? 2.0 : 1.0) * fma(ex, ex, ey * ey) / (sc * sc);
      });
    }
    const double err = sqrt(sm[0] * sh.inv_nn);
    nsteps += 1;
    if (!(err < INFINITY)) {
      status = DQB_INST_NONFINITE;
      break;
    }
    const bool keep = err < 1.0;
    const double dtnew = (kTd && made_jump ? dt_prop : h) * step_factor(o, err, keep);
    bool fresh = false;
    if (keep) {
      nacc += 1;
      if (kTape && a.tape_y && nacc <= a.tape_cap) {
        // gradient tape: the accepted step's start time, size and starting state
        const long long idx = nacc - 1;
        if (tid == 0) {
          a.tape_t[idx] = t;
          a.tape_h[idx] = h;
        }
        load_y();
        const float2* Y = stage(v);
        __syncthreads();
        float2* dst = a.tape_y + (a.inst * (long long)a.tape_cap + idx) * tape_np * tape_np;
        for (int e = tid; e < tape_np * tape_np; e += NT) {
          const int i = e / tape_np, j = e - i * tape_np;
          dst[e] = (i < n && j < n) ? Y[i * LD + j] : make_float2(0.f, 0.f);
        }
        __syncthreads();
      }
      // dense output at every save time in (t, tnext]
      while (sidx < a.ntsave && a.tsave[sidx] <= tnext) {
        double w[7];
        dense_weights(o.method, h > 0.0 ? (a.tsave[sidx] - t) / h : 1.0, w);
        load_y();
#pragma unroll
        for (int j = 0; j < 7; ++j) {
          const float cw = (float)(h * w[j]);
#pragma unroll
          for (int q = 0; q < Q; ++q) v[q] = caxpy(cw, kval(j, q), v[q]);
        }
        save(v);
      }
      // y1 again, by the same operations (rather than kept in registers meanwhile)
      load_y();
#pragma unroll
      for (int j = 0; j < 6; ++j) {
        const float cj = cfw[15 + j];
#pragma unroll
        for (int q = 0; q < Q; ++q) v[q] = caxpy(cj, kval(j, q), v[q]);
      }
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        y[q * NT] = v[q];
        k1[q * NT] = k[6][q];
      }
      // a step that ended just before a discontinuity: the next starts on it, with its
      // first stage evaluated there
      t = (kTd && made_jump) ? nextafter(tnext, INFINITY) : tnext;
      fresh = kTd && made_jump && t < sh.t1;
    }
    if constexpr (kTd) {
      dt_prop = dtnew;
      tnext = next_trial(a.jump_ts, a.n_jump, t, dtnew, sh.t1, keep, made_jump);
    } else {
      tnext = next_tend(t, dtnew, sh.t1, keep);
    }
    if (fresh) {
      load_y();
      rhs(t);
      store_k1(v);
    }
  }

  // saves left over (t1 <= t0: every save is the initial state)
  if (status == DQB_INST_OK)
    while (sidx < a.ntsave && a.tsave[sidx] <= t) {
      load_y();
      save(v);
    }
  if (!a.save_states) {  // final state when only it is kept
    load_y();
    const float2* X = stage(v);
    __syncthreads();
    copy_out(X, a.states, n);
  }
  if (ls.given) save_given(a, sh, sidx, !(t > a.t0));
  // every output before the status (see solve_one)
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    a.infos[0] = (int)nsteps;
    a.infos[1] = (int)nacc;
    a.infos[2] = (int)(nsteps - nacc);
    __threadfence_system();
    a.status[0] = status;
  }
  return true;
}

// Resident CTAs that the register budget is set for: the elements of a thread decide (and
// T = 16 runs n <= 32 for at most two instances per SM).
template <int T, int R>
constexpr int min_ctas() {
  return T == 16 ? (R <= 2 ? 2 : 1) : (R == 1 ? 12 : (R == 2 ? 8 : (R == 3 ? 6 : 4)));
}

template <int T, int R, int FEAT, bool RAG>
__global__ void __launch_bounds__(T * T, min_ctas<T, R>()) mesolve_band_kernel(Args a) {
  extern __shared__ float4 smem_raw[];
  __shared__ Shared<T, R> sh;
  float2* dyn = reinterpret_cast<float2*>(smem_raw);
  for (;;) {
    if (threadIdx.x == 0) sh.inst = (long long)atomicAdd(a.counter, 1u);
    __syncthreads();
    const long long pos = sh.inst;
    if (pos >= a.d.batch) break;
    const long long inst = a.d.order ? (long long)a.d.order[pos] : pos;
    if (inst >= 0 && inst < a.d.batch) {
      if (threadIdx.x == 0) sh.v = RAG ? view_of_ragged(a.rag[inst], inst) : view_of(a.d, inst);
      __syncthreads();
      const bool done = sh.v.n <= Geo<T, R>::NP && solve<T, R, FEAT>(a.d.o, &a.d.td, sh, dyn, a.tape_np);
      if (threadIdx.x == 0 && (RAG || !done)) a.pend[inst * a.pend_stride] = done ? 0 : kPending;
    }
    __syncthreads();  // every thread has read sh.inst, and the tables are free
  }
}

// Launches the kernel on resident CTAs (at most one per instance).  Its attributes and
// occupancy are looked up once per device.
template <int T, int R, int FEAT, bool RAG>
static int launch(const Args& a, int dev, int sms, cudaStream_t s) {
  auto kern = mesolve_band_kernel<T, R, FEAT, RAG>;
  constexpr int smem = dyn_values<T, R>(FEAT == 1) * (int)sizeof(float2);
  static std::mutex mu;
  static int resident[kMaxDevices] = {};
  int per_sm = 0;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (resident[dev] == 0) {
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      prefer_max_shared(kern);
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident[dev], kern, T * T, smem);
    }
    per_sm = resident[dev];
  }
  if (per_sm < 1) return DQB_ERR_CUDA;
  const long long g = std::min<long long>((long long)per_sm * sms, a.d.batch);
  kern<<<(unsigned)g, T * T, smem, s>>>(a);
  return cudaGetLastError() == cudaSuccess ? DQB_OK : DQB_ERR_CUDA;
}

template <int FEAT, bool RAG>
static int launch_for(const Args& a, int n, cudaStream_t s) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return DQB_ERR_CUDA;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (n <= 32 && a.d.batch > 2 * sms) {
    if (n <= 8) return launch<8, 1, FEAT, RAG>(a, dev, sms, s);
    if (n <= 16) return launch<8, 2, FEAT, RAG>(a, dev, sms, s);
    if (n <= 24) return launch<8, 3, FEAT, RAG>(a, dev, sms, s);
    return launch<8, 4, FEAT, RAG>(a, dev, sms, s);
  }
  if (n <= 16) return launch<16, 1, FEAT, RAG>(a, dev, sms, s);
  if (n <= 32) return launch<16, 2, FEAT, RAG>(a, dev, sms, s);
  if (n <= 48) return launch<16, 3, FEAT, RAG>(a, dev, sms, s);
  return launch<16, 4, FEAT, RAG>(a, dev, sms, s);
}

int run(const Args& a, int n, int feat, cudaStream_t s) {
  if (a.rag) return launch_for<0, true>(a, n, s);
  switch (feat) {
    case 1: return launch_for<1, false>(a, n, s);
    case 2: return launch_for<2, false>(a, n, s);
    default: return launch_for<0, false>(a, n, s);
  }
}

}  // namespace band
}  // namespace dqb
