// Batched linear ODEs d y/dt = A y on the same Runge-Kutta engine as the master-equation
// kernels (the Tsit5 / Dopri5 tableaux, starting step, FP64 error norm, integral
// controller and dense output of dqb_common.cuh), in two forms:
//   * the Schroedinger equation d psi/dt = -i H psi (dynamiqs/integrators/core/
//     diffrax_integrator.py:221-228, sesolve.py), y = psi, expectation values
//     <psi|E|psi>;
//   * the vectorized master equation d vec(rho)/dt = S vec(rho) with the Lindbladian
//     superoperator S (diffrax_integrator.py:325-327, utils/vectorization.py:213-259),
//     y = vec(rho) (columns stacked), expectation values tr(E rho) = sum_ij E[i][j]
//     rho[j][i], a dot product of y with E read row by row.
//
// Two kernels share the solve (solve_instance), by the operator of the instance:
//   * band_kernel: H in dense storage with at most kMaxH nonzero diagonals (as bosonic
//     Hamiltonians have), listed on the device; the product is a stencil of those
//     diagonals, so a step is short and one warp takes an instance, lane l holding the
//     entries l + 32 r.  Its small shared memory (diagonals and stage input) lets every warp
//     slot of the SM hold an instance.  Instances with a full H of more than 32 rows are
//     marked in their step counts and left to
//   * full_kernel: one CTA per instance, one thread per row, the operator in shared memory
//     (rows at an odd stride, so that the lanes' reads down a column are free of bank
//     conflicts) or, beyond 128 rows, read from global memory along its columns.
// Both sum a row's products by ascending column -- the stencil leaves out the zeros --, and
// keep the entries' Runge-Kutta state in registers; the stage input is exchanged through two
// shared buffers used in turn, one barrier per right-hand side.  Everything an instance
// decides -- error norm, accept or reject, next step, save points -- is computed by all of
// its threads from the same reduced values.
//
// Bound: band_kernel by the latency of the longest instance's steps (their FP64 controller
// above all), full_kernel by shared-memory bandwidth (n^2 values of the operator per product).
// Measured (one B200), kernels alone: n = 64 driven Kerr, 1500 instances: 0.77 ms against
// 2.57 ms for one kernel with a warp and a 33 KB tile per instance (six per SM); n = 101 full,
// 400 instances: 0.63 against 2.12 ms (one 132 KB tile, so one warp, per SM).
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "dqb_common.cuh"

namespace dqb {

namespace se {

constexpr int kMaxH = 8;      // diagonals of a banded H (what BandOp's two words hold; at
                              //   eight, n = 64, 1500 instances: 77 against 167 us full)
constexpr int kPending = -1;  // mark (in infos[0]) of an instance left to full_kernel
constexpr int kMaxDevices = 64;

enum Mode { kSchrodinger = 0, kLinear = 1 };

struct Args {
  int n, nE, ntsave;  // n: length of y (the Hilbert dimension, or its square when vectorized)
  int mode;           // Mode
  const float2* AT;   // kLinear: A transposed, complex64 [*, n, n] (A[i][m] at AT[m * n + i])
  long long batch;
  const float2* H;
  const float2* psi0;
  const float2* E;
  const double* tsave;
  const int* Hidx;
  const int* pidx;
  float2* states;
  float2* expects;
  int* infos;
  int* status;
  unsigned int* counter;
  int pending_only;  // full_kernel: take the marked instances only
  CtrlOpts o;
};

// The threads that solve one instance: a warp (R entries per lane), or a CTA of whole warps
// (R = 1).  `red`: 2 x 8 partial sums of a CTA, used in turn (the set is rewritten only after
// a barrier that every reader has passed).
template <int R_, bool kBlock>
struct Team {
  static constexpr int R = R_;
  double* red;
  int par;
  __device__ int rank() const { return kBlock ? threadIdx.x : threadIdx.x & 31; }
  __device__ int size() const { return kBlock ? blockDim.x : 32; }
  __device__ void sync() const {
    if (kBlock) __syncthreads();
    else __syncwarp();
  }
  __device__ double sum(double v) {
    v = warp_sum(v);
    if (!kBlock || blockDim.x == 32) return v;
    if ((threadIdx.x & 31) == 0) red[par * 8 + (threadIdx.x >> 5)] = v;
    __syncthreads();
    v = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += red[par * 8 + w];
    par ^= 1;
    return v;
  }
};

// H given by its diagonals: row i's entries at columns i + off[d], by ascending d (d[q * ld + i]).
struct BandOp {
  const float2* d;
  int ld, nd;
  unsigned long long off;  // one signed 16-bit value each in two words: |off| < 128
  unsigned long long off_hi;
  template <int R>
  __device__ __forceinline__ void mul(const float2* sx, int n, int rank, int size, float2 (&acc)[R]) const {
    // four diagonals per pass, all their reads in flight (the table's rows beyond nd are zero)
#pragma unroll 1
    for (int q0 = 0; q0 < nd; q0 += 4) {
      float2 c[4][R], x[4][R];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int o = (int)(short)((q0 == 0 ? off : off_hi) >> (16 * q));
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int i = rank + size * r;  // beyond the matrix the coefficient is zero, any entry will do
          c[q][r] = d[(q0 + q) * ld + i];
          x[q][r] = sx[min(max(i + o, 0), n - 1)];
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int r = 0; r < R; ++r) cmac(acc[r], c[q][r], x[q][r]);
    }
  }
};

// A full operator: row i at s + i * ld (shared memory), or A[i][m] at g[m * n + i].
struct FullOp {
  const float2* s;
  const float2* g;
  int ld;
  template <int R>
  __device__ __forceinline__ void mul(const float2* sx, int n, int rank, int, float2 (&acc)[R]) const {
    static_assert(R == 1, "one row per thread");
    const int i = min(rank, n - 1);
    if (s) {
      const float2* row = s + i * ld;
#pragma unroll 8
      for (int m = 0; m < n; ++m) cmac(acc[0], row[m], sx[m]);
    } else {
#pragma unroll 8
      for (int m = 0; m < n; ++m) cmac(acc[0], __ldg(g + (long long)m * n + i), sx[m]);
    }
  }
};

// out_r = (A x)_r for the thread's rows (times -i for the Schroedinger form), x staged in sx.
template <int R, class Op>
__device__ __forceinline__ void matvec(const Op& A, int mode, const float2* sx, int n, int rank, int size,
                                       float2 (&out)[R]) {
  float2 acc[R];
#pragma unroll
  for (int r = 0; r < R; ++r) acc[r] = make_float2(0.f, 0.f);
  A.mul(sx, n, rank, size, acc);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    out[r] = mode == kSchrodinger ? make_float2(acc[r].y, -acc[r].x) : acc[r];
    if (rank + size * r >= n) out[r] = make_float2(0.f, 0.f);
  }
}

// One instance's whole solve.  sx: two buffers of `ldx` values; cf: this warp's copy of the
// stage coefficients (24 floats); a21: the tableau's a[s][j], j < s, row by row.
template <class TeamT, class Op>
__device__ void solve_instance(const Args& a, long long inst, const Op& A, TeamT& tm, float2* sx, int ldx,
                               float* cf, const double* a21) {
  constexpr int R = TeamT::R;
  const int n = a.n, rank = tm.rank(), size = tm.size(), lane = threadIdx.x & 31;
  const CtrlOpts& o = a.o;
  const Tableau& T = c_tab[o.method];
  const double inv_n = 1.0 / (double)n;
  const long long pi = a.pidx ? a.pidx[inst] : inst;
  int buf = 0;
  float2 y[R], k[7][R], y1[R], x[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = rank + size * r;
    y[r] = i < n ? a.psi0[pi * n + i] : make_float2(0.f, 0.f);
  }
  // the next buffer <- x, visible to the team
  auto stage = [&](const float2 (&u)[R]) {
    buf ^= 1;
    float2* s = sx + buf * ldx;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = rank + size * r;
      if (i < n) s[i] = u[r];
    }
    tm.sync();
    return s;
  };
  auto rhs = [&](const float2 (&u)[R], float2 (&out)[R]) {
    const float2* s = stage(u);
    matvec<R>(A, a.mode, s, n, rank, size, out);
  };
  // State at save index `sidx` (entries v) and its expectation values (FP64 sums): <v|E_m|v> =
  // sum_ij conj(v_i) E_m[i][j] v_j, or tr(E rho) = sum_k E_k y_k with E read row by row.
  int sidx = 0;
  auto save = [&](const float2 (&v)[R]) {
    if (o.save_states) {
      float2* dst = a.states + (inst * a.ntsave + sidx) * (long long)n;
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (rank + size * r < n) dst[rank + size * r] = v[r];
    }
    const float2* s = (a.nE > 0 && a.mode == kSchrodinger) ? stage(v) : nullptr;
    for (int m = 0; m < a.nE; ++m) {
      double er = 0.0, ei = 0.0;
      const float2* Em = a.E + (long long)m * (a.mode == kLinear ? n : (long long)n * n);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int j = rank + size * r;
        if (j >= n) continue;
        float2 e = make_float2(0.f, 0.f);
        if (a.mode == kLinear) {
          e = Em[j];
        } else {
#pragma unroll 8
          for (int i = 0; i < n; ++i) cmac(e, cconj(s[i]), __ldg(Em + (long long)i * n + j));
        }
        er += (double)e.x * v[r].x - (double)e.y * v[r].y;
        ei += (double)e.x * v[r].y + (double)e.y * v[r].x;
      }
      er = tm.sum(er);
      ei = tm.sum(ei);
      if (rank == 0) a.expects[(inst * a.nE + m) * a.ntsave + sidx] = make_float2((float)er, (float)ei);
    }
    ++sidx;
  };

  // ---- starting step (Hairer-Norsett-Wanner, RMS norm) --------------------------------
  rhs(y, k[0]);
  double s0 = 0.0, s1 = 0.0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (rank + size * r >= n) continue;
    const double sc = o.atol + o.rtol * (double)cabsf(y[r]);
    s0 += (double)cabs2f(y[r]) / (sc * sc);
    s1 += (double)cabs2f(k[0][r]) / (sc * sc);
  }
  s0 = tm.sum(s0);
  s1 = tm.sum(s1);
  const double d0 = sqrt(s0 * inv_n), d1 = sqrt(s1 * inv_n);
  const double h0 = (d0 < 1e-5 || d1 < 1e-5) ? 1e-6 : 0.01 * d0 / d1;
#pragma unroll
  for (int r = 0; r < R; ++r) x[r] = caxpy((float)h0, k[0][r], y[r]);
  rhs(x, k[1]);
  double s2 = 0.0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (rank + size * r >= n) continue;
    const double sc = o.atol + o.rtol * (double)cabsf(y[r]);
    const double dx = (double)k[1][r].x - (double)k[0][r].x, dy = (double)k[1][r].y - (double)k[0][r].y;
    s2 += (dx * dx + dy * dy) / (sc * sc);
  }
  s2 = tm.sum(s2);
  const double t1 = a.tsave[a.ntsave - 1];
  double t = o.t0, tnext;
  {
    const double d2 = sqrt(s2 * inv_n) / h0;
    const double md = d1 > d2 ? d1 : d2;
    const double h1 = md <= 1e-15 ? fmax(1e-6, h0 * 1e-3) : pow(0.01 / md, 0.25);
    const double dt = fmin(100.0 * h0, h1);
    double tn = t + dt;
    if (tn > t1 - 1e-10) tn = t1;
    tnext = tn < t1 ? tn : t1;
  }
  long long nsteps = 0, nacc = 0;
  int status = DQB_INST_OK;

  // ---- main loop ----------------------------------------------------------------------
  while (t < t1) {
    if (nsteps >= o.max_steps) {
      status = DQB_INST_MAX_STEPS;
      break;
    }
    const double h = tnext - t;
    __syncwarp();
    if (lane < 21) cf[lane] = (float)(h * a21[lane]);
    __syncwarp();
#pragma unroll
    for (int s = 1; s < 7; ++s) {
#pragma unroll
      for (int r = 0; r < R; ++r) x[r] = y[r];
#pragma unroll
      for (int j = 0; j < 6; ++j)
        if (j < s) {
          const float cj = cf[s * (s - 1) / 2 + j];
#pragma unroll
          for (int r = 0; r < R; ++r) x[r] = caxpy(cj, k[j][r], x[r]);
        }
      if (s == 6) {
#pragma unroll
        for (int r = 0; r < R; ++r) y1[r] = x[r];  // row 6 of a is b (FSAL)
      }
      rhs(x, k[s]);  // (the unrolled stage loop keeps k[] in registers)
    }
    double se = 0.0;
    double cb[7];
#pragma unroll
    for (int j = 0; j < 7; ++j) cb[j] = h * T.btilde[j];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      double ex = 0.0, ey = 0.0;
#pragma unroll
      for (int j = 0; j < 7; ++j) {
        ex = fma(cb[j], (double)k[j][r].x, ex);
        ey = fma(cb[j], (double)k[j][r].y, ey);
      }
      const float ya = cabsf(y[r]), y1a = cabsf(y1[r]);
      const double sc = o.atol + o.rtol * (double)(ya > y1a ? ya : y1a);
      if (rank + size * r < n) se += ratio(ex * ex + ey * ey, sc * sc);
    }
    se = tm.sum(se);
    const double err = sqrt(se * inv_n);
    nsteps += 1;
    if (!(err < INFINITY)) {
      status = DQB_INST_NONFINITE;
      break;
    }
    const bool keep = err < 1.0;
    const double dtnew = h * step_factor(o, err, keep);
    if (keep) {
      nacc += 1;
      while (sidx < a.ntsave && a.tsave[sidx] <= tnext) {
        double w[7];
        const double theta = h > 0.0 ? (a.tsave[sidx] - t) / h : 1.0;
        dense_weights(o.method, theta, w);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          x[r] = y[r];
#pragma unroll
          for (int j = 0; j < 7; ++j) x[r] = caxpy((float)(h * w[j]), k[j][r], x[r]);
        }
        save(x);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        y[r] = y1[r];
        k[0][r] = k[6][r];
      }
      t = tnext;
    }
    tnext = next_tend(t, dtnew, t1, keep);
  }
  // saves left over (t1 <= t0: every save is the initial state)
  if (status == DQB_INST_OK)
    while (sidx < a.ntsave && a.tsave[sidx] <= t) save(y);
  if (!o.save_states) {
    float2* dst = a.states + inst * (long long)n;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (rank + size * r < n) dst[rank + size * r] = y[r];
  }
  __threadfence();
  tm.sync();
  if (rank == 0) {
    a.infos[inst * 3 + 0] = (int)nsteps;
    a.infos[inst * 3 + 1] = (int)nacc;
    a.infos[inst * 3 + 2] = (int)(nsteps - nacc);
    __threadfence_system();
    a.status[inst] = status;
  }
}

__device__ __forceinline__ void load_tableau(double* a21, int method) {
  for (int e = threadIdx.x; e < 21; e += blockDim.x) {
    int s = 1;
    while (e >= s * (s + 1) / 2) ++s;
    a21[e] = c_tab[method].a[s][e - s * (s - 1) / 2];
  }
}

// One warp per CTA and instance; n <= 32 R.  Shared memory: kMaxH diagonals, two x buffers.
// kFull (R = 1): a full H is solved here, too, its operator in dynamic shared memory, and
// full_kernel is not launched: up to 32 rows a warp has a row per lane and the operator costs
// few resident warps.  One instance of n = 5, full H: 43 us against 52 with the second launch
// (40 in a kernel with a 33 KB tile per warp); n = 32: 67 and 79; 20000 of n = 16: 436 and
// 535, banded 243 and 261.
constexpr int kFullMaxN = 32;

template <int R, bool kFull>
__global__ void __launch_bounds__(32, kFull ? 20 : (R == 2 ? 16 : 12)) band_kernel(Args a) {
  static_assert(!kFull || R == 1, "one row per lane");
  constexpr int NP = 32 * R;
  extern __shared__ float4 se_smem[];
  __shared__ float2 sd[kMaxH * NP];
  __shared__ float2 sx[2 * NP];
  __shared__ double a21[21];
  __shared__ float cf[24];
  __shared__ unsigned mask[8];
  const int lane = threadIdx.x, n = a.n;
  load_tableau(a21, a.o.method);
  for (;;) {
    unsigned int v = 0;
    if (lane == 0) v = atomicAdd(a.counter, 1u);
    const long long inst = (long long)__shfl_sync(0xffffffffu, v, 0);
    if (inst >= a.batch) break;
    const float2* H = a.H + (a.Hidx ? a.Hidx[inst] : inst) * (long long)n * n;
    __syncwarp();
    if (lane < 8) mask[lane] = 0u;
    __syncwarp();
    // the nonzeros of one row lie on as many diagonals: full matrices are told by one row
    int mid = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float2 e = lane + 32 * r < n ? __ldg(H + (long long)(n / 2) * n + lane + 32 * r) : make_float2(0.f, 0.f);
      mid += __popc(__ballot_sync(0xffffffffu, e.x != 0.f || e.y != 0.f));
    }
    BandOp A;
    A.d = sd;
    A.ld = NP;
    A.nd = 0;
    A.off = A.off_hi = 0;
    bool ok = mid <= kMaxH;
    if (ok) {
      // nonzero diagonals (bit j - i + n - 1)
      constexpr int U = 8 / R;  // rows in flight
      for (int i0 = 0; i0 < n; i0 += U) {
        float2 e[U][R];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const int i = i0 + u, j = lane + 32 * r;
            e[u][r] = (i < n && j < n) ? __ldg(H + (long long)i * n + j) : make_float2(0.f, 0.f);
          }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int r = 0; r < R; ++r)
            if (e[u][r].x != 0.f || e[u][r].y != 0.f) {
              const int b = lane + 32 * r - (i0 + u) + n - 1;
              if (!(*(volatile unsigned*)&mask[b >> 5] >> (b & 31) & 1u)) atomicOr(&mask[b >> 5], 1u << (b & 31));
            }
      }
      for (int e = lane; e < kMaxH * NP; e += 32) sd[e] = make_float2(0.f, 0.f);
      __syncwarp();
      for (int w = 0; w < 8; ++w)
        for (unsigned x = mask[w]; x; x &= x - 1) {
          if (A.nd == kMaxH) {
            ok = false;
            break;
          }
          const int off = 32 * w + __ffs((int)x) - 1 - (n - 1);
          const unsigned long long f = (unsigned long long)(off & 0xffff) << (16 * (A.nd & 3));
          if (A.nd < 4) A.off |= f;
          else A.off_hi |= f;
          for (int i = lane; i < NP; i += 32) {
            const int j = i + off;
            sd[A.nd * NP + i] = (i < n && j >= 0 && j < n) ? __ldg(H + (long long)i * n + j) : make_float2(0.f, 0.f);
          }
          ++A.nd;
        }
      __syncwarp();
    }
    if (!ok) {
      if constexpr (kFull) {
        const int ld = n | 1;
        float2* sA = reinterpret_cast<float2*>(se_smem);
        for (int p = 0; p < n; ++p)
          if (lane < n) sA[p * ld + lane] = __ldg(H + p * n + lane);
        __syncwarp();
        const FullOp F{sA, nullptr, ld};
        Team<1, false> tm{nullptr, 0};
        solve_instance(a, inst, F, tm, sx, NP, cf, a21);
      } else if (lane == 0) {
        a.infos[inst * 3] = kPending;
      }
      continue;
    }
    Team<R, false> tm{nullptr, 0};
    solve_instance(a, inst, A, tm, sx, NP, cf, a21);
  }
}

// One CTA per instance, one thread per row (blockDim.x = n rounded up to whole warps).
// G: the operator stays in global memory (A^T), else in dynamic shared memory.
template <bool G>
__global__ void __launch_bounds__(256) full_kernel(Args a) {
  extern __shared__ float4 se_smem[];
  __shared__ double red[16];
  __shared__ double a21[21];
  __shared__ float cf[8][24];
  __shared__ unsigned int next;
  const int n = a.n, ld = n | 1;
  float2* sx = reinterpret_cast<float2*>(se_smem);  // two buffers of n (rounded up to even) values
  const int ldx = (n + 1) & ~1;
  float2* sA = sx + 2 * ldx;
  load_tableau(a21, a.o.method);
  for (;;) {
    if (threadIdx.x == 0) next = atomicAdd(a.counter, 1u);
    __syncthreads();
    const long long inst = next;
    if (inst >= a.batch) break;
    const bool mine = !a.pending_only || a.infos[inst * 3] == kPending;
    __syncthreads();  // every thread has read `next`, and the previous instance's tile is free
    if (!mine) continue;
    const long long hi = a.Hidx ? a.Hidx[inst] : inst;
    FullOp A{nullptr, nullptr, ld};
    if (G) {
      A.g = a.AT + hi * (long long)n * n;
    } else {
      const float2* src = (a.mode == kLinear ? a.AT : a.H) + hi * (long long)n * n;
      for (int p = threadIdx.x >> 5; p < n; p += blockDim.x >> 5)
        for (int q = threadIdx.x & 31; q < n; q += 32) {
          const float2 v = src[p * n + q];
          if (a.mode == kLinear) sA[q * ld + p] = v;  // A[q][p] = AT[p][q]
          else sA[p * ld + q] = v;
        }
      A.s = sA;
    }
    __syncthreads();
    Team<1, true> tm{red, 0};
    solve_instance(a, inst, A, tm, sx, ldx, cf[threadIdx.x >> 5], a21);
    __syncthreads();
  }
}

// One right-hand side -i H psi per instance (no RK loop): one CTA, one thread per row.
__global__ void __launch_bounds__(128) schrodinger_rhs_kernel(Args a, const float2* psi, float2* out) {
  __shared__ float2 sx[128];
  const long long b = blockIdx.x;
  const int n = a.n, i = threadIdx.x;
  if (i < n) sx[i] = psi[b * n + i];
  __syncthreads();
  if (i >= n) return;
  const float2* row = a.H + (a.Hidx ? a.Hidx[b] : b) * (long long)n * n + (long long)i * n;
  float2 acc = make_float2(0.f, 0.f);
#pragma unroll 8
  for (int m = 0; m < n; ++m) cmac(acc, __ldg(row + m), sx[m]);
  out[b * n + i] = make_float2(acc.y, -acc.x);
}

size_t max_optin_smem() {
  int dev = 0, v = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  return v > 0 ? (size_t)v : (size_t)232448;
}

// Launches a persistent kernel on its resident CTAs (at most one per instance).
template <void (*kern)(Args)>
int launch(const Args& a, int threads, size_t smem, cudaStream_t s) {
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return DQB_ERR_CUDA;
  static std::mutex mu;
  static bool raised[kMaxDevices] = {};
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!raised[dev]) {  // the attribute is raised once per device, never lowered
      cudaFuncAttributes fa;
      cudaFuncGetAttributes(&fa, kern);
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)max_optin_smem() - (int)fa.sharedSizeBytes);
      prefer_max_shared(kern);
      raised[dev] = true;
    }
  }
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
  if (per_sm < 1) return DQB_ERR_UNSUPPORTED;
  const long long grid = std::max<long long>(std::min<long long>((long long)sms * per_sm, a.batch), 1);
  kern<<<(unsigned)grid, threads, smem, s>>>(a);
  return cudaGetLastError() == cudaSuccess ? DQB_OK : DQB_ERR_CUDA;
}

// Shared memory of full_kernel: two x buffers, and the operator's tile.
size_t full_smem(int n, bool tile) {
  return (2 * (size_t)((n + 1) & ~1) + (tile ? (size_t)n * (n | 1) : 0)) * sizeof(float2);
}

int check(const dqb_dense_problem* p, int max_n) {
  if (!p) return DQB_ERR_INVALID_ARGUMENT;
  if (p->n < 1 || p->n_jumps != 0 || p->n_exp < 0 || p->n_tsave < 1 || p->batch < 0) return DQB_ERR_INVALID_ARGUMENT;
  if (p->batch >= (int64_t)0x7fffffff) return DQB_ERR_INVALID_ARGUMENT;
  if (!p->H || !p->rho0 || !p->tsave || (p->n_exp > 0 && !p->E)) return DQB_ERR_INVALID_ARGUMENT;
  if (p->n > max_n) return DQB_ERR_UNSUPPORTED;
  return DQB_OK;
}

int check_run(const dqb_dense_problem* p, const dqb_ode_options* o, const dqb_outputs* out, int max_n) {
  int rc = check(p, max_n);
  if (rc) return rc;
  if (!o || !out || !out->states || !out->infos || !out->status || (p->n_exp > 0 && !out->expects))
    return DQB_ERR_INVALID_ARGUMENT;
  if (o->method != DQB_METHOD_TSIT5 && o->method != DQB_METHOD_DOPRI5) return DQB_ERR_INVALID_ARGUMENT;
  if (!(o->rtol >= 0) || !(o->atol >= 0) || o->max_steps < 0) return DQB_ERR_INVALID_ARGUMENT;
  return DQB_OK;
}

Args make(const dqb_dense_problem* p) {
  Args a;
  a.mode = kSchrodinger;
  a.AT = nullptr;
  a.n = p->n;
  a.nE = p->n_exp;
  a.ntsave = p->n_tsave;
  a.batch = p->batch;
  a.H = (const float2*)p->H;
  a.psi0 = (const float2*)p->rho0;
  a.E = (const float2*)p->E;
  a.tsave = p->tsave;
  a.Hidx = p->H_index;
  a.pidx = p->rho0_index;
  a.states = a.expects = nullptr;
  a.infos = a.status = nullptr;
  a.counter = nullptr;
  a.pending_only = 0;
  return a;
}

}  // namespace se
}  // namespace dqb

using namespace dqb;

extern "C" size_t dqb_sesolve_dense_workspace_size(void) { return 256; }

static int run(se::Args& a, const dqb_dense_problem* p, const dqb_ode_options* o, const dqb_outputs* out,
               void* workspace, size_t workspace_bytes, cudaStream_t s) {
  if (p->batch == 0) return DQB_OK;
  if (!workspace || workspace_bytes < 256) return DQB_ERR_WORKSPACE_TOO_SMALL;
  a.states = (float2*)out->states;
  a.expects = (float2*)out->expects;
  a.infos = out->infos;
  a.status = out->status;
  a.counter = (unsigned int*)workspace;
  a.o = make_ctrl(*o);
  const int n = p->n, threads = 32 * ((n + 31) / 32);
  zero_words_kernel<<<1, 64, 0, s>>>((unsigned int*)workspace, 64);
  if (a.mode == se::kSchrodinger && n <= se::kFullMaxN)
    return se::launch<se::band_kernel<1, true>>(a, 32, (size_t)n * (n | 1) * sizeof(float2), s);
  if (a.mode == se::kSchrodinger) {  // the banded instances first; the others are marked
    const int rc = n <= 64 ? se::launch<se::band_kernel<2, false>>(a, 32, 0, s)
                           : se::launch<se::band_kernel<4, false>>(a, 32, 0, s);
    if (rc) return rc;
    a.counter += 1;
    a.pending_only = 1;
  }
  if (n <= 128) return se::launch<se::full_kernel<false>>(a, threads, se::full_smem(n, true), s);
  return se::launch<se::full_kernel<true>>(a, threads, se::full_smem(n, false), s);
}

extern "C" int dqb_sesolve_dense(const dqb_dense_problem* p, const dqb_ode_options* o, const dqb_outputs* out,
                                 void* workspace, size_t workspace_bytes, void* stream) {
  int rc = se::check_run(p, o, out, 128);
  if (rc) return rc;
  se::Args a = se::make(p);
  return run(a, p, o, out, workspace, workspace_bytes, (cudaStream_t)stream);
}

extern "C" int dqb_mesolve_vectorized(const dqb_dense_problem* p, const void* superop_t, const dqb_ode_options* o,
                                      const dqb_outputs* out, void* workspace, size_t workspace_bytes,
                                      void* stream) {
  int rc = se::check_run(p, o, out, 256);
  if (rc) return rc;
  if (!superop_t) return DQB_ERR_INVALID_ARGUMENT;
  se::Args a = se::make(p);
  a.mode = se::kLinear;
  a.AT = (const float2*)superop_t;
  return run(a, p, o, out, workspace, workspace_bytes, (cudaStream_t)stream);
}

extern "C" int dqb_schrodinger_rhs_dense(const dqb_dense_problem* p, const void* psi, void* outp, void* stream) {
  int rc = se::check(p, 128);
  if (rc) return rc;
  if (!psi || !outp) return DQB_ERR_INVALID_ARGUMENT;
  if (p->batch == 0) return DQB_OK;
  const se::Args a = se::make(p);
  cudaStream_t s = (cudaStream_t)stream;
  se::schrodinger_rhs_kernel<<<(unsigned)p->batch, 128, 0, s>>>(a, (const float2*)psi, (float2*)outp);
  return cudaGetLastError() == cudaSuccess ? DQB_OK : DQB_ERR_CUDA;
}
