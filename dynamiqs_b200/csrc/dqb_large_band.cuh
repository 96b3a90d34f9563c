// Banded operators on the dense n > 64 path (included by dqb_dense_large.cu).
//
// Operators in dense storage are usually banded (kron products of ladder and number
// operators); their products with X are stencils of a few terms per element, against n
// terms per product.  At the start of a solve the nonzero diagonals of every instance's
// operators are listed on the device; instances with at most kBandMaxH of them in
// Hnh and kBandMaxL in the jump operators take their right-hand sides from
// band_rhs_kernel, one pass over X, and every product
// kernel skips them.  Nothing is decided on the host: the graph holds a loop with the
// product launches, one with the stencil and one with both, and runs the one that the
// instances need (an empty launch costs about 2 us, three per right-hand side).
//
// The stencil forms the sums of the FP32 product path term by term -- a product's sum by
// ascending inner index, then the terms in their order, then tmp + tmp^+ -- so for a
// hermitian X the result is the same to the last bit.  (With a tensor-core precision the
// banded instances are computed in FP32, which is at least as exact.)
//
// Measured (one B200): transmon x cavity, n = 256, two jumps, 64 instances: 19.0 ms per
// solve of 12 steps with 3xTF32 products, 4.5 ms with the stencil (24 us a right-hand side
// against 196 us).  Bound: instructions and latency of the displaced reads (every operand
// comes from L1 or L2); the floor is X read once and k
// written once, on the 32 x 32 tiles on and above the diagonal where only the
// hermitian-half kernels read it.
#pragma once

// What the records hold; at eight diagonals of Hnh, no jump, the stencil is still 1.8 (n = 100,
// 32 instances) to 3.9 (n = 256, 32) times as fast as the products.
constexpr int kBandMaxH = 8;  // nonzero diagonals of Hnh
constexpr int kBandMaxL = 8;  // nonzero diagonals of the jump operators together
constexpr int kBandMaxK = 8;  // jump operators

struct BandRec {  // one instance
  int ok;         // banded: taken by the stencil, skipped by the products
  int nh, nk;
  int hoff[kBandMaxH];                          // ascending
  int loff[kBandMaxL], lstart[kBandMaxK + 1];   // per jump operator, ascending
};

struct BandTabs {
  BandRec* rec;    // [B], or null: every instance takes the products
  unsigned* mask;  // [B][1 + K][words]: nonzero diagonals of H and the jumps (bit j - i + n - 1)
  int words;
  float2* hd;      // [B][kBandMaxH][n]: Hnh[i][i + off] at i
  float2* ld;      // [B][kBandMaxL][n]: L[i][i + off] at i
  int* work;       // Work bits (dqb_dense_large.cu) of all instances: full operators, banded
};
