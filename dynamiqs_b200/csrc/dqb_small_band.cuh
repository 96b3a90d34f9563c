// Interface between the banded kernel (dqb_dense_small_band.cu) and the product kernel
// (dqb_dense_small.cu) of the n <= 64 path: the first solves the instances whose operators
// have few nonzero diagonals and marks the others, the second takes the marked ones.
#pragma once

#include "dqb_small.cuh"

namespace dqb {
namespace band {

constexpr int kPending = -1;  // mark of an instance left to the product kernel

struct Args {
  DenseSmallArgs d;                // (ragged launches: batch and o only)
  const dqb_ragged_instance* rag;  // per-instance descriptors, or null
  unsigned int* counter;           // work counter, zeroed
  int* pend;                       // mark of instance b at pend[b * pend_stride]; a solved instance's
  int pend_stride;                 //   own outputs may lie there instead (never negative)
  int tape_np;                     // row length of the tape's states
};

// Enqueues the banded kernel for instances of dimension at most n (n <= 64), hermitian
// form.  feat: 0 = plain, 1 = time-dependent H, 2 = gradient tape (as mesolve_small_kernel).
int run(const Args& a, int n, int feat, cudaStream_t s);

}  // namespace band
}  // namespace dqb
