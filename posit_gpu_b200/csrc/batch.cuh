// batch.cuh -- batched posit32 factor-and-solve problems (batch.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace pg {

constexpr int BATCH_LU = 0;
constexpr int BATCH_CHOL = 1;
constexpr int BATCH_MAX_N = 4096; // largest n a batched problem may have
constexpr int BATCH_LARGE_N = 224;  // a problem of more rows takes an SM for itself
constexpr int BATCH_WARP_N = 32;    // a problem of up to this many rows may be a warp's
// From this many right-hand sides on a warp is the slower place for such a problem, unless there
// are so many of them that CTAs take more than three turns.  One problem of n = 32 with 300 right-hand
// sides: 1520 us by a warp, 462 by a CTA; 2000 of them: 2571 us by warps, about 3400 by CTAs.
constexpr int BATCH_WARP_RHS = 16;
constexpr int BATCH_CTA_TURNS = 3;
// One problem: A (n x n, column-major, lda) is factored in place, B (n x nrhs, ldb)
// overwritten with the solution; ipiv (LU) receives n 1-based pivots, info the
// reference's info.  All pointers are device pointers.
constexpr int BATCH_SOLVE_ONLY = 2; // flag added to kind: A (and ipiv) already factored

struct BatchProblem {
    int kind; // BATCH_LU or BATCH_CHOL, plus BATCH_SOLVE_ONLY
    int n, lda, nrhs, ldb;
    uint32_t *A;
    uint32_t *B;
    int *ipiv;
    int *info;
};

// Runs problems probs[order[i]] (order null: probs[i]), first <= i < last, on persistent CTAs;
// `order` sorts by decreasing n.  `large`: one CTA per SM (problems of more than
// BATCH_LARGE_N rows), else two smaller ones; those from warp_from on (of up to BATCH_WARP_N
// rows) go to a warp each.  `spread`: by the kernels that spread right-hand sides over the threads
// (batch_spread_pays; the bits are the same).  `next` is a device counter the launch zeroes first.  A null order may be in any order, of any sizes, with warp_from = last.
cudaError_t batch_factor_launch(bool large, bool spread, const BatchProblem *probs, int first, int last, const int *order,
                                int warp_from, int *next, int sms, cudaStream_t st);

// Whether such a launch of the host array's problems probs[order[i]] (order null: probs[i]), first <=
// i < last, is shorter with the kernels that spread right-hand sides over the threads.
bool batch_spread_pays(bool large, const BatchProblem *probs, int first, int last, const int *order, int sms);

} // namespace pg
