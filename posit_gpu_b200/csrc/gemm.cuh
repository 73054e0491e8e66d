// gemm.cuh -- posit32 GEMM kernels for sm_100a (declarations shared by the C ABI).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "gemm_tile.cuh"

namespace pg {

// The staged route's output tile: 16*TM x 16*TN outputs per CTA of 256 threads, TM x TN per
// thread (gemm_tile.cuh).  4x4 at 2 CTAs per SM (up to 128 registers: the accumulators, their
// values at the k tile's start and the operands of a step).
constexpr int TM = 4; // rows per thread
constexpr int TN = 4; // columns per thread
constexpr int STAGES = 3;
constexpr int MIN_CTAS_PER_SM = 2;
constexpr int SM_COUNT = 148;

// How a product is computed (gemm_route); the bits are the same.
enum GemmRoute { GEMM_STAGED, GEMM_FUSED_64x32, GEMM_FUSED_32x32 };

// Error flags a kernel can raise (read back with posit_get_device_error).
constexpr int DEV_ERR_WAIT_TIMEOUT = 1;

struct GemmPlan {
    int m, n, k;
    int mb, nb, kt; // 32-row blocks of op(A), 32-column blocks of op(B), k tiles
    size_t a_bytes, b_bytes, flag_bytes;
};

GemmPlan gemm_plan(int m, int n, int k);

// The Rgemm argument checks (Rgemm.cpp:90-128) in the reference's order: 0, or the info
// code of the first bad argument.  Sets nota/notb ('N' or 'n').
int rgemm_check_args(char ta, char tb, int m, int n, int k, int lda, int ldb, int ldc, bool &nota, bool &notb);
size_t gemm_workspace_bytes(int m, int n, int k);

// The route of one product.  `disjoint`: the caller knows that no entry of C is one of A or
// B; otherwise a C whose address range meets A's or B's takes the staged route, which has
// read both before it writes C.
GemmRoute gemm_route(bool nota, bool notb, int m, int n, int k, const uint32_t *A, int lda, const uint32_t *B,
                     int ldb, const uint32_t *C, int ldc, bool disjoint);

// C <- alpha*op(A)*op(B) + beta*C.  Device pointers; stream-ordered.  The workspace
// (gemm_workspace_bytes) is used by the staged route only.
cudaError_t gemm_launch(bool nota, bool notb, int m, int n, int k, uint32_t alpha,
                        const uint32_t *A, int lda, const uint32_t *B, int ldb, uint32_t beta,
                        uint32_t *C, int ldc, void *workspace, cudaStream_t stream, bool disjoint);

// Same, on disjoint operands, writing all of C, its lower or its upper triangle (TRI_*), and
// doing nothing when *stop != 0 (stop may be null).
cudaError_t gemm_launch_tri(int tri, bool nota, bool notb, int m, int n, int k, uint32_t alpha,
                            const uint32_t *A, int lda, const uint32_t *B, int ldb, uint32_t beta,
                            uint32_t *C, int ldc, void *workspace, cudaStream_t stream, const int *stop);

// The calls that form no product (alpha == 0, or k == 0), on the m x n submatrix:
// C <- 0 or beta*C; with `dot` (TN/TT and k == 0, alpha != 0) C <- alpha*0 or
// alpha*0 + beta*C, which is NaR everywhere when alpha is NaR.
cudaError_t scale_launch(int m, int n, bool dot, uint32_t alpha, uint32_t beta, uint32_t *C, int ldc,
                         cudaStream_t stream);

// Element-wise IEEE double <-> posit32 conversion on device buffers.
cudaError_t convert_launch(bool to_posit, const void *in, void *out, size_t n, cudaStream_t stream);

int read_device_error(bool clear);
// Device address of the kernels' error flag (for stream-ordered copies of it).
cudaError_t device_error_address(int **p);

// Optional instrumentation: CUDA events around each multiplying kernel (main or fused), recorded on
// the launch stream, plus a count of this library's kernel launches.
void profile_enable(bool on);
int profile_read(double *main_ms, long long *main_launches, long long *all_launches, bool reset);

} // namespace pg
