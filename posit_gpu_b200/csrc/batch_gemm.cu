// batch_gemm.cu -- many independent posit32 GEMMs of uneven shapes in one persistent
// launch fed by a device work queue of output tiles.
//
// The queue holds (problem, tile row, tile column, tile shape) items sorted by
// decreasing k.  A CTA takes the next item and runs it as a tile of the single GEMM's fused
// route (gemm_tile.cuh, fused_tile: operands converted from the problem's own matrices,
// transposes and alpha*B for the NN/NT order handled during the load), so every C is bit-identical to posit_rgemm_dev's, i.e. to the CPU Rgemm.  Three tile
// shapes (64x32, 32x32, 32x64 outputs per CTA) cover small and skinny problems; which one
// a problem uses comes from a table indexed by its (m, n) size bucket, produced by the
// autotuner (posit_gpu_b200/autotune.py).
#include "batch_gemm.cuh"
#include "gemm.cuh"
#include "gemm_tile.cuh"
#include "posit32.cuh"

namespace pg {

namespace {

constexpr int BG_THREADS = TILE_THREADS;

// alpha == 0 or k == 0 with beta != 1, on the tile: C <- 0 or beta*C (alpha == 0,
// Rgemm.cpp:142-156; NN/NT with k == 0, Rgemm.cpp:169-177).  TN/TT with k == 0 and
// alpha != 0 form alpha*0 and combine it with beta*C (Rgemm.cpp:193-201): NaR when alpha
// is NaR.
__device__ void batch_scale_tile(const BatchGemmDesc &P, int mt, int nt, int bm, int bn)
{
    const bool dot = P.alpha != 0 && !P.nota;
    const uint32_t t = pmul(P.alpha, 0u);
    for (int e = threadIdx.x; e < bm * bn; e += BG_THREADS) {
        const int row = mt * bm + e % bm, col = nt * bn + e / bm;
        if (row < P.m && col < P.n) {
            uint32_t *cp = P.C + (size_t)row + (size_t)col * P.ldc;
            if (dot)
                *cp = (P.beta == 0) ? t : padd(t, pmul(P.beta, *cp));
            else
                *cp = (P.beta == 0) ? 0u : pmul(P.beta, *cp);
        }
    }
}

} // namespace

template <int TM_, int TN_>
__device__ __forceinline__ void batch_tile(const BatchGemmDesc &P, int mt, int nt, unsigned char *smem)
{
    const TileArgs T{P.nota != 0, P.notb != 0, P.m,   P.n, P.k,           P.alpha, P.beta,
                     P.A,         (size_t)P.lda, P.B, (size_t)P.ldb, P.C, (size_t)P.ldc};
    fused_tile<TRI_FULL, TM_, TN_, false>(T, mt, nt, smem);
}

__global__ void __launch_bounds__(BG_THREADS, BATCH_GEMM_CTAS_PER_SM)
    batch_gemm_kernel(const BatchGemmDesc *__restrict__ probs, const BatchTile *__restrict__ tiles, int ntiles,
                      int *__restrict__ next)
{
    extern __shared__ __align__(128) unsigned char smem[]; // tile_smem_bytes(4, 2)
    __shared__ int s_item;
    step_tables_fill(smem, threadIdx.x, BG_THREADS);
    for (;;) {
        if (threadIdx.x == 0)
            s_item = atomicAdd(next, 1);
        __syncthreads();
        const int item = s_item;
        __syncthreads();
        if (item >= ntiles)
            return;
        const BatchTile t = tiles[item];
        const BatchGemmDesc P = probs[t.prob];
        const int bm = batch_tile_rows(t.cfg), bn = batch_tile_cols(t.cfg);
        if (P.alpha == 0 || P.k == 0)
            batch_scale_tile(P, t.mt, t.nt, bm, bn);
        else if (t.cfg == 0)
            batch_tile<4, 2>(P, t.mt, t.nt, smem);
        else if (t.cfg == 1)
            batch_tile<2, 2>(P, t.mt, t.nt, smem);
        else
            batch_tile<2, 4>(P, t.mt, t.nt, smem);
        __syncthreads();
    }
}

size_t batch_gemm_smem_bytes() { return tile_smem_bytes(4, 2); }

cudaError_t batch_gemm_launch(const BatchGemmDesc *probs, const BatchTile *tiles, int ntiles, int *next, int ctas,
                              cudaStream_t st)
{
    const size_t smem = batch_gemm_smem_bytes();
    cudaError_t e = cudaFuncSetAttribute(batch_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess)
        return e;
    e = cudaMemsetAsync(next, 0, sizeof(int), st);
    if (e != cudaSuccess)
        return e;
    batch_gemm_kernel<<<ctas, BG_THREADS, smem, st>>>(probs, tiles, ntiles, next);
    return cudaGetLastError();
}

} // namespace pg
