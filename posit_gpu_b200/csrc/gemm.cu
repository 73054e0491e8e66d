// gemm.cu -- bit-exact posit32 GEMM for sm_100a.
//
// Reproduces the per-element operation order of the reference CPU Rgemm
// (libRpack/Rgemm.cpp:163-247):
//   NN / NT  "scale, then accumulate":  c <- beta*c (0 if beta == 0, untouched if
//            beta == 1), then c <- c + (alpha*b_lj)*a_il for l = 0..k-1;
//   TN / TT  "dot, then combine":       t <- 0, t <- t + a_li*b_lj for l = 0..k-1,
//            then c <- alpha*t (beta == 0) or alpha*t + beta*c.
// Both are one chain of "acc <- acc + x_l*y_l" per output; they differ only in the
// operand prescale (alpha*B for NN/NT), the accumulator's start value and the
// epilogue.  Two routes, the same k-step (gemm_tile.cuh) and the same bits:
//
//  * staged (see gemm_route): a pre-pass converts op(A) and op(B) (times alpha for NN/NT,
//    rounded exactly as the reference rounds alpha*b_lj) ONCE per element to FP64 (posit32
//    values are exact there) into a workspace of 32 x 16 blocks, [block][k-tile][l][32],
//    plus a NaR flag per row and column; transposition is absorbed here.  The main kernel,
//    one CTA of 256 threads per 64x64 tile of C, 2 CTAs per SM, brings each k tile's four
//    4 KB blocks into shared memory by the bulk-copy (TMA) engine (cp.async.bulk + mbarrier
//    transaction counts, 3 stages, every wait bounded);
//  * fused (small and skinny products): one launch, no workspace; a CTA reads the patterns of its own
//    operand blocks and converts them itself (gemm_tile.cuh, fused_tile).
#include "gemm.cuh"
#include "gemm_tile.cuh"
#include "posit32.cuh"

#include <algorithm>
#include <atomic>
#include <mutex>
#include <vector>

namespace pg {

__device__ int g_dev_error;

// ---------------------------------------------------------------------------
// PTX helpers: mbarrier + bulk async copy (TMA engine, no multicast)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_fence_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done)
                 : "r"(smem_u32(bar)), "r"(parity)
                 : "memory");
    return done != 0;
}

// Every wait is bounded: a copy that never lands turns into an error flag, not a hang.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity)
{
    for (uint32_t it = 0; it < (1u << 24); ++it)
        if (mbar_try_wait(bar, parity))
            return true;
    return false;
}

__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

GemmPlan gemm_plan(int m, int n, int k)
{
    GemmPlan p;
    p.m = m;
    p.n = n;
    p.k = k;
    p.mb = (m + BLK - 1) / BLK;
    p.nb = (n + BLK - 1) / BLK;
    p.kt = (k + BK - 1) / BK;
    // op(A)'s blocks are padded to pairs, so that a workspace of the size the callers are
    // told holds any tile shape's operands
    p.a_bytes = (size_t)((p.mb + 1) / 2 * 2) * p.kt * BK * BLK * sizeof(double);
    p.b_bytes = (size_t)p.nb * p.kt * BK * BLK * sizeof(double);
    p.flag_bytes = (size_t)((p.mb + 1) / 2 * 2 + p.nb) * BLK;
    return p;
}

size_t gemm_workspace_bytes(int m, int n, int k)
{
    GemmPlan p = gemm_plan(m, n, k);
    return p.a_bytes + p.b_bytes + p.flag_bytes;
}

// ---------------------------------------------------------------------------
// Staged route: the conversion pre-pass
// ---------------------------------------------------------------------------
// op(A) (m x k) -> Ad[block][kt][l][i], op(B) (k x n) -> Td[block][kt][l][j], the latter
// times alpha when `scale`, in one launch (indexes below `na` are A's).  Rows and columns
// beyond the matrix hold 1.0 so that padded lanes stay on the fast path (their results are
// never stored), steps past k hold 0.  A NaR operand makes every output of its row (column) NaR (p32_mul and
// p32_add propagate NaR, kernel_entry.cl:385-390, 414-417); that is recorded in the flags
// and the operand is decoded as 1.0 so the row's arithmetic stays on the fast path.
__global__ void decode_kernel(bool nota, bool notb, int m, int n, int k, const uint32_t *__restrict__ A, size_t lda,
                              const uint32_t *__restrict__ B, size_t ldb, bool scale, uint32_t alpha, int KT,
                              size_t na, size_t total, double *__restrict__ Ad, double *__restrict__ Td,
                              unsigned char *__restrict__ row_nar, unsigned char *__restrict__ col_nar)
{
    for (size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x; g < total; g += (size_t)gridDim.x * blockDim.x) {
        const bool is_a = g < na;
        const size_t idx = is_a ? g : g - na;
        const int i = (int)(idx % BLK);
        size_t q = idx / BLK;
        const int l = (int)(q % BK);
        q /= BK;
        const int kt = (int)(q % KT);
        const int row = (int)(q / KT) * BLK + i, kk = kt * BK + l;
        const bool rows_contiguous = is_a ? nota : !notb;
        const uint32_t *X = is_a ? A : B;
        const size_t ld = is_a ? lda : ldb;
        double v = kk < k ? 1.0 : 0.0;
        if (row < (is_a ? m : n) && kk < k) {
            v = p32_to_double(rows_contiguous ? X[(size_t)row + (size_t)kk * ld] : X[(size_t)kk + (size_t)row * ld]);
            if (!is_a && scale)
                v = scale_operand(v, alpha);
        }
        if (v != v) {
            (is_a ? row_nar : col_nar)[row] = 1;
            v = 1.0;
        }
        (is_a ? Ad : Td)[idx] = v;
    }
}

// ---------------------------------------------------------------------------
// Staged route: the main kernel
// ---------------------------------------------------------------------------
// TRI selects the entries written: TRI_FULL all of C; TRI_LOWER only row >= column (the
// symmetric trailing update of a lower Cholesky factorization); TRI_UPPER only row <=
// column (Rsyrk('U', 'T') of an upper one).  Tiles wholly outside the triangle exit at once.
// `stop`, if given, is a device flag (a factorization's info) that turns the call into a
// no-op when it is nonzero.
template <int TRI>
__global__ void __launch_bounds__(TILE_THREADS, MIN_CTAS_PER_SM)
    gemm_main_kernel(bool dot, int m, int n, int k, int KT, int mb, int nb, uint32_t alpha, uint32_t beta,
                     const double *__restrict__ Ad, const double *__restrict__ Td, uint32_t *__restrict__ C,
                     size_t ldc, const unsigned char *__restrict__ row_nar,
                     const unsigned char *__restrict__ col_nar, const int *__restrict__ stop)
{
    constexpr int BM = 16 * TM, BN = 16 * TN;
    if (stop && *stop != 0)
        return;
    if (TRI == TRI_LOWER && (int)(blockIdx.x * BM + BM - 1) < (int)(blockIdx.y * BN))
        return; // every row of the tile is above its first column
    if (TRI == TRI_UPPER && (int)(blockIdx.x * BM) > (int)(blockIdx.y * BN + BN - 1))
        return; // every row of the tile is below its last column
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char *tab = smem_raw;
    constexpr int NBLK = TM / 2 + TN / 2;   // operand blocks of a stage
    constexpr int BLK_DBL = BK * BLK;       // doubles of a block
    double *stages = reinterpret_cast<double *>(smem_raw + STEP_TAB_BYTES);
    __shared__ __align__(8) uint64_t full[STAGES];

    const int tid = threadIdx.x;
    const int tx = tid % 16, ty = tid / 16;
    const int mt = blockIdx.x, nt = blockIdx.y;
    constexpr uint32_t kBlkBytes = BLK_DBL * sizeof(double);
    // the tile's blocks that exist (the last tile of an odd count has one block less)
    const int na = min(TM / 2, mb - mt * (TM / 2)), nbk = min(TN / 2, nb - nt * (TN / 2));
    auto fetch = [&](int kt, int s) {
        mbar_arrive_expect_tx(&full[s], (uint32_t)(na + nbk) * kBlkBytes);
        double *dst = stages + (size_t)s * NBLK * BLK_DBL;
        for (int q = 0; q < na; ++q)
            bulk_g2s(dst + q * BLK_DBL, Ad + ((size_t)(mt * (TM / 2) + q) * KT + kt) * BLK_DBL, kBlkBytes, &full[s]);
        for (int q = 0; q < nbk; ++q)
            bulk_g2s(dst + (TM / 2 + q) * BLK_DBL, Td + ((size_t)(nt * (TN / 2) + q) * KT + kt) * BLK_DBL, kBlkBytes,
                     &full[s]);
    };

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s)
            mbar_init(&full[s], 1);
        mbar_fence_init();
        for (int s = 0; s < STAGES && s < KT; ++s)
            fetch(s, s);
    }
    step_tables_fill(tab, tid, TILE_THREADS);
    // blocks that do not exist hold 1.0 throughout: their lanes stay on the fast path
    if (na < TM / 2 || nbk < TN / 2)
        for (int e = tid; e < STAGES * NBLK * BLK_DBL; e += TILE_THREADS) {
            const int q = e / BLK_DBL % NBLK;
            if (q < TM / 2 ? q >= na : q - TM / 2 >= nbk)
                stages[e] = 1.0;
        }
    __syncthreads(); // the barriers are initialised, the tables filled
    double acc[TM][TN];
    uint32_t nar_bits;
    {
        uint32_t cu[TM][TN];
        tile_load_c<TM, TN>(!dot && beta != 0, cu, mt * BM, nt * BN, m, n, C, ldc, tx, ty);
        tile_start<TM, TN>(dot, acc, nar_bits, beta, cu);
    }

    // One block barrier per k tile, although a barrier per stage would do: it keeps the warps
    // in step, and with them the unrolled steps (14 KB) in the instruction cache (warps
    // that ran on by themselves took 333 ms for 8192^3 instead of 289).
    bool bad = false, slow = false;
    int kt_stop = 0, s = 0;
    uint32_t parity = 0;
#pragma unroll 1
    for (int kt = 0; kt < KT; ++kt) {
        kt_stop = kt;
        const bool arrived = mbar_wait_bounded(&full[s], parity);
        const double *as = stages + (size_t)s * NBLK * BLK_DBL;
        tile_steps<4>(acc, as, as + (TM / 2) * BLK_DBL, tile_step_count<4>(k - kt * BK), tab, tx, ty,
                      BlockedOps<BLK>{}, slow);
        // every thread is done with stage s before it is refilled
        bad = __syncthreads_or(!arrived) != 0;
        if (bad)
            break;
        if (tid == 0 && kt + STAGES < KT)
            fetch(kt + STAGES, s);
        if (++s == STAGES) {
            s = 0;
            parity ^= 1u;
        }
    }

    if (bad) {
        if (tid == 0) {
            atomicOr(&g_dev_error, DEV_ERR_WAIT_TIMEOUT);
            // let copies already in flight land before the CTA's shared memory goes away
            for (int q = kt_stop + 1; q < KT && q < kt_stop + STAGES; ++q)
                (void)mbar_wait_bounded(&full[q % STAGES], (uint32_t)(q / STAGES) & 1u);
        }
        return;
    }
    tile_finish<TRI, TM, TN>(dot, acc, nar_bits, mt * BM, nt * BN, m, n, alpha, beta, C, ldc, tx, ty,
                             [&](int i, int j) { return (row_nar[mt * BM + i] | col_nar[nt * BN + j]) != 0; });
}

// ---------------------------------------------------------------------------
// Fused route
// ---------------------------------------------------------------------------
template <int TRI, int TM_, int TN_>
__global__ void __launch_bounds__(TILE_THREADS, TM_ * TN_ >= 16 ? 2 : (TM_ * TN_ >= 8 ? 3 : 4))
    gemm_fused_kernel(const __grid_constant__ TileArgs P, const int *__restrict__ stop)
{
    constexpr int BM = 16 * TM_, BN = 16 * TN_;
    if (stop && *stop != 0)
        return;
    if (TRI == TRI_LOWER && (int)(blockIdx.x * BM + BM - 1) < (int)(blockIdx.y * BN))
        return;
    if (TRI == TRI_UPPER && (int)(blockIdx.x * BM) > (int)(blockIdx.y * BN + BN - 1))
        return;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    fused_tile<TRI, TM_, TN_, true>(P, blockIdx.x, blockIdx.y, smem_raw);
}

// C <- 0 or beta*C (alpha == 0, Rgemm.cpp:142-156; NN/NT with k == 0, Rgemm.cpp:169-177), or,
// with `dot`, the dot-then-combine epilogue of an empty sum (TN/TT with k == 0,
// Rgemm.cpp:193-201): t = alpha*0, then c = t (beta == 0) or t + beta*c.  alpha*0 is NaR
// when alpha is NaR (p32_mul tests NaR before zero, kernel_entry.cl:414-421).
__global__ void scale_kernel(int m, int n, bool dot, uint32_t alpha, uint32_t beta, uint32_t *__restrict__ C,
                             size_t ldc)
{
    size_t total = (size_t)m * n;
    const uint32_t t = pmul(alpha, 0u);
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        size_t i = idx % m, j = idx / m;
        uint32_t *cp = C + i + j * ldc;
        if (dot)
            *cp = (beta == 0) ? t : padd(t, pmul(beta, *cp));
        else
            *cp = (beta == 0) ? 0u : pmul(beta, *cp);
    }
}

// ---------------------------------------------------------------------------
// Instrumentation
// ---------------------------------------------------------------------------
namespace {
std::mutex g_prof_mu;
std::atomic<bool> g_prof_on{false};
std::vector<std::pair<cudaEvent_t, cudaEvent_t>> g_prof_events;
double g_prof_ms = 0.0;
long long g_prof_main = 0, g_prof_all = 0;

void prof_count(int launches)
{
    if (!g_prof_on)
        return;
    std::lock_guard<std::mutex> lk(g_prof_mu);
    g_prof_all += launches;
}

cudaEvent_t prof_mark(cudaStream_t st)
{
    cudaEvent_t ev = nullptr;
    if (cudaEventCreate(&ev) != cudaSuccess)
        return nullptr;
    cudaEventRecord(ev, st);
    return ev;
}
} // namespace

void profile_enable(bool on)
{
    std::lock_guard<std::mutex> lk(g_prof_mu);
    g_prof_on = on;
}

int profile_read(double *main_ms, long long *main_launches, long long *all_launches, bool reset)
{
    std::lock_guard<std::mutex> lk(g_prof_mu);
    for (auto &pr : g_prof_events) {
        float ms = 0.f;
        if (pr.first && pr.second && cudaEventSynchronize(pr.second) == cudaSuccess &&
            cudaEventElapsedTime(&ms, pr.first, pr.second) == cudaSuccess)
            g_prof_ms += ms;
        if (pr.first)
            cudaEventDestroy(pr.first);
        if (pr.second)
            cudaEventDestroy(pr.second);
        g_prof_main += 1;
    }
    g_prof_events.clear();
    if (main_ms)
        *main_ms = g_prof_ms;
    if (main_launches)
        *main_launches = g_prof_main;
    if (all_launches)
        *all_launches = g_prof_all;
    if (reset) {
        g_prof_ms = 0.0;
        g_prof_main = 0;
        g_prof_all = 0;
    }
    return 0;
}

__global__ void from_double_kernel(const double *__restrict__ x, uint32_t *__restrict__ out, size_t n)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = p32_from_double(x[i]);
}

__global__ void to_double_kernel(const uint32_t *__restrict__ x, double *__restrict__ out, size_t n)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = p32_to_double(x[i]);
}

static int grid_for(size_t total, int threads)
{
    size_t b = (total + threads - 1) / threads;
    size_t cap = 148 * 16;
    return (int)(b < cap ? (b ? b : 1) : cap);
}

static bool spans_overlap(const void *x, size_t xn, const void *y, size_t yn)
{
    const uintptr_t a = (uintptr_t)x, b = (uintptr_t)y;
    return a < b + yn * 4 && b < a + xn * 4;
}

// Entries from the first to the last of a rows x cols matrix.
static size_t span(int rows, int cols, int ld) { return (size_t)(cols - 1) * ld + rows; }

static long long ceil_div(long long a, long long b) { return (a + b - 1) / b; }

GemmRoute gemm_route(bool nota, bool notb, int m, int n, int k, const uint32_t *A, int lda, const uint32_t *B,
                     int ldb, const uint32_t *C, int ldc, bool disjoint)
{
    if (!disjoint &&
        (spans_overlap(C, span(m, n, ldc), A, nota ? span(m, k, lda) : span(k, m, lda)) ||
         spans_overlap(C, span(m, n, ldc), B, notb ? span(k, n, ldb) : span(n, k, ldb))))
        return GEMM_STAGED;
    // A call's time on each route: launches (and the conversion pre-pass), then the tiles of the
    // fullest SM, one after the other as far as the FP64 issue slots go; an SM with one or two tiles
    // does not hide their latencies and takes a little longer for each.  Fitted to 895 shapes (k to
    // 8192; m = n to 8128; n = 1 to 512 by m to 100,000 and the reverse), each timed on all three
    // routes: the route it names is 0.4 % slower than the best on average, at most 8 %.  Edge
    // tiles count as whole ones, which is what they cost: 12800 x 32 x 512 staged 397 us, 64x32 226,
    // 32x32 197; 16384 x 1 x 1024 staged 780, 64x32 433; 3200 x 129 x 512 371 / 226 / 257; 1371 x 400
    // x 32 47 / 26 / 29.  Full tiles in numbers are staged: 1024^2 x 300 228 / 258 / 257, 2500^2
    // x 300 1117 / 1297 / 1474.
    struct Cost {
        double call, per_k, per_tile; // us
        double one, two, more;        // an SM's tiles, in tiles: one, two, or t + more
        double of(long long tiles, int k) const
        {
            const long long t = ceil_div(tiles, SM_COUNT);
            return call + (t == 1 ? one : t == 2 ? two : (double)t + more) * (per_k * k + per_tile);
        }
    };
    static const Cost staged = {20.4, 0.3172, 3.83, 1.17, 2.12, 0.25}, f64x32 = {10.4, 0.1834, 1.73, 1.50, 2.22, 0.30},
                      f32x32 = {10.1, 0.1076, 0.96, 1.57, 2.43, 0.31};
    if (ceil_div(n, 32) > 65535) // columns of 32-wide tiles: more than a grid has in y
        return GEMM_STAGED;
    const double cs = staged.of(ceil_div(m, 64) * ceil_div(n, 64), k),
                 c42 = f64x32.of(ceil_div(m, 64) * ceil_div(n, 32), k),
                 c22 = f32x32.of(ceil_div(m, 32) * ceil_div(n, 32), k);
    return cs < std::min(c42, c22) ? GEMM_STAGED : (c42 < c22 ? GEMM_FUSED_64x32 : GEMM_FUSED_32x32);
}

template <class Kernel>
static cudaError_t allow_smem(Kernel fn, size_t smem)
{
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

template <int TRI, int TM_, int TN_>
static cudaError_t fused_launch(const TileArgs &P, cudaStream_t stream, const int *stop)
{
    const size_t smem = tile_smem_bytes(TM_, TN_);
    cudaError_t e = allow_smem(gemm_fused_kernel<TRI, TM_, TN_>, smem);
    if (e != cudaSuccess)
        return e;
    const dim3 grid((unsigned)ceil_div(P.m, 16 * TM_), (unsigned)ceil_div(P.n, 16 * TN_));
    gemm_fused_kernel<TRI, TM_, TN_><<<grid, TILE_THREADS, smem, stream>>>(P, stop);
    return cudaGetLastError();
}

template <int TRI>
static cudaError_t staged_launch(const TileArgs &P, void *workspace, cudaStream_t stream, const int *stop,
                                 cudaEvent_t *start)
{
    const GemmPlan p = gemm_plan(P.m, P.n, P.k);
    unsigned char *ws = reinterpret_cast<unsigned char *>(workspace);
    double *Ad = reinterpret_cast<double *>(ws);
    double *Td = reinterpret_cast<double *>(ws + p.a_bytes);
    unsigned char *row_nar = ws + p.a_bytes + p.b_bytes;
    unsigned char *col_nar = row_nar + (size_t)((p.mb + 1) / 2 * 2) * BLK;
    const size_t na = (size_t)p.mb * p.kt * BK * BLK, nb = (size_t)p.nb * p.kt * BK * BLK;
    cudaError_t e = cudaMemsetAsync(row_nar, 0, p.flag_bytes, stream);
    if (e != cudaSuccess)
        return e;
    decode_kernel<<<grid_for(na + nb, 256), 256, 0, stream>>>(P.nota, P.notb, P.m, P.n, P.k, P.A, P.lda, P.B, P.ldb,
                                                              P.nota, P.alpha, p.kt, na, na + nb, Ad, Td, row_nar,
                                                              col_nar);
    const size_t smem = STEP_TAB_BYTES + (size_t)STAGES * (TM / 2 + TN / 2) * BK * BLK * sizeof(double);
    e = allow_smem(gemm_main_kernel<TRI>, smem);
    if (e != cudaSuccess)
        return e;
    if (start)
        *start = prof_mark(stream); // the main kernel alone is timed
    const dim3 grid((unsigned)ceil_div(P.m, 16 * TM), (unsigned)ceil_div(P.n, 16 * TN));
    gemm_main_kernel<TRI><<<grid, TILE_THREADS, smem, stream>>>(!P.nota, P.m, P.n, P.k, p.kt, p.mb, p.nb, P.alpha,
                                                                P.beta, Ad, Td, P.C, P.ldc, row_nar, col_nar, stop);
    return cudaGetLastError();
}

template <int TRI>
static cudaError_t gemm_launch_route(GemmRoute route, const TileArgs &P, void *workspace, cudaStream_t stream,
                                     const int *stop)
{
    const bool prof = g_prof_on;
    cudaEvent_t e0 = prof && route != GEMM_STAGED ? prof_mark(stream) : nullptr;
    const cudaError_t e = route == GEMM_STAGED ? staged_launch<TRI>(P, workspace, stream, stop, prof ? &e0 : nullptr)
                        : route == GEMM_FUSED_64x32 ? fused_launch<TRI, 4, 2>(P, stream, stop)
                                                    : fused_launch<TRI, 2, 2>(P, stream, stop);
    if (prof) {
        cudaEvent_t e1 = prof_mark(stream);
        std::lock_guard<std::mutex> lk(g_prof_mu);
        g_prof_events.emplace_back(e0, e1);
    }
    prof_count(route == GEMM_STAGED ? 2 : 1);
    return e;
}

template <int TRI>
static cudaError_t gemm_launch_impl(bool nota, bool notb, int m, int n, int k, uint32_t alpha, const uint32_t *A,
                                    int lda, const uint32_t *B, int ldb, uint32_t beta, uint32_t *C, int ldc,
                                    void *workspace, cudaStream_t stream, const int *stop, bool disjoint)
{
    const GemmRoute route = gemm_route(nota, notb, m, n, k, A, lda, B, ldb, C, ldc, disjoint);
    const TileArgs P{nota, notb, m, n, k, alpha, beta, A, (size_t)lda, B, (size_t)ldb, C, (size_t)ldc};
    return gemm_launch_route<TRI>(route, P, workspace, stream, stop);
}

cudaError_t gemm_launch(bool nota, bool notb, int m, int n, int k, uint32_t alpha, const uint32_t *A, int lda,
                        const uint32_t *B, int ldb, uint32_t beta, uint32_t *C, int ldc, void *workspace,
                        cudaStream_t stream, bool disjoint)
{
    return gemm_launch_impl<TRI_FULL>(nota, notb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, workspace, stream,
                                      nullptr, disjoint);
}

cudaError_t gemm_launch_tri(int tri, bool nota, bool notb, int m, int n, int k, uint32_t alpha, const uint32_t *A,
                            int lda, const uint32_t *B, int ldb, uint32_t beta, uint32_t *C, int ldc,
                            void *workspace, cudaStream_t stream, const int *stop)
{
    if (tri == TRI_LOWER)
        return gemm_launch_impl<TRI_LOWER>(nota, notb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, workspace,
                                           stream, stop, true);
    if (tri == TRI_UPPER)
        return gemm_launch_impl<TRI_UPPER>(nota, notb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, workspace,
                                           stream, stop, true);
    return gemm_launch_impl<TRI_FULL>(nota, notb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, workspace, stream,
                                      stop, true);
}

cudaError_t scale_launch(int m, int n, bool dot, uint32_t alpha, uint32_t beta, uint32_t *C, int ldc,
                         cudaStream_t stream)
{
    scale_kernel<<<grid_for((size_t)m * n, 256), 256, 0, stream>>>(m, n, dot, alpha, beta, C, (size_t)ldc);
    prof_count(1);
    return cudaGetLastError();
}

cudaError_t convert_launch(bool to_posit, const void *in, void *out, size_t n, cudaStream_t stream)
{
    if (n == 0)
        return cudaSuccess;
    if (to_posit)
        from_double_kernel<<<grid_for(n, 256), 256, 0, stream>>>((const double *)in, (uint32_t *)out, n);
    else
        to_double_kernel<<<grid_for(n, 256), 256, 0, stream>>>((const uint32_t *)in, (double *)out, n);
    prof_count(1);
    return cudaGetLastError();
}

cudaError_t device_error_address(int **p) { return cudaGetSymbolAddress((void **)p, g_dev_error); }

int read_device_error(bool clear)
{
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_dev_error, sizeof(int)) != cudaSuccess)
        return -1;
    if (clear && v) {
        int z = 0;
        cudaMemcpyToSymbol(g_dev_error, &z, sizeof(int));
    }
    return v;
}

} // namespace pg
