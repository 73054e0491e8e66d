// batch.cu -- many independent posit32 LU / Cholesky factor-and-solve problems in one
// persistent launch fed by a device work queue.
//
// Each CTA takes the next problem from the queue (an atomic counter over a list sorted by
// decreasing size, so the largest problems start first) and factors and solves it alone.
// Per-element operation order is the reference's (see lapack.cu), so every factor, pivot and
// solution is bit-identical to the per-call path (posit_rgetrf_dev + posit_rgetrs_dev,
// posit_rpotrf_dev + posit_rpotrs_dev) and to the CPU routines.
//
// A problem is factored by panels of up to 16 or 32 columns: the panel in shared memory as FP64,
// the trailing matrix in global memory (L2) as patterns, updated by 64x64 tiles in the GEMM's
// k-step (gemm_tile.cuh).  So an element is converted once per panel and its 16 or 32
// multiply-adds run from registers; one column per step, the form this replaced, converted
// every element for every multiply-add (about 80 instructions each).  The right-hand sides
// follow in shared memory, the L^T solve by warp_chain (one thread's chain before).
#include "batch.cuh"
#include "gemm_tile.cuh"
#include "posit32.cuh"
#include "trsm_chain.cuh"

#include <algorithm>
#include <limits.h>

namespace pg {

namespace {

// Two shapes of CTA.  Problems of more than BATCH_LARGE_N rows: 512 threads, panels of up to
// 32 columns, one CTA per SM -- the longest problem bounds the launch, so it gets a whole SM.
// The rest: 256 threads, panels of up to 16, two CTAs per SM.  (One shape of 256 threads for
// all: an LU of n = 512 took 12.1 ms alone and 17.8 with a second CTA on its SM, as long as
// all 2000 problems of the mix together.)
template <int THREADS, int JB_, int AREA>
struct BatchCfg {
    static constexpr int T = THREADS;
    static constexpr int GROUPS = T / 256;  // 256 threads work on a trailing tile
    static constexpr int JB = JB_;          // most columns of a panel
    static constexpr int CH = 64 * GROUPS;  // columns of the trailing matrix taken together
    static constexpr int UL = CH + 2;       // doubles per row of U12 in shared memory
    // Shared memory: tables; the rows of U12 of one stretch of columns; the rest: a panel
    // [jb][PL], or the right-hand sides, or the L^T solves' columns and terms.
    static constexpr int U_BYTES = (JB * UL * 8 + 127) / 128 * 128;
    static constexpr int AREA_BYTES = AREA;
    static constexpr int SMEM = STEP_TAB_BYTES + U_BYTES + AREA_BYTES;
};
using LargeCfg = BatchCfg<512, 32, (512 * 32 + 64) * 8>;
using SmallCfg = BatchCfg<256, 16, 512 * 16 * 8 + 10 * 1024>;
static_assert(LargeCfg::SMEM + 4096 <= 227 * 1024, "one CTA per SM");
static_assert(2 * (SmallCfg::SMEM + 3072) <= 228 * 1024, "two CTAs per SM");
constexpr int BJB = 32; // the larger JB

__device__ __forceinline__ double pd(uint32_t u) { return p32_to_double(u); }

struct BatchShared {
    int hi[16], row[16]; // the warps' pivot candidates
    uint32_t lo[16];
    double val[16];
    LtxRow ltx[2];
    int piv[BJB];                     // the panel's pivots (rows of the matrix, 0-based)
    int src[BJB], dst[BJB], from[BJB]; // net interchange: block row i <- src[i]; row dst[i] <- from[i] (dst < 0: none)
};

// The panel's operands in a trailing tile: as = panel rows, ts = U12 or the panel again.
struct PanelOps {
    static constexpr bool NEG = true;  // c + (-u)*l
    static constexpr bool NANS = true; // NaR travels as NaN
    int pl, ul;
    __device__ __forceinline__ int a(int q, int l) const { return l * pl + q * BLK; }
    __device__ __forceinline__ int t(int q, int l) const { return l * ul + q * BLK; }
};

// rw[c * T] += -u[c] * l for c in [c0, c1).
__device__ __forceinline__ void row_update(double *rw, int T, const double *u, double l, int c0, int c1,
                                           const unsigned char *tab)
{
    constexpr int U = 4;
    int c = c0;
#pragma unroll 1
    for (; c + U <= c1; c += U) {
        double y[U], *p = rw + c * T;
        bool bad = false;
#pragma unroll
        for (int q = 0; q < U; ++q) {
            y[q] = step_one(p[q * T], -u[c + q], l, tab);
            bad |= y[q] != y[q];
        }
        if (bad)
            break; // the rest one by one
#pragma unroll
        for (int q = 0; q < U; ++q)
            p[q * T] = y[q];
    }
#pragma unroll 1
    for (; c < c1; ++c)
        rw[c * T] = mac_any(rw[c * T], -u[c], l, tab);
}

// The largest |x| (NaN below everything), the lowest row among equal ones, over the warp.
struct Best {
    int hi, row;
    uint32_t lo;
};
__device__ __forceinline__ int best_lane(const Best &b)
{
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const int hi = __reduce_max_sync(FULL, b.hi);
    const uint32_t lo = __reduce_max_sync(FULL, b.hi == hi ? b.lo : 0u);
    const int row = __reduce_min_sync(FULL, b.hi == hi && b.lo == lo ? b.row : INT_MAX);
    return __ffs(__ballot_sync(FULL, b.hi == hi && b.lo == lo && b.row == row)) - 1;
}

// The panel of columns [j, j+jb): factored in shared memory, panel row r being matrix row j+r.
// LU: s.piv; Cholesky: returns the column whose diagonal failed, or jb.  `info` (LU): the
// first zero pivot, 1-based.
template <class C, bool LU>
__device__ __forceinline__ int factor_panel(double *pan, int PL, int M, int j, int jb, int &info, BatchShared &s,
                                            const unsigned char *tab)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto cand_init = [](Best &b, double &bv) {
        b = Best{INT_MIN, INT_MAX, 0u};
        bv = 0.0;
    };
    auto cand_add = [](Best &b, double &bv, double v, int r) { // rows in increasing order
        const int hi = v != v ? -1 : __double2hiint(fabs(v));
        const uint32_t lo = v != v ? 0u : (uint32_t)__double2loint(v);
        if (hi > b.hi || (hi == b.hi && lo > b.lo)) {
            b = Best{hi, r, lo};
            bv = v;
        }
    };
    auto cand_put = [&](const Best &b, double bv) {
        if (lane == best_lane(b)) {
            s.hi[warp] = b.hi;
            s.lo[warp] = b.lo;
            s.row[warp] = b.row;
            s.val[warp] = bv;
        }
    };
    Best b;
    double bv;
    if (LU) {
        cand_init(b, bv);
        for (int r = tid; r < M; r += C::T)
            cand_add(b, bv, pan[r], r);
        cand_put(b, bv);
        __syncthreads();
    }
    for (int k = 0; k < jb; ++k) {
        double *ck = pan + k * PL;
        double mult;
        if (LU) {
            Best cd = {INT_MIN, INT_MAX, 0u};
            if (lane < C::T / 32)
                cd = Best{s.hi[lane], s.row[lane], s.lo[lane]};
            const int w = best_lane(cd), p = s.row[w];
            const double v = s.val[w];
            if (v == 0.0 && info == 0)
                info = j + k + 1;
            // a zero pivot leaves its own column in place (Rgetrf2.cpp:107-117)
            if (p != k && tid < jb && !(tid == k && v == 0.0)) {
                double *c2 = pan + tid * PL;
                const double t = c2[k];
                c2[k] = c2[p];
                c2[p] = t;
            }
            if (tid == 0)
                s.piv[k] = j + p;
            // nothing scaled under a zero pivot; a NaR one makes the column NaR, as dividing by it does
            mult = v == 0.0 ? 1.0 : f64_posit_div(1.0, v, 1.0 / v);
            __syncthreads(); // the rows have changed places
        } else {
            const double akk = ck[k];
            if (!(akk > 0.0)) // Rpotrf2.cpp:90-93; the same in every thread
                return k;
            const double lkk = f64_posit_sqrt(akk);
            mult = f64_posit_div(1.0, lkk, 1.0 / lkk);
            __syncthreads(); // every thread has read a_kk
            if (tid == 0)
                ck[k] = lkk;
            for (int r = k + 1 + tid; r < M; r += C::T)
                ck[r] = mul_any(ck[r], mult, tab);
            __syncthreads(); // the column's l_ck
        }
        const double *u = LU ? pan + k : ck; // u[c]: row k's column c (LU), or l_ck
        cand_init(b, bv);
        for (int r = tid; r < M; r += C::T)
            if (r > k) {
                double l = ck[r];
                if (LU) {
                    l = mul_any(l, mult, tab);
                    ck[r] = l;
                    // row k's columns lie PL apart: through registers, four at a time
                    int c = k + 1;
#pragma unroll 1
                    for (; c < jb; c += 4) {
                        double y[4];
                        bool bad = false;
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const int cc = min(c + q, jb - 1);
                            y[q] = step_one(pan[cc * PL + r], -u[cc * PL], l, tab);
                            bad |= y[q] != y[q];
                        }
                        if (bad) {
#pragma unroll 1
                            for (int q = 0; q < 4 && c + q < jb; ++q)
                                pan[(c + q) * PL + r] = mac_any(pan[(c + q) * PL + r], -u[(c + q) * PL], l, tab);
                        } else {
#pragma unroll
                            for (int q = 0; q < 4; ++q)
                                if (c + q < jb)
                                    pan[(c + q) * PL + r] = y[q];
                        }
                    }
                    if (k + 1 < jb)
                        cand_add(b, bv, pan[(k + 1) * PL + r], r);
                } else {
                    row_update(pan + r, PL, u, l, k + 1, min(jb, r + 1), tab);
                }
            }
        if (LU && k + 1 < jb)
            cand_put(b, bv);
        __syncthreads();
    }
    return jb;
}

// The panel's interchanges as one permutation (s.src, s.dst, s.from), by the first warp: the
// interchanges in order as exchanges between lanes, of row numbers (lapack.cu, lu_rows_kernel).
__device__ __forceinline__ void net_interchange(int j, int jb, BatchShared &s)
{
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const int t = lane < jb ? s.piv[lane] : -1;
    int alias = -1; // pivots below the block: the first lane with that row keeps its content
    if (t >= j + jb) {
        alias = lane;
        for (int q = 0; q < lane; ++q)
            if (s.piv[q] == t) {
                alias = q;
                break;
            }
    }
    int v = j + lane, w = t;
    for (int i = 0; i < jb; ++i) {
        const int ti = __shfl_sync(FULL, t, i), ai = __shfl_sync(FULL, alias, i);
        if (ti == j + i)
            continue;
        const bool in = ti < j + jb;
        const int o = in ? ti - j : ai;
        const int vi = __shfl_sync(FULL, v, i), vo = __shfl_sync(FULL, in ? v : w, o);
        if (lane == o) {
            if (in)
                v = vi;
            else
                w = vi;
        }
        if (lane == i)
            v = vo;
    }
    if (lane < jb) {
        s.src[lane] = v;
        s.dst[lane] = alias == lane ? t : -1;
        s.from[lane] = w;
    }
}

// One column outside the panel through its interchanges.  Every value is read before one is
// written.
template <int JB>
__device__ __forceinline__ void permute_column(uint32_t *col, int j, int jb, const BatchShared &s)
{
    uint32_t v[JB], w[JB];
#pragma unroll
    for (int i = 0; i < JB; ++i) {
        v[i] = i < jb && s.src[i] != j + i ? col[s.src[i]] : 0u;
        w[i] = i < jb && s.dst[i] >= 0 ? col[s.from[i]] : 0u;
    }
#pragma unroll
    for (int i = 0; i < JB; ++i)
        if (i < jb) {
            if (s.dst[i] >= 0)
                col[s.dst[i]] = w[i];
            if (s.src[i] != j + i)
                col[j + i] = v[i];
        }
}

// The unit-lower solve of the block's rows of one column, in place: x_i += -l_ik * x_k in the
// order of k (no multiplier is skipped: the factorization's rank-1 updates).  `u`: the block's
// rows of the column; pan[k * PL + i] = l_ik.  By 16 rows in registers.
__device__ __forceinline__ void u12_column(uint32_t *u, const double *pan, int PL, int jb, const unsigned char *tab)
{
    constexpr int R = 16;
    bool bad = false;
#pragma unroll 1
    for (int i0 = 0; i0 < jb; i0 += R) {
        double x[R];
#pragma unroll
        for (int i = 0; i < R; ++i)
            x[i] = i0 + i < jb ? pd(u[i0 + i]) : 0.0;
#pragma unroll 1
        for (int k = 0; k < i0; ++k) {
            const double xk = -pd(u[k]), *l = pan + k * PL + i0;
#pragma unroll
            for (int i = 0; i < R; ++i) // (past jb: a row below the block, into an x not stored)
                x[i] = step_one(x[i], xk, l[i], tab);
        }
#pragma unroll
        for (int k = 0; k + 1 < R; ++k)
            if (i0 + k < jb) {
                const double xk = -x[k], *l = pan + (i0 + k) * PL + i0;
#pragma unroll
                for (int i = k + 1; i < R; ++i)
                    x[i] = step_one(x[i], xk, l[i], tab);
            }
#pragma unroll
        for (int i = 0; i < R; ++i)
            bad |= i0 + i < jb && x[i] != x[i];
        if (bad) { // step by step, in place
#pragma unroll 1
            for (int k = 0; k < min(jb, i0 + R); ++k) {
                const double xk = -pd(u[k]);
#pragma unroll 1
                for (int i = max(k + 1, i0); i < min(jb, i0 + R); ++i)
                    u[i] = p32_from_double_exact(mac_any(pd(u[i]), xk, pan[k * PL + i], tab));
            }
            bad = false;
        } else {
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (i0 + i < jb)
                    u[i0 + i] = p32_from_double_exact(x[i]);
        }
    }
}

// 64x64 outputs of the trailing matrix at (row0, col0): C += -(rows of the panel) * (ts), jb
// steps.  LOWER: only row >= column.
template <bool LOWER>
__device__ __forceinline__ void trailing_tile(uint32_t *A, size_t lda, int n, int row0, int col0, const double *as,
                                              const double *ts, PanelOps ops, int steps, const unsigned char *tab)
{
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16 % 16;
    double acc[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = row0 + own_off(tx, i), col = col0 + own_off(ty, q);
            const bool in = row < n && col < n && (!LOWER || row >= col);
            acc[i][q] = in ? pd(A[row + (size_t)col * lda]) : 1.0;
        }
    bool slow = false;
    tile_steps<2>(acc, as, ts, steps, tab, tx, ty, ops, slow);
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = row0 + own_off(tx, i), col = col0 + own_off(ty, q);
            if (row < n && col < n && (!LOWER || row >= col))
                A[row + (size_t)col * lda] = p32_from_double_exact(acc[i][q]);
        }
}

// Rgetrf / Rpotrf('L') of one problem; returns info.
template <class C, bool LU>
__device__ __forceinline__ int factor_one(const BatchProblem &pr, unsigned char *smem, BatchShared &s)
{
    const int n = pr.n, tid = threadIdx.x;
    uint32_t *A = pr.A;
    const size_t lda = (size_t)pr.lda;
    const unsigned char *tab = smem;
    double *U = reinterpret_cast<double *>(smem + STEP_TAB_BYTES);
    double *pan = reinterpret_cast<double *>(smem + STEP_TAB_BYTES + C::U_BYTES);
    const int group = tid / 256;
    int info = 0;
    for (int j = 0, jb = 0; j < n; j += jb) {
        const int M = n - j, PL = (M + 1) & ~1;
        // (64 doubles over: a tile at the edge reads past the panel's last row)
        const int fit = ((int)(C::AREA_BYTES / sizeof(double)) - 64) / PL & ~1;
        jb = min(min(C::JB, fit), M);
        for (int c = 0; c < jb; ++c)
            for (int r = tid; r < M; r += C::T)
                pan[c * PL + r] = (LU || r >= c) ? pd(A[(j + r) + (size_t)(j + c) * lda]) : 0.0;
        __syncthreads();
        const int done = factor_panel<C, LU>(pan, PL, M, j, jb, info, s, tab);
        if (!LU && done < jb) // the columns before the failed one still update the rest
            info = j + done + 1;
        for (int c = 0; c < jb; ++c)
            for (int r = tid; r < M; r += C::T)
                if (LU || r >= c)
                    A[(j + r) + (size_t)(j + c) * lda] = p32_from_double_exact(pan[c * PL + r]);
        if (LU) {
            if (tid < jb)
                pr.ipiv[j + tid] = s.piv[tid] + 1;
            if (tid < 32)
                net_interchange(j, jb, s);
            __syncthreads();
            // the columns outside the panel: interchanges and, right of it, U12
            for (int c = tid; c < n - jb; c += C::T) {
                uint32_t *col = A + (size_t)(c < j ? c : c + jb) * lda;
                permute_column<C::JB>(col, j, jb, s);
                if (c >= j)
                    u12_column(col + j, pan, PL, jb, tab);
            }
            __syncthreads();
        }
        const int steps = (done + 1) & ~1;
        if (steps > done) { // an odd count of steps: one more of zeros
            __syncthreads();
            for (int r = tid; r < M; r += C::T)
                if (done < jb || fit > jb) // (a panel of an odd count is the last one or a failed one)
                    pan[done * PL + r] = 0.0;
            __syncthreads();
        }
        const PanelOps ops{PL, LU ? C::UL : PL};
        for (int c0 = j + jb; c0 < n; c0 += C::CH) {
            if (LU) { // U12 of these columns, from where the step above left it
                for (int e = tid; e < jb * C::CH; e += C::T) {
                    const int k = e % jb, c = e / jb;
                    U[k * C::UL + c] = c0 + c < n ? pd(A[(j + k) + (size_t)(c0 + c) * lda]) : 0.0;
                }
                __syncthreads();
            }
            const int cg = c0 + 64 * group; // this group's 64 columns
            if (cg < n)
                for (int r0 = LU ? j + jb : cg; r0 < n; r0 += 64)
                    trailing_tile<!LU>(A, lda, n, r0, cg, pan + (r0 - j), LU ? U + 64 * group : pan + (cg - j), ops, steps,
                                       tab);
            if (LU)
                __syncthreads(); // U is done with
        }
        if (!LU && done < jb)
            break;
        __syncthreads();
    }
    return info;
}

// ---------------------------------------------------------------------------
// The right-hand sides
// ---------------------------------------------------------------------------
// The threads that solve one problem: a CTA, or a warp of one.
template <int THREADS>
struct Team {
    static constexpr int T = THREADS;
    __device__ __forceinline__ static int tid() { return THREADS == 32 ? threadIdx.x & 31 : threadIdx.x; }
    __device__ __forceinline__ static void sync()
    {
        if (THREADS == 32)
            __syncwarp();
        else
            __syncthreads();
    }
};

// Right-hand sides between global memory (patterns) and X (shared memory, FP64, ldx apart).
template <class TM, bool MANY>
__device__ __forceinline__ void load_rhs(double *X, int ldx, const uint32_t *B, size_t ldb, int n, int cnt)
{
    if (!MANY) {
        for (int r = 0; r < cnt; ++r)
            for (int i = TM::tid(); i < n; i += TM::T)
                X[r * ldx + i] = pd(B[r * ldb + i]);
    } else {
#pragma unroll 4
        for (int e = TM::tid(); e < n * cnt; e += TM::T)
            X[e / n * ldx + e % n] = pd(B[(size_t)(e / n) * ldb + e % n]);
    }
}
template <class TM, bool MANY>
__device__ __forceinline__ void store_rhs(const double *X, int ldx, uint32_t *B, size_t ldb, int n, int cnt)
{
    if (!MANY) {
        for (int r = 0; r < cnt; ++r)
            for (int i = TM::tid(); i < n; i += TM::T)
                B[r * ldb + i] = p32_from_double_exact(X[r * ldx + i]);
    } else {
#pragma unroll 4
        for (int e = TM::tid(); e < n * cnt; e += TM::T)
            B[(size_t)(e / n) * ldb + e % n] = p32_from_double_exact(X[e / n * ldx + e % n]);
    }
}

// Rlaswp, in order, a thread per right-hand side.
template <class TM>
__device__ __forceinline__ void swap_rhs(double *X, int ldx, const int *piv, int n, int cnt)
{
    for (int r = TM::tid(); r < cnt; r += TM::T) {
        double *x = X + r * ldx;
        for (int i = 0; i < n; ++i) {
            const int p = piv[i];
            const double t = x[i];
            x[i] = x[p];
            x[p] = t;
        }
    }
}

// Rtrsm('L', LOWER ? 'L' : 'U', 'N') on the columns X: b_i - b_k*a_ik for the rows of one step,
// then (non-unit) the next row's division (Rtrsm.cpp:127, 145; a zero is left alone, as the
// reference skips it).  A thread has row `row` of every RG-th right-hand side: few rows leave
// threads over, which take other right-hand sides (a thread per row alone, whatever the
// number of right-hand sides, took 4.0 ms for an LU of n = 33 with 300 of them; this takes 0.36).
template <class TM, bool LOWER, bool UNIT>
__device__ __forceinline__ void axpy_solve(const uint32_t *A, size_t lda, int n, double *X, int ldx, int nrhs,
                                           const unsigned char *tab)
{
    const int tid = TM::tid();
    const int W = 2 * n <= TM::T ? n : TM::T, RG = TM::T / W;
    const int row = tid % W, r0 = tid / W < RG ? tid / W : nrhs;
    auto col_of = [&](int st) { return LOWER ? st : n - 1 - st; };
    // a step's first coefficient and the next division's a_ii are loaded a step ahead
    uint32_t cur = row < n ? A[row + (size_t)col_of(0) * lda] : 0u, dn = UNIT ? 0u : A[(size_t)col_of(0) * (lda + 1)];
    for (int st = 0; st < n; ++st) {
        const int k = col_of(st), kn = col_of(st + 1);
        const bool more = st + 1 < n;
        if (!UNIT) {
            const double d = pd(dn), rc = 1.0 / d;
            TM::sync(); // row k is up to date
            for (int r = tid; r < nrhs; r += TM::T) {
                double *x = X + r * ldx;
                if (x[k] != 0.0)
                    x[k] = f64_posit_div(x[k], d, rc);
            }
            dn = more ? A[(size_t)kn * (lda + 1)] : 0u;
        }
        TM::sync();
        const uint32_t *ak = A + (size_t)k * lda;
        const uint32_t nxt = more && row < n ? A[row + (size_t)kn * lda] : 0u;
#pragma unroll 1
        for (int i = row; i < n; i += W) {
            if (LOWER ? i <= k : i >= k)
                continue;
            const double l = pd(i == row ? cur : ak[i]);
            constexpr int U = 4;
            int r = r0;
#pragma unroll 1
            for (; r + (U - 1) * RG < nrhs; r += U * RG) { // several at once, tested together
                double y[U];
                bool bad = false;
#pragma unroll
                for (int q = 0; q < U; ++q) {
                    const double *x = X + (r + q * RG) * ldx;
                    y[q] = step_one(x[i], -x[k], l, tab);
                    bad |= y[q] != y[q];
                }
                if (bad)
                    break; // the rest one by one
#pragma unroll
                for (int q = 0; q < U; ++q)
                    X[(r + q * RG) * ldx + i] = y[q];
            }
#pragma unroll 1
            for (; r < nrhs; r += RG) {
                double *x = X + r * ldx;
                const double xk = x[k];
                if (xk != 0.0) // zero multipliers skipped (Rtrsm.cpp:125-126, 143-144)
                    x[i] = mac_any(x[i], -xk, l, tab);
            }
        }
        cur = nxt;
    }
    TM::sync();
}

constexpr int AXPY_FEW = 4;
constexpr int B_PRE = 2; // rows per thread whose coefficients are loaded a step ahead
// The same for up to AXPY_FEW right-hand sides by a CTA: a thread per row, no other barrier than
// the step's; the thread with row `next` divides it when it has updated it.
template <class C, bool LOWER, bool UNIT>
__device__ __forceinline__ void axpy_few(const uint32_t *A, size_t lda, int n, double *X, int ldx, int nrhs,
                                         const unsigned char *tab)
{
    const int tid = threadIdx.x;
    auto col_of = [&](int st) { return LOWER ? st : n - 1 - st; };
    auto finish = [&](int i) {
        const double d = pd(A[i + (size_t)i * lda]), rc = 1.0 / d;
        for (int r = 0; r < nrhs; ++r) {
            double *x = X + r * ldx;
            if (x[i] != 0.0)
                x[i] = f64_posit_div(x[i], d, rc);
        }
    };
    uint32_t cur[B_PRE], nxt[B_PRE];
#pragma unroll
    for (int q = 0; q < B_PRE; ++q)
        cur[q] = tid + q * C::T < n ? A[(tid + q * C::T) + (size_t)col_of(0) * lda] : 0u;
    if (!UNIT) {
        if (tid == col_of(0) % C::T)
            finish(col_of(0));
        __syncthreads();
    }
    for (int st = 0; st < n; ++st) {
        const int k = col_of(st), kn = col_of(st + 1);
        const uint32_t *ak = A + (size_t)k * lda;
#pragma unroll
        for (int q = 0; q < B_PRE; ++q)
            nxt[q] = (st + 1 < n && tid + q * C::T < n) ? A[(tid + q * C::T) + (size_t)kn * lda] : 0u;
        auto update = [&](int i, uint32_t a) {
            if (LOWER ? i > k : i < k) {
                const double l = pd(a);
                for (int r = 0; r < nrhs; ++r) {
                    double *x = X + r * ldx;
                    const double xk = x[k];
                    if (xk != 0.0) // zero multipliers skipped (Rtrsm.cpp:125-126, 143-144)
                        x[i] = mac_any(x[i], -xk, l, tab);
                }
            }
        };
#pragma unroll
        for (int q = 0; q < B_PRE; ++q)
            if (tid + q * C::T < n)
                update(tid + q * C::T, cur[q]);
#pragma unroll 1
        for (int i = tid + B_PRE * C::T; i < n; i += C::T)
            update(i, ak[i]);
        if (!UNIT && st + 1 < n && tid == kn % C::T)
            finish(kn);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < B_PRE; ++q)
            cur[q] = nxt[q];
    }
}

// Rtrsm('L', 'L', 'T') (Rtrsm.cpp:175-186) on one column x by one thread: t = b_i,
// t = t - a_ki*b_k for k = i+1 .. n-1 in order, b_i = t / a_ii.  `coef(k, i)` is a_ki in FP64.
// Eight steps are tested together, the next eight's coefficients loaded meanwhile.
template <class Coef>
__device__ __forceinline__ void thread_llt(double *x, int n, Coef coef, const unsigned char *tab)
{
    constexpr int U = 8;
#pragma unroll 1
    for (int i = n - 1; i >= 0; --i) {
        double t = x[i], a[U], an[U];
        const double d = coef(i, i), rc = 1.0 / d;
#pragma unroll
        for (int q = 0; q < U; ++q)
            an[q] = coef(min(i + 1 + q, n - 1), i);
#pragma unroll 1
        for (int k = i + 1; k < n; k += U) {
#pragma unroll
            for (int q = 0; q < U; ++q)
                a[q] = an[q];
            if (k + U < n) {
#pragma unroll
                for (int q = 0; q < U; ++q)
                    an[q] = coef(min(k + U + q, n - 1), i);
            }
            const double t0 = t;
#pragma unroll
            for (int q = 0; q < U; ++q) {
                const double r = step_one(t, -x[min(k + q, n - 1)], a[q], tab);
                t = k + q < n ? r : t;
            }
            if (t != t) {
                t = t0;
#pragma unroll 1
                for (int q = k; q < min(k + U, n); ++q)
                    t = mac_any(t, -x[q], coef(q, i), tab);
            }
        }
        x[i] = f64_posit_div(t, d, rc);
    }
}

// Whether the L^T solve of `nrhs` columns goes by a thread each (thread_llt, up to `threads` at a
// time) instead of a warp each (`warps` at a time) or, `block`, the CTA for one after the other.
// In ns, measured: a thread's chain 70 n^2 and a little (n = 64 290 us, 128 1150), a warp's solve
// 1900 n + 7.5 n^2 (64 150, 200 770), a CTA's 1400 n + 4.5 n^2.  n = 64: 16 columns 440 us by warps and
// 487 by threads, 100 columns 1851 and 562.
__device__ __forceinline__ bool llt_by_thread(int n, int nrhs, int threads, int warps, bool block)
{
    const long long by_thread = (long long)((nrhs + threads - 1) / threads) * n * 80;
    const long long other = block ? nrhs * (1400 + n * 9 / 2)
                                  : (long long)((nrhs + warps - 1) / warps) * (1900 + n * 15 / 2);
    return by_thread < other;
}

// The right-hand sides: Rgetrs('N') or Rpotrs('L').  MANY: many of them, spread over the
// threads (batch_spread_pays).
template <class C, bool LU, bool MANY>
__device__ __forceinline__ void solve_one(const BatchProblem &pr, unsigned char *smem, BatchShared &s)
{
    using TM = Team<C::T>;
    const int n = pr.n, tid = threadIdx.x;
    const size_t lda = (size_t)pr.lda, ldb = (size_t)pr.ldb;
    const unsigned char *tab = smem;
    unsigned char *area = smem + STEP_TAB_BYTES + C::U_BYTES;
    double *X = reinterpret_cast<double *>(area);
    const int ldx = MANY ? n | 1 : n; // odd: a thread per column meets no bank conflicts
    const int group = max(1, (int)((C::AREA_BYTES - 4 * (size_t)n) / (8 * (size_t)ldx)));
    // L^T backward.  Few right-hand sides: one after the other, a warp adding and the others
    // forming terms; more: a warp for each, as many at a time as fit; short columns or many
    // of them: a thread for each.
    const size_t one = 2 * ChainTerms64::bytes(n) + (size_t)n * 8;
    const size_t per = ChainTerms64::bytes(n) + (((size_t)n * 8 + 15) & ~(size_t)15);
    const bool by_block = pr.nrhs <= 2 && one <= (size_t)C::AREA_BYTES;
    const int warps = min(C::T / 32, (int)(C::AREA_BYTES / per));
    const bool by_thread = MANY && !LU && llt_by_thread(n, pr.nrhs, min(group, C::T), warps, by_block);
    for (int r0 = 0; r0 < pr.nrhs; r0 += group) {
        const int cnt = min(group, pr.nrhs - r0);
        uint32_t *B = pr.B + r0 * ldb;
        load_rhs<TM, MANY>(X, ldx, B, ldb, n, cnt);
        if (LU) {
            int *piv = reinterpret_cast<int *>(X + (size_t)cnt * ldx);
            for (int i = tid; i < n; i += C::T)
                piv[i] = pr.ipiv[i] - 1;
            __syncthreads();
            swap_rhs<TM>(X, ldx, piv, n, cnt);
        }
        __syncthreads();
        if (!MANY || cnt <= AXPY_FEW) {
            axpy_few<C, true, LU>(pr.A, lda, n, X, ldx, cnt, tab);
            if (LU)
                axpy_few<C, false, false>(pr.A, lda, n, X, ldx, cnt, tab);
        } else {
            axpy_solve<TM, true, LU>(pr.A, lda, n, X, ldx, cnt, tab);
            if (LU)
                axpy_solve<TM, false, false>(pr.A, lda, n, X, ldx, cnt, tab);
        }
        if (by_thread) {
            const uint32_t *A = pr.A;
            for (int r = tid; r < cnt; r += C::T)
                thread_llt(X + r * ldx, n, [=](int k, int i) { return pd(A[k + i * lda]); }, tab);
            __syncthreads();
        }
        store_rhs<TM, MANY>(X, ldx, B, ldb, n, cnt);
        __syncthreads();
    }
    if (LU || by_thread)
        return;
    if (by_block) {
        LtxCol64 x;
        x.b = reinterpret_cast<double *>(area + 2 * ChainTerms64::bytes(n));
        for (int r = 0; r < pr.nrhs; ++r) {
            uint32_t *b = pr.B + r * ldb;
            for (int i = tid; i < n; i += C::T)
                x.set(i, pd(b[i]));
            block_ltx_solve<C::T, false, ChainTerms64>(pr.A, lda, x, n, false, area, s.ltx);
            for (int i = tid; i < n; i += C::T)
                b[i] = p32_from_double_exact(x.get(i));
            __syncthreads();
        }
        return;
    }
    const int warp = tid >> 5, lane = tid & 31;
    if (warp < warps) {
        ChainTerms64 q;
        q.q = reinterpret_cast<double *>(area + warp * per);
        double *x = reinterpret_cast<double *>(area + warp * per + ChainTerms64::bytes(n));
        for (int r = warp; r < pr.nrhs; r += warps) {
            uint32_t *b = pr.B + r * ldb;
            for (int i = lane; i < n; i += 32)
                x[i] = pd(b[i]);
            __syncwarp();
            warp_llt_solve(pr.A, lda, x, n, q);
            for (int i = lane; i < n; i += 32)
                b[i] = p32_from_double_exact(x[i]);
            __syncwarp();
        }
    }
}

// ---------------------------------------------------------------------------
// Problems of up to 32 rows: a warp each, a row per lane, the matrix in shared memory.
// ---------------------------------------------------------------------------
// A CTA's barriers cost such a problem more than its arithmetic; eight of them run side by
// side in a CTA instead.
constexpr int SMALL_N = BATCH_WARP_N;
constexpr int SMALL_LD = SMALL_N + 1;
struct SmallArea {
    double a[SMALL_N * SMALL_LD + SMALL_N]; // a_ic at [c * SMALL_LD + i]; then, many right-hand sides
    double x[SMALL_N];
    int piv[SMALL_N];
};
static_assert(sizeof(SmallArea) * (SmallCfg::T / 32) <= SmallCfg::U_BYTES + SmallCfg::AREA_BYTES, "a problem per warp");
// From this many right-hand sides on they go through side by side.  n = 24, three and four of them:
// LU 85 us one by one and 97 side by side, 94 / 84; Cholesky 144 / 133, 174 / 127.
constexpr int SMALL_MANY_LU = 4, SMALL_MANY_CHOL = 3;

template <bool LU>
__device__ __forceinline__ int small_factor(SmallArea &w, int n, const unsigned char *tab)
{
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    int info = 0;
    for (int k = 0; k < n; ++k) {
        double *ck = w.a + k * SMALL_LD;
        double mult;
        const double mine = ck[lane];
        if (LU) {
            Best b = {INT_MIN, INT_MAX, 0u};
            if (lane >= k && lane < n)
                b = Best{mine != mine ? -1 : __double2hiint(fabs(mine)), lane,
                         mine != mine ? 0u : (uint32_t)__double2loint(mine)};
            const int p = best_lane(b);
            const double v = __shfl_sync(FULL, mine, p);
            if (v == 0.0 && info == 0)
                info = k + 1;
            if (p != k && lane < n && !(lane == k && v == 0.0)) { // a column per lane
                double *c2 = w.a + lane * SMALL_LD;
                const double t = c2[k];
                c2[k] = c2[p];
                c2[p] = t;
            }
            if (lane == 0)
                w.piv[k] = p;
            mult = v == 0.0 ? 1.0 : f64_posit_div(1.0, v, 1.0 / v);
            __syncwarp();
        } else {
            const double akk = __shfl_sync(FULL, mine, k);
            if (!(akk > 0.0))
                return k + 1;
            const double lkk = f64_posit_sqrt(akk);
            mult = f64_posit_div(1.0, lkk, 1.0 / lkk);
            if (lane == k)
                ck[k] = lkk;
        }
        double l = 0.0;
        if (lane > k && lane < n) {
            l = mul_any(ck[lane], mult, tab);
            ck[lane] = l;
        }
        __syncwarp(); // LU: row k in place; Cholesky: the column's l_ck
#pragma unroll 1
        for (int c = k + 1; c < n; c += 4) {
            double y[4];
            bool bad = false;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int cc = min(c + q, n - 1);
                y[q] = step_one(w.a[cc * SMALL_LD + lane], -(LU ? w.a[cc * SMALL_LD + k] : ck[cc]), l, tab);
                bad |= y[q] != y[q];
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                double *e = w.a + (c + q) * SMALL_LD;
                if (c + q < n && lane < n && (LU ? lane > k : lane >= c + q))
                    e[lane] = bad ? mac_any(e[lane], -(LU ? e[k] : ck[c + q]), l, tab) : y[q];
            }
        }
        __syncwarp();
    }
    return info;
}

template <bool LU, bool MANY>
__device__ __forceinline__ void run_small(const BatchProblem &pr, SmallArea &w, const unsigned char *tab)
{
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const int n = pr.n, lane = threadIdx.x & 31;
    const size_t lda = (size_t)pr.lda;
    const bool factor = !(pr.kind & BATCH_SOLVE_ONLY);
    for (int c = 0; c < n; ++c)
        w.a[c * SMALL_LD + lane] = (lane < n && (LU || lane >= c)) ? pd(pr.A[lane + (size_t)c * lda]) : 0.0;
    __syncwarp();
    if (factor) {
        const int info = small_factor<LU>(w, n, tab);
        for (int c = 0; c < n; ++c)
            if (lane < n && (LU || lane >= c))
                pr.A[lane + (size_t)c * lda] = p32_from_double_exact(w.a[c * SMALL_LD + lane]);
        if (LU && lane < n)
            pr.ipiv[lane] = w.piv[lane] + 1;
        if (lane == 0)
            *pr.info = info;
        if (!LU && info != 0)
            return;
    } else if (LU) {
        if (lane < n)
            w.piv[lane] = pr.ipiv[lane] - 1;
    }
    __syncwarp();
    if (MANY && pr.nrhs >= (LU ? SMALL_MANY_LU : SMALL_MANY_CHOL)) {
        using TM = Team<32>;
        const int ldx = n | 1, group = (int)(sizeof(w.a) / sizeof(double)) / ldx;
        const uint32_t *A = pr.A; // the factor, from global memory: X takes its place
        for (int r0 = 0; r0 < pr.nrhs; r0 += group) {
            const int cnt = min(group, pr.nrhs - r0);
            uint32_t *B = pr.B + (size_t)r0 * pr.ldb;
            load_rhs<TM, true>(w.a, ldx, B, (size_t)pr.ldb, n, cnt);
            __syncwarp();
            if (LU) {
                swap_rhs<TM>(w.a, ldx, w.piv, n, cnt);
                __syncwarp();
            }
            axpy_solve<TM, true, LU>(A, lda, n, w.a, ldx, cnt, tab);
            if (LU)
                axpy_solve<TM, false, false>(A, lda, n, w.a, ldx, cnt, tab);
            else
                for (int r = lane; r < cnt; r += 32)
                    thread_llt(w.a + r * ldx, n, [=](int k, int i) { return pd(A[k + i * lda]); }, tab);
            __syncwarp();
            store_rhs<TM, true>(w.a, ldx, B, (size_t)pr.ldb, n, cnt);
            __syncwarp();
        }
        return;
    }
    double d = 1.0;
    if (lane < n)
        d = w.a[lane * SMALL_LD + lane];
    const double rc = 1.0 / d;
    for (int r = 0; r < pr.nrhs; ++r) {
        uint32_t *b = pr.B + (size_t)r * pr.ldb;
        double x = lane < n ? pd(b[lane]) : 0.0;
        if (LU)
            for (int i = 0; i < n; ++i) { // Rlaswp
                const int p = w.piv[i];
                const double xi = __shfl_sync(FULL, x, i), xp = __shfl_sync(FULL, x, p);
                x = lane == i ? xp : (lane == p ? xi : x);
            }
        for (int k = 0; k < n; ++k) { // L forward, zero multipliers skipped
            if (!LU && lane == k && x != 0.0)
                x = f64_posit_div(x, d, rc);
            const double xk = __shfl_sync(FULL, x, k);
            if (xk != 0.0 && lane > k && lane < n)
                x = mac_any(x, -xk, w.a[k * SMALL_LD + lane], tab);
        }
        if (LU) { // U backward
            for (int k = n - 1; k >= 0; --k) {
                if (lane == k && x != 0.0)
                    x = f64_posit_div(x, d, rc);
                const double xk = __shfl_sync(FULL, x, k);
                if (xk != 0.0 && lane < k)
                    x = mac_any(x, -xk, w.a[k * SMALL_LD + lane], tab);
            }
        } else {
            w.x[lane] = x;
            __syncwarp();
            const double *a = w.a;
            if (lane == 0)
                thread_llt(w.x, n, [=](int k, int i) { return a[i * SMALL_LD + k]; }, tab);
            __syncwarp();
            x = w.x[lane];
            __syncwarp();
        }
        if (lane < n)
            b[lane] = p32_from_double_exact(x);
    }
}

template <class C, bool LU, bool MANY>
__device__ __forceinline__ void run_one(const BatchProblem &pr, unsigned char *smem, BatchShared &s)
{
    int info = 0;
    if (!(pr.kind & BATCH_SOLVE_ONLY)) {
        info = factor_one<C, LU>(pr, smem, s);
        if (threadIdx.x == 0)
            *pr.info = info;
        __syncthreads();
    }
    if (pr.n > 0 && pr.nrhs > 0 && (LU || info == 0))
        solve_one<C, LU, MANY>(pr, smem, s);
}

} // namespace

// The problems [first, last) of the list, from the queue `next` (which counts from 0); from
// warp_from on a warp takes each.
template <class C, bool MANY>
__global__ void __launch_bounds__(C::T, 512 / C::T) batch_factor_kernel(const BatchProblem *__restrict__ probs, int first,
                                                                        int last, const int *__restrict__ order,
                                                                        int warp_from, int *__restrict__ next)
{
    extern __shared__ __align__(128) unsigned char smem_batch[];
    __shared__ BatchShared s;
    __shared__ int s_item;
    step_tables_fill(smem_batch, threadIdx.x, C::T);
    for (;;) {
        if (threadIdx.x == 0)
            s_item = first + atomicAdd(next, 1);
        __syncthreads();
        const int item = s_item;
        __syncthreads();
        if (item >= last)
            return;
        const BatchProblem pr = probs[order ? order[item] : item];
        if (C::T == SmallCfg::T && item >= warp_from) {
            SmallArea &w = reinterpret_cast<SmallArea *>(smem_batch + STEP_TAB_BYTES)[threadIdx.x >> 5];
            const bool lead = (threadIdx.x & 31) == 0;
            auto take = [&]() { return __shfl_sync(0xFFFFFFFFu, lead ? first + atomicAdd(next, 1) : 0, 0); };
            for (int mine = threadIdx.x < 32 ? item : take(); mine < last; mine = take()) {
                const BatchProblem ps = probs[order[mine]];
                if (ps.n > 0) {
                    if ((ps.kind & 1) == BATCH_LU)
                        run_small<true, MANY>(ps, w, smem_batch);
                    else
                        run_small<false, MANY>(ps, w, smem_batch);
                    __syncwarp();
                } else if (lead && !(ps.kind & BATCH_SOLVE_ONLY)) {
                    *ps.info = 0;
                }
            }
            return;
        }
        if ((pr.kind & 1) == BATCH_LU)
            run_one<C, true, MANY>(pr, smem_batch, s);
        else
            run_one<C, false, MANY>(pr, smem_batch, s);
        __syncthreads();
    }
}

template <class C, bool MANY>
static cudaError_t launch_cfg(const BatchProblem *probs, int first, int last, const int *order, int warp_from, int *next,
                              int ctas, cudaStream_t st)
{
    cudaError_t e = cudaFuncSetAttribute(batch_factor_kernel<C, MANY>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    if (e == cudaSuccess)
        e = cudaMemsetAsync(next, 0, sizeof(int), st);
    if (e != cudaSuccess)
        return e;
    const int count = last - first;
    batch_factor_kernel<C, MANY><<<count < ctas ? count : ctas, C::T, C::SMEM, st>>>(probs, first, last, order, warp_from, next);
    return cudaGetLastError();
}

// The kernels without the code that spreads right-hand sides solve any number of them too, a thread
// per row (a warp's one by one), and factor faster: with that code in, the compiler spills more, and an
// LU of n = 512 takes 9.1 ms instead of 8.2 (two CTAs an SM: n = 200 1.75 instead of 1.70). So it is
// a matter of the launch's longest problem, or of all of them over its CTAs.  Times in us, fitted to
// problems of 33 to 512 rows and 1 to 300 right-hand sides.
bool batch_spread_pays(bool large, const BatchProblem *probs, int first, int last, const int *order, int sms)
{
    double longest[2] = {0.0, 0.0}, sum[2] = {0.0, 0.0};
    bool many = false;
    for (int i = first; i < last; ++i) {
        const BatchProblem &q = probs[order ? order[i] : i];
        const double n = q.n, rhs = q.nrhs, f = (q.kind & BATCH_SOLVE_ONLY) ? 0.0 : (large ? 0.030 : 0.039) * n * n;
        const bool spread = q.nrhs > (q.n > BATCH_WARP_N ? AXPY_FEW : 2);
        many |= spread;
        const double each = q.n <= BATCH_WARP_N && (q.kind & 1) == BATCH_CHOL ? 1.5 : 0.41; // a right-hand side, us a row
        const double t[2] = {f + each * n * rhs, f * (large ? 1.10 : 1.03) + (spread ? 0.12 : each) * n * rhs};
        for (int w = 0; w < 2; ++w) {
            longest[w] = std::max(longest[w], t[w]);
            sum[w] += t[w];
        }
    }
    const double ctas = large ? sms : 2.0 * sms;
    return many && std::max(longest[1], sum[1] / ctas) < std::max(longest[0], sum[0] / ctas);
}

cudaError_t batch_factor_launch(bool large, bool spread, const BatchProblem *probs, int first, int last, const int *order,
                                int warp_from, int *next, int sms, cudaStream_t st)
{
    if (last <= first)
        return cudaSuccess;
    if (large)
        return spread ? launch_cfg<LargeCfg, true>(probs, first, last, order, warp_from, next, sms, st)
                    : launch_cfg<LargeCfg, false>(probs, first, last, order, warp_from, next, sms, st);
    return spread ? launch_cfg<SmallCfg, true>(probs, first, last, order, warp_from, next, 2 * sms, st)
                : launch_cfg<SmallCfg, false>(probs, first, last, order, warp_from, next, 2 * sms, st);
}

} // namespace pg
