// lapack.cu -- device-resident posit32 LU (Rgetrf) and Cholesky (Rpotrf), and their
// solves (Rgetrs, Rpotrs), bit-exact against the reference's CPU routines.
//
// Operation order.  In the reference every entry of L and U receives its updates as
// a <- a + (-u)*l (Rgemm's c + (alpha*b)*a with alpha = -1, Rgemm.cpp:180-182; Rtrsm's
// b - b_k*a, Rtrsm.cpp:151, is the same bits because posit multiplication is symmetric in
// sign) in ascending k, however Rgetrf/Rgetrf2/Rpotrf/Rpotrf2 group the columns into
// blocks; L entries are then multiplied by the reciprocal of the pivot (Rgetrf2.cpp:121-122,
// Rscal) or of the Cholesky diagonal (Rtrsm.cpp:265-268), diagonals of a Cholesky factor
// take a square root (Rpotrf2.cpp:97).  So LU and lower Cholesky are independent of the
// block size bit for bit (the zero-multiplier skips of Rtrsm/Rsyrk add zero and change
// nothing unless a NaR is present), and the device code may block the work its own way:
//
//   panel (nb columns)   one launch: LU on a thread-block cluster holding up to 32 columns in
//                        shared memory (wider or taller blocks by inner panels), Cholesky
//                        on independent CTAs; LU panels of more rows than fit take two
//                        launches per column, ordered by the kernel boundary alone (the
//                        pivot step of one CTA, then the scaling and the rank-1 update over
//                        all rows in parallel);
//   U block row          Rtrsm("L","L","N","U"), a warp or a CTA per column;
//   row interchanges     Rlaswp on the columns outside the panel;
//   trailing update      the posit32 GEMM of gemm.cu (NN for LU; NT restricted to the
//                        lower triangle for Cholesky).
// The matrix never leaves the device.  Upper Cholesky (dot-then-combine order, block size
// dependent) follows the caller's block size.
#include "gemm.cuh"
#include "lapack.cuh"

#include <algorithm>
#include <limits.h>
#include <cooperative_groups.h>
#include "posit32.cuh"
#include "trsm_chain.cuh"

namespace pg {

// ---------------------------------------------------------------------------
// LU panel
// ---------------------------------------------------------------------------
// Two launches per panel column k, synchronised only by the kernel boundary:
//   lu_update_kernel  blocks over (rows > k) x (groups of PANEL_CG columns in (k, jb)):
//                     l_i = a_ik scaled as Rgetrf2 does, a_ic += (-u_kc)*l_i.  Column k is
//                     only read; the first column group writes l_i to a scratch column.
//   lu_pivot_kernel   one block: the scratch column into column k, then the pivot step of
//                     column k+1 -- iRamax over the updated column, the interchange of the
//                     pivot row across the panel, the scaling decision.
constexpr int PANEL_ROWS = 128; // rows per update block (one per thread)
constexpr int PANEL_CG = 4;     // panel columns per update block

// Pivot decision of one column, shared by the two kernels of a panel step.
struct PivotInfo {
    int row;       // panel-local row of the pivot
    uint32_t piv;  // pivot value (after the interchange it sits at row k)
    int mode;      // 0: zero pivot (no scaling), 1: multiply by reciprocal, 2: divide
    uint32_t recip;
};

// Workspace of the panel kernels: the pivot/diagonal record and a scratch column of m
// entries, then the trailing GEMM's workspace.
static size_t panel_ws_bytes(int m) { return 256 + (((size_t)m * 4 + 255) & ~(size_t)255); }

// Copies the scaled multipliers of column `copy_col` (rows copy_col+1 .. M-1) from the
// scratch column into place (copy_col < 0: none), then, when k < jb, the pivot step of
// column k: iRamax (iRamax.cpp:65-71) over panel-local rows [k, M) -- the first index of
// the strict maximum of abs() in posit order (signed integer order of the patterns, NaR
// lowest) -- the interchange of rows k and p over the panel's jb columns
// (Rgetrf2.cpp:107-117; with a zero pivot, over every column but k) and the scaling
// decision (Rgetrf2.cpp:119-131).
__global__ void __launch_bounds__(1024) lu_pivot_kernel(uint32_t *__restrict__ P, size_t lda, int M, int jb, int k,
                                                        int row0, int *__restrict__ ipiv, int *__restrict__ info,
                                                        PivotInfo *__restrict__ pinfo,
                                                        const uint32_t *__restrict__ lcol, int copy_col)
{
    __shared__ int32_t s_key[1024];
    __shared__ int s_idx[1024];
    if (*info < 0)
        return; // an earlier failure stops the factorization
    const int tid = threadIdx.x;
    if (copy_col >= 0) {
        uint32_t *pc = P + (size_t)copy_col * lda;
        for (int r = copy_col + 1 + tid; r < M; r += blockDim.x)
            pc[r] = lcol[r];
        __syncthreads(); // the interchange below moves two of these entries
    }
    if (k >= jb)
        return;
    int32_t best = INT32_MIN;
    int bidx = -1;
    const uint32_t *col = P + (size_t)k * lda;
    for (int i = k + tid; i < M; i += blockDim.x) {
        int32_t key = (int32_t)pabs(col[i]);
        if (bidx < 0 || key > best) { // rows visited in increasing order per thread
            best = key;
            bidx = i;
        }
    }
    // larger key wins, equal keys the smaller row; warp shuffles, then one warp over the
    // warps' results (blockDim.x == 1024: 32 warps)
    const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int round = 0; round < 2; ++round) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const int32_t k2 = __shfl_down_sync(0xFFFFFFFFu, best, off);
            const int i2 = __shfl_down_sync(0xFFFFFFFFu, bidx, off);
            if (i2 >= 0 && (bidx < 0 || k2 > best || (k2 == best && i2 < bidx))) {
                best = k2;
                bidx = i2;
            }
        }
        if (round == 0) {
            if (lane == 0) {
                s_key[warp] = best;
                s_idx[warp] = bidx;
            }
            __syncthreads();
            best = s_key[lane];
            bidx = s_idx[lane];
        }
    }
    if (tid == 0)
        s_idx[32] = bidx;
    __syncthreads();
    const int p = s_idx[32];
    const uint32_t piv = col[p];
    if (tid == 0) {
        ipiv[row0 + k] = row0 + p + 1; // 1-based, global
        PivotInfo pi;
        pi.row = p;
        pi.piv = piv;
        if (piv == 0) {
            pi.mode = 0;
            pi.recip = 0;
            if (*info == 0)
                *info = row0 + k + 1;
        } else if ((int32_t)pabs(piv) >= (int32_t)1u) { // |pivot| >= sfmin = FLT_MIN -> minpos
            pi.mode = 1;
            pi.recip = pdiv_est(P32_ONE, piv);
        } else {
            pi.mode = 2; // NaR pivot: element-wise division (Rgetrf2.cpp:124-126)
            pi.recip = 0;
        }
        *pinfo = pi;
    }
    __syncthreads(); // every thread has read the pivot before the rows move
    if (p != k) {
        // A zero pivot leaves its own column in place (Rgetrf2.cpp:107-117) while the
        // recursion's Rlaswp calls (Rgetrf2.cpp:141-150, 167-176) still move rows k and p in
        // every other column of the panel, and Rgetrf's outside it.
        for (int c = tid; c < jb; c += blockDim.x) {
            if (c == k && piv == 0)
                continue;
            uint32_t *pc = P + (size_t)c * lda;
            uint32_t t = pc[k];
            pc[k] = pc[p];
            pc[p] = t;
        }
    }
}

PG_HD uint32_t lu_scaled(uint32_t a, const PivotInfo &pi)
{
    if (pi.mode == 1)
        return pmul(pi.recip, a); // Rscal: da*dx
    if (pi.mode == 2)
        return pdiv_est(a, pi.piv);
    return a;
}

__global__ void __launch_bounds__(PANEL_ROWS) lu_update_kernel(uint32_t *__restrict__ P, size_t lda, int M, int jb,
                                                               int k, const int *__restrict__ info,
                                                               const PivotInfo *__restrict__ pinfo,
                                                               uint32_t *__restrict__ lcol)
{
    __shared__ double s_u[PANEL_CG]; // -u_kc for this block's columns, FP64
    if (*info < 0)
        return;
    const PivotInfo pi = *pinfo;
    const int c0 = k + 1 + blockIdx.y * PANEL_CG;
    if (threadIdx.x < PANEL_CG && c0 + (int)threadIdx.x < jb)
        s_u[threadIdx.x] = -p32_to_double(P[k + (size_t)(c0 + threadIdx.x) * lda]); // row k after the interchange
    __syncthreads();
    const int i = k + 1 + blockIdx.x * PANEL_ROWS + threadIdx.x;
    if (i >= M)
        return;
    const uint32_t l = lu_scaled(P[i + (size_t)k * lda], pi);
    if (blockIdx.y == 0)
        lcol[i] = l;
    const double dl = p32_to_double(l);
    const int cn = min(PANEL_CG, jb - c0);
    for (int j = 0; j < cn; ++j) { // a_ic + (-u_kc)*l_i in the FP64 step (posit32.cuh)
        uint32_t *pc = P + i + (size_t)(c0 + j) * lda;
        *pc = p32_from_double_exact(f64_posit_mac_checked(p32_to_double(*pc), s_u[j], dl));
    }
}

// ---------------------------------------------------------------------------
// LU panel in one thread-block cluster, held in shared memory: the per-column steps of
// lu_pivot_kernel + lu_update_kernel -- iRamax with first-max tie-break, the interchange
// across the panel, the scaling decision, the scaled column, the rank-1 update in the FP64
// step -- in the same per-element order, one launch per panel.  Up to 8 CTAs of T threads
// (T a multiple of 32, up to 1024), each holding a stretch of the panel's rows: row i of it
// in slot r of thread t, i = r*T + t, jb FP64 values each, in shared memory.  Rows never
// move: an interchange of rows k and p swaps the logical row numbers the two slots hold
// (each thread keeps its slots' numbers in registers, and every thread knows k and p, so
// each applies the swap to its own slots), and the write-back stores each slot at the row
// it holds at the end.
//
// What bounds it: latency, column after column.  So the next pivot is looked for as early as
// it can be and the bulk of the update runs while it travels.  Per column k:
//   * wait for the CTAs' candidates of column k, pushed with their reciprocals and whole
//     rows into every CTA's shared memory; every warp picks the winner (three warp
//     reductions: the key's two words, the lowest logical row);
//   * each thread scales its rows' column k and updates column k+1 only; the largest of
//     column k+1 over the warp, the CTA (one block barrier); the warp that holds the CTA's
//     candidate brings that one row up to date (a column per lane), forms the reciprocal
//     (f64_posit_div) and pushes both to all CTAs;
//   * arrive at the cluster barrier, and only then update columns k+2 .. of all rows.
// The pushed rows are triple-buffered: a CTA may push column k+1's while another, past its
// arrival for column k, still reads column k-1's.  The pivot row's slot is not written again
// in the panel (but for a zero pivot below row k, where the two slots trade back their
// column-k values: that column stays in place, Rgetrf2.cpp:107-117).  A final cluster barrier
// keeps every CTA's shared memory alive until no other CTA writes it.
// At n = 1024 a panel of 24 columns took 103 us when the update of all columns, one multiply-add
// at a time, came before the search, the pivot row was read from its owner afterwards and
// the reciprocal by pdiv_est stood in between: 4.2 us a column.  Now 55 us: about 400 cycles
// to pick the winner, 500 to scale and update one column, 600 to find the CTA's candidate,
// 500 for its row and reciprocal, 700 until every CTA has it, the update of the rest beside.
// LU n = 1024: 5.3 -> 3.4 ms, 4096: 51.6 -> 32.7.
// ---------------------------------------------------------------------------
constexpr int PANEL1_THREADS = 1024; // most threads per CTA
constexpr int PANEL1_MAX_JB = 32;        // wider blocks go by inner panels (panel_width)
constexpr int PANEL1_MAX_CTAS = 8;
constexpr int PANEL1_MAX_R = 4;          // slots per thread (the LU panel keeps their row numbers in registers)
constexpr int PANEL1_ROWS_PER_CTA = 128; // the rows one CTA takes before another joins
constexpr size_t PANEL1_SMEM = 227 * 1024 - 4096; // dynamic shared memory of a panel CTA

// The barrier of a cluster: the cluster's, or the block's when the cluster is one CTA.
__device__ __forceinline__ void panel_sync(cooperative_groups::cluster_group &cl, int ncta)
{
    if (ncta == 1)
        __syncthreads();
    else
        cl.sync();
}

// A pivot candidate.  The key is |x| as FP64 bits, NaR below everything (iRamax.cpp:65-71
// compares abs() in posit order); among equal keys the lowest logical row wins.
struct PivotCand {
    int hi;      // high word of |x|; -1 for NaR, INT_MIN for no candidate
    uint32_t lo; // low word of |x|
    int row;     // logical row
    int slot;    // (r << 16) | thread of the slot holding it
};
struct PivotPush {
    PivotCand c;
    double val, recip; // the pivot; what the column below it is multiplied by
};

__device__ __forceinline__ bool cand_better(const PivotCand &a, const PivotCand &b) // a over b
{
    return a.hi != b.hi ? a.hi > b.hi : (a.lo != b.lo ? a.lo > b.lo : a.row < b.row);
}

// The lane holding the warp's best candidate.
__device__ __forceinline__ int cand_best_lane(const PivotCand &c)
{
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const int hi = __reduce_max_sync(FULL, c.hi);
    const uint32_t lo = __reduce_max_sync(FULL, c.hi == hi ? c.lo : 0u);
    const int row = __reduce_min_sync(FULL, c.hi == hi && c.lo == lo ? c.row : INT_MAX);
    return __ffs(__ballot_sync(FULL, c.hi == hi && c.lo == lo && c.row == row)) - 1;
}

// The columns of a row are updated PANEL_U at a time; up to PANEL_U - 1 columns past jb are read
// and written too (u is zero there).
constexpr int PANEL_U = 8;
__host__ __device__ constexpr int panel_cols(int jb) { return jb + PANEL_U - 1; } // columns a row takes in shared memory
inline size_t lu_panel_smem(int R, int T, int jb, int ncta)
{
    return STEP_TAB_BYTES + ((size_t)R * T + 3 * (size_t)ncta) * panel_cols(jb) * sizeof(double);
}

// rw[c*T] += -u[c] * l for the columns [c0, jb) of one row.
__device__ __forceinline__ void panel_row_update(double *rw, int T, const double *u, double l, int c0, int jb,
                                                 const unsigned char *tab)
{
#pragma unroll 1
    for (int c = c0; c < jb; c += PANEL_U) {
        double y[PANEL_U];
        double *p = rw + c * T;
        bool bad = false;
#pragma unroll
        for (int q = 0; q < PANEL_U; ++q) {
            y[q] = step_one(p[q * T], -u[c + q], l, tab);
            bad |= y[q] != y[q];
        }
        if (!bad) {
#pragma unroll
            for (int q = 0; q < PANEL_U; ++q)
                p[q * T] = y[q];
        } else {
            bool out;
#pragma unroll 1
            for (int q = 0; q < PANEL_U; ++q)
                p[q * T] = step_any<true>(p[q * T], -u[c + q], l, tab, out);
        }
    }
}

// One row of jb columns from the matrix into shared memory, zeros behind it; eight loads in
// flight.
__device__ __forceinline__ void panel_load_row(double *rw, int T, const uint32_t *p, size_t lda, int jb)
{
    constexpr int U = 8;
#pragma unroll 1
    for (int c = 0; c < panel_cols(jb); c += U) {
        uint32_t v[U];
#pragma unroll
        for (int q = 0; q < U; ++q)
            v[q] = c + q < jb ? p[(size_t)(c + q) * lda] : 0u;
#pragma unroll
        for (int q = 0; q < U; ++q)
            if (c + q < panel_cols(jb))
                rw[(c + q) * T] = p32_to_double(v[q]);
    }
}

// MAXT: the most threads a CTA of this instance has, MAXR: the most slots of a thread.  One CTA
// per SM is said to the compiler so that it spends registers on overlapping a row's columns (62
// instead of 40: 355 cycles for 8 columns of a warp instead of 511).
template <int MAXT, int MAXR>
__global__ void __launch_bounds__(MAXT, 1) lu_panel_cluster_kernel(uint32_t *__restrict__ P, size_t lda, int M, int jb,
                                                                   int R, int row0, int *__restrict__ ipiv,
                                                                   int *__restrict__ info)
{
    namespace cgs = cooperative_groups;
    cgs::cluster_group cluster = cgs::this_cluster();
    const int rank = (int)cluster.block_rank(), ncta = (int)cluster.num_blocks();
    extern __shared__ __align__(128) unsigned char smem_panel[];
    __shared__ PivotCand s_wc[2][32];                  // each warp's candidate, by column parity
    __shared__ PivotPush s_push[3][PANEL1_MAX_CTAS]; // the CTAs' candidates, by column mod 3
    if (*info < 0) // written only by earlier launches: the same in every CTA
        return;
    const int T = (int)blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = T >> 5;
    const unsigned char *tab = smem_panel;
    double *s_rows = reinterpret_cast<double *>(smem_panel + STEP_TAB_BYTES); // [R][W][T]: this CTA's slots
    const int W = panel_cols(jb);
    double *s_cu = s_rows + (size_t)R * W * T; // [3][ncta][W]: the candidates' rows
    __shared__ int s_piv[PANEL1_MAX_JB];       // the pivots' rows (written out at the end: a global store
                                               // would hold up the next arrival)
    step_tables_fill(smem_panel, tid, T);
    auto slot_row = [&](int r, int t) { return s_rows + r * W * T + t; }; // column c at [c * T]
    for (int e = tid; e < 3 * ncta * W; e += T)
        s_cu[e] = 0.0; // past jb it stays
    const int base = rank * (R * T);
    int row[MAXR]; // the logical row each slot holds (-1: none)
#pragma unroll
    for (int r = 0; r < MAXR; ++r) {
        const int i = base + r * T + tid;
        row[r] = (r < R && i < M) ? i : -1;
        if (row[r] >= 0)
            panel_load_row(slot_row(r, tid), T, P + i, lda, jb);
    }
    panel_sync(cluster, ncta); // the tables are filled; every CTA has started

    PivotCand cand;
    auto cand_none = [&]() { cand = PivotCand{INT_MIN, 0u, INT_MAX, 0}; };
    auto cand_add = [&](double v, int r) {
        const double a = fabs(v);
        const PivotCand c = {v != v ? -1 : __double2hiint(a), v != v ? 0u : (uint32_t)__double2loint(a), row[r],
                             (r << 16) | tid};
        if (cand_better(c, cand))
            cand = c;
    };
    // The CTA's candidate of column c into every CTA; `u` and the rows' column c-1 bring its
    // row up to date (c > 0).  Then the arrival for column c.
    auto publish = [&](int c, const double *u) {
        const int bl = cand_best_lane(cand);
        if (lane == bl)
            s_wc[c & 1][warp] = cand;
        __syncthreads();
        PivotCand best = lane < nw ? s_wc[c & 1][lane] : PivotCand{INT_MIN, 0u, INT_MAX, 0};
        const int bw = cand_best_lane(best);
        if (warp == bw) {
            best = s_wc[c & 1][bw];
            const double *rw = slot_row(best.slot >> 16, best.slot & 0xFFFF);
            double v = 0.0;
            if (best.hi != INT_MIN) {
                const double l = c > 0 ? rw[(c - 1) * T] : 0.0;
                v = rw[c * T];
                for (int q = c + lane; q < jb; q += 32) {
                    double x = rw[q * T];
                    if (c > 0 && q > c)
                        x = mac_any(x, -u[q], l, tab);
                    double *to = s_cu + ((c % 3) * ncta + rank) * W + q;
                    for (int r = 0; r < ncta; ++r)
                        *cluster.map_shared_rank(to, r) = x;
                }
            }
            // 1/pivot (Rgetrf2.cpp:119-131: |pivot| >= sfmin = FLT_MIN, minpos as a posit, holds for
            // all but zero and NaR; a NaR pivot divides every element, which gives NaR as
            // multiplying by NaR does; a zero one scales nothing)
            const double recip = v == 0.0 ? 1.0 : f64_posit_div(1.0, v, 1.0 / v);
            if (lane < ncta) {
                PivotPush *to = cluster.map_shared_rank(&s_push[c % 3][rank], lane);
                to->c = best;
                to->val = v;
                to->recip = recip;
            }
        }
        __syncwarp();
        if (ncta > 1)
            cgs::this_cluster().barrier_arrive();
    };
    cand_none();
#pragma unroll
    for (int r = 0; r < MAXR; ++r)
        if (row[r] >= 0)
            cand_add(slot_row(r, tid)[0], r);
    publish(0, nullptr);
    for (int k = 0; k < jb; ++k) {
        if (ncta > 1)
            cgs::this_cluster().barrier_wait();
        else
            __syncthreads();
        const PivotCand mine = lane < ncta ? s_push[k % 3][lane].c : PivotCand{INT_MIN, 0u, INT_MAX, 0};
        const int win = cand_best_lane(mine);
        const PivotPush pv = s_push[k % 3][win];
        const double *u = s_cu + ((k % 3) * ncta + win) * W; // the pivot row, columns k ..
        const int p = pv.c.row;
        if (rank == 0 && tid == 0) {
            s_piv[k] = row0 + p + 1; // 1-based, global
            if (pv.val == 0.0 && *info == 0)
                *info = row0 + k + 1;
        }
        if (p != k) {
            if (pv.val == 0.0) {
                // A zero pivot leaves its own column in place (Rgetrf2.cpp:107-117) while the
                // recursion's Rlaswp calls move rows k and p in every other column: the two
                // slots trade their column-k values back, by row k's holder.
                double *src = cluster.map_shared_rank(s_rows, win) + (pv.c.slot >> 16) * W * T + (pv.c.slot & 0xFFFF);
#pragma unroll
                for (int r = 0; r < MAXR; ++r)
                    if (row[r] == k) {
                        src[k * T] = slot_row(r, tid)[k * T];
                        slot_row(r, tid)[k * T] = pv.val;
                    }
            }
#pragma unroll
            for (int r = 0; r < MAXR; ++r)
                row[r] = row[r] == k ? p : (row[r] == p ? k : row[r]);
        }
        const bool more = k + 1 < jb;
        const double un = more ? -u[k + 1] : 0.0;
        cand_none();
#pragma unroll
        for (int r = 0; r < MAXR; ++r)
            if (row[r] > k) {
                double *rw = slot_row(r, tid);
                const double l = mul_any(rw[k * T], pv.recip, tab); // Rscal
                rw[k * T] = l;
                if (more) {
                    const double x = mac_any(rw[(k + 1) * T], un, l, tab);
                    rw[(k + 1) * T] = x;
                    cand_add(x, r);
                }
            }
        if (more) {
            publish(k + 1, u);
            __syncwarp(); // the candidate's row has been read
        }
#pragma unroll
        for (int r = 0; r < MAXR; ++r)
            if (row[r] > k) {
                double *rw = slot_row(r, tid);
                panel_row_update(rw, T, u, rw[k * T], k + 2, jb, tab);
            }
    }
    panel_sync(cluster, ncta); // no CTA leaves while another may still write its shared memory
    if (rank == 0)
        for (int c = tid; c < jb; c += T)
            ipiv[row0 + c] = s_piv[c];
#pragma unroll
    for (int r = 0; r < MAXR; ++r)
        if (row[r] >= 0)
            for (int c = 0; c < jb; ++c)
                P[row[r] + (size_t)c * lda] = p32_from_double_exact(slot_row(r, tid)[c * T]);
}

// After a panel of columns [j, j+jb) (jb <= ROWS_JB_MAX): the panel's row interchanges
// (Rlaswp, Rlaswp.cpp:77-107, in ascending order) on every column outside the panel, and
// the unit-lower solve of the U12 block (Rtrsm('L', 'L', 'N', 'U'), Rtrsm.cpp:139-154, zero
// multipliers skipped as there) on the columns right of it, in one launch: one warp per
// column, lane i holding row j+i and (for an interchange with a row below the block) that
// row's value, loaded together; the interchanges run in order as exchanges between lanes,
// the solve as jb steps of one multiply-add per lane with the step's b_k from its lane.
// For an inner panel of a wider block (rgetrf_launch), A is the block's corner, at row and column
// `off` of the matrix, n its width, and `skip` false: a panel's own updates skip no multiplier.
constexpr int ROWS_JB_MAX = 32;
constexpr int ROWS_THREADS = 256; // 8 columns per block

__global__ void __launch_bounds__(ROWS_THREADS) lu_rows_kernel(uint32_t *__restrict__ A, size_t lda, int n, int j,
                                                               int jb, const int *__restrict__ ipiv, int off,
                                                               bool skip)
{
    constexpr unsigned FULL = 0xFFFFFFFFu;
    __shared__ double s_L[ROWS_JB_MAX * ROWS_JB_MAX]; // l_ik at [i * ROWS_JB_MAX + k], FP64
    __shared__ int s_t[ROWS_JB_MAX];                  // interchange i: row j+i <-> row s_t[i] (0-based)
    __shared__ int s_alias[ROWS_JB_MAX];              // below the block: the first interchange with that row
    const int tid = threadIdx.x, lane = tid & 31;
    for (int e = tid; e < jb * jb; e += ROWS_THREADS) {
        const int i = e % jb, k = e / jb;
        s_L[i * ROWS_JB_MAX + k] = p32_to_double(A[(j + i) + (size_t)(j + k) * lda]);
    }
    for (int i = tid; i < jb; i += ROWS_THREADS)
        s_t[i] = ipiv[j + i] - 1 - off;
    __syncthreads();
    for (int i = tid; i < jb; i += ROWS_THREADS) {
        int a = -1;
        if (s_t[i] >= j + jb) {
            a = i;
            for (int q = 0; q < i; ++q)
                if (s_t[q] == s_t[i]) {
                    a = q;
                    break;
                }
        }
        s_alias[i] = a;
    }
    __syncthreads();
    const int ci = blockIdx.x * (ROWS_THREADS / 32) + (tid >> 5);
    if (ci >= n - jb)
        return; // the whole warp
    const int c = ci < j ? ci : ci + jb; // the columns outside the panel
    uint32_t *col = A + (size_t)c * lda;
    const bool row = lane < jb;
    const int my_t = row ? s_t[lane] : 0, my_alias = row ? s_alias[lane] : -1;
    uint32_t v = row ? col[j + lane] : 0u;               // row j+lane
    uint32_t w = (my_alias == lane) ? col[my_t] : 0u;  // row my_t (below the block)
    for (int i = 0; i < jb; ++i) {
        const int t = s_t[i];
        if (t == j + i)
            continue;
        const bool in = t < j + jb;
        const int o = in ? t - j : s_alias[i];
        const uint32_t vi = __shfl_sync(FULL, v, i);
        const uint32_t vo = __shfl_sync(FULL, in ? v : w, o);
        if (lane == o) {
            if (in)
                v = vi;
            else
                w = vi;
        }
        if (lane == i)
            v = vo;
    }
    if (my_alias == lane)
        col[my_t] = w;
    if (c > j) { // U12 <- L11^-1 A12, column-oriented as Rtrsm.cpp:139-154 (unit diagonal)
        double x = row ? p32_to_double(v) : 0.0;
        for (int k = 0; k < jb; ++k) {
            const double bk = __shfl_sync(FULL, x, k);
            if ((bk != 0.0 || !skip) && lane > k && row)
                x = f64_posit_mac_checked(x, -bk, s_L[lane * ROWS_JB_MAX + k]);
        }
        v = p32_from_double(x);
    }
    if (row)
        col[j + lane] = v;
}

// ---------------------------------------------------------------------------
// Rlaswp (Rlaswp.cpp:77-107): interchanges k1..k2 (1-based, global ipiv) applied in order
// to `ncols` columns starting at A; one thread per column.
// ---------------------------------------------------------------------------
__global__ void laswp_kernel(uint32_t *__restrict__ A, size_t lda, int ncols, int k1, int k2,
                             const int *__restrict__ ipiv, int incx, const int *__restrict__ info)
{
    if (info && *info < 0)
        return;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncols)
        return;
    uint32_t *col = A + (size_t)c * lda;
    if (incx > 0) {
        for (int i = k1; i <= k2; ++i) {
            int ip = ipiv[i - 1];
            if (ip != i) {
                uint32_t t = col[i - 1];
                col[i - 1] = col[ip - 1];
                col[ip - 1] = t;
            }
        }
    } else {
        for (int i = k2; i >= k1; --i) {
            int ip = ipiv[i - 1];
            if (ip != i) {
                uint32_t t = col[i - 1];
                col[i - 1] = col[ip - 1];
                col[ip - 1] = t;
            }
        }
    }
}

// The same on a few columns of B, all n interchanges of a solve: one CTA per column, the
// column and a stretch of ipiv in shared memory, one thread doing the swaps there (about 60
// cycles each, against an L2 round trip each for laswp_kernel).
constexpr int LASWP_COL_THREADS = 256;
constexpr int LASWP_COL_MAX = 48 * 1024; // rows: 4 bytes each, beside the stretch
constexpr int LASWP_STRETCH = 1024;

__global__ void __launch_bounds__(LASWP_COL_THREADS) laswp_col_kernel(uint32_t *__restrict__ B, size_t ldb, int n,
                                                                      const int *__restrict__ ipiv, bool forward)
{
    extern __shared__ uint32_t s_c[]; // [n]
    __shared__ int s_p[LASWP_STRETCH];
    uint32_t *col = B + (size_t)blockIdx.x * ldb;
    for (int i = threadIdx.x; i < n; i += LASWP_COL_THREADS)
        s_c[i] = col[i];
    for (int d0 = 0; d0 < n; d0 += LASWP_STRETCH) {
        const int cnt = min(LASWP_STRETCH, n - d0);
        __syncthreads(); // the column is staged; the last stretch is done with
        for (int d = threadIdx.x; d < cnt; d += LASWP_COL_THREADS)
            s_p[d] = ipiv[forward ? d0 + d : n - 1 - d0 - d] - 1;
        __syncthreads();
        if (threadIdx.x == 0)
            for (int d = 0; d < cnt; ++d) {
                const int i = forward ? d0 + d : n - 1 - d0 - d, p = s_p[d];
                const uint32_t x = s_c[i];
                s_c[i] = s_c[p];
                s_c[p] = x;
            }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += LASWP_COL_THREADS)
        col[i] = s_c[i];
}

// Rlaswp of a solve's right-hand sides (Rgetrs.cpp:84-114).
static cudaError_t launch_laswp_rhs(uint32_t *B, int ldb, int nrhs, int n, const int *ipiv, bool forward,
                                    cudaStream_t st)
{
    if (n <= LASWP_COL_MAX) {
        const cudaError_t e = cudaFuncSetAttribute(laswp_col_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   LASWP_COL_MAX * 4);
        if (e != cudaSuccess)
            return e;
        laswp_col_kernel<<<nrhs, LASWP_COL_THREADS, (size_t)n * 4, st>>>(B, ldb, n, ipiv, forward);
    } else {
        laswp_kernel<<<(nrhs + 127) / 128, 128, 0, st>>>(B, ldb, nrhs, 1, n, ipiv, forward ? 1 : -1, nullptr);
    }
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// The axpy-form solves: lower forwards (Rtrsm.cpp:139-154) and upper backwards
// (Rtrsm.cpp:121-136), side = L, trans = N.
// ---------------------------------------------------------------------------
// Each b_i takes its updates b_i - b_k*a_ik in the order of k, then (non-unit) one division;
// a zero b_k is skipped.  Which other rows are updated when does not matter, so the column
// is cut into blocks of 32 rows: a warp solves the next block's 32 rows by itself, a lane
// each, b_k by shuffle, publishes them, and every warp then runs its own rows through those
// 32 columns.  One thread-block cluster of up to 8 CTAs of 16 warps per right-hand side, the
// blocks dealt out CTA by CTA, then warp by warp; a published block goes to every CTA's
// shared memory, double-buffered, with one cluster barrier (one CTA: a block barrier) per
// block.  The owner of the block after the published one updates that first and solves it
// while the others update the rest.
// What bounds it: the chain of one row after the other, about 70 cycles for an update whose
// multiplier is there and 150 for one whose b_k was the last step's (260 with the division),
// i.e. 230 (340) cycles per row and no more barriers than blocks.  A column per step of one
// CTA of 1024 threads, with a barrier each, took 1.9 us per row at n = 4096.  Rgetrs, one
// right-hand side: n = 1024 1.84 -> 0.79 ms, 4096 15.4 -> 3.1 ms, 8192 48.8 -> 8.4 ms.
// Updates and solves run in step_one (gemm_tile.cuh): a value outside the fast window or a
// NaR turns into NaN, is noticed at the end of the block and done again step by step.
constexpr int COL_BLK = 32;
constexpr int COL_WARPS = 16;
constexpr int COL_MAX_CTAS = 8;
constexpr size_t COL_SMEM_MAX = 227 * 1024 - 1024;

// Shared memory of a CTA: tables, a diagonal block's patterns per warp, the CTA's rows.
static size_t col_smem_bytes(int nb, int ncta, int warps)
{
    const int per = (nb + ncta - 1) / ncta;
    return STEP_TAB_BYTES + (size_t)warps * COL_BLK * COL_BLK * 4 + (size_t)per * COL_BLK * 8;
}

template <bool UPPER, bool UNIT>
__global__ void __launch_bounds__(COL_WARPS * 32, 1) trsm_block_kernel(const uint32_t *__restrict__ A, size_t lda,
                                                                       uint32_t *__restrict__ B, size_t ldb, int m,
                                                                       const int *__restrict__ info)
{
    namespace cgs = cooperative_groups;
    cgs::cluster_group cluster = cgs::this_cluster();
    constexpr unsigned FULL = 0xFFFFFFFFu;
    extern __shared__ __align__(128) unsigned char smem_col[];
    __shared__ double s_sol[2][COL_BLK]; // the published block, by step parity
    if (info && *info < 0) // written by earlier launches: the same in every CTA
        return;
    const int rank = (int)cluster.block_rank(), ncta = (int)cluster.num_blocks();
    const int nw = (int)blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nb = (m + COL_BLK - 1) / COL_BLK;
    const unsigned char *tab = smem_col;
    uint32_t *tile = reinterpret_cast<uint32_t *>(smem_col + STEP_TAB_BYTES) + warp * COL_BLK * COL_BLK;
    double *s_x = reinterpret_cast<double *>(smem_col + STEP_TAB_BYTES + (size_t)nw * COL_BLK * COL_BLK * 4);
    uint32_t *bcol = B + (size_t)(blockIdx.x / ncta) * ldb;
    step_tables_fill(smem_col, threadIdx.x, blockDim.x);

    // block j is this warp's when mine(j); the warp's blocks in the order they are solved
    auto mine = [&](int j) { return j % ncta == rank && (j / ncta) % nw == warp; };
    auto block_of = [&](int step) { return UPPER ? nb - 1 - step : step; };
    const int first = rank + ncta * warp, stride = ncta * nw;
    const int count = first < nb ? (nb - 1 - first) / stride + 1 : 0;
    auto own = [&](int s) { return first + stride * (UPPER ? count - 1 - s : s); };
    auto xrow = [&](int j) -> double & { return s_x[(j / ncta) * COL_BLK + lane]; };
    auto load_tile = [&](int j) { // the diagonal block: lane's row, all columns
        const int i = j * COL_BLK + lane;
        for (int k = 0; k < COL_BLK; ++k) {
            const int c = j * COL_BLK + k;
            tile[k * COL_BLK + lane] = (i < m && c < m) ? A[i + (size_t)c * lda] : 0u;
        }
    };
    // Solves block j (its tile loaded, its updates done) and publishes it into `buf`.
    auto solve = [&](int j, int buf) {
        const double x0 = xrow(j);
        const bool live = j * COL_BLK + lane < m;
        double x = x0, d = 1.0, rc = 1.0;
        if (!UNIT && live) {
            d = p32_to_double(tile[lane * COL_BLK + lane]);
            rc = 1.0 / d;
        }
#pragma unroll 4
        for (int q = 0; q < COL_BLK; ++q) {
            const int k = UPPER ? COL_BLK - 1 - q : q;
            if (!UNIT && lane == k && x != 0.0)
                x = f64_posit_div(x, d, rc);
            const double xk = __shfl_sync(FULL, x, k);
            const double r = step_one(x, -xk, p32_to_double(tile[k * COL_BLK + lane]), tab);
            if (UPPER ? lane < k : lane > k)
                x = r;
        }
        if (__any_sync(FULL, live && x != x)) { // step by step, as the reference skips and rounds
            x = x0;
#pragma unroll 1
            for (int q = 0; q < COL_BLK; ++q) {
                const int k = UPPER ? COL_BLK - 1 - q : q;
                if (!UNIT && lane == k && x != 0.0)
                    x = f64_posit_div(x, d, rc);
                const double xk = __shfl_sync(FULL, x, k);
                if (xk != 0.0 && (UPPER ? lane < k : lane > k))
                    x = f64_posit_mac_checked(x, -xk, p32_to_double(tile[k * COL_BLK + lane]));
            }
        }
        if (!live)
            x = 0.0;
        xrow(j) = x;
        for (int r = 0; r < ncta; ++r)
            *cluster.map_shared_rank(&s_sol[buf][lane], r) = x;
    };
    // Block j's coefficients of the columns of block c, a row per lane.
    auto load_coef = [&](int j, int c, uint32_t (&l)[COL_BLK]) {
        const int i = j * COL_BLK + lane;
        const uint32_t *p = A + i + (size_t)c * COL_BLK * lda;
#pragma unroll
        for (int k = 0; k < COL_BLK; ++k)
            l[k] = (i < m && c * COL_BLK + k < m) ? p[(size_t)k * lda] : 0u;
    };
    for (int s = 0; s < count; ++s) {
        const int j = own(s), i = j * COL_BLK + lane;
        xrow(j) = i < m ? p32_to_double(bcol[i]) : 0.0;
    }
    if (count > 0)
        load_tile(own(0));
    panel_sync(cluster, ncta); // the tables are filled; every CTA has started
    int done = 0; // the warp's blocks solved so far
    if (mine(block_of(0))) {
        solve(block_of(0), 0);
        if (++done < count)
            load_tile(own(done));
    }
    for (int step = 0; step + 1 < nb; ++step) {
        const int c = block_of(step);
        uint32_t l[COL_BLK];
        if (done < count)
            load_coef(own(done), c, l); // in flight across the barrier
        panel_sync(cluster, ncta); // block c is published
        const double *sol = s_sol[step & 1];
        for (int s = done; s < count; ++s) {
            const int j = own(s);
            if (s > done)
                load_coef(j, c, l);
            const double x0 = xrow(j);
            double x = x0;
#pragma unroll
            for (int q = 0; q < COL_BLK; ++q) {
                const int k = UPPER ? COL_BLK - 1 - q : q;
                x = step_one(x, -sol[k], p32_to_double(l[k]), tab);
            }
            if (x != x) {
                x = x0;
                const int i = j * COL_BLK + lane;
#pragma unroll 1
                for (int q = 0; q < COL_BLK; ++q) {
                    const int k = UPPER ? COL_BLK - 1 - q : q;
                    const double xk = sol[k];
                    if (xk != 0.0 && i < m)
                        x = f64_posit_mac_checked(x, -xk, p32_to_double(A[i + (size_t)(c * COL_BLK + k) * lda]));
                }
            }
            xrow(j) = x;
            __syncwarp();
            if (s == done && j == block_of(step + 1))
                solve(j, (step + 1) & 1);
        }
        if (done < count && own(done) == block_of(step + 1))
            if (++done < count)
                load_tile(own(done));
    }
    panel_sync(cluster, ncta); // no CTA leaves while another may still write its shared memory
    for (int s = 0; s < count; ++s) {
        const int j = own(s), i = j * COL_BLK + lane;
        if (i < m)
            bcol[i] = p32_from_double_exact(xrow(j));
    }
}

// A column that does not fit in the shared memory of 8 CTAs (more than 202,752 rows: a triangle of
// 164 GB): the column stays in B, one CTA of 1024 threads per right-hand side, a row a step.
template <bool UPPER>
__global__ void __launch_bounds__(1024) trsm_long_kernel(const uint32_t *__restrict__ A, size_t lda, uint32_t *B,
                                                         size_t ldb, int m, bool unit, const int *__restrict__ info)
{
    if (info && *info < 0)
        return;
    uint32_t *x = B + (size_t)blockIdx.x * ldb;
    for (int s = 0; s < m; ++s) {
        const int k = UPPER ? m - 1 - s : s;
        const uint32_t *ak = A + (size_t)k * lda;
        uint32_t bk = x[k];
        if (bk != 0) {
            if (!unit) {
                bk = pdiv_est(bk, ak[k]);
                __syncthreads(); // every thread has read x[k]
                if (threadIdx.x == 0)
                    x[k] = bk;
            }
            const int end = UPPER ? k : m;
            for (int i = (UPPER ? 0 : k + 1) + (int)threadIdx.x; i < end; i += (int)blockDim.x)
                x[i] = padd(x[i], pmul(0u - bk, ak[i]));
        }
        __syncthreads();
    }
}

// CTAs of a right-hand side's cluster: up to one per 16 blocks (512 rows) and 8, but not so many
// that the right-hand sides take more turns for it.  A cluster's time goes as 1 + m / (1800 ctas): its
// chain of rows, and the updates its CTAs share.  Rgetrs, n = 4096: one right-hand side 3.1 ms with 8
// CTAs, 4.1 with 4, 8.0 with 1; 1024 of them 204 ms with 8, 123 with 4, 55 with 1 (107 in the
// form before this one, a CTA each); n = 2048, 1024 of them: 47 ms with 4, 18 with 1.
int solve_cluster_ctas(int m, int nrhs)
{
    // clusters on the GPU at a time by size, one CTA per SM (a cluster lies within one GPC)
    static const int at_once[COL_MAX_CTAS + 1] = {0, 148, 74, 44, 32, 20, 20, 15, 15};
    const int nb = (m + COL_BLK - 1) / COL_BLK;
    const int most = std::max(1, std::min(COL_MAX_CTAS, (nb + COL_WARPS - 1) / COL_WARPS));
    int best = most;
    double best_cost = 0.0;
    for (int c = most; c >= 1; --c) {
        if (c < most && col_smem_bytes(nb, c, std::min(COL_WARPS, (nb + c - 1) / c)) > COL_SMEM_MAX)
            break; // long columns: fewer CTAs would hold fewer warps
        const double cost = (double)((nrhs + at_once[c] - 1) / at_once[c]) * (1.0 + m / (1800.0 * c));
        if (c == most || cost < best_cost) {
            best = c;
            best_cost = cost;
        }
    }
    return best;
}

// One cluster per right-hand side.
static cudaError_t launch_col(bool upper, bool unit, int nrhs, const uint32_t *A, size_t lda, uint32_t *B, size_t ldb,
                              int m, const int *info, cudaStream_t st)
{
    const int nb = (m + COL_BLK - 1) / COL_BLK;
    const int ncta = solve_cluster_ctas(m, nrhs);
    auto *fn = upper ? (unit ? trsm_block_kernel<true, true> : trsm_block_kernel<true, false>)
                     : (unit ? trsm_block_kernel<false, true> : trsm_block_kernel<false, false>);
    // no more warps than a CTA has blocks (nor, for the longest columns, than fit)
    int warps = std::min(COL_WARPS, (nb + ncta - 1) / ncta);
    while (warps > 1 && col_smem_bytes(nb, ncta, warps) > COL_SMEM_MAX)
        --warps;
    const size_t smem = col_smem_bytes(nb, ncta, warps);
    if (smem > COL_SMEM_MAX) {
        if (upper)
            trsm_long_kernel<true><<<nrhs, 1024, 0, st>>>(A, lda, B, ldb, m, unit, info);
        else
            trsm_long_kernel<false><<<nrhs, 1024, 0, st>>>(A, lda, B, ldb, m, unit, info);
        return cudaGetLastError();
    }
    // Here and elsewhere the limit is set to the most the kernel can take, not to this launch's size:
    // another thread's launch of the same kernel may come between this call and the launch.
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)COL_SMEM_MAX);
    if (e != cudaSuccess)
        return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nrhs * ncta));
    cfg.blockDim = dim3((unsigned)(warps * 32));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)ncta;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, fn, A, lda, B, ldb, m, info);
}

// Lower, transposed (Rtrsm.cpp:175-186): one block per right-hand side; the column is
// staged in shared memory (when it fits) and one thread runs the whole dependent chain
// (trsm_chain.cuh).
constexpr int LLT_SMEM_MAX = 227 * 1024 - 128; // dynamic, beside a row's scalars

__global__ void __launch_bounds__(32) trsm_llt_kernel(const uint32_t *__restrict__ L, size_t ldl,
                                                      uint32_t *__restrict__ B, size_t ldb, int m, bool staged,
                                                      bool unit, bool upper, const int *__restrict__ info)
{
    extern __shared__ uint32_t s_col[];
    if (info && *info != 0) // a factorization stopped before this solve
        return;
    uint32_t *bcol = B + (size_t)blockIdx.x * ldb;
    if (!staged) {
        if (threadIdx.x == 0)
            llt_chain(L, ldl, bcol, m, unit, upper);
        return;
    }
    for (int i = threadIdx.x; i < m; i += 32)
        s_col[i] = bcol[i];
    __syncwarp();
    if (threadIdx.x == 0)
        llt_chain(L, ldl, s_col, m, unit, upper);
    __syncwarp();
    for (int i = threadIdx.x; i < m; i += 32)
        bcol[i] = s_col[i];
}

// ---------------------------------------------------------------------------
// The dot-form solves, one block per right-hand side.
// ---------------------------------------------------------------------------
// Rtrsm('L', 'L', 'T'), Rtrsm.cpp:175-186: for i = m-1 down to 0, t = b_i, t = t - a_ki*b_k
// for k = i+1 .. m-1 in order, b_i = t / a_ii (UPPER: Rtrsm('L', 'U', 'T'),
// Rtrsm.cpp:160-173, rows in increasing order, terms k = 0 .. i-1).  A right-hand side is one
// chain of m(m-1)/2 dependent additions, so the warp that adds (warp 0) bounds the solve;
// the other three compute the next row's terms -a_k * b_k (all whose b_k are final) into the
// other half of a double buffer, and its diagonal's reciprocal, meanwhile.  Warp 0 sums a row
// with warp_chain (trsm_chain.cuh); the term of the b just finished (the first one, UPPER:
// the last) it forms itself.  Four warps: one per sub-partition of the SM, so nothing else
// issues where the chain runs.  Rpotrs, one right-hand side, against four warps that scanned one
// step map per addend: n = 1024 10.5 -> 5.7 ms, 4096 92 -> 52 ms.
// NaR travels as NaN; a NaR term sets its row's flag and is replaced by 0.
constexpr int LTX_THREADS = 128;

template <class Terms, class Col>
static size_t ltx_smem_bytes(int m)
{
    return 2 * Terms::bytes(m) + (Col::GLOBAL ? 0 : (size_t)m * 8);
}

template <class Terms, class Col, bool UPPER>
__global__ void __launch_bounds__(LTX_THREADS) trsm_ltx_kernel(const uint32_t *__restrict__ L, size_t ldl,
                                                               uint32_t *__restrict__ B, size_t ldb, int m, bool unit,
                                                               const int *__restrict__ info)
{
    extern __shared__ __align__(16) unsigned char smem_ltx[];
    __shared__ LtxRow s_row[2];
    if (info && *info != 0) // a factorization stopped before this solve
        return;
    Col x;
    uint32_t *bcol = B + (size_t)blockIdx.x * ldb;
    if constexpr (Col::GLOBAL) {
        x.b = bcol;
        block_ltx_solve<LTX_THREADS, UPPER, Terms>(L, ldl, x, m, unit, smem_ltx, s_row);
    } else {
        x.b = reinterpret_cast<double *>(smem_ltx + 2 * Terms::bytes(m));
        for (int k = threadIdx.x; k < m; k += LTX_THREADS)
            x.set(k, p32_to_double(bcol[k]));
        block_ltx_solve<LTX_THREADS, UPPER, Terms>(L, ldl, x, m, unit, smem_ltx, s_row);
        for (int k = threadIdx.x; k < m; k += LTX_THREADS)
            bcol[k] = p32_from_double_exact(x.get(k));
    }
}

// ---------------------------------------------------------------------------
// Cholesky panel (lower)
// ---------------------------------------------------------------------------
// Lower Cholesky panel of up to 32 columns in one launch.  Below the diagonal block every row goes its own way once the block is
// factored, so each CTA of 128 threads factors the block for itself, in shared memory, and
// then takes 128 rows through it, one per thread: l_ik = (1/l_kk)*a_ik (Rtrsm.cpp:265-268),
// a_ic += (-l_ck)*l_ik for c > k, in the FP64 step.  No CTA waits for another.
// The block's factor: per column every warp forms l_kk (Rpotrf2.cpp:90-97) and 1/l_kk and
// scales the column for itself, a row per lane, and updates every fourth of the columns right
// of it; one block barrier.  A failed diagonal (a_kk <= 0, NaR included) stops with info after
// the columns before it, in the rows below too.
// Other CTAs still read the block when the first one is done, so its factor goes to `out`
// and the next panel's launch (the next to touch the matrix there) puts it in place; the last
// panel has one CTA and writes it itself.
// What bounds it: the block's chain, about 850 cycles a column (root, reciprocal, scaling,
// update, one after the other), then 15,000 for 32 columns of a row.  The cluster form this
// replaced took two cluster barriers and one update at a time per column: Cholesky n = 1024
// 3.9 -> 2.5 ms, 4096 27.6 -> 19.2.
constexpr int CHOL_JB_MAX = 32;
constexpr int CHOL_T = 128;
constexpr int CHOL_LD = CHOL_JB_MAX + 1;
constexpr size_t CHOL_BLOCKS_BYTES = 2 * CHOL_JB_MAX * CHOL_JB_MAX * 4; // two panels' blocks in the workspace

static size_t chol_panel_smem(int jb)
{
    return STEP_TAB_BYTES + ((size_t)CHOL_JB_MAX * CHOL_LD + PANEL_U + CHOL_JB_MAX + (size_t)panel_cols(jb) * CHOL_T) * sizeof(double);
}

__global__ void __launch_bounds__(CHOL_T, 1) chol_panel_kernel(uint32_t *__restrict__ P, size_t lda, int M, int jb,
                                                            int row0, int *__restrict__ info,
                                                            uint32_t *__restrict__ out, uint32_t *__restrict__ prev,
                                                            int prev_jb, const uint32_t *__restrict__ in)
{
    extern __shared__ __align__(128) unsigned char smem_chol[];
    const unsigned char *tab = smem_chol;
    double *s_d = reinterpret_cast<double *>(smem_chol + STEP_TAB_BYTES); // the block: a_ic at [c * CHOL_LD + i]
    double *s_r = s_d + CHOL_JB_MAX * CHOL_LD + PANEL_U;                  // 1/l_kk
    double *s_rows = s_r + CHOL_JB_MAX;                                   // [panel_cols(jb)][CHOL_T]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // info within this panel is this launch's own, by the first CTA
    const int seen = *info;
    if (blockIdx.x == 0 && prev_jb > 0 && (seen == 0 || seen > row0 - prev_jb))
        for (int e = tid; e < prev_jb * prev_jb; e += CHOL_T) {
            const int i = e % prev_jb, c = e / prev_jb;
            if (i >= c)
                prev[i + (size_t)c * lda] = in[e];
        }
    if (seen != 0 && seen <= row0)
        return;
    step_tables_fill(smem_chol, tid, CHOL_T);
    for (int e = tid; e < CHOL_JB_MAX * CHOL_LD + PANEL_U; e += CHOL_T)
        s_d[e] = 0.0; // past a column's end it stays, or meets a column past jb
    __syncthreads();
    for (int e = tid; e < jb * jb; e += CHOL_T) {
        const int i = e % jb, c = e / jb;
        if (i >= c)
            s_d[c * CHOL_LD + i] = p32_to_double(P[i + (size_t)c * lda]);
    }
    const int i = jb + blockIdx.x * CHOL_T + tid; // this thread's row
    if (i < M)
        panel_load_row(s_rows + tid, CHOL_T, P + i, lda, jb);
    __syncthreads();
    int stop = jb; // the first column whose diagonal fails
    for (int k = 0; k < jb; ++k) {
        const double *dk = s_d + k * CHOL_LD;
        const double akk = dk[k];
        if (!(akk > 0.0)) { // the same in every thread
            stop = k;
            break;
        }
        const double lkk = f64_posit_sqrt(akk);
        const double recip = f64_posit_div(1.0, lkk, 1.0 / lkk);
        double l = 0.0;
        if (lane > k && lane < jb)
            l = mul_any(dk[lane], recip, tab);
        // columns k+1+warp, +4, ...: rows lane >= column; l_ck is lane c's l
        for (int c0 = k + 1 + warp; c0 < jb; c0 += 16) {
            double y[4];
            bool bad = false;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int c = c0 + 4 * q;
                const double t = -__shfl_sync(0xFFFFFFFFu, l, c & 31);
                const bool in_block = c < jb && lane >= c && lane < jb;
                const double x = in_block ? s_d[c * CHOL_LD + lane] : 0.0;
                y[q] = step_one(x, t, l, tab);
                bad |= in_block && y[q] != y[q];
            }
            if (__any_sync(0xFFFFFFFFu, bad)) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int c = c0 + 4 * q;
                    const double t = -__shfl_sync(0xFFFFFFFFu, l, c & 31);
                    if (c < jb && lane >= c && lane < jb)
                        y[q] = mac_any(s_d[c * CHOL_LD + lane], t, l, tab);
                }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int c = c0 + 4 * q;
                if (c < jb && lane >= c && lane < jb)
                    s_d[c * CHOL_LD + lane] = y[q];
            }
        }
        __syncthreads(); // column k has been read, the columns right of it are up to date
        if (warp == (k & 3) && lane >= k && lane < jb)
            s_d[k * CHOL_LD + lane] = lane == k ? lkk : l;
        if (tid == 0)
            s_r[k] = recip;
    }
    __syncthreads();
    if (blockIdx.x == 0) {
        if (stop < jb && tid == 0)
            *info = row0 + stop + 1;
        for (int e = tid; e < jb * jb; e += CHOL_T) {
            const int r = e % jb, c = e / jb;
            if (r >= c) {
                const uint32_t v = p32_from_double_exact(s_d[c * CHOL_LD + r]);
                if (out)
                    out[e] = v;
                else
                    P[r + (size_t)c * lda] = v;
            }
        }
    }
    if (i >= M)
        return;
    double *rw = s_rows + tid;
    for (int k = 0; k < stop; ++k) {
        const double l = mul_any(rw[k * CHOL_T], s_r[k], tab);
        rw[k * CHOL_T] = l;
        panel_row_update(rw, CHOL_T, s_d + k * CHOL_LD, l, k + 1, jb, tab);
    }
    for (int c = 0; c < jb; ++c)
        P[i + (size_t)c * lda] = p32_from_double_exact(rw[c * CHOL_T]);
}

// ---------------------------------------------------------------------------
// Upper Cholesky diagonal block: Rpotrf2('U') (Rpotrf2.cpp:86-131) in one CTA
// ---------------------------------------------------------------------------
// The recursion exactly as the reference runs it, since the upper factor's bits depend on
// how the work is grouped: a 1x1 block takes the square root (a <= 0, NaR included, stops
// with info); a larger one splits n1 = n/2, n2 = n - n1, factors A11, solves
// A12 <- U11^-T A12 (Rtrsm('L', 'U', 'T', 'N'), Rtrsm.cpp:160-173: per column, for each
// row i, t = b_i, t = t - u_ki*b_k over k < i in order, b_i = t / u_ii), updates
// A22 <- -(A12^T A12) + A22 on and above the diagonal (Rsyrk('U', 'T'), Rsyrk.cpp:182-195:
// each entry's dot product summed from zero in order, then alpha*t + beta*c) and factors
// A22.  The recursion runs on an explicit stack in shared memory; the solves are one
// thread per column, the update one thread per entry, with barriers in between.
constexpr int POTRF2_CTA_THREADS = 256;
constexpr int POTRF2_CTA_MAX = 128; // larger blocks recurse on the host with many-block kernels

__global__ void __launch_bounds__(POTRF2_CTA_THREADS) potrf2_upper_cta_kernel(uint32_t *__restrict__ A, size_t lda,
                                                                              int n, int row0, int *__restrict__ info)
{
    constexpr int DEPTH = 16;
    __shared__ int s_off[DEPTH], s_n[DEPTH], s_stage[DEPTH];
    __shared__ int s_sp, s_stop;
    if (*info != 0)
        return;
    const int tid = threadIdx.x;
    if (tid == 0) {
        s_sp = 1;
        s_off[0] = 0;
        s_n[0] = n;
        s_stage[0] = 0;
        s_stop = 0;
    }
    __syncthreads();
    for (;;) {
        const int sp = s_sp;
        if (sp == 0)
            break;
        const int off = s_off[sp - 1], nn = s_n[sp - 1], stage = s_stage[sp - 1];
        __syncthreads(); // the frame is read before thread 0 changes the stack
        if (nn == 1) {
            if (tid == 0) {
                uint32_t *d = A + off + (size_t)off * lda;
                const uint32_t a = *d;
                if ((int32_t)a <= 0) { // Rpotrf2.cpp:90-93 (NaR is below zero in posit order)
                    *info = row0 + off + 1;
                    s_stop = 1;
                } else {
                    *d = psqrt_est(a);
                }
                s_sp = sp - 1;
            }
        } else {
            const int n1 = nn / 2, n2 = nn - n1;
            uint32_t *a11 = A + off + (size_t)off * lda;
            uint32_t *a12 = A + off + (size_t)(off + n1) * lda;
            uint32_t *a22 = A + (off + n1) + (size_t)(off + n1) * lda;
            if (stage == 0) {
                if (tid == 0) {
                    s_stage[sp - 1] = 1;
                    s_off[sp] = off;
                    s_n[sp] = n1;
                    s_stage[sp] = 0;
                    s_sp = sp + 1;
                }
            } else if (stage == 1) {
                for (int j = tid; j < n2; j += POTRF2_CTA_THREADS) { // A12 <- U11^-T A12
                    uint32_t *b = a12 + (size_t)j * lda;
                    for (int i = 0; i < n1; ++i) {
                        const uint32_t *ui = a11 + (size_t)i * lda;
                        double t = p32_to_double(b[i]);
                        for (int k = 0; k < i; ++k)
                            t = f64_posit_mac_checked(t, -p32_to_double(b[k]), p32_to_double(ui[k]));
                        b[i] = pdiv_est(p32_from_double(t), ui[i]);
                    }
                }
                __syncthreads();
                const int cnt = n2 * (n2 + 1) / 2; // A22 <- -(A12^T A12) + A22, i <= j
                for (int e = tid; e < cnt; e += POTRF2_CTA_THREADS) {
                    int j = (int)((sqrtf(8.0f * (float)e + 1.0f) - 1.0f) * 0.5f); // e = j(j+1)/2 + i
                    while (j * (j + 1) / 2 > e)
                        --j;
                    while ((j + 1) * (j + 2) / 2 <= e)
                        ++j;
                    const int i = e - j * (j + 1) / 2;
                    const uint32_t *ci = a12 + (size_t)i * lda, *cj = a12 + (size_t)j * lda;
                    double t = 0.0;
                    for (int l = 0; l < n1; ++l)
                        t = f64_posit_mac_checked(t, p32_to_double(ci[l]), p32_to_double(cj[l]));
                    uint32_t *c = a22 + i + (size_t)j * lda;
                    *c = padd(pmul(0xC0000000u /* -1 */, p32_from_double(t)), pmul(P32_ONE, *c));
                }
                __syncthreads();
                if (tid == 0) {
                    s_stage[sp - 1] = 2;
                    s_off[sp] = off + n1;
                    s_n[sp] = n2;
                    s_stage[sp] = 0;
                    s_sp = sp + 1;
                }
            } else if (tid == 0) {
                s_sp = sp - 1;
            }
        }
        __syncthreads();
        if (s_stop)
            return;
    }
}

// ---------------------------------------------------------------------------
// Host orchestration
// ---------------------------------------------------------------------------
static int imin(int a, int b) { return a < b ? a : b; }
static int imax(int a, int b) { return a > b ? a : b; }

// Panel width for an n x n factorization when the caller passes nb <= 0: the widths the
// autotuner (posit_gpu_b200/autotune.py) measured fastest on B200, by size bucket.  LU and
// lower Cholesky give the same bits at every width.
int tuned_panel_width(bool lu, int n)
{
    struct Row {
        int n, lu, chol;
    };
    static const Row rows[] = {{0, 32, 32},    {512, 32, 32},  {1024, 32, 16},   {2048, 32, 32},
                               {4096, 32, 32}, {8192, 32, 32}, {16384, 128, 32}};
    int nb = 16;
    for (const Row &r : rows)
        if (n >= r.n)
            nb = lu ? r.lu : r.chol;
    return nb;
}

// The LU panel's form: the cluster panel held in shared memory when its rows fit (ncta CTAs,
// one per PANEL1_ROWS_PER_CTA rows up to 8, T threads each -- the CTA's rows rounded up to
// whole warps, at most 1024 -- R slots per thread), else the two-launch form (ncta = 0).
struct PanelForm {
    int ncta, R, T; // CTAs (0: the panel does not fit), slots per thread, threads per CTA
};
static PanelForm panel_form(int M, int jb)
{
    if (jb > PANEL1_MAX_JB)
        return {0, 0, 0};
    const int ncta = std::max(1, std::min(PANEL1_MAX_CTAS, (M + PANEL1_ROWS_PER_CTA - 1) / PANEL1_ROWS_PER_CTA));
    const int rpc = (M + ncta - 1) / ncta; // rows per CTA
    const int T = std::min(PANEL1_THREADS, (rpc + 31) / 32 * 32), R = (rpc + T - 1) / T;
    if (lu_panel_smem(R, T, jb, ncta) > PANEL1_SMEM || R > PANEL1_MAX_R)
        return {0, 0, 0};
    return {ncta, R, T};
}

// The columns of a block of jb that one panel launch takes: all, if they are at most 32 and fit in a
// cluster (tables, padding columns and pushed rows beside them leave room for 4864 rows of 32
// columns, 6144 of 24, 8192 of 16); else inner panels of 32, 24 or 16, the widest that fits, the
// block's columns updated between them; else all, in two launches per column.  A block's update of
// the rest of the matrix stays one of jb columns.
// Two launches per column cost 14 us a column, and one launch for all columns of a wide block gains
// less with each: 6144 x 32 0.47 ms in two launches a column (0.83 in the cluster of all 32 that fitted
// without the padding) and 0.15 by inner panels, 3072 x 64 0.82 (0.71) and 0.20, 1536 x 128 1.58 (1.46)
// and 0.39; LU n = 8192 197 -> 161 ms, n = 1024 with the caller's nb = 256 14.1 -> 4.5, with nb = 128 (one
// launch a panel) 5.5 -> 4.6.
static int panel_width(int M, int jb)
{
    if (panel_form(M, jb).ncta == 0)
        for (int w : {32, 24, 16})
            if (w < jb && panel_form(M, w).ncta > 0)
                return w;
    return jb;
}

size_t rgetrf_workspace_bytes(int m, int n, int nb)
{
    int mn = imin(m, n);
    if (nb < 1)
        nb = 1;
    int jb = imin(nb, mn);
    size_t g = mn > jb ? gemm_workspace_bytes(m - jb > 0 ? m - jb : 1, n - jb > 0 ? n - jb : 1, jb) : 0;
    if (jb > 16) // inner panels
        g = std::max(g, gemm_workspace_bytes(m, jb, PANEL1_MAX_JB));
    return panel_ws_bytes(m) + g;
}

template <class... Args>
static cudaError_t launch_panel_cluster(void (*kernel)(Args...), PanelForm f, size_t smem, cudaStream_t st,
                                        Args... args)
{
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PANEL1_SMEM);
    if (e != cudaSuccess)
        return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)f.ncta);
    cfg.blockDim = dim3((unsigned)f.T);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)f.ncta;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

static dim3 panel_grid(int M, int jb, int k)
{
    return dim3((unsigned)imax((M - k - 1 + PANEL_ROWS - 1) / PANEL_ROWS, 1),
                (unsigned)imax((jb - k - 1 + PANEL_CG - 1) / PANEL_CG, 1));
}

// Rgetrf.cpp:95-132 with the device kernels above.  `ws` holds the pivot record, the
// scratch column and the trailing GEMM's workspace.
cudaError_t rgetrf_launch(int m, int n, uint32_t *A, int lda, int *ipiv, int nb, int *info, void *ws,
                          cudaStream_t st)
{
    const int mn = imin(m, n);
    if (nb < 1)
        nb = 1;
    PivotInfo *pinfo = reinterpret_cast<PivotInfo *>(ws);
    uint32_t *lcol = reinterpret_cast<uint32_t *>(reinterpret_cast<unsigned char *>(ws) + 256);
    void *gws = reinterpret_cast<unsigned char *>(ws) + panel_ws_bytes(m);
    const size_t L = (size_t)lda;
    for (int j = 0; j < mn; j += nb) {
        const int jb = imin(mn - j, nb);
        const int M = m - j;
        uint32_t *P = A + j + (size_t)j * L;
        uint32_t *lc = lcol + j; // indexed by panel-local row
        const int w = panel_width(M, jb);
        for (int q = 0; q < jb; q += w) { // the block's inner panels (one, where w == jb)
            const int wj = imin(w, jb - q), rest = jb - q - wj;
            uint32_t *Pq = P + q + (size_t)q * L;
            const PanelForm pf = panel_form(M - q, wj);
            if (pf.ncta > 0) {
                cudaError_t e = launch_panel_cluster(pf.R > 1      ? lu_panel_cluster_kernel<PANEL1_THREADS, PANEL1_MAX_R>
                                                     : pf.T <= 128 ? lu_panel_cluster_kernel<128, 1>
                                                     : pf.T <= 512 ? lu_panel_cluster_kernel<512, 1>
                                                                   : lu_panel_cluster_kernel<PANEL1_THREADS, 1>,
                                                     pf, lu_panel_smem(pf.R, pf.T, wj, pf.ncta), st, Pq, L, M - q, wj,
                                                     pf.R, j + q, ipiv, info);
                if (e != cudaSuccess)
                    return e;
            } else { // (never an inner panel)
                lu_pivot_kernel<<<1, 1024, 0, st>>>(P, L, M, jb, 0, j, ipiv, info, pinfo, lc, -1);
                for (int k = 0; k < jb; ++k) {
                    lu_update_kernel<<<panel_grid(M, jb, k), PANEL_ROWS, 0, st>>>(P, L, M, jb, k, info, pinfo, lc);
                    lu_pivot_kernel<<<1, 1024, 0, st>>>(P, L, M, jb, k + 1, j, ipiv, info, pinfo, lc, k);
                }
            }
            if (wj == jb)
                break;
            lu_rows_kernel<<<(jb - wj + ROWS_THREADS / 32 - 1) / (ROWS_THREADS / 32), ROWS_THREADS, 0, st>>>(
                P, L, jb, q, wj, ipiv + j, j, false);
            if (rest > 0 && M - q > wj) {
                cudaError_t e = gemm_launch(true, true, M - q - wj, rest, wj, 0xC0000000u /* -1 */, Pq + wj, lda,
                                            Pq + (size_t)wj * L, lda, P32_ONE, Pq + wj + (size_t)wj * L, lda, gws, st, true);
                if (e != cudaSuccess)
                    return e;
            }
        }
        if (jb <= ROWS_JB_MAX) {
            if (n > jb)
                lu_rows_kernel<<<(n - jb + ROWS_THREADS / 32 - 1) / (ROWS_THREADS / 32), ROWS_THREADS, 0, st>>>(
                    A, L, n, j, jb, ipiv, 0, true);
        } else {
            if (j > 0)
                laswp_kernel<<<(j + 127) / 128, 128, 0, st>>>(A, L, j, j + 1, j + jb, ipiv, 1, info);
            if (j + jb < n) {
                const int nr = n - j - jb;
                laswp_kernel<<<(nr + 127) / 128, 128, 0, st>>>(A + (size_t)(j + jb) * L, L, nr, j + 1, j + jb, ipiv,
                                                              1, info);
                cudaError_t e = launch_col(false, true, nr, P, L, A + j + (size_t)(j + jb) * L, L, jb, info, st);
                if (e != cudaSuccess)
                    return e;
            }
        }
        if (j + jb < n) {
            const int nr = n - j - jb;
            uint32_t *A12 = A + j + (size_t)(j + jb) * L;
            cudaError_t e = cudaSuccess;
            if (j + jb < m) {
                e = gemm_launch(true, true, m - j - jb, nr, jb, 0xC0000000u /* -1 */,
                                            A + (j + jb) + (size_t)j * L, lda, A12, lda, P32_ONE,
                                            A + (j + jb) + (size_t)(j + jb) * L, lda, gws, st, true);
                if (e != cudaSuccess)
                    return e;
            }
        }
    }
    return cudaGetLastError();
}

size_t rpotrf_workspace_bytes(int n, int nb)
{
    const int jb = imin(imin(imax(nb, 1), CHOL_JB_MAX), n);
    return CHOL_BLOCKS_BYTES + (n > jb ? gemm_workspace_bytes(n - jb, n - jb, jb) : 0);
}

// Lower Cholesky (Rpotrf.cpp:124-142 / Rpotrf2.cpp:132-146 order, blocked right-looking).
cudaError_t rpotrf_lower_launch(int n, uint32_t *A, int lda, int nb, int *info, void *ws, cudaStream_t st)
{
    if (nb < 1)
        nb = 1;
    // The factor does not depend on the panel width, and wider panels in one launch per
    // column are slower at every size (n = 1024: 2.5 ms at 32, 11 at 48).
    nb = imin(nb, CHOL_JB_MAX);
    uint32_t *blocks = reinterpret_cast<uint32_t *>(ws);
    void *gws = reinterpret_cast<unsigned char *>(ws) + CHOL_BLOCKS_BYTES;
    const size_t L = (size_t)lda;
    for (int j = 0; j < n; j += nb) {
        const int jb = imin(n - j, nb);
        const int M = n - j;
        uint32_t *P = A + j + (size_t)j * L;
        const bool last = j + jb >= n, first = j == 0;
        cudaError_t e = cudaFuncSetAttribute(chol_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)chol_panel_smem(CHOL_JB_MAX));
        if (e != cudaSuccess)
            return e;
        const int turn = j / nb & 1;
        chol_panel_kernel<<<imax(1, (M - jb + CHOL_T - 1) / CHOL_T), CHOL_T, chol_panel_smem(jb), st>>>(
            P, L, M, jb, j, info, last ? nullptr : blocks + turn * CHOL_JB_MAX * CHOL_JB_MAX,
            first ? nullptr : P - (size_t)nb * (L + 1), first ? 0 : nb,
            blocks + (turn ^ 1) * CHOL_JB_MAX * CHOL_JB_MAX);
        if (j + jb < n) {
            const int nr = n - j - jb;
            const uint32_t *L21 = A + (j + jb) + (size_t)j * L;
            e = gemm_launch_tri(TRI_LOWER, true, false, nr, nr, jb, 0xC0000000u /* -1 */, L21, lda, L21,
                                              lda, P32_ONE, A + (j + jb) + (size_t)(j + jb) * L, lda, gws, st, info);
            if (e != cudaSuccess)
                return e;
        }
    }
    return cudaGetLastError();
}

// Upper Cholesky (Rpotrf.cpp:96-118): left-looking and blocked by nb in the reference's
// order, which the upper factor's bits depend on.  For each block column j: the diagonal
// block's update by the rows above it (Rsyrk('U', 'T'): the TN GEMM on its upper
// triangle), its factorization (Rpotrf2('U'), recursive), the block row's update (Rgemm
// 'T', 'N') and solve (Rtrsm('L', 'U', 'T', 'N')).  nb <= 1 or nb >= n is Rpotrf2 on the
// whole matrix (Rpotrf.cpp:86-91).  Kernels after a failed diagonal do nothing.
static cudaError_t launch_ltx(bool upper, bool unit, int n, int nrhs, const uint32_t *A, int lda, uint32_t *B,
                              int ldb, const int *info, cudaStream_t st);

static void potrf2_upper_plan(int n, size_t *ws)
{
    if (n <= POTRF2_CTA_MAX)
        return;
    const int n1 = n / 2, n2 = n - n1;
    potrf2_upper_plan(n1, ws);
    *ws = std::max(*ws, gemm_workspace_bytes(n2, n2, n1));
    potrf2_upper_plan(n2, ws);
}

size_t rpotrf_upper_workspace_bytes(int n, int nb)
{
    size_t ws = 0;
    if (nb <= 1 || nb >= n) {
        potrf2_upper_plan(n, &ws);
        return ws;
    }
    for (int j = 0; j < n; j += nb) {
        const int jb = imin(nb, n - j);
        if (j > 0) {
            ws = std::max(ws, gemm_workspace_bytes(jb, jb, j));
            if (j + jb < n)
                ws = std::max(ws, gemm_workspace_bytes(jb, n - j - jb, j));
        }
        potrf2_upper_plan(jb, &ws);
    }
    return ws;
}

static cudaError_t potrf2_upper(uint32_t *A, int lda, int off, int n, int *info, void *ws, cudaStream_t st)
{
    const size_t L = (size_t)lda;
    if (n <= POTRF2_CTA_MAX) {
        potrf2_upper_cta_kernel<<<1, POTRF2_CTA_THREADS, 0, st>>>(A + off + (size_t)off * L, L, n, off, info);
        return cudaGetLastError();
    }
    const int n1 = n / 2, n2 = n - n1;
    cudaError_t e = potrf2_upper(A, lda, off, n1, info, ws, st);
    if (e == cudaSuccess)
        e = launch_ltx(true, false, n1, n2, A + off + (size_t)off * L, lda, A + off + (size_t)(off + n1) * L, lda,
                       info, st);
    if (e == cudaSuccess)
        e = gemm_launch_tri(TRI_UPPER, false, true, n2, n2, n1, 0xC0000000u /* -1 */,
                            A + off + (size_t)(off + n1) * L, lda, A + off + (size_t)(off + n1) * L, lda, P32_ONE,
                            A + (off + n1) + (size_t)(off + n1) * L, lda, ws, st, info);
    if (e == cudaSuccess)
        e = potrf2_upper(A, lda, off + n1, n2, info, ws, st);
    return e;
}

cudaError_t rpotrf_upper_launch(int n, uint32_t *A, int lda, int nb, int *info, void *ws, cudaStream_t st)
{
    if (nb <= 1 || nb >= n)
        return potrf2_upper(A, lda, 0, n, info, ws, st);
    const size_t L = (size_t)lda;
    for (int j = 0; j < n; j += nb) {
        const int jb = imin(nb, n - j);
        cudaError_t e = cudaSuccess;
        if (j > 0) // Rsyrk('U', 'T', jb, j, -1, A(0:j, j:j+jb), 1, A(j:j+jb, j:j+jb))
            e = gemm_launch_tri(TRI_UPPER, false, true, jb, jb, j, 0xC0000000u /* -1 */, A + (size_t)j * L, lda,
                                A + (size_t)j * L, lda, P32_ONE, A + j + (size_t)j * L, lda, ws, st, info);
        if (e == cudaSuccess)
            e = potrf2_upper(A, lda, j, jb, info, ws, st);
        if (e == cudaSuccess && j + jb < n) {
            const int nr = n - j - jb;
            if (j > 0) // Rgemm('T', 'N', jb, nr, j, -1, A(0:j, j:j+jb), A(0:j, j+jb:n), 1, A(j:j+jb, j+jb:n))
                e = gemm_launch_tri(TRI_FULL, false, true, jb, nr, j, 0xC0000000u /* -1 */, A + (size_t)j * L, lda,
                                    A + (size_t)(j + jb) * L, lda, P32_ONE, A + j + (size_t)(j + jb) * L, lda, ws, st,
                                    info);
            if (e == cudaSuccess) // Rtrsm('L', 'U', 'T', 'N', jb, nr, 1, A(j:j+jb, j:j+jb), A(j:j+jb, j+jb:n))
                e = launch_ltx(true, false, jb, nr, A + j + (size_t)j * L, lda, A + j + (size_t)(j + jb) * L, lda,
                               info, st);
        }
        if (e != cudaSuccess)
            return e;
    }
    return cudaGetLastError();
}

// Rgetrs.cpp:84-114 (trans = 'N'): interchanges, L (unit) forward, U backward.
cudaError_t rgetrs_launch(int n, int nrhs, const uint32_t *A, int lda, const int *ipiv, uint32_t *B, int ldb,
                          cudaStream_t st)
{
    cudaError_t e = launch_laswp_rhs(B, ldb, nrhs, n, ipiv, true, st);
    if (e == cudaSuccess)
        e = launch_col(false, true, nrhs, A, lda, B, ldb, n, nullptr, st);
    if (e == cudaSuccess)
        e = launch_col(true, false, nrhs, A, lda, B, ldb, n, nullptr, st);
    return e;
}

// The dot-form solves with the triangle transposed: L^-T B (Rtrsm('L', 'L', 'T'),
// Rtrsm.cpp:175-186) or, with `upper`, U^-T B (Rtrsm('L', 'U', 'T'), Rtrsm.cpp:160-173).
// One block per right-hand side: trsm_ltx_kernel where its terms fit in shared memory
// (FP64 where 26n bytes do, five bytes each where 10n do, n <= 23,232), else one thread's chain.
// A nonzero *info (when given) turns the solve into a no-op.
static cudaError_t launch_ltx(bool upper, bool unit, int n, int nrhs, const uint32_t *A, int lda, uint32_t *B,
                              int ldb, const int *info, cudaStream_t st)
{
    cudaError_t e = cudaSuccess;
    const size_t b64 = ltx_smem_bytes<ChainTerms64, LtxCol64>(n), b40 = ltx_smem_bytes<ChainTerms40, LtxColGlobal>(n);
    if (b64 <= (size_t)LLT_SMEM_MAX || b40 <= (size_t)LLT_SMEM_MAX) {
        const bool f64 = b64 <= (size_t)LLT_SMEM_MAX;
        const size_t bytes = f64 ? b64 : b40;
        auto *fn = f64 ? (upper ? trsm_ltx_kernel<ChainTerms64, LtxCol64, true>
                                : trsm_ltx_kernel<ChainTerms64, LtxCol64, false>)
                       : (upper ? trsm_ltx_kernel<ChainTerms40, LtxColGlobal, true>
                                : trsm_ltx_kernel<ChainTerms40, LtxColGlobal, false>);
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, LLT_SMEM_MAX);
        if (e != cudaSuccess)
            return e;
        fn<<<nrhs, LTX_THREADS, bytes, st>>>(A, lda, B, ldb, n, unit, info);
        return cudaGetLastError();
    }
    const size_t col = (size_t)n * 4;
    const bool staged = col <= (size_t)LLT_SMEM_MAX;
    if (staged && col > 48 * 1024) {
        e = cudaFuncSetAttribute(trsm_llt_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LLT_SMEM_MAX);
        if (e != cudaSuccess)
            return e;
    }
    trsm_llt_kernel<<<nrhs, 32, staged ? col : 0, st>>>(A, lda, B, ldb, n, staged, unit, upper, info);
    return cudaGetLastError();
}

// Rpotrs.cpp:95-106 (uplo = 'L'): L forward, L^T backward.
cudaError_t rpotrs_lower_launch(int n, int nrhs, const uint32_t *A, int lda, uint32_t *B, int ldb, cudaStream_t st)
{
    cudaError_t e = launch_col(false, false, nrhs, A, lda, B, ldb, n, nullptr, st);
    if (e != cudaSuccess)
        return e;
    return launch_ltx(false, false, n, nrhs, A, lda, B, ldb, nullptr, st);
}

// Rpotrs.cpp:84-95 (uplo = 'U'): U^T forward (Rtrsm('L', 'U', 'T', 'N')), then U backward
// (Rtrsm('L', 'U', 'N', 'N')).
cudaError_t rpotrs_upper_launch(int n, int nrhs, const uint32_t *A, int lda, uint32_t *B, int ldb, cudaStream_t st)
{
    cudaError_t e = launch_ltx(true, false, n, nrhs, A, lda, B, ldb, nullptr, st);
    if (e != cudaSuccess)
        return e;
    return launch_col(true, false, nrhs, A, lda, B, ldb, n, nullptr, st);
}

// Rgetrs.cpp:99-113 (trans = 'T' or 'C'): U^T forward (non-unit), L^T backward (unit),
// then the interchanges applied in reverse order (Rlaswp with incx = -1).
cudaError_t rgetrs_trans_launch(int n, int nrhs, const uint32_t *A, int lda, const int *ipiv, uint32_t *B, int ldb,
                                cudaStream_t st)
{
    cudaError_t e = launch_ltx(true, false, n, nrhs, A, lda, B, ldb, nullptr, st);
    if (e != cudaSuccess)
        return e;
    e = launch_ltx(false, true, n, nrhs, A, lda, B, ldb, nullptr, st);
    if (e != cudaSuccess)
        return e;
    return launch_laswp_rhs(B, ldb, nrhs, n, ipiv, false, st);
}

} // namespace pg
