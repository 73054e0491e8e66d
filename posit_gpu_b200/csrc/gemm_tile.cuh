// gemm_tile.cuh -- device pieces shared by the GEMM kernels (gemm.cu, batch_gemm.cu): the
// rounding-constant tables, thread ownership inside a tile, the k-step loop and the tile
// that converts its operands on the fly.
//
// What bounds the k-step.  A multiply-add is 6 FP64 instructions, two table look-ups
// (shift, mask, shared load) and at most one move.  On B200 an FP64 warp instruction takes
// two issue slots of its sub-partition and every other instruction one (measured: the time
// per multiply-add is 2 F + O cycles for F FP64 and O other instructions, within 3 %, in
// five variants), so a warp's multiply-add costs about 12 + 7.5 cycles, and what is not one
// of these instructions costs speed:
//   * the exactness test of the sum is not needed (posit32.cuh, f64_posit_mac): 4 FP64
//     instructions less;
//   * no step is tested on its own: a product or sum outside the fast window becomes NaN
//     and stays NaN, so the accumulators are looked at once per k tile, and a tile that
//     met one is done again from the accumulators' values at its start;
//   * look-ups mask the sign off: with both signs in the table, lanes whose values differ
//     in sign alone hit one bank (3320 against 1986 Gop/s in the isolated loop);
//   * the product's constants are 8-byte entries (one load gives the register pair), the
//     sum's 4-byte ones (half the bank cycles, one move for the zero low word): 3950 against
//     3700 (both 8-byte: shared-memory bandwidth) and 3850 Gop/s (both 4-byte);
//   * 4x4 outputs per thread and an unrolled k loop (4x2: 3800).
// ncu on the main kernel (4096^3 NN): 14.02 instructions per multiply-add (before: 22.4), 6.03 of
// them FP64, issue 71.7 % and the second FP64 slots 31 %: full.  8192^3 NN,
// the whole call: 470 -> 289 ms.  Wide-range data (10^U(-20,20), 2048^3, nearly every sum
// outside the fast window): 206 -> 20 ms, with g_outside_table (61 ms with the integer
// rounding on every such step).
#pragma once
#include "posit32.cuh"

namespace pg {

// Operand tiles are made of blocks of 32 rows (columns of B) by BK steps, [l][32] FP64.
constexpr int BLK = 32;
constexpr int BK = 16; // k-depth of one staged tile

// Thread (tx, ty) owns rows {2tx, 2tx+1} of each 32-row block and the same pattern of
// columns with ty: the 16-byte shared-memory loads of a warp then hit distinct banks.
__device__ __forceinline__ int own_off(int t, int q) { return (q >> 1) * BLK + 2 * t + (q & 1); }

// Rounding constants by exponent field (f64_round_const_top), in shared memory.
constexpr int STEP_TAB_P_BYTES = F64_CONST_ENTRIES * 8; // the product's, as FP64 values
constexpr int STEP_TAB_S_BYTES = F64_CONST_ENTRIES * 4; // the sum's, high words only
constexpr int STEP_TAB_BYTES = STEP_TAB_P_BYTES + STEP_TAB_S_BYTES;

__device__ __forceinline__ void step_tables_fill(unsigned char *tab, int tid, int nthreads)
{
    for (int i = tid; i < F64_CONST_ENTRIES; i += nthreads) {
        const uint32_t h = f64_round_const_top((uint32_t)i);
        reinterpret_cast<double *>(tab)[i] = f64_from_hi(h);
        reinterpret_cast<uint32_t *>(tab + STEP_TAB_P_BYTES)[i] = h;
    }
}

// c + t*a as f64_posit_mac, its constants from the tables; NaN where that one is flagged.
__device__ __forceinline__ double step_one(double c, double t, double a, const unsigned char *tab)
{
    const uint32_t hp = f64_hi(f64_mul(t, a));
    const double Cp = *reinterpret_cast<const double *>(tab + ((hp >> 17) & 0x3FF8));
    const double q = f64_add(f64_fma(t, a, Cp), -Cp);
    const double s = f64_add(c, q);
    const double Cs =
        f64_from_hi(*reinterpret_cast<const uint32_t *>(tab + STEP_TAB_P_BYTES + ((f64_hi(s) >> 18) & 0x1FFC)));
    return f64_add(f64_add(s, Cs), -Cs);
}

// f64_round_outside as a table, for the tiles where such steps are common (wide-range data:
// nearly every sum): per binade two results and the fraction from which the larger one is
// taken.  Entry 0 stands for all binades below -120, then -120 .. -109, 108 .. 119, and the
// last one for all from 120.  In global memory, read on the slow path only (L1-resident).
struct OutsideEntry {
    uint64_t thr;          // |x|'s bits from which it rounds up
    uint32_t dn_hi, up_hi; // high words of the two powers of two
};
struct OutsideTable {
    static constexpr int NEG = 13, N = 26;
    OutsideEntry e[N];
    constexpr OutsideTable() : e{}
    {
        for (int i = 0; i < N; ++i) {
            const int32_t ex = i < NEG ? i - 121 : i - NEG + 108;
            const uint64_t cand[4] = {0, 1, (uint64_t)1 << 51, ((uint64_t)1 << 51) + 1}; // where the rounding may turn
            const int32_t dn = outside_exponent(ex, 0), up = outside_exponent(ex, 0xFFFFFFFFFFFFFull);
            uint64_t thr = 0;
            for (int q = 3; q >= 0; --q)
                if (outside_exponent(ex, cand[q]) == up)
                    thr = cand[q];
            e[i].thr = ((uint64_t)(uint32_t)(ex + 1023) << 52) + thr;
            e[i].dn_hi = (uint32_t)(dn + 1023) << 20;
            e[i].up_hi = (uint32_t)(up + 1023) << 20;
        }
    }
};
static __device__ const OutsideTable g_outside_table;

// x rounded as f64_round_outside, by the table.  NANS: x may be NaN, and stays it.
template <bool NANS>
__device__ __forceinline__ double round_outside_tab(double x)
{
    if (NANS && x != x)
        return x;
    const uint64_t b = f64_bits(x) & 0x7FFFFFFFFFFFFFFFull;
    const int ex = (int)(b >> 52) - 1023;
    const int i = ex < 0 ? max(ex + 121, 0) : min(ex - 108 + OutsideTable::NEG, OutsideTable::N - 1);
    const OutsideEntry e = g_outside_table.e[i];
    return f64_from_hi((b >= e.thr ? e.up_hi : e.dn_hi) | (f64_hi(x) & 0x80000000u));
}

// The same step for any operands (f64_posit_mac_exact with its tables); `out` is set when the
// product or the sum was outside the fast window.
template <bool NANS>
__device__ __forceinline__ double step_any(double c, double t, double a, const unsigned char *tab, bool &out)
{
    const double p = f64_mul(t, a);
    const double Cp = *reinterpret_cast<const double *>(tab + ((f64_hi(p) >> 17) & 0x3FF8));
    double q = f64_add(f64_fma(t, a, Cp), -Cp);
    if (q != q) {
        q = round_outside_tab<NANS>(p);
        out = true;
    }
    const double s = f64_add(c, q);
    const double Cs =
        f64_from_hi(*reinterpret_cast<const uint32_t *>(tab + STEP_TAB_P_BYTES + ((f64_hi(s) >> 18) & 0x1FFC)));
    double r = f64_add(f64_add(s, Cs), -Cs);
    if (r != r) {
        r = round_outside_tab<NANS>(s);
        out = true;
    }
    return r;
}

// Where a tile's operands lie in shared memory: as = [TM_/2 blocks][step][32], ts likewise.
template <int LD> // a block's steps LD doubles apart, its blocks after one another
struct BlockedOps {
    static constexpr bool NEG = false;  // t is taken negated
    static constexpr bool NANS = false; // operands and accumulators may be NaN (NaR)
    __device__ __forceinline__ int a(int q, int l) const { return q * BK * LD + l * LD; }
    __device__ __forceinline__ int t(int q, int l) const { return q * BK * LD + l * LD; }
};

// The operands of step l.
template <int TM_, int TN_, class Ops>
__device__ __forceinline__ void load_operands(const double *as, const double *ts, int l, int tx, int ty, Ops ops,
                                              double (&a)[TM_], double (&t)[TN_])
{
#pragma unroll
    for (int q = 0; q < TM_ / 2; ++q) {
        const double2 v = *reinterpret_cast<const double2 *>(as + ops.a(q, l) + 2 * tx);
        a[2 * q] = v.x;
        a[2 * q + 1] = v.y;
    }
#pragma unroll
    for (int q = 0; q < TN_ / 2; ++q) {
        const double2 v = *reinterpret_cast<const double2 *>(ts + ops.t(q, l) + 2 * ty);
        t[2 * q] = Ops::NEG ? -v.x : v.x;
        t[2 * q + 1] = Ops::NEG ? -v.y : v.y;
    }
}

template <int TM_, int TN_, class Ops>
__device__ __forceinline__ void step_fast(double (&acc)[TM_][TN_], const double *as, const double *ts, int l,
                                          const unsigned char *tab, int tx, int ty, Ops ops)
{
    double a[TM_], t[TN_];
    load_operands<TM_, TN_>(as, ts, l, tx, ty, ops, a, t);
#pragma unroll
    for (int i = 0; i < TM_; ++i)
#pragma unroll
        for (int j = 0; j < TN_; ++j)
            acc[i][j] = step_one(acc[i][j], t[j], a[i], tab);
}

// The k-steps of a tile: one p32_mul and one p32_add per k and accumulator, in k order; the
// accumulators and operands are posit32 values held in FP64 (no NaR unless Ops::NANS: the
// callers carry it in flags).  `steps` is a multiple of UNR_; steps past k have t = 0, which leaves c as it
// is.  `slow` is the warp's state: after a tile with a step outside the fast window the next
// one is done step by step with a test, until a tile has none (data of a wide dynamic range
// has such steps everywhere, and doing those tiles twice would not pay).
template <int UNR_, int TM_, int TN_, class Ops>
__device__ __forceinline__ void tile_steps(double (&acc)[TM_][TN_], const double *as, const double *ts, int steps,
                                           const unsigned char *tab, int tx, int ty, Ops ops, bool &slow)
{
    constexpr unsigned FULL = 0xFFFFFFFFu;
    if (!slow) {
        double save[TM_][TN_];
#pragma unroll
        for (int i = 0; i < TM_; ++i)
#pragma unroll
            for (int j = 0; j < TN_; ++j)
                save[i][j] = acc[i][j];
#pragma unroll 1
        for (int l0 = 0; l0 < steps; l0 += UNR_) {
#pragma unroll
            for (int l = 0; l < UNR_; ++l)
                step_fast<TM_, TN_>(acc, as, ts, l0 + l, tab, tx, ty, ops);
        }
        bool any = false;
#pragma unroll
        for (int i = 0; i < TM_; ++i)
#pragma unroll
            for (int j = 0; j < TN_; ++j)
                any |= acc[i][j] != acc[i][j];
        if (!__any_sync(FULL, any))
            return;
        slow = true;
#pragma unroll
        for (int i = 0; i < TM_; ++i)
#pragma unroll
            for (int j = 0; j < TN_; ++j)
                acc[i][j] = save[i][j];
    }
    bool any = false;
#pragma unroll 1
    for (int l = 0; l < steps; ++l) {
        double a[TM_], t[TN_];
        load_operands<TM_, TN_>(as, ts, l, tx, ty, ops, a, t);
#pragma unroll
        for (int i = 0; i < TM_; ++i)
#pragma unroll
            for (int j = 0; j < TN_; ++j)
                acc[i][j] = step_any<Ops::NANS>(acc[i][j], t[j], a[i], tab, any);
    }
    slow = __any_sync(FULL, any);
}

// The number of steps run for the k left in a tile.
template <int UNR_>
__device__ __forceinline__ int tile_step_count(int left)
{
    return (min(BK, left) + UNR_ - 1) / UNR_ * UNR_;
}

// c + t*a and x*y rounded, for any operands: the fast step first, its rare exceptions after
// it in little code (the panel kernels run a few iterations of long loops: code that does
// not fit the instruction cache costs them more than it computes).
__device__ __forceinline__ double mac_any(double c, double t, double a, const unsigned char *tab)
{
    double r = step_one(c, t, a, tab);
    if (r != r) {
        bool out;
        r = step_any<true>(c, t, a, tab, out);
    }
    return r;
}
__device__ __forceinline__ double mul_any(double x, double y, const unsigned char *tab)
{
    const double p = f64_mul(x, y);
    const double C = *reinterpret_cast<const double *>(tab + ((f64_hi(p) >> 17) & 0x3FF8));
    const double q = f64_add(f64_fma(x, y, C), -C);
    return q == q ? q : round_outside_tab<true>(p);
}

// alpha*b_lj as the NN/NT order rounds it (Rgemm.cpp:180, 222), b in FP64; NaN for NaR.
__device__ __forceinline__ double scale_operand(double b, uint32_t alpha)
{
    if (alpha == P32_ONE)
        return b;
    if (alpha == 0u - P32_ONE)
        return -b;
    return f64_posit_mul_checked(p32_to_double(alpha), b, F64ConstComputed{});
}

// ---------------------------------------------------------------------------
// A tile of one GEMM that reads its operands as patterns and converts them itself.
// ---------------------------------------------------------------------------
struct TileArgs {
    bool nota, notb;
    int m, n, k;
    uint32_t alpha, beta;
    const uint32_t *A;
    size_t lda;
    const uint32_t *B;
    size_t ldb;
    uint32_t *C;
    size_t ldc;
};

constexpr int TILE_THREADS = 256;
// Doubles per step of a block in shared memory: two more than 32, so that a warp storing a
// transposed operand (lanes along k) spreads over the banks.
constexpr int TILE_LD = BLK + 2;
__host__ __device__ constexpr size_t tile_buffer_bytes(int TM_, int TN_)
{
    return 2 * (size_t)(TM_ / 2 + TN_ / 2) * BK * TILE_LD * sizeof(double);
}
// Shared memory of a kernel running tiles of up to TM_ x TN_: tables, two operand buffers,
// a NaR flag per row and column.
__host__ __device__ constexpr size_t tile_smem_bytes(int TM_, int TN_)
{
    return STEP_TAB_BYTES + tile_buffer_bytes(TM_, TN_) + (size_t)(16 * TM_ + 16 * TN_);
}

// Which entries of C are written (gemm_launch_tri).
constexpr int TRI_FULL = 0;
constexpr int TRI_LOWER = 1; // row >= column
constexpr int TRI_UPPER = 2; // row <= column

// One operand's raw patterns of k tile kt: X(r, kk) for the tile's rows r0.. (TQ_ * 16 of
// them) into `raw`, each thread TQ_ elements, along the contiguous direction of X.  Rows
// outside the matrix are 1 (their lanes stay on the fast path, their results are not
// stored), steps past k are 0.
template <int TQ_>
__device__ __forceinline__ void tile_load(uint32_t (&raw)[TQ_], const uint32_t *X, size_t ld, bool rows_contiguous,
                                          int r0, int rows, int k0, int k)
{
#pragma unroll
    for (int q = 0; q < TQ_; ++q) {
        const int e = threadIdx.x + q * TILE_THREADS;
        const int i = rows_contiguous ? e % (16 * TQ_) : e / BK, l = rows_contiguous ? e / (16 * TQ_) : e % BK;
        const int r = r0 + i, kk = k0 + l;
        raw[q] = kk < k ? P32_ONE : 0u;
        if (r < rows && kk < k)
            raw[q] = rows_contiguous ? X[(size_t)r + (size_t)kk * ld] : X[(size_t)kk + (size_t)r * ld];
    }
}

// Those patterns as FP64 into a shared buffer [TQ_/2][16][TILE_LD], times alpha where the
// order scales B first; NaR goes to the row's flag and is replaced by 1.
template <int TQ_>
__device__ __forceinline__ void tile_store(const uint32_t (&raw)[TQ_], double *dst, bool rows_contiguous, bool scale,
                                           uint32_t alpha, unsigned char *nar)
{
#pragma unroll
    for (int q = 0; q < TQ_; ++q) {
        const int e = threadIdx.x + q * TILE_THREADS;
        const int i = rows_contiguous ? e % (16 * TQ_) : e / BK, l = rows_contiguous ? e / (16 * TQ_) : e % BK;
        double v = p32_to_double(raw[q]);
        if (scale)
            v = scale_operand(v, alpha);
        if (v != v) {
            nar[i] = 1;
            v = 1.0;
        }
        dst[(i / BLK) * BK * TILE_LD + l * TILE_LD + i % BLK] = v;
    }
}

// The entries of C a tile starts from, as patterns: 1.0 outside the matrix and where C is not
// read.  Loaded ahead of everything else a CTA does; tile_start converts them.
template <int TM_, int TN_>
__device__ __forceinline__ void tile_load_c(bool reads_c, uint32_t (&u)[TM_][TN_], int row0, int col0, int m, int n,
                                            const uint32_t *C, size_t ldc, int tx, int ty)
{
#pragma unroll
    for (int i = 0; i < TM_; ++i)
#pragma unroll
        for (int j = 0; j < TN_; ++j) {
            const int row = row0 + own_off(tx, i), col = col0 + own_off(ty, j);
            u[i][j] = reads_c && row < m && col < n ? C[(size_t)row + (size_t)col * ldc] : P32_ONE;
        }
}

// The start values of a tile's accumulators: NN/NT beta*C (Rgemm.cpp:169-177, 211-219; with
// beta == 0, C is not read), TN/TT zero.  A NaR start value is remembered in nar_bits (the
// output stays NaR whatever follows) and replaced by 1.0.
template <int TM_, int TN_>
__device__ __forceinline__ void tile_start(bool dot, double (&acc)[TM_][TN_], uint32_t &nar_bits, uint32_t beta,
                                           const uint32_t (&c)[TM_][TN_])
{
    nar_bits = 0;
#pragma unroll
    for (int i = 0; i < TM_; ++i) {
#pragma unroll
        for (int j = 0; j < TN_; ++j) {
            uint32_t u = 0;
            if (!dot && beta != 0) {
                u = c[i][j];
                if (beta != P32_ONE)
                    u = pmul(beta, u);
                if (u == P32_NAR) {
                    nar_bits |= 1u << (i * TN_ + j);
                    u = P32_ONE;
                }
            }
            acc[i][j] = p32_to_double(u);
        }
    }
}

// The results of a tile into C; `nar(i, j)` tells whether row i or column j of the tile met
// a NaR operand.
template <int TRI, int TM_, int TN_, class Nar>
__device__ __forceinline__ void tile_finish(bool dot, const double (&acc)[TM_][TN_], uint32_t nar_bits,
                                            int row0, int col0, int m, int n, uint32_t alpha, uint32_t beta,
                                            uint32_t *C, size_t ldc, int tx, int ty, Nar nar_of)
{
#pragma unroll
    for (int i = 0; i < TM_; ++i) {
#pragma unroll
        for (int j = 0; j < TN_; ++j) {
            const int li = own_off(tx, i), lj = own_off(ty, j);
            const int row = row0 + li, col = col0 + lj;
            if (row < m && col < n && (TRI != TRI_LOWER || row >= col) && (TRI != TRI_UPPER || row <= col)) {
                uint32_t *cp = C + (size_t)row + (size_t)col * ldc;
                const bool nar = ((nar_bits >> (i * TN_ + j)) & 1u) || nar_of(li, lj);
                uint32_t v = nar ? P32_NAR : p32_from_double_exact(acc[i][j]);
                if (dot) { // Rgemm.cpp:197-201
                    const uint32_t at = pmul(alpha, v);
                    v = (beta == 0) ? at : padd(at, pmul(beta, *cp));
                }
                *cp = v;
            }
        }
    }
}

// Tile (mt, nt) of the product, 16*TM_ x 16*TN_ outputs, by 256 threads.  `smem` is laid out
// as tile_smem_bytes, its tables filled (FILL: here, while the first loads are in flight).  The
// next k tile's patterns are loaded while the
// current one is multiplied, converted into the other buffer: one barrier per k tile.
template <int TRI, int TM_, int TN_, bool FILL>
__device__ __forceinline__ void fused_tile(const TileArgs &P, int mt, int nt, unsigned char *smem)
{
    constexpr int BM_ = 16 * TM_, BN_ = 16 * TN_;
    constexpr int ABUF = (TM_ / 2) * BK * TILE_LD, BUF = (TM_ / 2 + TN_ / 2) * BK * TILE_LD;
    const unsigned char *tab = smem;
    double *buf = reinterpret_cast<double *>(smem + STEP_TAB_BYTES);
    unsigned char *rnar = smem + STEP_TAB_BYTES + tile_buffer_bytes(TM_, TN_), *cnar = rnar + BM_;
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    const int row0 = mt * BM_, col0 = nt * BN_;
    const bool dot = !P.nota; // TN / TT use the dot-then-combine order
    constexpr int UNR = 4;    // the batched kernel holds three tile shapes' loops: code that fits the I-cache
    uint32_t ra[TM_], rb[TN_];
    tile_load<TM_>(ra, P.A, P.lda, P.nota, row0, P.m, 0, P.k);
    tile_load<TN_>(rb, P.B, P.ldb, !P.notb, col0, P.n, 0, P.k);
    double acc[TM_][TN_];
    uint32_t nar_bits, cu[TM_][TN_];
    tile_load_c<TM_, TN_>(!dot && P.beta != 0, cu, row0, col0, P.m, P.n, P.C, P.ldc, tx, ty);
    for (int i = tid; i < BM_ + BN_; i += TILE_THREADS)
        rnar[i] = 0;
    if (FILL)
        step_tables_fill(smem, tid, TILE_THREADS);
    tile_start<TM_, TN_>(dot, acc, nar_bits, P.beta, cu);
    __syncthreads(); // the flags are clear, the tables filled
    bool slow = false;
    const int KT = (P.k + BK - 1) / BK;
#pragma unroll 1
    for (int kt = 0; kt < KT; ++kt) {
        double *b = buf + (kt & 1) * BUF;
        tile_store<TM_>(ra, b, P.nota, false, 0u, rnar);
        tile_store<TN_>(rb, b + ABUF, !P.notb, !dot, P.alpha, cnar);
        if (kt + 1 < KT) {
            tile_load<TM_>(ra, P.A, P.lda, P.nota, row0, P.m, (kt + 1) * BK, P.k);
            tile_load<TN_>(rb, P.B, P.ldb, !P.notb, col0, P.n, (kt + 1) * BK, P.k);
        }
        __syncthreads(); // this buffer is full; every thread is done with the other one
        tile_steps<UNR>(acc, b, b + ABUF, tile_step_count<UNR>(P.k - kt * BK), tab, tx, ty, BlockedOps<TILE_LD>{}, slow);
    }
    tile_finish<TRI, TM_, TN_>(dot, acc, nar_bits, row0, col0, P.m, P.n, P.alpha, P.beta, P.C, P.ldc, tx, ty,
                               [&](int i, int j) { return (rnar[i] | cnar[j]) != 0; });
}

} // namespace pg
