// trsm_chain.cuh -- the transposed lower triangular solve of Rpotrs: chains of dependent
// posit additions.
//
// Rtrsm('L', 'L', 'T', 'N'), Rtrsm.cpp:175-186: for i = m-1 down to 0,
//     t = b_i;  t = t - a_ki * b_k  for k = i+1 .. m-1 (ascending);  b_i = t / a_ii.
// Each b_i's sum starts from the b_{i+1} just finished, so one right-hand side is a single
// chain of m(m-1)/2 dependent multiply-subtracts with two roundings each.  Three forms:
//   * llt_chain: one thread runs a right-hand side's whole chain with the accumulator
//     held in the decoded integer form (very long columns);
//   * warp_chain (end of this file): a warp sums a row's additions with the running value
//     biased onto its binade's grid, one FP64 addition per step, and where the value is calm
//     as a parallel prefix of step maps (lapack.cu's transposed-solve kernel and the
//     batched kernels);
//   * the forms it grew from, for the host: chain_add_run and chain_add_run_reg (one thread's
//     chain, its products computed elsewhere) and the scan with one map per addend (SegFn).
//     No kernel runs them; the CPU tests do.
//
// For the one-thread chains latency is everything.  Only the addition depends on the previous step: loads,
// decoding and the product of step k+1 can overlap the addition of step k, but not across
// a branch (a GPU issues in order and does not run past an unresolved branch).  So the
// steps run in blocks of CHAIN_BLOCK without a branch: the fast path's failure flags are
// OR-ed over the block and tested once at its end; in the rare block that has one, the
// block is replayed from its start value one exactly checked step at a time.  The next
// block's operands are loaded (clamped to stay in bounds) while the current one runs.
#pragma once
#include "posit32.cuh"
#include "posit32_div.cuh"
#include <math.h>

namespace pg {

constexpr int CHAIN_BLOCK = 8;

PG_HD dp32 chain_neg_b(uint32_t bk) { return decode_dz_bf(bk == P32_NAR ? 0u : 0u - bk); }
PG_HD dp32 chain_a(uint32_t l) { return decode_dz_bf(l == P32_NAR ? 0u : l); }

// b (this thread's right-hand side, m entries; shared or global memory) is overwritten
// with L^-T b.  L is read-only.  Host and device (the host build is what the CPU tests run).
// With `upper`, the triangle is an upper one, U, and b is overwritten with U^-T b
// (Rtrsm('L', 'U', 'T'), Rtrsm.cpp:160-173): for i = 0 .. m-1, t = b_i, t = t - u_ki*b_k for
// k = 0 .. i-1 (ascending), b_i = t / u_ii -- the same chain run forwards.
PG_HD void llt_chain(const uint32_t *__restrict__ L, size_t ldl, uint32_t *b, int m, bool unit, bool upper = false)
{
    constexpr int U = CHAIN_BLOCK;
    for (int step = 0; step < m; ++step) {
        const int i = upper ? step : m - 1 - step;
        const uint32_t *li = L + (size_t)i * ldl; // column i: a_ki for k > i (lower) or k < i (upper)
        const uint32_t bi = b[i];                 // alpha*b with alpha == 1
        uint32_t nar = bi == P32_NAR;
        dp32 c = decode_dz(nar ? 0u : bi);
        int k = upper ? 0 : i + 1;
        const int kend = upper ? i : m;
        if (k + U <= kend) {
            uint32_t lv[U], bv[U];
#pragma unroll
            for (int j = 0; j < U; ++j) {
                lv[j] = li[k + j];
                bv[j] = b[k + j];
            }
            for (; k + U <= kend; k += U) {
                // next block's operands (indexes clamped into [0, kend))
                uint32_t ln[U], bn[U];
#pragma unroll
                for (int j = 0; j < U; ++j) {
                    const int kk = k + U + j < kend ? k + U + j : kend - 1;
                    ln[j] = li[kk];
                    bn[j] = b[kk];
                }
                const dp32 c0 = c;
                uint32_t bad = 0;
#pragma unroll
                for (int j = 0; j < U; ++j) {
                    // t - a_ki*b_k == t + (-b_k)*a_ki bit for bit: posit negation is exact
                    // and rounding is symmetric in sign.  NaR dominates
                    // (kernel_entry.cl:385-390, 414-417) and is carried in `nar`.
                    nar |= (lv[j] == P32_NAR) | (bv[j] == P32_NAR);
                    dp32 p, r;
                    uint32_t bm, ba;
                    dmul_core(chain_neg_b(bv[j]), chain_a(lv[j]), ComputedEntry{}, p, bm);
                    dadd_core(c, p, ComputedEntry{}, r, ba);
                    c = r;
                    bad |= bm | ba;
                }
                if (bad & 0x40000000u) {
                    c = c0;
                    for (int j = 0; j < U; ++j)
                        c = dmac_chain(c, chain_neg_b(bv[j]), chain_a(lv[j]));
                }
#pragma unroll
                for (int j = 0; j < U; ++j) {
                    lv[j] = ln[j];
                    bv[j] = bn[j];
                }
            }
        }
        for (; k < kend; ++k) {
            const uint32_t l = li[k], bk = b[k];
            nar |= (l == P32_NAR) | (bk == P32_NAR);
            c = dmac_chain(c, chain_neg_b(bk), chain_a(l));
        }
        uint32_t t = nar ? P32_NAR : encode(c);
        if (!unit)
            t = pdiv_est(t, li[i]);
        b[i] = t;
    }
}

// ---------------------------------------------------------------------------
// Split form: products computed elsewhere, the chain thread only adds -- in FP64.
// ---------------------------------------------------------------------------
// A posit32 value is exact in FP64 (at most 28 significant bits, scale within +-120).
// One step t + q of the chain is then:
//   s = fl64(t + q);
//   r = (s + C) - C        C = 1.5 * 2^(e + 52 - fb), e the binade of s and fb the posit's
//                          fraction width there: round to nearest even at the posit's last
//                          fraction bit (ties to the even pattern, whose parity is the
//                          fraction's).
// Where s is inexact it never lies half way between two posits (posit32.cuh,
// f64_posit_mac), so r is the exact sum rounded once, which is the reference's p32_add.  A
// step is handed to the exact path when the sum's scale is outside the fast window (regime
// longer than 27 bits, fewer than one fraction bit; this includes an exactly cancelling
// sum, whose FP64 value is 0).
// The dependent path per step: three FP64 additions and a handful of integer operations
// that build C from the exponent of s.
// t + q rounded to posit32, both posit values held in FP64; bit 30 of `bad` is set when
// the step must come from the exact path instead.
PG_HD double f64_posit_add(double t, double q, uint32_t &bad)
{
    const double s = f64_add(t, q);
    const int32_t eb = (int32_t)((f64_bits(s) >> 52) & 0x7FF); // biased binade of s
    const double C = f64_from_hi(f64_round_const_hi(eb));
    const double r = f64_add(f64_add(s, C), -C);
    bad |= f64_outside_fast(eb) ? 0x40000000u : 0u;
    return r;
}

// The exact step on patterns (rare).
PG_HD double f64_posit_add_exact(double t, double q)
{
    return p32_to_double(padd(p32_from_double(t), p32_from_double(q)));
}

// The term -a_ki*b_k of the dot-form solve as the reference rounds it (p32_mul,
// kernel_entry.cl:399-538), in FP64; *nar is set when it is NaR (the term is then 0).
PG_HD double llt_term(uint32_t l, uint32_t bk, uint32_t *nar)
{
    const uint32_t p = pmul(0u - bk, l); // (-b)*a == -(a*b) bit for bit
    *nar |= p == P32_NAR;
    return p32_to_double(p == P32_NAR ? 0u : p);
}

// t + q_0 + q_1 + ... + q_{count-1}, every addition rounded (p32_add), in that order; t
// and the q are posit32 values in FP64.  (The kernels use warp_chain below; this plain form is a
// sequence the tests hold chains to.)
// Blocks of CHAIN_BLOCK steps without a branch, the flags tested once per block, a
// flagged block replayed exactly from its start.
PG_HD double chain_add_run(double t, const double *q, int count)
{
    constexpr int U = CHAIN_BLOCK;
    int k = 0;
    if (count >= U) {
        double v[U];
#pragma unroll
        for (int j = 0; j < U; ++j)
            v[j] = q[j];
        for (; k + U <= count; k += U) {
            double nv[U];
#pragma unroll
            for (int j = 0; j < U; ++j)
                nv[j] = q[k + U + j < count ? k + U + j : count - 1];
            const double t0 = t;
            uint32_t bad = 0;
#pragma unroll
            for (int j = 0; j < U; ++j)
                t = f64_posit_add(t, v[j], bad);
            if (bad & 0x40000000u) {
                t = t0;
                for (int j = 0; j < U; ++j)
                    t = f64_posit_add_exact(t, v[j]);
            }
#pragma unroll
            for (int j = 0; j < U; ++j)
                v[j] = nv[j];
        }
    }
    for (; k < count; ++k) {
        uint32_t bad = 0;
        const double r = f64_posit_add(t, q[k], bad);
        t = (bad & 0x40000000u) ? f64_posit_add_exact(t, q[k]) : r;
    }
    return t;
}


// ---------------------------------------------------------------------------
// Scan form: one row's chain of additions as a parallel prefix over the row.
// ---------------------------------------------------------------------------
// While the running value t stays in one binade [2^e, 2^(e+1)) with sign sg, it is an
// integer multiple M of the posit spacing u = 2^(e - fb) there (fb = the fraction width at
// scale e, M in [2^fb, 2^(fb+1))), and the fraction's last bit -- the pattern's last bit --
// is M's.  A step t + q with the exact sum inside that binade rounds (to nearest, ties to
// the even pattern) as
//     M' = M + K + [F > 1/2] + [F == 1/2] * ((M + K) & 1),   sg * q / u = K + F, 0 <= F < 1,
// which is p32_add's result (kernel_entry.cl:370-397): with the addend at most 30 binades
// down no bit of it leaves the reference's 64-bit frame, and a bit that falls below the
// sticky window after normalisation leaves set bits inside the window (the addend spans
// at most 28 bits), so the rounding decision is that of the exact sum; an addend further
// down has |K + F| < 1/8 and leaves M unchanged, as the reference does.  Steps 25..30
// binades down are still handed to the exact path, as the FP64 step does.
// The exact sum stays in the binade iff 2^fb <= M + K < 2^(fb+1).
//
// So a step is the map M -> M + c[M & 1] (c[0] and c[1] differ only on a tie), and such
// maps compose into maps of the same form.  A thread composes the maps of its slice of the
// row, an exclusive scan over the threads gives each slice its start, and each thread then
// walks its slice with the true M and reports the first step that leaves the binade (or
// starts at its top edge, or is risky).  All steps before that one are exact; the row
// goes on from there with one exact step and a new scan in the new binade.  A map's
// displacements saturate at +-SEG_SAT: only a path that has already left the binade can
// reach that, and no value past the first invalid step is used.
constexpr int32_t SEG_SAT = 1 << 29;

struct SegFn {
    int32_t c0, c1; // displacement for even / odd M
};

// Parameters of a run of steps in t's binade.
struct SegParams {
    double w;       // sg * 2^(fb - e): q * w is q in units of u, sign-folded
    double us;      // sg * 2^(e - fb): t = us * M
    double rlo, rhi; // |q * w| in [rlo, rhi): the addend is 25..30 binades below the binade
    int32_t lo, hi;  // 2^fb, 2^(fb+1)
    int32_t M0;
};

PG_HD int32_t seg_sat(int32_t v) { return v > SEG_SAT ? SEG_SAT : (v < -SEG_SAT ? -SEG_SAT : v); }

// g after f
PG_HD SegFn seg_then(SegFn f, SegFn g)
{
    SegFn h;
    h.c0 = seg_sat(f.c0 + ((f.c0 & 1) ? g.c1 : g.c0));
    h.c1 = seg_sat(f.c1 + ((f.c1 & 1) ? g.c0 : g.c1));
    return h;
}

PG_HD double seg_pow2(int32_t x, uint32_t neg)
{
    return f64_from_bits(((uint64_t)neg << 63) | ((uint64_t)(uint32_t)(x + 1023) << 52));
}

// false when t is zero or its binade is outside the fast window (no scan then).
PG_HD bool seg_begin(double t, SegParams &sp)
{
    const uint64_t b = f64_bits(t);
    const int32_t e = (int32_t)((b >> 52) & 0x7FF) - 1023;
    if (t == 0.0 || e < FAST_LO || e > FAST_HI)
        return false;
    const uint32_t neg = (uint32_t)(b >> 63);
    const int32_t k = e >> 2;
    const int32_t fb = 28 - ((k ^ (k >> 31)) + 1);
    sp.w = seg_pow2(fb - e, neg);
    sp.us = seg_pow2(e - fb, neg);
    sp.rlo = seg_pow2(fb - 30, 0);
    sp.rhi = seg_pow2(fb - 24, 0);
    sp.lo = 1 << fb;
    sp.hi = 2 << fb;
    sp.M0 = (int32_t)(t * sp.w);
    return true;
}

// The step map of addend q; K and `risky` for the validity test.
PG_HD SegFn seg_fn(double q, const SegParams &sp, int32_t &K, bool &risky)
{
    const double Q = q * sp.w; // exact: a power-of-two scaling of a posit value
    const double aQ = Q < 0 ? -Q : Q;
    risky = (aQ >= sp.rlo) & (aQ < sp.rhi);
    const double Qc = Q > (double)SEG_SAT ? (double)SEG_SAT : (Q < -(double)SEG_SAT ? -(double)SEG_SAT : Q);
    const double Kd = floor(Qc);
    const double F = Qc - Kd; // exact
    K = (int32_t)Kd;
    const int32_t up = F > 0.5, tie = F == 0.5;
    SegFn f;
    f.c0 = K + (up | (tie & (K & 1)));
    f.c1 = K + (up | (tie & ((K + 1) & 1)));
    return f;
}

// Is the step from M exact in the scan form?
PG_HD bool seg_valid(int32_t M, int32_t K, bool risky, const SegParams &sp)
{
    return (M < sp.hi) & (M + K >= sp.lo) & (M + K < sp.hi) & !risky;
}

PG_HD int32_t seg_apply(SegFn f, int32_t M) { return M + ((M & 1) ? f.c1 : f.c0); }

// One step t + q with the exact path behind the FP64 form.
PG_HD double chain_add_one(double t, double q)
{
    uint32_t bad = 0;
    const double r = f64_posit_add(t, q, bad);
    return (bad & 0x40000000u) ? f64_posit_add_exact(t, q) : r;
}



// ---------------------------------------------------------------------------
// The chain step with the fraction width held fixed.
// ---------------------------------------------------------------------------
// In f64_posit_add the rounding constant is built from the sum's exponent with integer
// operations on the dependent path.  Within a range of scales of one fraction width fb the
// posit grid is every number with fb + 1 significant bits, so the rounding is that of the
// FP64 significand to 53 - sh bits (sh = 52 - fb), to nearest, ties to even (the last
// fraction bit is the pattern's), whatever the binade.  Veltkamp's splitting (Dekker, "A
// floating-point technique for extending the available precision", 1971) does exactly
// that in FP64 arithmetic rounded to nearest even: with C = 2^sh + 1, g = fl(C s),
// d = fl(s - g), the high part fl(g + d) is s rounded to 53 - sh bits (2 <= sh <= 51), ties
// to even.  So a step is s = fl(t + q) and three more FP64 operations, no exponent on the
// dependent path.  The fraction width is that of the value a block of steps starts at; it
// is the same in regimes k and -k-1 (both have a run of the same length), so the scales
// [2^-4, 2^4) around 1 form one such range of 8 binades, and the other ranges are single
// regimes.  A step whose sum lands at another fraction width (or is zero) is flagged, and the caller redoes the block with chain_add_one.
PG_HD int32_t f64_regime(double x) { return ((int32_t)((f64_bits(x) >> 52) & 0x7FF) - 1023) >> 2; }

// The regime run length of the scale of FP64 pattern sb (fb = 28 - run).
PG_HD int32_t f64_bits_run(uint64_t sb)
{
    const int32_t k = ((int32_t)((sb >> 52) & 0x7FF) - 1023) >> 2;
    return (k ^ (k >> 31)) + 1;
}

// C = 2^sh + 1 for regime run `run` (sh = 52 - fb = 24 + run).
PG_HD double f64_split_const(int32_t run) { return f64_add(f64_from_bits((uint64_t)(24 + run + 1023) << 52), 1.0); }

PG_HD double f64_posit_add_split(double t, double q, double C, int32_t run, uint32_t &bad)
{
    const double s = f64_add(t, q);
    const double g = f64_mul(C, s);
    const double r = f64_add(g, f64_add(s, -g));
    bad |= f64_bits_run(f64_bits(s)) != run ? 0x40000000u : 0u; // off the dependent path
    return r;
}

// t + q_0 + ... + q_{count-1} as chain_add_run, with the fixed-width step: blocks of
// CHAIN_BLOCK steps without a branch, a flagged block redone step by step exactly.
struct TermsF64 {
    const double *q;
    PG_HD_MEMBER double operator[](int i) const { return q[i]; }
    PG_HD_MEMBER TermsF64 operator+(int i) const { return TermsF64{q + i}; }
};

template <class Q>
PG_HD double chain_add_run_reg(double t, Q q, int count)
{
    constexpr int U = CHAIN_BLOCK;
    int k = 0;
    for (; k + U <= count; k += U) {
        const int32_t kreg = f64_regime(t);
        const bool in = (t != 0.0) & (kreg >= (FAST_LO >> 2)) & (kreg <= (FAST_HI >> 2));
        const int32_t run = (kreg ^ (kreg >> 31)) + 1;
        const double C = f64_split_const(run);
        double v[U];
#pragma unroll
        for (int j = 0; j < U; ++j)
            v[j] = q[k + j];
        const double t0 = t;
        uint32_t bad = in ? 0u : 0x40000000u;
#pragma unroll
        for (int j = 0; j < U; ++j)
            t = f64_posit_add_split(t, v[j], C, run, bad);
        if (bad & 0x40000000u) { // (from q: a dynamic index into v would put v in local memory)
            t = t0;
            for (int j = 0; j < U; ++j)
                t = chain_add_one(t, q[k + j]);
        }
    }
    for (; k < count; ++k)
        t = chain_add_one(t, q[k]);
    return t;
}

// ---------------------------------------------------------------------------
// A warp's chain of additions on the biased running value.
// ---------------------------------------------------------------------------
// While t stays in one binade, t = M u with the grid's spacing u = 2^(e - fb) and
// 2^fb <= |M| < 2^(fb+1).  Hold it as w = C + t, C = sign(t) 1.5 * 2^52 u: w is exact, its
// spacing as an FP64 number is u, and C/u is even, so the FP64 addition w + q, rounded to
// nearest even, IS the posit addition: one FP64 addition per step instead of the sum, its
// exponent, a constant and two more additions.  And |M| is w's low word: the step was inside
// the binade iff w's high word is C's and the low word in (2^fb, 2^(fb+1)) -- 2^fb itself is
// given up, since the exact sum may have been below it, where the grid is finer.
//
// So 512 addends are taken at once (a window), 16 per lane.  A step moves M by an amount that
// depends on M's parity alone (ties), so a lane's 16 steps are two displacements, found by
// running them from an even and from an odd M; a warp scan composes them (mod 2^32: past the
// first step that left the binade nothing is used), and each lane runs its steps again from
// its true start, tested at once.  The window ends where the first lane with a step outside
// starts.  There the value is near a power of two and often crosses it again soon: blocks of
// 16 in the fixed-width step (which crosses powers of two, not fraction widths; f64_posit_add
// does) follow until one stayed in its binade.
//
// What bounds it: latency.  A dependent FP64 addition takes 8.1 cycles, a window about 900, a
// fixed-width step 32 and its block's tests and branches 150 (so 16 steps, not 8).  (Blocks of 8 one-addition steps first, repeated where
// they left the binade, were slower: half of them did, and each start in a new binade cost
// 200.)
#if defined(__CUDACC__)
constexpr int CHAIN_E = 16;          // addends per lane of a window, 8 or 16
constexpr int CHAIN_WINDOW_MIN = 64; // addends left for a window to pay

// A row's addends in shared memory, in groups of 16.  FP64: a group every 18 doubles, so that
// the lanes of a warp reading a group each spread over the banks.
struct ChainTerms64 {
    double *q;
    static constexpr int GROUP_DOUBLES = 18;
    static __host__ __device__ size_t bytes(int n) { return (size_t)((n + 15) / 16) * GROUP_DOUBLES * sizeof(double); }
    using Word = double;
    __device__ static int at(int k) { return k + (k >> 4) * 2; }
    __device__ void set(int k, double v) const { q[at(k)] = v; }
    __device__ double get(int k) const { return q[at(k)]; }
    template <int N> // N addends from k, a multiple of N, N <= 16 a power of two
    __device__ void load(int k, double (&v)[N]) const
    {
        const double2 *p = reinterpret_cast<const double2 *>(q + at(k));
#pragma unroll
        for (int j = 0; j < N / 2; ++j) {
            const double2 x = p[j];
            v[2 * j] = x.x;
            v[2 * j + 1] = x.y;
        }
    }
};
// Five bytes an addend, for columns too long for FP64: a posit has at most 27 fraction bits, so
// the low word's upper byte holds all that the high word does not.  Patterns instead (4 bytes,
// converted by the adding warp at each load) took Rpotrs n = 16384 1618 ms; this takes 838.
struct ChainTerms40 {
    unsigned char *q; // a buffer of n addends: the high words, then the bytes
    int n16;          // n, up to a multiple of 16
    static __host__ __device__ size_t bytes(int n) { return (size_t)((n + 15) / 16) * 80; }
    using Word = uint32_t;
    __device__ uint32_t *hi() const { return reinterpret_cast<uint32_t *>(q); }
    __device__ unsigned char *lo() const { return q + (size_t)n16 * 4; }
    __device__ void set(int k, double v) const
    {
        hi()[k] = (uint32_t)__double2hiint(v);
        lo()[k] = (unsigned char)((uint32_t)__double2loint(v) >> 24);
    }
    __device__ double get(int k) const { return __hiloint2double((int)hi()[k], (int)((uint32_t)lo()[k] << 24)); }
    template <int N> // as above, N a multiple of 8
    __device__ void load(int k, double (&v)[N]) const
    {
        const uint4 *h = reinterpret_cast<const uint4 *>(hi() + k);
        const uint2 *l = reinterpret_cast<const uint2 *>(lo() + k);
#pragma unroll
        for (int j = 0; j < N / 4; ++j) {
            const uint4 x = h[j];
            const uint32_t y = j & 1 ? l[j / 2].y : l[j / 2].x;
            v[4 * j] = __hiloint2double((int)x.x, (int)(y << 24));
            v[4 * j + 1] = __hiloint2double((int)x.y, (int)__byte_perm(y, 0, 0x1444));
            v[4 * j + 2] = __hiloint2double((int)x.z, (int)__byte_perm(y, 0, 0x2444));
            v[4 * j + 3] = __hiloint2double((int)x.w, (int)(y & 0xFF000000u));
        }
    }
};

// t + q[pos] + ... + q[end-1], every addition rounded, in that order; t and the q are posit32
// values, none NaR.  In the groups that hold q[pos] and q[end-1], every other addend is zero
// (so nothing is masked).  Every lane of a full warp calls it with the same arguments and
// returns the same value.
template <class Q>
__device__ double warp_chain(double t, Q q, int pos, int end)
{
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    pos &= ~7; // from here on a multiple of 8: adding a zero changes nothing
    while (pos < end) {
        const uint32_t th = f64_hi(t);
        const int32_t eb = (int32_t)((th >> 20) & 0x7FF);
        if (end - pos >= CHAIN_WINDOW_MIN && !f64_outside_fast(eb)) {
            const uint32_t chi = f64_round_const_hi(eb) | (th & 0x80000000u);
            const double C = f64_from_hi(chi);
            const uint32_t lim = 1u << (28 - ((int32_t)((chi >> 20) & 0x7FF) - eb - 24)); // 2^fb
            double w = f64_add(C, t);
            bool left = false;
            do { // windows in this binade
                const int g0 = pos / CHAIN_E, k0 = (g0 + lane) * CHAIN_E;
                const int wend = min(end, (g0 + 32) * CHAIN_E);
                double v[CHAIN_E];
                if (k0 < end) {
                    q.load(k0, v);
                    if (CHAIN_E > 8 && k0 < pos) { // the group's first half is done
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            v[e] = 0.0;
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < CHAIN_E; ++e)
                        v[e] = 0.0;
                }
                // the lane's displacements: of an even M, and by how much an odd one's differs
                constexpr uint32_t M0 = 1u << 28;
                double w0 = __hiloint2double((int)chi, (int)M0), w1 = __hiloint2double((int)chi, (int)(M0 + 1));
#pragma unroll
                for (int e = 0; e < CHAIN_E; ++e) {
                    w0 = f64_add(w0, v[e]);
                    w1 = f64_add(w1, v[e]);
                }
                uint32_t c0 = (uint32_t)__double2loint(w0) - M0, d = (uint32_t)__double2loint(w1) - 1 - M0 - c0;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const uint32_t o0 = __shfl_up_sync(FULL, c0, off), od = __shfl_up_sync(FULL, d, off);
                    // this lane's steps after the earlier ones': M moves by o0 (+ od), then by
                    // c0, and by d more where M is odd then
                    const uint32_t p0 = o0 & 1, p1 = (o0 + od + 1) & 1;
                    const uint32_t n0 = o0 + c0 + p0 * d, nd = od + (p1 - p0) * d;
                    c0 = lane >= off ? n0 : c0;
                    d = lane >= off ? nd : d;
                }
                uint32_t x0 = __shfl_up_sync(FULL, c0, 1), xd = __shfl_up_sync(FULL, d, 1);
                if (lane == 0)
                    x0 = xd = 0;
                uint32_t M = (uint32_t)__double2loint(w);
                M += x0 + (M & 1) * xd;
                double y = __hiloint2double((int)chi, (int)M);
                uint32_t bad = 0, mn = 0xFFFFFFFFu, mx = 0;
#pragma unroll
                for (int e = 0; e < CHAIN_E; ++e) {
                    y = f64_add(y, v[e]);
                    const uint32_t lo = (uint32_t)__double2loint(y);
                    bad |= (uint32_t)__double2hiint(y) ^ chi;
                    mn = min(mn, lo);
                    mx = max(mx, lo);
                }
                const unsigned bal = __ballot_sync(FULL, bad != 0 || mn <= lim || mx >= 2 * lim);
                const uint32_t Mend = __shfl_sync(FULL, (uint32_t)__double2loint(y), 31);
                left = bal != 0;
                if (!left) {
                    w = __hiloint2double((int)chi, (int)Mend);
                    pos = wend;
                } else {
                    const int src = __ffs(bal) - 1;
                    w = __hiloint2double((int)chi, (int)__shfl_sync(FULL, M, src));
                    pos = max(pos, (g0 + src) * CHAIN_E);
                }
            } while (!left && end - pos >= CHAIN_WINDOW_MIN);
            t = f64_add(w, -C);
            if (pos >= end)
                break;
        }
        // blocks of 16 in the fixed-width step, its constant kept while the width is
        double v[8], v2[8], Cs = 0.0;
        uint32_t wlo = 1, wspan = 0; // |t|'s high words of this fraction width: [wlo, wlo + wspan)
        auto width = [&]() {
            const int32_t eb = f64_binade(t), k = (eb - 1023) >> 2, run = (k ^ (k >> 31)) + 1;
            // the binades of regime k; around 1, those of regimes 0 and -1
            wlo = (uint32_t)((run == 1 ? -4 : 4 * k) + 1023) << 20;
            wspan = f64_outside_fast(eb) ? 0u : (run == 1 ? 8u : 4u) << 20;
            Cs = f64_split_const(run);
        };
        auto fetch = [&]() {
            q.load(pos, v);
            if (pos + 8 < end) {
                q.load(pos + 8, v2);
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    v2[e] = 0.0;
            }
        };
        width();
        fetch();
        bool crossed;
        do {
            const double t0 = t;
            uint32_t out = wspan == 0, cross = 0;
            auto step = [&](double x) {
                const double s = f64_add(t, x);
                const double g = f64_mul(Cs, s);
                t = f64_add(g, f64_add(s, -g));
                // off the dependent path
                const uint32_t h = f64_hi(s);
                out |= (h & 0x7FFFFFFFu) - wlo >= wspan;
                cross |= h ^ f64_hi(t0);
            };
#pragma unroll
            for (int e = 0; e < 8; ++e)
                step(v[e]);
#pragma unroll
            for (int e = 0; e < 8; ++e)
                step(v2[e]);
            if (out) { // across fraction widths: with the constant of every step's own binade
                t = t0;
                uint32_t flag = 0;
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    t = f64_posit_add(t, v[e], flag);
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    t = f64_posit_add(t, v2[e], flag);
                if (flag & 0x40000000u) { // zero, or outside the fast window
                    t = t0;
                    for (int e = 0; e < 16; ++e)
                        if (pos + e < end)
                            t = f64_round_any(f64_add(t, q.get(pos + e)));
                }
                width();
            }
            crossed = (cross >> 20) != 0;
            pos += 16;
            if (pos < end)
                fetch();
        } while (pos < end && (crossed || end - pos < CHAIN_WINDOW_MIN));
    }
    return t;
}

// L^-T b for one right-hand side by one warp (Rtrsm('L', 'L', 'T', 'N'), as llt_chain): the
// terms of a row, one per lane and stretch of 32, then their chain.  x (shared memory, the
// column as FP64, NaN for NaR) is overwritten; `q` holds m terms, its buffer is cleared here.
template <class Q>
__device__ void warp_llt_solve(const uint32_t *__restrict__ L, size_t ldl, double *x, int m, Q q)
{
    constexpr unsigned FULL = 0xFFFFFFFFu;
    constexpr int PRE = 8; // a row's first coefficients, loaded while the row before it is summed
    const int lane = threadIdx.x & 31;
    for (int k = lane; k < (int)(Q::bytes(m) / sizeof(typename Q::Word)); k += 32)
        q.q[k] = 0;
    __syncwarp();
    uint32_t pre[PRE], dn = L[(m - 1) + (size_t)(m - 1) * ldl];
#pragma unroll
    for (int j = 0; j < PRE; ++j)
        pre[j] = 0;
    for (int i = m - 1; i >= 0; --i) {
        const uint32_t *li = L + (size_t)i * ldl;
        bool nar = false;
        auto term = [&](int k, uint32_t l) {
            double v = f64_posit_mul_checked(-x[k], p32_to_double(l), F64ConstComputed{});
            if (v != v) {
                nar = true;
                v = 0.0;
            }
            q.set(k, v);
        };
#pragma unroll
        for (int j = 0; j < PRE; ++j)
            if (i + 1 + lane + 32 * j < m)
                term(i + 1 + lane + 32 * j, pre[j]);
#pragma unroll 1
        for (int k = i + 1 + lane + 32 * PRE; k < m; k += 32)
            term(k, li[k]);
        const double d = p32_to_double(dn);
        if (i > 0) {
            dn = li[-(ptrdiff_t)ldl + i - 1];
#pragma unroll
            for (int j = 0; j < PRE; ++j) {
                const int k = i + lane + 32 * j;
                pre[j] = k < m ? li[k - (ptrdiff_t)ldl] : 0u;
            }
        }
        const double rc = 1.0 / d;
        nar = __any_sync(FULL, nar) || x[i] != x[i];
        __syncwarp(); // the terms are in place
        double t = nar ? 0.0 : warp_chain(x[i], q, i + 1, m);
        t = f64_posit_div(nar ? p32_to_double(P32_NAR) : t, d, rc);
        __syncwarp();
        if (lane == 0)
            x[i] = t;
        __syncwarp();
    }
}

// The solution column: FP64 in shared memory, or where the columns are long the patterns in
// global memory.
struct LtxCol64 {
    double *b;
    static constexpr bool GLOBAL = false;
    __device__ double get(int k) const { return b[k]; }
    __device__ void set(int k, double v) const { b[k] = v; }
};
struct LtxColGlobal {
    uint32_t *b;
    static constexpr bool GLOBAL = true;
    __device__ double get(int k) const { return p32_to_double(b[k]); }
    __device__ void set(int k, double v) const { b[k] = p32_from_double_exact(v); }
};
// What the adding warp needs of a row besides its terms.
struct LtxRow {
    double diag, recip; // a_ii and fl(1/a_ii)
    double near;        // the coefficient of the b finished last
    double b;           // the right-hand side's entry (Col::GLOBAL)
    int nar;            // a term was NaR
};

// L^-T x (UPPER: U^-T x) for one right-hand side by a block of NT threads: warp 0 sums a row's
// terms (warp_chain) while the others compute the next row's, all whose x_k are final, into
// the other half of a double buffer, and its diagonal's reciprocal; the term of the x_k just
// finished (the first one, UPPER: the last) warp 0 forms itself.  `buf`: 2 * Terms::bytes(m).
// NaR travels as NaN; a NaR term sets its row's flag and is replaced by 0.
template <int NT, bool UPPER, class Terms, class Col>
__device__ __forceinline__ void block_ltx_solve(const uint32_t *__restrict__ L, size_t ldl, Col x, int m, bool unit,
                                                unsigned char *buf, LtxRow *s_row)
{
    const int tid = threadIdx.x;
    auto terms = [&](int half) {
        Terms q;
        q.q = reinterpret_cast<decltype(q.q)>(buf + half * Terms::bytes(m));
        if constexpr (Col::GLOBAL)
            q.n16 = (m + 15) & ~15;
        return q;
    };
    // Terms outside a row's range are zero for warp_chain: rows grow, so what no earlier row
    // wrote is still this.
    for (int k = tid; k < (int)(2 * Terms::bytes(m) / sizeof(typename Terms::Word)); k += NT)
        reinterpret_cast<typename Terms::Word *>(buf)[k] = 0;
    auto row_of = [&](int step) { return UPPER ? step : m - 1 - step; };
    // the row's diagonal and nearest coefficient
    auto head = [&](int step) {
        const int i = row_of(step);
        const uint32_t *li = L + (size_t)i * ldl;
        LtxRow &r = s_row[step & 1];
        r.diag = unit ? 1.0 : p32_to_double(li[i]);
        r.recip = 1.0 / r.diag;
        r.near = step > 0 ? p32_to_double(li[UPPER ? i - 1 : i + 1]) : 0.0;
        if (Col::GLOBAL)
            r.b = x.get(i);
    };
    if (tid < 2)
        s_row[tid].nar = 0;
    if (tid == 32)
        head(0);
    __syncthreads();
    double last = 0.0; // the x_k finished last (warp 0)
    for (int step = 0; step < m; ++step) {
        const int i = row_of(step), cur = step & 1;
        if (tid < 32) {
            const LtxRow r = s_row[cur];
            double t = Col::GLOBAL ? r.b : x.get(i);
            bool nar = t != t || r.nar;
            double near = 0.0; // -a*x_k of the one just finished
            if (step > 0) {
                near = f64_posit_mul_checked(-last, r.near, F64ConstComputed{});
                if (near != near) {
                    nar = true;
                    near = 0.0;
                }
            }
            if (nar)
                t = 0.0;
            if (!UPPER && step > 0) {
                t = f64_round_any(f64_add(t, near));
                t = warp_chain(t, terms(cur), i + 2, m);
            }
            if (UPPER && step > 0) {
                t = warp_chain(t, terms(cur), 0, i - 1);
                t = f64_round_any(f64_add(t, near));
            }
            last = nar ? p32_to_double(P32_NAR) : t;
            if (!unit)
                last = f64_posit_div(last, r.diag, r.recip);
            __syncwarp(); // every lane has read the row
            if (tid == 0) {
                x.set(i, last);
                s_row[cur].nar = 0;
            }
        } else if (step + 1 < m) {
            // the terms of the next row whose x_k are final: k = i+1 .. m-1 of row i-1
            // (lower), k = 0 .. i-1 of row i+1 (upper)
            const int kbeg = UPPER ? 0 : i + 1, kend = UPPER ? i : m;
            const uint32_t *lp = L + (size_t)row_of(step + 1) * ldl;
            if (tid == 32)
                head(step + 1);
            const Terms q = terms(cur ^ 1);
            int nar = 0;
            constexpr int P = NT - 32, U = 8; // U loads in flight per thread
            for (int k = kbeg + (tid - 32); k < kend; k += U * P) {
                uint32_t l[U];
                double xk[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    l[u] = k + u * P < kend ? lp[k + u * P] : 0u;
                    xk[u] = Col::GLOBAL && k + u * P < kend ? x.get(k + u * P) : 0.0;
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (k + u * P < kend) {
                        if (!Col::GLOBAL)
                            xk[u] = x.get(k + u * P);
                        double v = f64_posit_mul_checked(-xk[u], p32_to_double(l[u]), F64ConstComputed{});
                        if (v != v) {
                            nar = 1;
                            v = 0.0;
                        }
                        q.set(k + u * P, v);
                    }
            }
            if (nar)
                s_row[cur ^ 1].nar = 1;
        }
        __syncthreads();
    }
}
#endif

} // namespace pg
