// Host build of the division and square root the kernels use (posit32_div.cuh), and the kernels'
// present algorithms restated in the same FP64 steps: the LU panel (lapack.cu,
// lu_panel_cluster_kernel), the Cholesky panel (chol_panel_kernel) and the adding warp
// (trsm_chain.cuh, warp_chain).  Compiled by tests/test_kernels_restated_cpu.py.
#include "../posit_gpu_b200/csrc/posit32.cuh"
#include "../posit_gpu_b200/csrc/posit32_div.cuh"
#include "../posit_gpu_b200/csrc/trsm_chain.cuh"
#include <math.h>
#include <stdint.h>
#include <algorithm>
#include <vector>
using namespace pg;

namespace {
double mac(double c, double t, double a) { return f64_posit_mac_checked(c, t, a, F64ConstComputed{}); }
double mul(double x, double y) { return f64_posit_mul_checked(x, y, F64ConstComputed{}); }
double recip(double x) { return f64_posit_div(1.0, x, 1.0 / x); }

// How far q is from half way between two posits, over its size: what f64_posit_div and
// f64_posit_sqrt compare with 2^-50.
bool near_half(double q)
{
    const uint32_t ch = f64_round_const_top(f64_hi(q) >> 20);
    const double C = f64_from_hi(ch), z = f64_add(f64_add(q, C), -C);
    const double half = f64_from_hi((ch & 0x7FF00000u) - (53u << 20));
    return !(fabs(fabs(q - z) - half) > fabs(q) * 8.8817841970012523e-16);
}
} // namespace

extern "C" {
// o = t / a; returns how many were too near half way for the FP64 quotient
long hk_div_n(const uint32_t *t, const uint32_t *a, uint32_t *o, long n)
{
    long near = 0;
    for (long i = 0; i < n; ++i) {
        const double x = p32_to_double(t[i]), y = p32_to_double(a[i]), rc = 1.0 / y;
        o[i] = p32_from_double(f64_posit_div(x, y, rc));
        near += x == x && y == y && x != 0.0 && y != 0.0 && near_half(x / y);
    }
    return near;
}
long hk_sqrt_n(const uint32_t *a, uint32_t *o, long n)
{
    long near = 0;
    for (long i = 0; i < n; ++i) {
        const double x = p32_to_double(a[i]);
        o[i] = p32_from_double(f64_posit_sqrt(x));
        near += near_half(sqrt(x));
    }
    return near;
}

// The LU panel: the pivot of column k+1 is looked for once that column alone is up to date, the
// candidate's row is then brought up to date by itself and travels ahead; the other columns of
// the rows follow.  Rows keep their slots, interchanges swap the slots' logical rows.
int hk_lu_panel(uint32_t *P, int M, int jb, int *ipiv)
{
    std::vector<double> S((size_t)M * jb); // slot s, column c at [s * jb + c]
    std::vector<int> row(M);
    for (int s = 0; s < M; ++s) {
        row[s] = s;
        for (int c = 0; c < jb; ++c)
            S[(size_t)s * jb + c] = p32_to_double(P[s + (size_t)c * M]);
    }
    int info = 0, cand = -1;
    std::vector<double> u(jb, 0.0), next(jb, 0.0);
    auto better = [&](int s, int than, int c) {
        auto key = [&](int q) {
            const double v = S[(size_t)q * jb + c];
            return v != v ? -1.0 : fabs(v);
        };
        return than < 0 || key(s) > key(than) || (key(s) == key(than) && row[s] < row[than]);
    };
    // the candidate's row, columns c .. (its columns past c: with the step of column c - 1)
    auto publish = [&](int c) {
        const double *rw = &S[(size_t)cand * jb];
        for (int q = c; q < jb; ++q)
            next[q] = c > 0 && q > c ? mac(rw[q], -u[q], rw[c - 1]) : rw[q];
    };
    for (int s = 0; s < M; ++s)
        if (better(s, cand, 0))
            cand = s;
    publish(0);
    for (int k = 0; k < jb; ++k) {
        const int win = cand, p = row[win];
        u = next;
        const double val = u[k], rc = val == 0.0 ? 1.0 : recip(val);
        ipiv[k] = p + 1;
        if (val == 0.0 && info == 0)
            info = k + 1;
        if (p != k) {
            if (val == 0.0)
                for (int s = 0; s < M; ++s)
                    if (row[s] == k) {
                        S[(size_t)win * jb + k] = S[(size_t)s * jb + k];
                        S[(size_t)s * jb + k] = val;
                    }
            for (int s = 0; s < M; ++s)
                row[s] = row[s] == k ? p : (row[s] == p ? k : row[s]);
        }
        cand = -1;
        for (int s = 0; s < M; ++s)
            if (row[s] > k) {
                double *rw = &S[(size_t)s * jb];
                rw[k] = mul(rw[k], rc);
                if (k + 1 < jb)
                    rw[k + 1] = mac(rw[k + 1], -u[k + 1], rw[k]);
            }
        if (k + 1 < jb) {
            for (int s = 0; s < M; ++s)
                if (row[s] > k && better(s, cand, k + 1))
                    cand = s;
            if (cand >= 0)
                publish(k + 1);
            else
                std::fill(next.begin(), next.end(), 0.0); // no row left: not used, M >= jb
        }
        for (int s = 0; s < M; ++s)
            if (row[s] > k)
                for (int c = k + 2; c < jb; ++c)
                    S[(size_t)s * jb + c] = mac(S[(size_t)s * jb + c], -u[c], S[(size_t)s * jb + k]);
    }
    for (int s = 0; s < M; ++s)
        for (int c = 0; c < jb; ++c)
            P[row[s] + (size_t)c * M] = p32_from_double_exact(S[(size_t)s * jb + c]);
    return info;
}

// The Cholesky panel: the diagonal block factored by itself (by every CTA), then each row below
// taken through it alone; a failed diagonal stops both after the columns before it.
int hk_chol_panel(uint32_t *P, int M, int jb)
{
    std::vector<double> D((size_t)jb * jb, 0.0), rc(jb, 0.0); // a_ic of the block at [c * jb + i]
    for (int c = 0; c < jb; ++c)
        for (int i = c; i < jb; ++i)
            D[(size_t)c * jb + i] = p32_to_double(P[i + (size_t)c * M]);
    int stop = jb;
    for (int k = 0; k < jb; ++k) {
        double *dk = &D[(size_t)k * jb];
        if (!(dk[k] > 0.0)) {
            stop = k;
            break;
        }
        const double lkk = f64_posit_sqrt(dk[k]);
        rc[k] = recip(lkk);
        std::vector<double> l(jb, 0.0);
        for (int i = k + 1; i < jb; ++i)
            l[i] = mul(dk[i], rc[k]);
        for (int c = k + 1; c < jb; ++c)
            for (int i = c; i < jb; ++i)
                D[(size_t)c * jb + i] = mac(D[(size_t)c * jb + i], -l[c], l[i]);
        for (int i = k; i < jb; ++i)
            dk[i] = i == k ? lkk : l[i];
    }
    for (int c = 0; c < jb; ++c)
        for (int i = c; i < jb; ++i)
            P[i + (size_t)c * M] = p32_from_double_exact(D[(size_t)c * jb + i]);
    for (int i = jb; i < M; ++i)
        for (int k = 0; k < stop; ++k) {
            const double l = mul(p32_to_double(P[i + (size_t)k * M]), rc[k]);
            P[i + (size_t)k * M] = p32_from_double_exact(l);
            for (int c = k + 1; c < jb; ++c) {
                uint32_t &x = P[i + (size_t)c * M];
                x = p32_from_double_exact(mac(p32_to_double(x), -D[(size_t)k * jb + c], l));
            }
        }
    return stop < jb ? stop + 1 : 0;
}

// warp_chain, its 32 lanes one after the other: t + q[pos] + ... + q[end-1] (q zero outside, up
// to the multiples of 16 around).  stats: windows kept whole, windows cut, blocks, blocks redone.
uint32_t hk_warp_chain(uint32_t t0, const uint32_t *qp, int pos, int end, long *stats)
{
    constexpr int E = 16, WINDOW_MIN = 64;
    const int n16 = (end + E - 1) / E * E;
    std::vector<double> q(n16 + 32 * E, 0.0);
    for (int k = pos; k < end; ++k)
        q[k] = p32_to_double(qp[k]);
    auto lo = [](double x) { return (uint32_t)f64_bits(x); };
    auto hilo = [](uint32_t h, uint32_t l) { return f64_from_bits(((uint64_t)h << 32) | l); };
    double t = p32_to_double(t0);
    pos &= ~7;
    while (pos < end) {
        const uint32_t th = f64_hi(t);
        const int32_t eb = (int32_t)((th >> 20) & 0x7FF);
        if (end - pos >= WINDOW_MIN && !f64_outside_fast(eb)) {
            const uint32_t chi = f64_round_const_hi(eb) | (th & 0x80000000u);
            const double C = f64_from_hi(chi);
            const uint32_t lim = 1u << (28 - ((int32_t)((chi >> 20) & 0x7FF) - eb - 24));
            double w = f64_add(C, t);
            bool left = false;
            do {
                const int g0 = pos / E, wend = std::min(end, (g0 + 32) * E);
                constexpr uint32_t M0 = 1u << 28;
                double v[32][E];
                uint32_t c0[32], d[32];
                for (int lane = 0; lane < 32; ++lane) {
                    const int k0 = (g0 + lane) * E;
                    double w0 = hilo(chi, M0), w1 = hilo(chi, M0 + 1);
                    for (int e = 0; e < E; ++e) {
                        v[lane][e] = k0 < end && !(k0 < pos && e < 8) ? q[k0 + e] : 0.0;
                        w0 = f64_add(w0, v[lane][e]);
                        w1 = f64_add(w1, v[lane][e]);
                    }
                    c0[lane] = lo(w0) - M0;
                    d[lane] = lo(w1) - 1 - M0 - c0[lane];
                }
                for (int off = 1; off < 32; off <<= 1)
                    for (int lane = 31; lane >= off; --lane) { // downwards: the lanes below are still the old ones
                        const uint32_t o0 = c0[lane - off], od = d[lane - off];
                        const uint32_t p0 = o0 & 1, p1 = (o0 + od + 1) & 1;
                        const uint32_t n0 = o0 + c0[lane] + p0 * d[lane], nd = od + (p1 - p0) * d[lane];
                        c0[lane] = n0;
                        d[lane] = nd;
                    }
                int src = -1;
                uint32_t Msrc = 0, Mend = 0;
                for (int lane = 0; lane < 32; ++lane) {
                    const uint32_t x0 = lane ? c0[lane - 1] : 0, xd = lane ? d[lane - 1] : 0;
                    uint32_t M = lo(w);
                    M += x0 + (M & 1) * xd;
                    double y = hilo(chi, M);
                    uint32_t bad = 0, mn = 0xFFFFFFFFu, mx = 0;
                    for (int e = 0; e < E; ++e) {
                        y = f64_add(y, v[lane][e]);
                        bad |= f64_hi(y) ^ chi;
                        mn = std::min(mn, lo(y));
                        mx = std::max(mx, lo(y));
                    }
                    if (src < 0 && (bad || mn <= lim || mx >= 2 * lim)) {
                        src = lane;
                        Msrc = M;
                    }
                    Mend = lo(y);
                }
                left = src >= 0;
                ++stats[left ? 1 : 0];
                w = hilo(chi, left ? Msrc : Mend);
                pos = left ? std::max(pos, (g0 + src) * E) : wend;
            } while (!left && end - pos >= WINDOW_MIN);
            t = f64_add(w, -C);
            if (pos >= end)
                break;
        }
        bool crossed;
        do {
            ++stats[2];
            const double start = t;
            const int32_t b = f64_binade(t), k = (b - 1023) >> 2, run = (k ^ (k >> 31)) + 1;
            const uint32_t wlo = (uint32_t)((run == 1 ? -4 : 4 * k) + 1023) << 20;
            const uint32_t wspan = f64_outside_fast(b) ? 0u : (run == 1 ? 8u : 4u) << 20;
            const double Cs = f64_split_const(run);
            bool out = wspan == 0;
            uint32_t cross = 0;
            double v[16];
            for (int e = 0; e < 16; ++e)
                v[e] = e < 8 || pos + 8 < end ? q[pos + e] : 0.0;
            for (int e = 0; e < 16; ++e) {
                const double s = f64_add(t, v[e]), g = f64_mul(Cs, s);
                t = f64_add(g, f64_add(s, -g));
                out |= (f64_hi(s) & 0x7FFFFFFFu) - wlo >= wspan;
                cross |= f64_hi(s) ^ f64_hi(start);
            }
            if (out) {
                ++stats[3];
                t = start;
                uint32_t flag = 0;
                for (int e = 0; e < 16; ++e)
                    t = f64_posit_add(t, v[e], flag);
                if (flag & 0x40000000u) {
                    t = start;
                    for (int e = 0; e < 16 && pos + e < end; ++e)
                        t = f64_round_any(f64_add(t, q[pos + e]));
                }
            }
            crossed = (cross >> 20) != 0;
            pos += 16;
        } while (pos < end && (crossed || end - pos < WINDOW_MIN));
    }
    return p32_from_double(t);
}
// the same chain one addition after the other, on patterns
uint32_t hk_plain_chain(uint32_t t, const uint32_t *q, int pos, int end)
{
    for (int k = pos; k < end; ++k)
        t = padd(t, q[k]);
    return t;
}
}
