// FP32 complex FFT building blocks for the fused slice passes.
//
// An N-point transform is computed by a "team" of G threads, each holding
// E = N/G points in registers, as a two-level Cooley-Tukey factorisation
// N = E x G:
//   1. each thread g takes x[g + G j] (j < E) and runs an E-point DFT in
//      registers (radix-4 decimation in frequency, constant twiddles from
//      __constant__ memory, fully unrolled);
//   2. the E outputs are multiplied by the inter-level twiddles W_N^(g k1)
//      (a shared-memory table laid out [k1][g] so a team reads it without
//      bank conflicts);
//   3. one transpose through shared memory (padded rows) hands every thread
//      the G values of E/G columns k1, and a G-point register DFT finishes
//      each.
// The result is X[g + G j'] in thread g, i.e. the same distribution as the
// input, so an inverse transform, a pointwise multiply and a forward
// transform chain in registers with no data movement.  Forward transforms
// use exp(-2 pi i jk/N) and are unnormalised, like CUFFT_FORWARD.
#pragma once
#include <cuda_runtime.h>

#include "fft_layout.hpp"

namespace msb {

// The parts of W_64^m = exp(-2 pi i m / 64) are +-cos(k pi / 32), k = 0..16, kept as an unevaluated
// sum hi + lo of two floats: hi is the double value rounded to float, lo the rounded remainder.  One
// table of cosines serves real and imaginary parts, so a 32-point DFT touches 7 distinct pairs.  The
// values are computed at compile time (tw64::cos_m: the octant by an exact rotation, the remainder
// angle below pi/4 by its Taylor series in double), so every translation unit's copy of the table is
// initialised in its module image and nothing is uploaded at run time.
namespace tw64 {
constexpr double kPi = 3.14159265358979323846264338327950288;
constexpr double kRsqrt2 = 0.70710678118654752440084436210484903928;
// sin a and cos a for 0 <= a <= pi/4 (terms to a^41: truncation far below double rounding)
constexpr double sin_series(double a)
{
    double t = a, s = a;
    for (int k = 1; k <= 20; k++) {
        t *= -a * a / ((2.0 * k) * (2.0 * k + 1.0));
        s += t;
    }
    return s;
}
constexpr double cos_series(double a)
{
    double t = 1.0, s = 1.0;
    for (int k = 1; k <= 20; k++) {
        t *= -a * a / ((2.0 * k - 1.0) * (2.0 * k));
        s += t;
    }
    return s;
}
// cos and sin of 2 pi m / 64 = q pi/4 + r pi/32 with q = m / 8, r = m % 8
constexpr double cq_of(int q) { return q == 0 ? 1.0 : q == 1 ? kRsqrt2 : q == 2 ? 0.0 : q == 3 ? -kRsqrt2 : q == 4 ? -1.0 : q == 5 ? -kRsqrt2 : q == 6 ? 0.0 : kRsqrt2; }
constexpr double sq_of(int q) { return q == 0 ? 0.0 : q == 1 ? kRsqrt2 : q == 2 ? 1.0 : q == 3 ? kRsqrt2 : q == 4 ? 0.0 : q == 5 ? -kRsqrt2 : q == 6 ? -1.0 : -kRsqrt2; }
constexpr double cos_m(int m)
{
    const double a = kPi * (m % 8) / 32.0;
    return cq_of(m / 8) * cos_series(a) - sq_of(m / 8) * sin_series(a);
}
struct Table {
    float hi[16], lo[16];
};
constexpr Table table()
{
    Table t{};
    for (int k = 0; k < 16; k++) {
        t.hi[k] = (float)cos_m(k);
        t.lo[k] = (float)(cos_m(k) - (double)(float)cos_m(k));
    }
    return t;
}
}  // namespace tw64
static __constant__ tw64::Table c_cos32 = tw64::table();
// cos(k pi / 32), any k >= 0 (a compile-time constant once the callers are unrolled)
__device__ __forceinline__ float cos32_of(const float (&c)[16], int k)
{
    k &= 63;
    if (k > 32) k = 64 - k;
    return k == 16 ? 0.0f : k < 16 ? c[k] : -c[32 - k];
}
// W_64^m, hi and lo parts: (cos, -sin) with sin(m pi / 32) = cos((m - 16) pi / 32)
__device__ __forceinline__ float2 tw64_hi(int m) { return make_float2(cos32_of(c_cos32.hi, m), -cos32_of(c_cos32.hi, m + 48)); }
__device__ __forceinline__ float2 tw64_lo(int m) { return make_float2(cos32_of(c_cos32.lo, m), -cos32_of(c_cos32.lo, m + 48)); }

// Complex sums, and the products with one real factor, act on both parts at once: one packed FP32
// instruction instead of two.  The packed forms run at the multiply-add rate of the scalar ones with
// half the issue slots (measured: 2.0 packed against 2 x 1.9 scalar sums per clock and SM), and
// issue slots bound the passes: 1024^2, 8 waves, row step 36.1 -> 31.9 us, column step 45.2 -> 40.5,
// the same bits.
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a * conj(b)
__device__ __forceinline__ float2 cmulc(float2 a, float2 b)
{
    return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
// a * conj(b), rounded as conj(cmul(conj(a), b)) is: an inverse transform with these products gives
// the bits of a forward one between two conjugations
__device__ __forceinline__ float2 cmulc_mirror(float2 a, float2 b)
{
    return make_float2(fmaf(a.x, b.x, __fmul_rn(a.y, b.y)), fmaf(-a.x, b.y, __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }

// Twiddle multiply d * (hi + lo) with the twiddle carried to about 48 bits.  Rounding a
// twiddle to one float is a fixed error of the transform operator; applied the same way at
// every slice of a crystal it adds up coherently (about 6e-5 relative after 240 slices at
// 1024^2, against 5e-6 with the split).  The low part enters through an FMA chain:
// re = vx hx - vy hy + (vx lx - vy ly), im = vx hy + vy hx + (vx ly + vy lx).  (Scalar:
// packing these products needs exchanged or doubled parts of d, which cost what they save.)
__device__ __forceinline__ float2 cmul_split(float2 d, float2 hi, float2 lo)
{
    const float cre = fmaf(d.x, lo.x, -(d.y * lo.y));
    const float cim = fmaf(d.x, lo.y, d.y * lo.x);
    return make_float2(fmaf(d.x, hi.x, fmaf(-d.y, hi.y, cre)), fmaf(d.x, hi.y, fmaf(d.y, hi.x, cim)));
}
__device__ __forceinline__ float2 cmulc_split(float2 d, float2 hi, float2 lo)
{
    return cmul_split(d, make_float2(hi.x, -hi.y), make_float2(lo.x, -lo.y));
}

// Multiply by W_64^m (DIR < 0) or its conjugate (DIR > 0); m is a compile-time
// constant once the callers are unrolled.
template <int DIR>
__device__ __forceinline__ float2 tw_apply(float2 d, int m)
{
    if (m == 0) return d;
    if (m == 16) return DIR < 0 ? make_float2(d.y, -d.x) : make_float2(-d.y, d.x);
    if (m == 8 || m == 24) {
        // W_64^8 = (1 - i)/sqrt2 and W_64^24 = (-1 - i)/sqrt2 (their conjugates for DIR > 0): a sum
        // and a difference of the two parts, each scaled by 1/sqrt2 carried as hi + lo
        const float hs = c_cos32.hi[8], ls = c_cos32.lo[8];
        float re, im;
        if (DIR < 0) {
            re = (m == 8) ? d.x + d.y : d.y - d.x;
            im = (m == 8) ? d.y - d.x : -(d.x + d.y);
        } else {
            re = (m == 8) ? d.x - d.y : -(d.x + d.y);
            im = (m == 8) ? d.x + d.y : d.x - d.y;
        }
        const float2 r = make_float2(re, im);
        return __ffma2_rn(r, make_float2(hs, hs), __fmul2_rn(r, make_float2(ls, ls)));
    }
    return DIR < 0 ? cmul_split(d, tw64_hi(m), tw64_lo(m)) : cmulc_split(d, tw64_hi(m), tw64_lo(m));
}

template <int E>
__host__ __device__ constexpr int brev(int k)
{
    int r = 0;
    for (int b = 1; b < E; b <<= 1) {
        r = (r << 1) | (k & 1);
        k >>= 1;
    }
    return r;
}

// multiply by -i (DIR < 0) or +i (DIR > 0)
template <int DIR>
__device__ __forceinline__ float2 mul_mi(float2 d)
{
    return DIR < 0 ? make_float2(d.y, -d.x) : make_float2(-d.y, d.x);
}

// In-register E-point DFT, E a power of two <= 64, by radix-4 decimation in frequency (a final
// radix-2 stage when log2 E is odd).  A radix-4 step is two radix-2 stages with their twiddles
// combined (W^(j+len/4) = -i W^j and W^j W^2j = W^3j), so it needs three twiddle products per four points
// instead of four, and most of its twiddles are trivial or eighth-turn.  Output in bit-reversed
// order, as the radix-2 form: after the call a[brev<E>(k)] holds X[k].
template <int E, int DIR>
__device__ __forceinline__ void dft_reg(float2 (&a)[E])
{
    // radix-4 steps, each equal to two radix-2 decimation-in-frequency stages (same output order):
    // x0..x3 at j, j+q, j+2q, j+3q become (x0+x2)+(x1+x3), ((x0+x2)-(x1+x3)) W^2j,
    // ((x0-x2) -+ i (x1-x3)) W^j, ((x0-x2) +- i (x1-x3)) W^3j with W = W_len (forward: -i first)
#pragma unroll
    for (int len = E; len >= 4; len >>= 2) {
        const int q = len >> 2;
#pragma unroll
        for (int base = 0; base < E; base += len) {
#pragma unroll
            for (int j = 0; j < q; j++) {
                const float2 x0 = a[base + j], x1 = a[base + j + q], x2 = a[base + j + 2 * q], x3 = a[base + j + 3 * q];
                // t3 exchanges the parts of x1 - x3, so the sums with it are scalar
                const float2 t0 = cadd(x0, x2), t1 = csub(x0, x2), t2 = cadd(x1, x3), t3 = mul_mi<DIR>(csub(x1, x3));
                const int m = j * (64 / len);
                a[base + j] = cadd(t0, t2);
                a[base + j + q] = tw_apply<DIR>(csub(t0, t2), (2 * m) & 63);
                a[base + j + 2 * q] = tw_apply<DIR>(make_float2(t1.x + t3.x, t1.y + t3.y), m);
                a[base + j + 3 * q] = tw_apply<DIR>(make_float2(t1.x - t3.x, t1.y - t3.y), (3 * m) & 63);
            }
        }
    }
    // a remaining radix-2 stage when log2(E) is odd
    constexpr int LOG = (E >= 64) ? 6 : (E >= 32) ? 5 : (E >= 16) ? 4 : (E >= 8) ? 3 : (E >= 4) ? 2 : 1;
    if constexpr (LOG % 2 == 1) {
#pragma unroll
        for (int base = 0; base < E; base += 2) {
            const float2 u = a[base], v = a[base + 1];
            a[base] = cadd(u, v);
            a[base + 1] = csub(u, v);
        }
    }
}

// Team transform.  On entry v[j] = x[g + G j]; on exit v[j] = X[g + G j].
// `tw` is the shared table W_N^(g k1) at tw[k1 * G + g] (one of the dithered sets: the
// engine's slices take the sets in turn, see kTwSets).  `scr(k1, g)` returns
// the shared-memory slot for the transpose; `sync()` orders the team's shared
// accesses (a warp barrier when the team is inside one warp, a block barrier
// otherwise).  DIR: -1 forward, +1 inverse, +2 inverse with cmulc_mirror's products (the slice steps).
template <int N, int G, int DIR, class Scr, class Sync>
__device__ __forceinline__ void team_fft(float2 (&v)[N / G], int g, const float2* __restrict__ tw, Scr scr,
                                         Sync sync)
{
    constexpr int E = N / G;
    static_assert(E >= G && E % G == 0, "team layout needs E >= G");
    dft_reg<E, DIR>(v);
#pragma unroll
    for (int k1 = 1; k1 < E; k1++) {
        const float2 w = tw[k1 * G + g];
        float2& x = v[brev<E>(k1)];
        x = DIR < 0 ? cmul(x, w) : DIR == 2 ? cmulc_mirror(x, w) : cmulc(x, w);
    }
    sync();
#pragma unroll
    for (int k1 = 0; k1 < E; k1++) *scr(k1, g) = v[brev<E>(k1)];
    sync();
    constexpr int M = E / G;
#pragma unroll
    for (int m = 0; m < M; m++) {
        float2 u[G];
#pragma unroll
        for (int q = 0; q < G; q++) u[q] = *scr(g + G * m, q);
        dft_reg<G, DIR>(u);
#pragma unroll
        for (int k2 = 0; k2 < G; k2++) v[m + M * k2] = u[brev<G>(k2)];
    }
}

// ---------------------------------------------------------------------------
// 2048 points on a team of 64 threads, 32 points each.  The two-level scheme above needs 64 points per
// thread, which leaves room for 8 warps per SM; this one runs 16 and pays half a transpose and one
// twiddle layer more.  3 waves of 2048^2: row step 78.0 -> 64.7 us, column step 108 -> 98, both in turn
// 210 -> 162; one wave 73.9 -> 55.1; the same error against 64 bits (2.1e-7 per slice, 3.87e-6 after
// 240; forward calls of 2048 x 128 over 48 inputs 2.38e-7 and 2.37e-7).  2048 = 32 x 8 x 8:
//   1. thread g holds x[g + 64 j] (j < 32): 32-point DFT over j, twiddle W_2048^(g k1);
//   2. transpose (k1, g) so that thread t holds k1 = t mod 32 and, of g = 8 a + b, every a for the
//      four b = t / 32 + 2 m: 8-point DFTs over a, twiddle W_64^(b c);
//   3. threads t and t xor 32 share k1: each gives the other the half of its values whose c has the
//      other's parity, then holds every b for c = t / 32 + 2 m: 8-point DFTs over b give
//      X[k1 + 32 c + 256 d] = X[t + 64 (m + 4 d)], the input's distribution.
// `scr(k1, g)` is the transpose's slot, `xch(q, t)` a slot of the exchange (q < 16, may overlap scr);
// `sync()` orders the 64 threads.
// ---------------------------------------------------------------------------
// the twiddles W_64^(b c) of the four b = P + 2 m, carried as hi + lo
template <int P, int DIR>
__device__ __forceinline__ void team64_twiddle(float2 (&u)[4][8])
{
#pragma unroll
    for (int m = 0; m < 4; m++)
#pragma unroll
        for (int c = 1; c < 8; c++) u[m][brev<8>(c)] = tw_apply<DIR>(u[m][brev<8>(c)], ((P + 2 * m) * c) & 63);
}
template <int DIR, class Scr, class Xch, class Sync>
__device__ __forceinline__ void team64_fft(float2 (&v)[32], int t, const float2* __restrict__ tw, Scr scr, Xch xch,
                                           Sync sync)
{
    constexpr int D = DIR < 0 ? -1 : 1;
    dft_reg<32, D>(v);
#pragma unroll
    for (int k1 = 1; k1 < 32; k1++) {
        const float2 w = tw[k1 * 64 + t];
        float2& x = v[brev<32>(k1)];
        x = DIR < 0 ? cmul(x, w) : cmulc_mirror(x, w);
    }
    sync();
#pragma unroll
    for (int k1 = 0; k1 < 32; k1++) *scr(k1, t) = v[brev<32>(k1)];
    sync();
    const int k1 = t & 31, p = t >> 5;
    float2 u[4][8];
#pragma unroll
    for (int m = 0; m < 4; m++)
#pragma unroll
        for (int a = 0; a < 8; a++) u[m][a] = *scr(k1, 8 * a + 2 * m + p);
#pragma unroll
    for (int m = 0; m < 4; m++) dft_reg<8, D>(u[m]);
    if (p == 0) team64_twiddle<0, D>(u);
    else team64_twiddle<1, D>(u);
    sync();
    // u[m][brev(c)] is value (b = p + 2 m, c); give those with c of the other parity
#pragma unroll
    for (int m = 0; m < 4; m++)
#pragma unroll
        for (int i = 0; i < 4; i++) *xch(4 * m + i, t) = p == 0 ? u[m][brev<8>(2 * i + 1)] : u[m][brev<8>(2 * i)];
    sync();
    // w[b] for c = p + 2 i: the own b = p + 2 m and the partner's b = 1 - p + 2 m
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float2 w[8];
#pragma unroll
        for (int m = 0; m < 4; m++) {
            const float2 own = p == 0 ? u[m][brev<8>(2 * i)] : u[m][brev<8>(2 * i + 1)];
            const float2 oth = *xch(4 * m + i, t ^ 32);
            w[2 * m] = p == 0 ? own : oth;
            w[2 * m + 1] = p == 0 ? oth : own;
        }
        dft_reg<8, D>(w);
#pragma unroll
        for (int d = 0; d < 8; d++) v[i + 4 * d] = w[brev<8>(d)];
    }
}

// ---------------------------------------------------------------------------
// Short steps for small batches: N = 512, 256 or 128 points on T = N / 8 threads, 8 points each.  A
// batch of one or two waves leaves most of the GPU idle with 16 or 32 points per thread, and a step
// takes as long as one thread's chain of operations; this form has a quarter of the chain and four
// times the threads, for one transpose more.  N = 8 x RA x RB with T = RA RB:
//   1. thread t holds x[t + T j]: 8-point DFT over j, twiddle W_N^(t k1);
//   2. transpose; k1 = t mod 8 and, of t' = RB a + b, every a: RA-point DFTs, twiddle W_T^(b c);
//   3. transpose; every b of a c: RB-point DFTs give X[k1 + 8 c + 8 RA d], the input's distribution.
// Both twiddles are carried as hi + lo (`tw`: N entries at [k1][t], then T at [b][c]).
// Per slice of one wave, chained: 512^2 10.6 -> 6.4 us, 256^2 5.9 -> 5.2, 128^2 6.3 -> 4.7; two waves
// 512^2 12.3 -> 9.2; but four 15.2 -> 16.4, and eight of 256^2 8.6 -> 9.3.
// ---------------------------------------------------------------------------
template <int DIR>
__device__ __forceinline__ float2 short_twiddle(float2 x, float4 w)
{
    const float2 hi = make_float2(w.x, w.y), lo = make_float2(w.z, w.w);
    return DIR < 0 ? cmul_split(x, hi, lo) : cmulc_split(x, hi, lo);
}
template <int N, int DIR, class Scr, class Sync>
__device__ __forceinline__ void short_fft(float2 (&v)[8], int t, const float4* __restrict__ tw, Scr scr, Sync sync)
{
    using S = ShortCfg<N>;
    constexpr int T = S::T, RA = S::RA, RB = S::RB, MA = 8 / RA, MB = 8 / RB;
    dft_reg<8, DIR>(v);
#pragma unroll
    for (int k1 = 1; k1 < 8; k1++) {
        v[brev<8>(k1)] = short_twiddle<DIR>(v[brev<8>(k1)], __ldg(tw + k1 * T + t));
    }
    sync();
#pragma unroll
    for (int k1 = 0; k1 < 8; k1++) *scr(k1, t) = v[brev<8>(k1)];
    sync();
    // this thread: k1 = t mod 8, and of t' = RB a + b every a for b = t / 8 + (T / 8) m
    const int k1 = t & 7, q = t >> 3;
    float2 u[MA][RA];
#pragma unroll
    for (int m = 0; m < MA; m++)
#pragma unroll
        for (int a = 0; a < RA; a++) u[m][a] = *scr(k1, RB * a + q + (T / 8) * m);
#pragma unroll
    for (int m = 0; m < MA; m++) {
        dft_reg<RA, DIR>(u[m]);
#pragma unroll
        for (int c = 1; c < RA; c++) {
            float2& x = u[m][brev<RA>(c)];
            x = short_twiddle<DIR>(x, __ldg(tw + N + (q + (T / 8) * m) * RA + c));
        }
    }
    sync();
#pragma unroll
    for (int m = 0; m < MA; m++)
#pragma unroll
        for (int c = 0; c < RA; c++) *scr(k1, RB * c + q + (T / 8) * m) = u[m][brev<RA>(c)];
    sync();
    // every b for c = t / 8 + (T / 8) m: X[k1 + 8 c + 8 RA d] = X[t + T (m + MB d)]
#pragma unroll
    for (int m = 0; m < MB; m++) {
        float2 w[RB];
#pragma unroll
        for (int b = 0; b < RB; b++) w[b] = *scr(k1, RB * (q + (T / 8) * m) + b);
        dft_reg<RB, DIR>(w);
#pragma unroll
        for (int d = 0; d < RB; d++) v[m + MB * d] = w[brev<RB>(d)];
    }
}

}  // namespace msb
