// FP64 Wigner-d recursion: starts and exponent rescaling (legendre.cu,
// legendre_tc64.cu, legendre_tc64_adj.cu), and the integer-pipe split of a
// double into seven 8-bit digits for the tensor-core forms.
#pragma once
#include "common.cuh"

namespace cunusht {

// Start of the recursion at l0 = max(m, s): (-1)^m 2^lg0 sh^(m+s) ch^|m-s| as
// mantissa (cur) times 2^e, e a non-positive multiple of 512 so that sin^m
// never underflows; values are accumulated once e has climbed back to 0
// (before that they are below 2^-312 and cannot contribute).
__device__ __forceinline__ void rec_start(double lg0, int m, int s, double sh, double ch,
                                          double &cur, double &prev, int &e) {
    prev = 0.0;
    double lg = lg0;
    bool zero = false;
    if (m + s > 0) {
        if (sh <= 0.0) zero = true;
        else lg += (double)(m + s) * log2(sh);
    }
    if (m != s) {
        if (ch <= 0.0) zero = true;
        else lg += (double)abs(m - s) * log2(ch);
    }
    if (zero) {
        cur = 0.0;
        e = 0;
        return;
    }
    int k = 0;
    if (lg < -400.0) k = (int)ceil((-400.0 - lg) / 512.0);
    e = -512 * k;
    cur = exp2(lg + 512.0 * (double)k);
    if (m & 1) cur = -cur;
}

#define REC_RESCALE(cur, prev, e)                                                        \
    if ((e) < 0 && fabs(cur) > 0x1p200) {                                               \
        (cur) *= 0x1p-512;                                                               \
        (prev) *= 0x1p-512;                                                              \
        (e) += 512;                                                                      \
    }

// ---------------------------------------------------------------- double-double (plan set-up)
// Pairs hi + lo of FP64 (about 106 bits; Dekker 1971, Knuth's TwoSum, FMA
// TwoProduct) for tables built once per plan, where rounding in FP64 would
// reach the results: the relative error of a start value is |log2| 2^-53, and
// that of c_l grows with the number of its factors.
struct dd {
    double h, l;
};
__device__ __forceinline__ dd dd_fast(double a, double b) {
    const double s = a + b;
    return dd{s, b - (s - a)};
}
__device__ __forceinline__ dd dd_add(dd a, dd b) {
    const double s = a.h + b.h, bb = s - a.h;
    return dd_fast(s, ((a.h - (s - bb)) + (b.h - bb)) + (a.l + b.l));
}
__device__ __forceinline__ dd dd_mul(dd a, dd b) {
    const double p = a.h * b.h;
    return dd_fast(p, fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h));
}
__device__ __forceinline__ dd dd_div(dd a, dd b) {
    const double q = a.h / b.h;
    const dd r = dd_add(a, dd_mul(dd{-q, 0.0}, b));
    return dd_fast(q, (r.h + r.l) / b.h);
}
__device__ __forceinline__ dd dd_sqrt(dd a) {  // a > 0
    const double q = sqrt(a.h);
    const dd r = dd_add(a, dd_mul(dd{-q, 0.0}, dd{q, 0.0}));
    return dd_fast(q, (r.h + r.l) / (2.0 * q));
}

// rec_start with log2 of the normalisation (lg0) and of sin, cos(theta / 2)
// (ls, lc; hi, lo pairs) summed in double-double: relative error of the start
// 2^-52 instead of about |lg| 2^-53.  zs, zc: sin / cos exactly zero.
__device__ __forceinline__ void rec_start_dd(double2 lg0, int m, int s, double2 ls, double2 lc, bool zs, bool zc,
                                             double &cur, double &prev, int &e) {
    prev = 0.0;
    cur = 0.0;
    e = 0;
    if ((m + s > 0 && zs) || (m != s && zc)) return;
    dd lg{lg0.x, lg0.y};
    if (m + s > 0) lg = dd_add(lg, dd_mul(dd{(double)(m + s), 0.0}, dd{ls.x, ls.y}));
    if (m != s) lg = dd_add(lg, dd_mul(dd{(double)abs(m - s), 0.0}, dd{lc.x, lc.y}));
    int k = 0;
    if (lg.h < -400.0) k = (int)ceil((-400.0 - lg.h) / 512.0);
    e = -512 * k;
    const double v = lg.h + 512.0 * (double)k;  // exact: both on the grid of lg.h, |v| <= 400 + 512
    const double r = rint(v);
    cur = scalbn(exp2(v - r) * (1.0 + lg.l * 0.69314718055994530942), (int)r);
    if (m & 1) cur = -cur;
}

// start at ring theta (side 0) or pi - theta of a pair
__device__ __forceinline__ void tc64_start(double2 lg0, int m, int s, RingLog q, int side, double &cur, double &prev,
                                           int &e) {
    const double2 a = make_double2(q.sh, q.sl), b = make_double2(q.ch, q.cl);
    if (side) rec_start_dd(lg0, m, s, b, a, isinf(b.x), isinf(a.x), cur, prev, e);
    else rec_start_dd(lg0, m, s, a, b, isinf(a.x), isinf(b.x), cur, prev, e);
}

// Coefficients alpha_l, gamma_l, beta_l of the double-float recursion of the
// mixed plans, laid out for the packed steps: windows of 128 l from l0 = max(m,
// s), window k of order m at woff[m] + k, twelve floats per pair of l (a_l.h,
// a_{l+1}.h, a_l.l, a_{l+1}.l, then gamma, then beta), zero from l = L on.
constexpr int CO_WIN = 64 * 12;  // floats per window
__device__ __forceinline__ void co_load(const float *__restrict__ com, int i, dfl &a, dfl &g, dfl &b) {
    const float *q = com + (i >> 1) * 12 + (i & 1);  // i = l - l0, com: the order's first window
    a = dfl{q[0], q[2]};
    g = dfl{q[4], q[6]};
    b = dfl{q[8], q[10]};
}

// 2^El > |mu_l| from the bound sqrt((2l + 1) / (4 pi)) / c_l
__device__ __forceinline__ int tc_bound_exp(float c, int l) {
    int e;
    frexpf(1.0001f * sqrtf((2.f * l + 1.f) * 0.0795774715459476679f) / c, &e);
    return e;
}

// ---------------------------------------------------------------- digits
// v = 2^Eb 2^-7 sum_{i<7} d_i 2^-8i with integer digits |d_i| <= 128: the
// fixed-point value X = v 2^(55 - Eb) (truncated; |v| < 2^Eb, so |X| <= 2^55)
// plus 0x80 in each of the seven low bytes, whose bytes are then the digits
// biased by 128 (d_6 lowest; d_0 = top 16 bits, 0 .. 256).  Sign, shift and
// bias run on the integer pipe: an FP64 instruction costs 32 of its
// instructions (2 lanes per SM and clock against 64, measured).  nb = 1030 +
// Eb - (exponent of the recursion value, a non-positive multiple of 512);
// zero and values below 2^(Eb - 55) give X = 0.
constexpr unsigned long long FIX_BIAS = 0x0080808080808080ull;
__device__ __forceinline__ unsigned long long fix55_biased(double v, int nb) {
    const int hi = __double2hiint(v);
    const unsigned lo = (unsigned)__double2loint(v);
    const unsigned n = min((unsigned)(nb - ((hi >> 20) & 0x7FF)), 63u);  // >= 8 for |v| < 2^Eb
    const unsigned mh = ((unsigned)hi & 0xFFFFFu) | 0x100000u;
    const unsigned long long M = ((unsigned long long)__funnelshift_l(lo, mh, 10) << 32) | (lo << 10);
    const long long s = (long long)(hi >> 31);
    return ((M >> n) ^ (unsigned long long)s) + (FIX_BIAS - (unsigned long long)s);
}

// ---------------------------------------------------------------- fixed-point recursion
// Past its turning point a ring's mu stays within a few binary orders of its
// bound, so the recursion can run in 64-bit fixed point on the integer pipes:
// U = mu 2^(62 - Es) with 2^Es > |mu| up to lmax, x in Q61, a in Q58 (a < 8), g
// and t = a x + g in Q60 (|t| < 4).  Products of 31-bit halves (three
// IMAD.WIDE each; the low x low term enters by its mean) leave an error of
// about one unit per step, 2^-62 of the bound or 2^-56 of the amplitude at
// lmax 2047, against 2^-54 of an FP64 step.  About 30 integer instructions per
// step and ring, digits included, at 64 lanes per SM and clock, in place of
// two FP64 instructions at 2.
struct alignas(16) FixCoef {
    int ah, al;    // a 2^58 = ah 2^31 + al
    long long g;   // g 2^60
};
__device__ __forceinline__ FixCoef fix_load(const FixCoef *p) {
    const int4 q = __ldg(reinterpret_cast<const int4 *>(p));
    return FixCoef{q.x, q.y, (long long)(((unsigned long long)(unsigned)q.w << 32) | (unsigned)q.z)};
}
// v 2^(62 - Eb) for |v| < 2^Eb, truncated
__device__ __forceinline__ long long fix62(double v, int Eb) {
    const int hi = __double2hiint(v);
    const unsigned n = min((unsigned)(1023 + Eb - ((hi >> 20) & 0x7FF)), 63u);  // >= 1
    const unsigned long long M =
        (((unsigned long long)(((unsigned)hi & 0xFFFFFu) | 0x100000u) << 32) | (unsigned)__double2loint(v)) << 10;
    const long long s = (long long)(hi >> 31);
    return (long long)((M >> n) ^ (unsigned long long)s) - s;
}
__device__ __forceinline__ FixCoef fix_coef(double a, double g) {
    const long long A = a < 8.0 ? fix62(a, 4) : 0;  // Q58
    return FixCoef{(int)(A >> 31), (int)(A & 0x7FFFFFFF), fabs(g) < 4.0 ? fix62(g, 2) : 0};
}
// rnd: FIX_ROUND, or 0 for a ring that stays zero (a rounding constant would grow where |t| > 2)
constexpr long long FIX_ROUND = (1LL << 28) + (1LL << 29);
__device__ __forceinline__ void fix_step(const FixCoef q, int xh, int xl, long long rnd, long long &U, long long &V) {
    const long long p = (long long)q.ah * xh;
    const long long cr = (long long)q.al * xh + ((long long)q.ah * xl + rnd);
    const long long T = (q.g + (p * 8)) + (cr >> 28);
    const int th = (int)(T >> 31), tl = (int)T & 0x7FFFFFFF, uh = (int)(U >> 31), ul = (int)U & 0x7FFFFFFF;
    const long long p2 = (long long)uh * th;
    const long long c2 = (long long)ul * th + ((long long)uh * tl + rnd);
    // modulo 2^64: t U may pass 2^63, mu_{l+1} does not
    const unsigned long long N = (((unsigned long long)p2 << 2) - (unsigned long long)V) + (unsigned long long)(c2 >> 29);
    V = U;
    U = (long long)N;
}
// Whether a ring may go over to fixed point at a chunk with digit exponent El:
// |mu| or |previous mu| at least 2^(Es - 9), a and |t| small enough from here
// on (both fall towards 2 and 2 |x|), the digits a right shift of U by 0 .. 7.
__device__ __forceinline__ bool fix_ready(double cur, double prev, int e, double a, double g, double x, int Es, int El) {
    const int ec = (__double2hiint(cur) >> 20) & 0x7FF, ep = (__double2hiint(prev) >> 20) & 0x7FF;
    return e == 0 && max(ec, ep) - 1023 >= Es - 9 && a < 7.5 && fabs(fma(a, x, g)) < 3.0 && El + 7 >= Es;
}

// digit K of the biased words of two values as packed fp16 (a low, b high):
// the bit pattern 0x6400 | (digit + 128) is 1024 + (digit + 128); minus 1152, exact
template <int K> __device__ __forceinline__ uint32_t digit_pair(unsigned long long a, unsigned long long b) {
    constexpr int by = (6 - K) & 3;  // byte of the 32-bit half that holds d_K
    const uint32_t wa = K <= 2 ? (uint32_t)(a >> 32) : (uint32_t)a;
    const uint32_t wb = K <= 2 ? (uint32_t)(b >> 32) : (uint32_t)b;
    uint32_t p, r;
    if constexpr (K == 0) p = __byte_perm(wa, wb, 0x7632) | 0x64006400u;
    else p = (__byte_perm(wa, wb, by | ((4 + by) << 8)) & 0x00FF00FFu) | 0x64006400u;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(p), "r"(0xE480E480u));
    return r;
}

}  // namespace cunusht
