// Point coordinates and exponential-of-semicircle kernel values on the
// oversampled theta / phi torus, shared by the interpolation and spreading
// kernels (nufft.cu, spread_bins.cu).
#pragma once
#include "common.cuh"
#include "df.cuh"

namespace cunusht {

constexpr int NU_TPB = 256;
constexpr int MAXW = 16;

template <typename T> __device__ __forceinline__ T es_kernel(T z, T beta) {
    const T q = (T)1 - z * z;
    return q > (T)0 ? exp(beta * (sqrt(q) - (T)1)) : (T)0;
}

struct PointCoords {
    int r0;  // first fine row (relative to n_lo)
    int p0;  // first fine column (may be negative / >= Npf: wrap)
    double ft, fp;  // (n0 - t), (p0 - p): offsets of the first tap
};

__device__ __forceinline__ PointCoords point_coords(double th, double ph, int Ntf, int Npf, int n_lo,
                                                    int nrows, int w) {
    PointCoords pc;
    // non-finite or far out-of-range coordinates are clamped so every index
    // below stays inside the grid (the result for such points is garbage-in)
    if (!isfinite(th)) th = 0.0;
    if (!isfinite(ph) || fabs(ph) > 1e12) ph = 0.0;
    double t = th * ((double)Ntf / TWOPI);
    t = fmin(fmax(t, -1.0), 0.5 * Ntf + 1.0);
    double p = ph * ((double)Npf / TWOPI);
    p -= floor(p * (1.0 / (double)Npf)) * (double)Npf;  // Npf a power of two: exact
    p = fmin(fmax(p, 0.0), (double)Npf);
    const double hw = 0.5 * w;
    const int n0 = (int)ceil(t - hw);
    const int p0 = (int)ceil(p - hw);
    pc.ft = (double)n0 - t;
    pc.fp = (double)p0 - p;
    int r0 = n0 - n_lo;
    r0 = r0 < 0 ? 0 : (r0 > nrows - w ? nrows - w : r0);  // stays in bounds for any input
    pc.r0 = r0;
    pc.p0 = p0;
    return pc;
}

// The same coordinates in double-float arithmetic, for the mixed-precision
// kernels: no FP64 instruction (GB300 issues FP64 at 1/64 of the FP32 rate,
// and point_coords' FP64 products, division, rounding and clamps made the
// interpolation kernel FP64-pipe bound).  theta and phi become double-floats
// on the integer pipe (df_from), are scaled by Ntf / 2 pi and Npf / 2 pi
// (1 / 2 pi as a double-float constant, Ntf and Npf powers of two), and the
// first taps and offsets follow as in point_coords: ceil of a normalised
// double-float is ceilf(h) unless h is an integer and l > 0, and the offsets
// n0 - t, p0 - p are formed exactly (|n0 - t.h| <= w / 2 + 1 is a multiple of
// ulp(t.h)) and renormalised.  Positions carry about 2^-47 of the grid size
// (6e-11 cells at 8192) instead of 2^-53.
struct PointCoordsDf {
    int r0;      // first fine row (relative to n_lo), clamped into the grid
    int p0;      // first fine column (may be negative / >= Npf: wrap)
    dfl ft, fp;  // (n0 - t), (p0 - p)
};

__device__ __forceinline__ float df_ceil(dfl x) {
    const float c = ceilf(x.h);
    return (c == x.h && x.l > 0.f) ? c + 1.f : c;
}

__device__ __forceinline__ PointCoordsDf point_coords_df(double th, double ph, int Ntf, int Npf, int n_lo,
                                                         int nrows, int w) {
    const dfl inv2pi{0x1.45f306p-3f, 0x1.b93910p-28f};  // 1 / 2 pi
    dfl a = df_from(th), b = df_from(ph);
    // non-finite or far out-of-range coordinates are clamped so every index
    // below stays inside the grid (the result for such points is garbage-in)
    if (!isfinite(a.h) || !isfinite(a.l)) a = dfl{0.f, 0.f};
    if (!isfinite(b.h) || !isfinite(b.l) || fabsf(b.h) > 1e12f) b = dfl{0.f, 0.f};
    dfl t = df_scale(df_mul(a, inv2pi), (float)Ntf);
    const float thi = 0.5f * (float)Ntf + 1.f;
    if (t.h < -1.f) t = dfl{-1.f, 0.f};
    else if (t.h > thi) t = dfl{thi, 0.f};
    dfl p = df_scale(df_mul(b, inv2pi), (float)Npf);
    const float k = floorf(p.h / (float)Npf);  // Npf a power of two: exact quotient
    p = df_add(p, dfl{-k * (float)Npf, 0.f});
    if (p.h < 0.f) p = df_add(p, dfl{(float)Npf, 0.f});  // p.h an integer multiple of Npf with p.l < 0
    if (p.h < 0.f) p = dfl{0.f, 0.f};
    else if (p.h > (float)Npf) p = dfl{(float)Npf, 0.f};
    const float hw = 0.5f * (float)w;
    const float n0 = df_ceil(df_add(t, dfl{-hw, 0.f}));
    const float q0 = df_ceil(df_add(p, dfl{-hw, 0.f}));
    PointCoordsDf pc;
    pc.ft = df_fast(n0 - t.h, -t.l);  // |n0 - t.h| >= w / 2 - 1 > |t.l|
    pc.fp = df_fast(q0 - p.h, -p.l);
    int r0 = (int)n0 - n_lo;
    r0 = r0 < 0 ? 0 : (r0 > nrows - w ? nrows - w : r0);  // stays in bounds for any input
    pc.r0 = r0;
    pc.p0 = (int)q0;
    return pc;
}

__device__ __forceinline__ void load_point(const double *loc, long long j, long long npts, int layout,
                                           double &th, double &ph) {
    if (layout == 0) {
        th = loc[2 * j];
        ph = loc[2 * j + 1];
    } else {
        th = loc[j];
        ph = loc[npts + j];
    }
}

// FP32 kernel value from the cancellation-free exponent
// beta (sqrt(1 - z^2) - 1) = -beta z^2 / (1 + sqrt(1 - z^2))
__device__ __forceinline__ float es_kernel_acc(float z, float beta) {
    const float q = 1.f - z * z;
    if (q <= 0.f) return 0.f;
    const float r = sqrtf(q);
    return expf(-beta * (z * z) / (1.f + r));
}

// 2^(j / 128) as double-floats: the table of Tang's exponential (ACM TOMS 15, 144, 1989)
__device__ const float2 ES_EXP2[128] = {
    {0x1.0p+0f, 0x0.0p+0f}, {0x1.0163dap+0f, 0x1.3f6666p-25f}, {0x1.02c9a4p+0f, -0x1.887fap-28f},
    {0x1.04315ep+0f, 0x1.0dcffp-25f}, {0x1.059b0ep+0f, -0x1.9d4f52p-25f}, {0x1.0706b2p+0f, 0x1.3bbedcp-25f},
    {0x1.087452p+0f, -0x1.e2990ep-26f}, {0x1.09e3ecp+0f, 0x1.58de7p-25f}, {0x1.0b5586p+0f, 0x1.9f3122p-25f},
    {0x1.0cc922p+0f, 0x1.6e48fep-25f}, {0x1.0e3ec4p+0f, -0x1.a585ccp-25f}, {0x1.0fb66ap+0f, 0x1.ffda64p-25f},
    {0x1.11301ep+0f, -0x1.fdb496p-25f}, {0x1.12abdcp+0f, 0x1.b0c73p-30f}, {0x1.1429aap+0f, 0x1.d525bcp-25f},
    {0x1.15a98cp+0f, 0x1.14b1cap-25f}, {0x1.172b84p+0f, -0x1.c15742p-27f}, {0x1.18af94p+0f, -0x1.dcdc86p-26f},
    {0x1.1a35bep+0f, 0x1.6df96ep-25f}, {0x1.1bbe08p+0f, 0x1.011734p-26f}, {0x1.1d4874p+0f, -0x1.d2e8cap-25f},
    {0x1.1ed502p+0f, 0x1.7e6c8ep-27f}, {0x1.2063b8p+0f, 0x1.0c519ap-25f}, {0x1.21f49ap+0f, -0x1.d0446ep-25f},
    {0x1.2387a6p+0f, 0x1.ceac48p-25f}, {0x1.251ce4p+0f, 0x1.f654c8p-25f}, {0x1.26b456p+0f, 0x1.789f38p-26f},
    {0x1.284dfep+0f, 0x1.f5638p-28f}, {0x1.29e9ep+0f, -0x1.5c0424p-25f}, {0x1.2b87fep+0f, -0x1.e4a4cep-25f},
    {0x1.2d285ap+0f, 0x1.b900c2p-26f}, {0x1.2ecafap+0f, 0x1.27c5eap-25f}, {0x1.306fep+0f, 0x1.4636e2p-25f},
    {0x1.32171p+0f, -0x1.d993e8p-27f}, {0x1.33c08cp+0f, -0x1.b37d2p-25f}, {0x1.356c56p+0f, -0x1.b5803cp-30f},
    {0x1.371a74p+0f, -0x1.18aac6p-25f}, {0x1.38cae6p+0f, 0x1.a0bb0cp-25f}, {0x1.3a7db4p+0f, -0x1.634c02p-25f},
    {0x1.3c32dcp+0f, 0x1.89d472p-27f}, {0x1.3dea64p+0f, 0x1.824684p-25f}, {0x1.3fa45p+0f, 0x1.2b2006p-26f},
    {0x1.4160a2p+0f, 0x1.f72e2ap-28f}, {0x1.431f5ep+0f, -0x1.abd5dap-26f}, {0x1.44e086p+0f, 0x1.8624b4p-30f},
    {0x1.46a41ep+0f, 0x1.a3a00ap-25f}, {0x1.486a2cp+0f, -0x1.47d866p-25f}, {0x1.4a32bp+0f, -0x1.e50584p-25f},
    {0x1.4bfdaep+0f, -0x1.593abcp-25f}, {0x1.4dcb2ap+0f, -0x1.8088bcp-26f}, {0x1.4f9b28p+0f, -0x1.2c5a6cp-25f},
    {0x1.516daap+0f, 0x1.67b32p-27f}, {0x1.5342b6p+0f, -0x1.2c561p-25f}, {0x1.551a4cp+0f, 0x1.4bb242p-25f},
    {0x1.56f474p+0f, -0x1.295b04p-25f}, {0x1.58d12ep+0f, -0x1.6d07p-25f}, {0x1.5ab07ep+0f, -0x1.5bd5ecp-27f},
    {0x1.5c9268p+0f, 0x1.4b28d6p-25f}, {0x1.5e76f2p+0f, -0x1.4a5bd6p-25f}, {0x1.605e1cp+0f, -0x1.a248fep-26f},
    {0x1.6247ecp+0f, -0x1.f8b55p-25f}, {0x1.643464p+0f, -0x1.66679cp-25f}, {0x1.662388p+0f, 0x1.2a9112p-27f},
    {0x1.68155ep+0f, -0x1.766ad2p-25f}, {0x1.6a09e6p+0f, 0x1.9fcef4p-26f}, {0x1.6c0128p+0f, -0x1.5e84a8p-25f},
    {0x1.6dfb24p+0f, -0x1.cd72e8p-27f}, {0x1.6ff7ep+0f, -0x1.ab9aep-26f}, {0x1.71f75ep+0f, 0x1.1d8beep-25f},
    {0x1.73f9a4p+0f, 0x1.14b02ep-25f}, {0x1.75feb6p+0f, -0x1.37b306p-25f}, {0x1.780694p+0f, 0x1.fbcba8p-25f},
    {0x1.7a1148p+0f, -0x1.829fdp-25f}, {0x1.7c1edp+0f, 0x1.30c132p-28f}, {0x1.7e2f34p+0f, -0x1.261634p-25f},
    {0x1.804276p+0f, -0x1.783cbep-25f}, {0x1.82589ap+0f, -0x1.accc7cp-26f}, {0x1.8471a4p+0f, 0x1.88f1ecp-26f},
    {0x1.868d9ap+0f, -0x1.2edb44p-26f}, {0x1.88ac7ep+0f, -0x1.9d665ap-26f}, {0x1.8ace54p+0f, 0x1.15506ep-27f},
    {0x1.8cf322p+0f, -0x1.29576ep-25f}, {0x1.8f1aeap+0f, -0x1.baa232p-26f}, {0x1.9145bp+0f, 0x1.723ff8p-25f},
    {0x1.93737cp+0f, -0x1.e64744p-25f}, {0x1.95a44cp+0f, 0x1.790a42p-25f}, {0x1.97d82ap+0f, -0x1.0d8d84p-31f},
    {0x1.9a0f18p+0f, -0x1.e6bf08p-25f}, {0x1.9c4918p+0f, 0x1.51f848p-27f}, {0x1.9e8632p+0f, -0x1.873738p-26f},
    {0x1.a0c668p+0f, -0x1.2886a6p-26f}, {0x1.a309bep+0f, 0x1.8945a6p-25f}, {0x1.a5503cp+0f, -0x1.b83b54p-25f},
    {0x1.a799e2p+0f, -0x1.99e994p-25f}, {0x1.a9e6b6p+0f, -0x1.50c048p-25f}, {0x1.ac36bcp+0f, -0x1.606432p-31f},
    {0x1.ae89fap+0f, -0x1.a94b14p-26f}, {0x1.b0e072p+0f, 0x1.31b6ccp-25f}, {0x1.b33a2cp+0f, -0x1.ec3a82p-26f},
    {0x1.b59728p+0f, 0x1.bcab28p-25f}, {0x1.b7f77p+0f, -0x1.a09438p-25f}, {0x1.ba5b04p+0f, -0x1.ebdf36p-25f},
    {0x1.bcc1eap+0f, -0x1.f687c6p-25f}, {0x1.bf2c26p+0f, -0x1.0a387ep-26f}, {0x1.c199bep+0f, -0x1.3d56b2p-27f},
    {0x1.c40ab6p+0f, -0x1.7c2c98p-39f}, {0x1.c67f12p+0f, 0x1.cafa2ap-25f}, {0x1.c8f6dap+0f, -0x1.7f230ap-25f},
    {0x1.cb720ep+0f, -0x1.8837ccp-27f}, {0x1.cdf0b6p+0f, -0x1.54478p-25f}, {0x1.d072d4p+0f, 0x1.40f13p-25f},
    {0x1.d2f87p+0f, 0x1.01b13ep-25f}, {0x1.d5818ep+0f, -0x1.822dbcp-27f}, {0x1.d80e32p+0f, -0x1.26cf8ep-25f},
    {0x1.da9e6p+0f, 0x1.ed9942p-27f}, {0x1.dd322p+0f, -0x1.9fc974p-25f}, {0x1.dfc974p+0f, -0x1.908c94p-25f},
    {0x1.e26462p+0f, -0x1.614bdap-25f}, {0x1.e502eep+0f, 0x1.e2cffep-26f}, {0x1.e7a52p+0f, -0x1.0e2cep-26f},
    {0x1.ea4afap+0f, 0x1.52486cp-27f}, {0x1.ecf482p+0f, 0x1.b1ccfep-25f}, {0x1.efa1bep+0f, 0x1.cc2b44p-25f},
    {0x1.f252b4p+0f, -0x1.1288aep-25f}, {0x1.f50766p+0f, -0x1.246ebp-26f}, {0x1.f7bfdap+0f, 0x1.b397c2p-25f},
    {0x1.fa7c18p+0f, 0x1.9e90d8p-28f}, {0x1.fd3c22p+0f, 0x1.71ee3ep-25f}};

// The kernel value of the FP64 plans from double-float arithmetic on the FP32
// pipe: about 115 FP32 instructions for the value (absolute error up to 2.4e-14, of
// values up to 1) in place of about 33 FP64 instructions of exp, sqrt and
// products, each of which takes the issue time of 64 (2 FP64 lanes per SM and
// clock, measured).  z = (a + f) s with f the offset of the first tap and s =
// 2 / w; u = 1 - |z|, q = 1 - z^2 = u (2 - u); exponent y = -beta z^2 / (1 + sqrt(q)) (no
// cancellation); e^y = 2^k (2^(j/128)) e^f from the table T in shared memory with |f| < 0.0028, ln 2
// / 128 split so that the first two products are exact.  Used for widths up to
// ES_SPLIT_MAXW (eps >= 1e-10), where the kernel's own aliasing error is over a
// hundred times larger (with FP64 weights the errors of both transform types and of
// the gradients at eps 1e-7 to 1e-10 are the same to four digits); wider kernels
// keep the FP64 functions.
constexpr int ES_SPLIT_MAXW = 12;
struct EsParams {
    dfl s, nbeta;  // 2 / w, -beta
    float hw;      // w / 2
    float edge;    // derivatives: 1 - |z| up to here counts as 0
};
template <bool DERIV>
__device__ __forceinline__ dfl es_kernel_df(dfl f0, float a, const EsParams &E, const float2 *T, dfl *dlog) {
    const dfl x = df_add(dfl{a, 0.f}, f0);
    const dfl z = df_mul(x, E.s);
    const dfl z2 = df_mul(z, z);
    // u = 1 - |z| from the distance to the kernel's edge, exact: zero there (1 - z^2 of the
    // rounded z is up to 2e-15, where the derivative's 1 / sqrt(q) is at its largest)
    const dfl u = df_mul(df_add(dfl{E.hw, 0.f}, x.h < 0.f ? x : df_neg(x)), E.s);
    const dfl q = df_mul(u, df_add(dfl{2.f, 0.f}, df_neg(u)));
    if (DERIV) *dlog = dfl{0.f, 0.f};
    if (!(q.h > 0.f)) return dfl{0.f, 0.f};
    const float r0 = sqrtf(q.h);
    const dfl r = df_fast(r0, (fmaf(-r0, r0, q.h) + q.l) / (2.f * r0));
    dfl d = df_fast(1.f, r.h);
    d.l += r.l;
    const dfl bz = df_mul(E.nbeta, z2);
    const float i0 = 1.f / d.h;
    const float y0 = bz.h * i0;
    const dfl y = df_fast(y0, (fmaf(-y0, d.l, fmaf(-y0, d.h, bz.h)) + bz.l) * i0);
    if (DERIV && u.h > E.edge) {  // d log(psi) / dz = -beta z / sqrt(1 - z^2)
        const dfl n = df_mul(E.nbeta, z);
        const float g0 = n.h / r.h;
        *dlog = df_fast(g0, (fmaf(-g0, r.l, fmaf(-g0, r.h, n.h)) + n.l) / r.h);
    }
    const float k = rintf(y.h * 184.664965f);  // 128 / ln 2
    const float f1 = fmaf(-k, 0x1.62cp-8f, y.h);
    const dfl f2 = df_add_u(dfl{f1, y.l}, dfl{-(k * 0x1.214p-19f), -(k * 0x1.fbe8e8p-30f)});
    const dfl f = df_fast(f2.h, f2.l);
    const float qq = f.h * f.h;
    const float qe = fmaf(f.h, f.l + f.l, fmaf(f.h, f.h, -qq));
    const float c3 = f.h * qq * (1.f / 6.f);
    const float small = fmaf(0.5f, qe, fmaf(c3, 0.25f * f.h, c3)) + f.l;
    const dfl p = df_fast(f.h, 0.5f * qq);  // e^f - 1 = p.h + (p.l + small)
    const int ki = (int)k;
    const float2 t = T[ki & 127];
    const dfl tp = df_mul_u(dfl{t.x, t.y}, dfl{p.h, p.l + small});
    dfl v = df_fast(t.x, tp.h);
    v.l += tp.l + t.y;
    return df_scale(v, __int_as_float((127 + (ki >> 7)) << 23));  // k / 128 >= -54
}

// Fixed-point accumulation of the deterministic spreading: every cell sum is
// at most npts x (the largest rotated value, below 2 vmax) < 2^(E + 61), with
// lgn = ceil(log2(npts + 1)); values are added as round(v 2^-E) in int64.
__device__ __forceinline__ int fix_exp(float vmax, int lgn) {
    int ev = 0;
    if (vmax > 0.f) frexpf(2.f * vmax, &ev);
    return ev + lgn - 61;
}
__device__ __forceinline__ long long to_fix(float v, int E) { return __float2ll_rn(ldexpf(v, -E)); }
__device__ __forceinline__ long long to_fix(double v, int E) { return __double2ll_rn(ldexp(v, -E)); }

}  // namespace cunusht
