// Legendre synthesis of the FP64 plans on the tensor cores (tcgen05): FP64
// recursion on the CUDA cores, contraction by exact integer digit products.
// Replaces the SHTns synthesis calls of the reference
// (cunusht/sht/GPU_sht_transformer.py:56-62, :88-97).
//
// GB300 issues FP64 at 2 lanes per SM and clock, so the FP64 pipe bounds the
// CUDA-core kernel (legendre.cu): 14 FP64 instructions per (l, m, ring pair)
// for spin s, 8 of them the contraction and 6 the two recursions (88.7 ms at
// lmax 2047 spin 2).  Here
//   * the recursion is rescaled, lambda_l = c_l mu_l with c_{l+1} = beta_l
//     c_{l-1}, to mu_{l+1} = (a_l x + g_l) mu_l - mu_{l-1}: 2 FP64
//     instructions per step and ring instead of 3 (c_l goes into the alm), and
//     past the turning point it runs in 64-bit fixed point without any
//     (rec64.cuh); a warp goes over when all its rings have;
//   * mu and the alm are split into seven 8-bit digits on the integer pipe
//     (rec64.cuh) and multiplied on the tensor cores,
//         mu = 2^El 2^-7 sum_i d_i 2^-8i,   c a = 2^Ea 2^-7 sum_j t_j 2^-8j,
//     El per 16 l from the bound sqrt((2l + 1) / (4 pi)) / c_l, Ea per window
//     and column from the largest |c a|.  The digits are exact in fp16,
//     their products of equal weight g = i + j <= 6 (28 of the 49 pairs, the
//     rest below 2^-56) are summed over 128 l in FP32 tensor memory: at most
//     7 x 128 products below 2^14, an integer below 2^24, so no rounding
//     occurs.  Per window the seven sums are combined in 64-bit integers and
//     added to FP64 accumulators (two fused multiply-adds per output).
// The products carry 2^-56 of the bounds and the sum over l rounds twice per
// 128 terms instead of once per term.
//
// lmax 2047 spin 2, one request: 9.7 ms (FP64 recursion throughout, one block
// of 512 rings per SM: 13.2 ms; two of 256: 12.3 ms; fixed point in half of the
// warps, to share the work between the FP64 and integer pipes: 9.9 ms).  At
// lmax 1023 spin 2 (1.39 ms): issue slots 55 %, ALU pipe 53 %, FP64 pipe 33 %,
// tensor pipe 7 %; long scoreboard and dependent issue lead the stalls.
//
// Layout as in legendre_tc.cu: one order m and 256 rings per block as two
// 128-row MMA tiles, two blocks per SM, one ring per thread (spin s: 128 pairs,
// both rings; spin 0: 256 pairs, the theta ring only), chunks of 8 l: A rows hold eight 16-byte
// K-cores (digit i, 8 l), the eighth zero, so a chunk is four MMA K-steps; B'
// rows (weight g, column) hold t_{g-i} at K-core i.  Two A / B' buffers with
// full (one arrival per ring warp) and empty (commit) mbarriers; the window
// records (k_tc64_records) arrive by bulk copy, the next one prefetched.
// Every wait is bounded; a block whose wait runs out sets bit 0 of the plan's
// status word, writes NaN to its rings (no caller polls that word), waits once
// more for its own copies and MMAs, frees its tensor memory and returns.
#include "common.cuh"
#include "kernels.cuh"
#include "rec64.cuh"
#include "tcgen05.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

namespace cunusht {

constexpr int T6_W = 128;                 // l window accumulated in tensor memory
constexpr int T6_KC = 8;                  // l per chunk
constexpr int T6_CPW = T6_W / T6_KC;      // chunks per window
constexpr int T6_ND = 7;                  // digits, and digit-product weights kept
constexpr int T6_NO = 4;                  // outputs per ring
constexpr int T6_NN = 32;                 // MMA N: 7 x 4 weights x outputs, padded
constexpr int T6_NT = 2;                  // 128-ring tiles per block
constexpr int T6_T = 128 * T6_NT;         // ring threads
constexpr int T6_BLOCK = T6_T + 32;       // + the MMA warp
constexpr int T6_TILE = 128 * 128;        // A tile: 128 rows x 8 K-cores x 16 bytes
constexpr int T6_SBO = 1024;              // 8-row group stride
constexpr int T6_ABUF = T6_NT * T6_TILE;
constexpr int T6_BBUF = T6_NN * 128;
constexpr int T6_TPS = T6_W + 8;          // digit-plane row stride (elements)
// window record: fp16 digit planes [7][4][TPS], double epilogue scales [2][4],
// mu exponents per 16 l, double2 (a, g) [W + 1] (zero past the window), FixCoef [W]
constexpr int T6_RSC = T6_ND * T6_NO * T6_TPS * 2;
constexpr int T6_REL = T6_RSC + 2 * T6_NO * 8;
constexpr int T6_RCO = T6_REL + 32;
constexpr int T6_RFX = T6_RCO + (T6_W + 1) * 16;
constexpr int T6_RSZ = T6_RFX + T6_W * 16;
constexpr int T6_OFF_B = 2 * T6_ABUF;
constexpr int T6_OFF_R = T6_OFF_B + 2 * T6_BBUF;
constexpr int T6_OFF_BAR = T6_OFF_R + 2 * T6_RSZ;   // full[2], empty[2], record[2]
constexpr int T6_OFF_TM = T6_OFF_BAR + 48;          // tensor-memory base, give-up flag, first chunk
constexpr int T6_BYTES = T6_OFF_TM + 16;
static_assert(T6_BYTES <= 227 * 1024, "dynamic shared memory of one block");
static_assert(T6_RCO % 16 == 0 && T6_RSZ % 16 == 0 && T6_OFF_R % 16 == 0, "bulk copies on 16 bytes");
static_assert(T6_OFF_BAR % 8 == 0, "mbarriers are 8-byte words");

// ---------------------------------------------------------------- plan tables
// Recursion factors as double-doubles: alpha_l = (l+1) sqrt((2l+1)(2l+3)) / d_l,
// gamma_l = alpha_l m s / (l (l+1)), beta_l = f_l / f_{l+1} sqrt((2l+3) / (2l-1))
// with f_l = sqrt((l^2 - m^2)(l^2 - s^2)) / l, d_l = (l+1) f_{l+1}.  The integers
// under the roots stay below 2^53 for l <= 16383 in each factor.
__device__ __forceinline__ dd tc64_sq(int l, int m, int s) {  // (l^2 - m^2)(l^2 - s^2)
    return dd_mul(dd{(double)((long long)l * l - (long long)m * m), 0.0},
                  dd{(double)((long long)l * l - (long long)s * s), 0.0});
}
__device__ __forceinline__ dd tc64_beta(int l, int m, int s) {
    dd n = dd_mul(tc64_sq(l, m, s), dd_mul(dd{(double)(l + 1) * (l + 1), 0.0}, dd{2.0 * l + 3.0, 0.0}));
    dd d = dd_mul(tc64_sq(l + 1, m, s), dd_mul(dd{(double)l * l, 0.0}, dd{2.0 * l - 1.0, 0.0}));
    return dd_sqrt(dd_div(n, d));
}
__device__ __forceinline__ dd tc64_alpha(int l, int m, int s) {
    const double lp = l + 1.0;
    return dd_sqrt(dd_div(dd_mul(dd{lp * lp, 0.0}, dd{(2.0 * l + 1.0) * (2.0 * l + 3.0), 0.0}), tc64_sq(l + 1, m, s)));
}

// beta_l of every (l, m) (l > l0) into b (hi, lo), one thread each
__global__ void k_tc64_beta(int L, int s, double2 *__restrict__ b) {
    const int m = blockIdx.y, l = m + blockIdx.x * blockDim.x + threadIdx.x;
    if (l > L) return;
    dd v{1.0, 0.0};
    if (l > max(m, s)) v = tc64_beta(l, m, s);
    b[almidx(L, m, m) - m + l] = make_double2(v.h, v.l);
}

// c_l of one order per thread, in place of beta_l: c_{l0} = 1, c_{l+1} = beta_l
// c_{l-1}; the chain of l0 + 1 starts at the factor k that makes the two chains
// meet at l = L, so that c (and the coefficients) vary smoothly there.
__global__ void k_tc64_scale(int L, int s, double2 *__restrict__ b) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m > L) return;
    const int l0 = max(m, s);
    double2 *c = b + (almidx(L, m, m) - m);
    dd c0{1.0, 0.0}, c1{1.0, 0.0};  // c_{l-1}, c_l
    for (int l = l0 + 1; l < L; ++l) {
        const dd c2 = dd_mul(dd{c[l].x, c[l].y}, c0);
        c0 = c1;
        c1 = c2;
    }
    dd k{1.0, 0.0};
    if (L > l0) k = ((L - l0) & 1) == 0 ? dd_div(c1, c0) : dd_div(c0, c1);
    c0 = dd{1.0, 0.0};
    c1 = k;
    if (l0 < L) {
        dd bl{c[l0 + 1].x, c[l0 + 1].y};
        c[l0 + 1] = make_double2(c1.h, c1.l);
        for (int l = l0 + 1; l < L; ++l) {
            const dd c2 = dd_mul(bl, c0);
            bl = dd{c[l + 1].x, c[l + 1].y};
            c[l + 1] = make_double2(c2.h, c2.l);
            c0 = c1;
            c1 = c2;
        }
    }
}

// a_l = alpha_l c_l / c_{l+1}, g_l = gamma_l c_l / c_{l+1} and c_l, rounded once
__global__ void k_tc64_coef(int L, int s, const double2 *__restrict__ c, double2 *__restrict__ ag,
                            double *__restrict__ cl, FixCoef *__restrict__ fx) {
    const int m = blockIdx.y, l = m + blockIdx.x * blockDim.x + threadIdx.x;
    if (l > L) return;
    const long long ix = almidx(L, m, m) - m + l;
    double2 v = make_double2(0.0, 0.0);
    if (l < L && l >= max(m, s)) {
        const dd a = dd_mul(tc64_alpha(l, m, s), dd_div(dd{c[ix].x, c[ix].y}, dd{c[ix + 1].x, c[ix + 1].y}));
        v.x = a.h;
        if (l > 0)
            v.y = dd_div(dd_mul(a, dd{(double)m * s, 0.0}), dd{(double)l * (l + 1), 0.0}).h;
    }
    ag[ix] = v;
    fx[ix] = fix_coef(v.x, v.y);
    cl[ix] = c[ix].x;
}

// El of every chunk of 16 l (from l0) of every order: entry 8 woff[m] + chunk
__global__ void k_tc64_chunk_exp(int L, int s, const double *__restrict__ cl, const int *__restrict__ woff,
                                 short *__restrict__ eb) {
    const int m = blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x;
    const int lb = max(m, s) + 16 * c;
    if (lb > L) return;
    const long long b = almidx(L, m, m) - m;
    int e = -1000;
    for (int l = lb; l <= min(lb + 15, L); ++l) e = max(e, tc_bound_exp((float)cl[b + l], l));
    eb[8 * (long long)woff[m] + c] = (short)e;
}

// Es of every order: 2^Es > |mu_l| for all its l
__global__ void k_tc64_order_exp(int L, int s, const int *__restrict__ woff, const short *__restrict__ eb,
                                 short *__restrict__ es) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m > L) return;
    int e = -1000;
    for (int c = 0, lb = max(m, s); lb <= L; ++c, lb += 16) e = max(e, (int)eb[8 * (long long)woff[m] + c]);
    es[m] = (short)e;
}

// Start states: per (m, side, pair) the first chunk of 16 l (from l0) in which
// mu exceeds 2^-64 of its bound at exponent 0, and the recursion state at its
// start, by the same steps as the kernels.  A ring's functions are below that
// while sin(theta) < m / l by a margin; a ring that never gets there has c0 =
// TC_NEVER.
__global__ void k_tc64_starts(int L, int spin, const double2 *__restrict__ lg0, int npairs,
                              const double *__restrict__ x, const RingLog *__restrict__ lsc,
                              const double2 *__restrict__ ag, double2 *__restrict__ v, short2 *__restrict__ ec) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2LL * npairs * (L + 1)) return;
    const int p = (int)(i % npairs);
    const long long ms = i / npairs;
    const int side = (int)(ms & 1), m = (int)(ms >> 1);
    const int l0 = max(m, spin);
    double cur, prev;
    int e;
    tc64_start(lg0[m], m, spin, lsc[p], side, cur, prev, e);
    const double xs = side ? -x[p] : x[p];
    const long long b = almidx(L, m, m) - m;
    const int nchk = l0 <= L ? (L - l0 + 16) / 16 : 0;
    int c = 0;
    for (; c < nchk; ++c) {
        const double c0 = cur, p0 = prev;
        const int e0 = e, lb = l0 + 16 * c;
        bool seen = false;
        for (int j = 0; j < 16 && lb + j <= L; ++j) {
            seen |= e == 0 && ((__double2hiint(cur) >> 20) & 0x7FF) > 1023 - 66;
            const double2 a = ag[b + lb + j];
            const double nxt = fma(fma(a.x, xs, a.y), cur, -prev);
            prev = cur;
            cur = nxt;
        }
        if (e < 0 && ((__double2hiint(cur) >> 20) & 0x7FF) > 1023 + 200) {
            cur *= 0x1p-512;
            prev *= 0x1p-512;
            e += 512;
        }
        if (seen) {
            cur = c0, prev = p0, e = e0;
            break;
        }
    }
    const bool never = c >= nchk || (cur == 0.0 && prev == 0.0);
    v[i] = make_double2(cur, prev);
    ec[i] = make_short2((short)(e / 512), never ? TC_NEVER : (short)c);
}

// ---------------------------------------------------------------- window records
// One block of 128 threads per (window k, order m), thread i for l = wb + i:
// the four alm combinations of legendre.cu times c_l, their column exponents
// and digit planes, the epilogue scales 2^(Ea - 14 - 24) and 2^(Ea - 14 - 48) (NaN when the window's column holds a non-finite value, so that it
// reaches every ring of the order), the mu exponents and the window's
// recursion coefficients.  Spin 0: the columns are the alm split by the parity
// of l + m, (E re, E im, O re, O im).
__global__ void __launch_bounds__(T6_W)
    k_tc64_records(int L, int spin, const double2 *__restrict__ G, const double2 *__restrict__ C,
                   const double *__restrict__ lfac, const double2 *__restrict__ ag, const double *__restrict__ cl,
                   const int *__restrict__ woff, unsigned char *__restrict__ rec) {
    __shared__ int s_mx[T6_W / 32][T6_NO];
    __shared__ int s_ea[T6_NO];
    const int m = blockIdx.y, k = blockIdx.x;
    if (k >= woff[m + 1] - woff[m]) return;
    const int wb = max(m, spin) + k * T6_W, cnt = min(T6_W, L - wb + 1);
    unsigned char *R = rec + (size_t)(woff[m] + k) * T6_RSZ;
    const int i = threadIdx.x, lane = i & 31, warp = i >> 5;
    const int l = wb + i;
    const long long ix = almidx(L, m, m) - m + l;
    double2 *co = reinterpret_cast<double2 *>(R + T6_RCO);
    const double2 agi = i < cnt ? ag[ix] : make_double2(0.0, 0.0);
    co[i] = agi;
    reinterpret_cast<FixCoef *>(R + T6_RFX)[i] = fix_coef(agi.x, agi.y);
    if (i == 0) co[T6_W] = make_double2(0.0, 0.0);
    double v[T6_NO] = {0.0, 0.0, 0.0, 0.0};
    int eb = -1000;
    if (i < cnt) {
        const double c = cl[ix], f = (lfac ? lfac[l] : 1.0) * c;
        const bool odd = (l + m) & 1;
        const double2 g = G[ix];
        eb = tc_bound_exp((float)c, l);
        if (spin == 0) {
            v[odd ? 2 : 0] = f * g.x;
            v[odd ? 3 : 1] = f * g.y;
        } else {
            const double2 cc = C ? C[ix] : make_double2(0.0, 0.0);
            const double par = odd ? -f : f;
            v[0] = f * (g.x - cc.y);
            v[1] = f * (g.y + cc.x);
            v[2] = par * (g.x + cc.y);
            v[3] = par * (cc.x - g.y);
        }
    }
    // digit exponent of mu over the chunk of 16 l, 2^El > |mu_l|; the alm take the factor 2^El, so
    // that c_l, which falls by a factor 3 over the first l of an order, costs no digit
#pragma unroll
    for (int sft = 8; sft > 0; sft >>= 1) eb = max(eb, __shfl_xor_sync(0xffffffffu, eb, sft));
    if (i % 16 == 0) reinterpret_cast<int *>(R + T6_REL)[i / 16] = eb;
#pragma unroll
    for (int o = 0; o < T6_NO; ++o) {
        if (i < cnt) v[o] = scalbn(v[o], eb);
        const int ex = __reduce_max_sync(0xffffffffu, (__double2hiint(v[o]) >> 20) & 0x7FF);
        if (lane == 0) s_mx[warp][o] = ex;
    }
    __syncthreads();
    if (i < T6_NO) {
        int ex = 0;
#pragma unroll
        for (int w = 0; w < T6_W / 32; ++w) ex = max(ex, s_mx[w][i]);
        double *sc = reinterpret_cast<double *>(R + T6_RSC);
        const int ea = max(ex, 64) - 1022;  // 2^ea > |v| (zero columns: digits 0)
        const bool bad = ex == 0x7FF;
        s_ea[i] = ea;
        sc[i] = bad ? nan("") : scalbn(1.0, ea - 14 - 24);
        sc[T6_NO + i] = bad ? nan("") : scalbn(1.0, ea - 14 - 48);
    }
    __syncthreads();
    unsigned short *tp = reinterpret_cast<unsigned short *>(R);
#pragma unroll
    for (int o = 0; o < T6_NO; ++o) {
        const unsigned long long X = fix55_biased(v[o], 1030 + s_ea[o]);
        const uint32_t d[7] = {digit_pair<0>(X, X), digit_pair<1>(X, X), digit_pair<2>(X, X), digit_pair<3>(X, X),
                               digit_pair<4>(X, X), digit_pair<5>(X, X), digit_pair<6>(X, X)};
#pragma unroll
        for (int j = 0; j < T6_ND; ++j) tp[(j * T6_NO + o) * T6_TPS + i] = (unsigned short)d[j];
    }
}

// ---------------------------------------------------------------- synthesis
template <bool S0>
__global__ void __launch_bounds__(T6_BLOCK, 2)
    k_leg_synth_tc64(int L, int spin, const unsigned char *__restrict__ rec, const int *__restrict__ woff,
                     const double2 *__restrict__ lg0, int npairs, const double *__restrict__ px,
                     const RingLog *__restrict__ lsc, const int *__restrict__ prn, const int *__restrict__ prs, const double2 *__restrict__ stv, const short2 *__restrict__ ste,
                     int st_ld, const short *__restrict__ es, double2 *__restrict__ H, int ldH, int wlim, int *status) {
    constexpr int T = T6_T;
    extern __shared__ __align__(1024) unsigned char sm[];
    uint32_t *s_tm = reinterpret_cast<uint32_t *>(sm + T6_OFF_TM);
    volatile int *s_bad = reinterpret_cast<volatile int *>(sm + T6_OFF_TM + 4);
    int *s_c0 = reinterpret_cast<int *>(sm + T6_OFF_TM + 8);
    const uint32_t sbase = smem_u32(sm);
    const uint32_t full0 = sbase + T6_OFF_BAR, empty0 = full0 + 16, rbar0 = full0 + 32;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m = blockIdx.y;
    const int l0 = max(m, spin);
    const unsigned char *recm = rec + (size_t)woff[m] * T6_RSZ;

    if (warp == T / 32) tmem_alloc(sbase + T6_OFF_TM, T6_NT * T6_NN);
    if (tid == 0) {
        mbar_init(full0, T / 32);
        mbar_init(full0 + 8, T / 32);
        mbar_init(empty0, 1);
        mbar_init(empty0 + 8, 1);
        mbar_init(rbar0, 1);
        mbar_init(rbar0 + 8, 1);
        *s_bad = 0;
        *s_c0 = TC_NEVER;
        mbar_init_fence();
    }
    // the eighth K-core of A and the B' positions with i > g stay zero for the whole kernel
    for (int i = tid; i < (2 * T6_ABUF + 2 * T6_BBUF) / 16; i += T6_BLOCK)
        reinterpret_cast<uint4 *>(sm)[i] = make_uint4(0u, 0u, 0u, 0u);

    const bool ring_thread = warp < T / 32;
    const int side = S0 ? 0 : tid / (T / 2);
    const int p = S0 ? blockIdx.x * T + tid : blockIdx.x * (T / 2) + tid % (T / 2);
    const bool act = ring_thread && p < npairs;
    // this ring's state at its first accumulated chunk of 16 l (the plan's table), or the start at l0
    double cur = 0.0, prev = 0.0;
    int e = 0, c_me = TC_NEVER;
    if (act) {
        if (stv) {
            const size_t ix = ((size_t)m * 2 + side) * st_ld + p;
            const double2 v = stv[ix];
            const short2 ec = ste[ix];
            cur = v.x;
            prev = v.y;
            e = 512 * (int)ec.x;
            c_me = ec.y;
        } else {
            tc64_start(lg0[m], m, spin, lsc[p], side, cur, prev, e);
            c_me = 0;
        }
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = *s_tm;
    {
        const int cm = __reduce_min_sync(0xffffffffu, c_me);
        if (lane == 0 && ring_thread && cm < TC_NEVER) atomicMin(s_c0, cm);
    }
    __syncthreads();
    // the block starts at the first chunk in which any of its rings accumulates
    const int nchk = l0 <= L ? (L - l0 + T6_KC) / T6_KC : 0;
    const int cb = 2 * *s_c0;
    const bool work = cb < nchk;
    const int kw0 = work ? cb / T6_CPW : 0, cs0 = cb - kw0 * T6_CPW;
    if (tid == 0 && work) bulk_g2s(sbase + T6_OFF_R, recm + (size_t)kw0 * T6_RSZ, T6_RSZ, rbar0);

    int issued = 0;  // chunks whose MMAs the MMA warp has issued
    if (warp == T / 32) {
        // ---------------- MMA warp: follows the chunk sequence (outcome warp-uniform), lane 0 issues
        constexpr uint32_t IDESC = idesc_f16_f32(128, T6_NN);
        int gc = 0;
        bool ok = true;
        for (int kw = kw0; work && l0 + kw * T6_W <= L && ok; ++kw) {
            const int wb = l0 + kw * T6_W;
            const int nch = (min(T6_W, L - wb + 1) + T6_KC - 1) / T6_KC;
            const int cs = kw == kw0 ? cs0 : 0;
            for (int c = cs; c < nch; ++c, ++gc) {
                const int buf = gc & 1;
                const bool got = !*s_bad && mbar_wait(full0 + 8 * buf, (gc >> 1) & 1, wlim);
                if (!__all_sync(0xffffffffu, got)) {
                    *s_bad = 1;
                    ok = false;
                    break;
                }
                if (lane == 0) {
                    tc_fence_after();
                    const uint32_t aa = sbase + buf * T6_ABUF, ba = sbase + T6_OFF_B + buf * T6_BBUF;
#pragma unroll
                    for (int t = 0; t < T6_NT; ++t)
#pragma unroll
                        for (int k = 0; k < 4; ++k)  // K-step k: digits 2k and 2k + 1, 8 l each
                            tc_mma(tbase + t * T6_NN, sdesc(aa + t * T6_TILE + k * 256, 128, T6_SBO),
                                   sdesc(ba + k * 256, 128, T6_SBO), IDESC, (c > cs || k > 0) ? 1u : 0u);
                    tc_commit(empty0 + 8 * buf);
                }
                __syncwarp();
            }
        }
        issued = gc;
    } else {
        // ---------------- ring warps
        const int tile = tid >> 7, row = tid & 127;
        const double xs = act ? (side ? -px[p] : px[p]) : 0.0;
        double acc[T6_NO] = {0.0, 0.0, 0.0, 0.0};
        // fixed point once every ring of the warp is past its turning point (cur, prev then hold U, V)
        const int Es = es[m];
        const long long X = fix62(xs, 1);  // Q61
        const int xh = (int)(X >> 31), xl = (int)X & 0x7FFFFFFF;
        const bool idle = c_me == TC_NEVER;  // never accumulates: stays zero
        const long long rnd = idle ? 0 : FIX_ROUND;
        bool fixed = false;
        const bool may_fix = __any_sync(0xffffffffu, !idle);
        // windows before the block's first: no digits, but a value in them that is not finite (scale NaN) counts
        bool nonfin = false;
        for (int k = lane; k < (work ? kw0 : woff[m + 1] - woff[m]); k += 32) {
            const double *sc = reinterpret_cast<const double *>(recm + (size_t)k * T6_RSZ + T6_RSC);
            nonfin |= isnan(sc[0] + sc[1] + sc[2] + sc[3]);
        }
        nonfin = __any_sync(0xffffffffu, nonfin);
        const uint32_t t_lane = tbase + ((uint32_t)((warp & 3) * 32) << 16) + tile * T6_NN;
        const uint32_t a_row = (uint32_t)tile * T6_TILE + (row >> 3) * T6_SBO + (row & 7) * 16;
        // this thread's B' copy: row n = g NO + o, K-core di = t_{g-di} of output o (28 pairs x 4 outputs)
        constexpr int NCOPY = T6_ND * (T6_ND + 1) / 2 * T6_NO;
        int b_src = 0, b_dst = -1;
        if (tid < NCOPY) {
            const int pr = tid / T6_NO, o = tid - pr * T6_NO;
            int g = 0;
            while ((g + 1) * (g + 2) / 2 <= pr) ++g;
            const int di = pr - g * (g + 1) / 2, n = g * T6_NO + o;
            b_src = ((g - di) * T6_NO + o) * T6_TPS;
            b_dst = (n >> 3) * T6_SBO + di * 128 + (n & 7) * 16;
        }
        int gc = 0, kw = kw0, kl = 0;
        int bad = 0;
        for (; work && l0 + kw * T6_W <= L; ++kw, ++kl) {
            const int wb = l0 + kw * T6_W;
            const int cnt = min(T6_W, L - wb + 1);
            // prefetch the next window's record (its buffer's readers finished at the previous closing barrier)
            if (tid == 0 && wb + T6_W <= L) {
                fence_async_smem();
                bulk_g2s(sbase + T6_OFF_R + ((kl + 1) & 1) * T6_RSZ, recm + (size_t)(kw + 1) * T6_RSZ, T6_RSZ,
                         rbar0 + 8 * ((kl + 1) & 1));
            }
            bad |= !mbar_wait(rbar0 + 8 * (kl & 1), (kl >> 1) & 1, wlim);
            const unsigned char *Rw = sm + T6_OFF_R + (kl & 1) * T6_RSZ;
            const unsigned short *s_tp = reinterpret_cast<const unsigned short *>(Rw);
            const double *s_sc = reinterpret_cast<const double *>(Rw + T6_RSC);
            const int *s_el = reinterpret_cast<const int *>(Rw + T6_REL);
            const double2 *s_ag = reinterpret_cast<const double2 *>(Rw + T6_RCO);
            const FixCoef *s_fx = reinterpret_cast<const FixCoef *>(Rw + T6_RFX);

            const int nch = (cnt + T6_KC - 1) / T6_KC;
            for (int c = kw == kw0 ? cs0 : 0; c < nch; ++c, ++gc) {
                const int buf = gc & 1;
                const bool live = kw * T6_CPW + c >= 2 * c_me;
                if (gc >= 2) bad |= !mbar_wait(empty0 + 8 * buf, ((gc - 2) >> 1) & 1, wlim);
                unsigned char *sA = sm + buf * T6_ABUF;
                unsigned char *sB = sm + T6_OFF_B + buf * T6_BBUF;
                if (b_dst >= 0)
                    *reinterpret_cast<uint4 *>(sB + b_dst) =
                        *reinterpret_cast<const uint4 *>(s_tp + b_src + c * T6_KC);
                const int El = s_el[c >> 1];
                if (may_fix && !fixed) {
                    const double2 a = s_ag[c * T6_KC];
                    fixed = __all_sync(0xffffffffu, idle || (live && fix_ready(cur, prev, e, a.x, a.y, xs, Es, El)));
                    if (fixed) {
                        cur = __longlong_as_double(idle ? 0 : fix62(cur, Es));
                        prev = __longlong_as_double(idle ? 0 : fix62(prev, Es));
                    }
                }
                if (fixed) {
                    const int sh = 7 + El - Es;
                    long long U = __double_as_longlong(cur), V = __double_as_longlong(prev);
                    uint32_t pk[T6_ND][4];
#pragma unroll
                    for (int j2 = 0; j2 < 4; ++j2) {
                        const FixCoef q0 = s_fx[c * T6_KC + 2 * j2], q1 = s_fx[c * T6_KC + 2 * j2 + 1];
                        const unsigned long long w0 = (unsigned long long)(U >> sh) + FIX_BIAS;
                        fix_step(q0, xh, xl, rnd, U, V);
                        const unsigned long long w1 = (unsigned long long)(U >> sh) + FIX_BIAS;
                        fix_step(q1, xh, xl, rnd, U, V);
                        pk[0][j2] = digit_pair<0>(w0, w1);
                        pk[1][j2] = digit_pair<1>(w0, w1);
                        pk[2][j2] = digit_pair<2>(w0, w1);
                        pk[3][j2] = digit_pair<3>(w0, w1);
                        pk[4][j2] = digit_pair<4>(w0, w1);
                        pk[5][j2] = digit_pair<5>(w0, w1);
                        pk[6][j2] = digit_pair<6>(w0, w1);
                    }
                    cur = __longlong_as_double(U);
                    prev = __longlong_as_double(V);
#pragma unroll
                    for (int k = 0; k < T6_ND; ++k)
                        *reinterpret_cast<uint4 *>(sA + a_row + k * 128) =
                            make_uint4(pk[k][0], pk[k][1], pk[k][2], pk[k][3]);
                } else if (live) {
                    const int nb = 1030 + El - e;  // e < 0: every digit 0
                    uint32_t pk[T6_ND][4];
#pragma unroll
                    for (int j2 = 0; j2 < 4; ++j2) {
                        // past the window's end the alm digits are zero, so these rows need no mask
                        unsigned long long w2[2];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const double2 a = s_ag[c * T6_KC + 2 * j2 + h];
                            w2[h] = fix55_biased(cur, nb);
                            const double nxt = fma(fma(a.x, xs, a.y), cur, -prev);
                            prev = cur;
                            cur = nxt;
                        }
                        pk[0][j2] = digit_pair<0>(w2[0], w2[1]);
                        pk[1][j2] = digit_pair<1>(w2[0], w2[1]);
                        pk[2][j2] = digit_pair<2>(w2[0], w2[1]);
                        pk[3][j2] = digit_pair<3>(w2[0], w2[1]);
                        pk[4][j2] = digit_pair<4>(w2[0], w2[1]);
                        pk[5][j2] = digit_pair<5>(w2[0], w2[1]);
                        pk[6][j2] = digit_pair<6>(w2[0], w2[1]);
                    }
#pragma unroll
                    for (int k = 0; k < T6_ND; ++k)
                        *reinterpret_cast<uint4 *>(sA + a_row + k * 128) =
                            make_uint4(pk[k][0], pk[k][1], pk[k][2], pk[k][3]);
                    // a step grows the value by less than 2^8.5: eight from below 2^200 stay in range
                    if (e < 0 && ((__double2hiint(cur) >> 20) & 0x7FF) > 1023 + 200) {
                        cur *= 0x1p-512;
                        prev *= 0x1p-512;
                        e += 512;
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < T6_ND; ++k)
                        *reinterpret_cast<uint4 *>(sA + a_row + k * 128) = make_uint4(0u, 0u, 0u, 0u);
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(full0 + 8 * buf);
            }
            // window epilogue: column n = g NO + o holds the exact sum of weight 2^-8g, |sum| < 2^24
            bad |= !mbar_wait(empty0 + 8 * ((gc - 1) & 1), ((gc - 1) >> 1) & 1, wlim);
            bad = __any_sync(0xffffffffu, bad);
            tc_fence_after();
            if (!bad) {
                long long hi[T6_NO], lo[T6_NO];
                float dv[16];
                tmem_ld16(t_lane, dv);
#pragma unroll
                for (int o = 0; o < T6_NO; ++o)
                    hi[o] = ((((long long)(int)dv[o] << 8) + (int)dv[4 + o]) << 16) +
                            (((long long)(int)dv[8 + o] << 8) + (int)dv[12 + o]);
                tmem_ld16(t_lane + 16, dv);
#pragma unroll
                for (int o = 0; o < T6_NO; ++o) {
                    lo[o] = ((((long long)(int)dv[o] << 8) + (int)dv[4 + o]) << 8) + (int)dv[8 + o];
                    acc[o] = fma((double)lo[o], s_sc[T6_NO + o], acc[o]);
                    acc[o] = fma((double)hi[o], s_sc[o], acc[o]);
                }
            }
            tc_fence_before();
            bad = bar_or_1(T, bad | *s_bad);
            if (bad) break;
        }
        if (bad) {
            *s_bad = 1;
            if (tid == 0) {
                if (status) atomicOr(status, 1);
                // the record copies of the last window entered and of the one after it may still be in flight
                mbar_wait(rbar0 + 8 * (kl & 1), (kl >> 1) & 1);
                if (l0 + (kw + 1) * T6_W <= L) mbar_wait(rbar0 + 8 * ((kl + 1) & 1), ((kl + 1) >> 1) & 1);
            }
        }
        if (bad || nonfin) {  // H holds an earlier call's columns: after a wait that ran out nothing may pass for this one's
#pragma unroll
            for (int o = 0; o < T6_NO; ++o) acc[o] = nan("");
        }
        if (act) {
            const int n = prn[p], s = prs[p];
            if (S0) {
                H[(long long)m * ldH + n] = make_double2(acc[0] + acc[2], acc[1] + acc[3]);
                if (s != n) H[(long long)m * ldH + s] = make_double2(acc[0] - acc[2], acc[1] - acc[3]);
            } else {
                const double sgs = (spin & 1) ? -1.0 : 1.0;
                const double2 A = make_double2(-acc[0], -acc[1]), B = make_double2(-sgs * acc[2], -sgs * acc[3]);
                if (side == 0) {
                    H[(long long)(L + m) * ldH + n] = A;
                    if (m > 0 && s != n) H[(long long)(L - m) * ldH + s] = B;
                } else {
                    if (s != n) H[(long long)(L + m) * ldH + s] = A;
                    if (m > 0) H[(long long)(L - m) * ldH + n] = B;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == T / 32) {
        // after a wait that ran out, wherever it did, the MMAs issued may still be in flight
        if (*s_bad && issued > 0) mbar_wait(empty0 + 8 * ((issued - 1) & 1), ((issued - 1) >> 1) & 1);
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tbase, T6_NT * T6_NN);
    }
}

// ---------------------------------------------------------------- host side
static void log2_pair(long double v, double &h, double &l) {
    const long double lg = std::log2(v);
    h = v > 0 ? (double)lg : -INFINITY;
    l = v > 0 ? (double)(lg - h) : 0.0;
}

// Tables, window records and start states (Gauss-Legendre spins 0 ..
// max(max_spin, 1), Clenshaw-Curtis 0 .. max_spin) in one allocation, rounded
// up to the 2 MB granularity of device memory; base NULL: size only.
static size_t tc64_layout(cunusht_plan_s *P, char *base, size_t &nrec) {
    const size_t L = P->lmax;
    size_t off = 0;
    auto take = [&](auto *&p, size_t n) {
        p = base ? reinterpret_cast<std::remove_reference_t<decltype(p)>>(base + off) : nullptr;
        off += (n * sizeof(*p) + 255) / 256 * 256;
    };
    take(P->d_t6_lsc[0], P->h_gl_theta.size());
    take(P->d_t6_lsc[1], P->h_cc_theta.size());
    nrec = 0;
    for (size_t s = 0; s <= 2 && s <= L; ++s) {
        size_t w = 0;
        for (size_t m = 0; m <= L; ++m) w += (L - std::max(m, s) + T6_W) / T6_W;
        nrec = std::max(nrec, w);
        take(P->d_t6_ag[s], P->nalm_tab);
        take(P->d_t6_cl[s], P->nalm_tab);
        take(P->d_t6_fx[s], P->nalm_tab);
        take(P->d_t6_lg0[s], L + 1);
        take(P->d_t6_eb[s], 8 * w);
        take(P->d_t6_woff[s], L + 2);
        take(P->d_t6_es[s], L + 1);
    }
    take(P->d_t6_rec, nrec * T6_RSZ);
    for (int g = 0; g < 2; ++g) {
        const size_t smax = g ? P->max_spin : std::max(P->max_spin, 1), n = 2 * (g ? P->cc_npairs : P->gl_npairs) * (L + 1);
        for (size_t s = 0; s <= smax && s <= L; ++s) {
            take(P->d_t6_stv[g][s], n);
            take(P->d_t6_ste[g][s], n);
        }
    }
    return (off + (2 << 20) - 1) >> 21 << 21;
}

// recursion tables of one spin (cdd: scratch of nalm_tab pairs)
static int tc64_tables(cunusht_plan_s *P, int s, double2 *cdd) {
    const int L = P->lmax;
    const dim3 grid((L + 256) / 256, L + 1);
    k_tc64_beta<<<grid, 256>>>(L, s, cdd);
    k_tc64_scale<<<(L + 32) / 32, 32>>>(L, s, cdd);
    k_tc64_coef<<<grid, 256>>>(L, s, cdd, P->d_t6_ag[s], P->d_t6_cl[s], P->d_t6_fx[s]);
    CU_LAUNCH_CHECK();
    // log2 of the start's normalisation sqrt((2 l0 + 1) / (4 pi) (2 l0)! / ((m + s)! |m - s|!)), l0 = max(m, s)
    std::vector<double2> lg(L + 1);
    std::vector<long double> lf(2 * std::max(L, s) + 3, 0.0L);  // log2 n!
    for (size_t n = 2; n < lf.size(); ++n) lf[n] = lf[n - 1] + std::log2((long double)n);
    std::vector<int> wo(L + 2, 0);
    for (int m = 0; m <= L; ++m) {
        const int l0 = std::max(m, s);
        const long double v = 0.5L * (std::log2((2.0L * l0 + 1.0L) / (4.0L * 3.14159265358979323846264338327950288L)) +
                                      lf[2 * l0] - lf[m + s] - lf[std::abs(m - s)]);
        lg[m].x = (double)v;
        lg[m].y = (double)(v - lg[m].x);
        wo[m + 1] = wo[m] + (L - l0 + T6_W) / T6_W;
    }
    CU_TRY(cudaMemcpy(P->d_t6_lg0[s], lg.data(), lg.size() * sizeof(double2), cudaMemcpyHostToDevice));
    CU_TRY(cudaMemcpy(P->d_t6_woff[s], wo.data(), wo.size() * sizeof(int), cudaMemcpyHostToDevice));
    k_tc64_chunk_exp<<<dim3((L / 16 + 64) / 64, L + 1), 64>>>(L, s, P->d_t6_cl[s], P->d_t6_woff[s], P->d_t6_eb[s]);
    k_tc64_order_exp<<<(L + 64) / 64, 64>>>(L, s, P->d_t6_woff[s], P->d_t6_eb[s], P->d_t6_es[s]);
    CU_LAUNCH_CHECK();
    return CUNUSHT_OK;
}

int tc64_plan_init(cunusht_plan_s *P) {
    const int L = P->lmax;
    size_t nrec = 0;
    const size_t bytes = tc64_layout(P, nullptr, nrec);
    void *slab = nullptr;
    RC_TRY(plan_alloc(P, &slab, bytes));
    P->d_t6_slab = slab;
    tc64_layout(P, (char *)slab, nrec);
    for (int g = 0; g < 2; ++g) {
        std::vector<RingLog> q;
        for (double th : g ? P->h_cc_theta : P->h_gl_theta) {
            RingLog v;
            log2_pair(std::sin(0.5L * th), v.sh, v.sl);
            log2_pair(std::cos(0.5L * th), v.ch, v.cl);
            q.push_back(v);
        }
        if (!q.empty())
            CU_TRY(cudaMemcpy(P->d_t6_lsc[g], q.data(), q.size() * sizeof(RingLog), cudaMemcpyHostToDevice));
    }
    // the record buffer, unused until the first call, holds the tables' double-doubles
    for (int s = 0; s <= 2 && s <= L; ++s) RC_TRY(tc64_tables(P, s, (double2 *)P->d_t6_rec));
    for (int g = 0; g < 2; ++g) {
        const int np = g ? P->cc_npairs : P->gl_npairs;
        const size_t n = 2 * (size_t)np * (L + 1);
        for (int s = 0; s <= 2; ++s) {
            if (!P->d_t6_stv[g][s] || n == 0) continue;
            k_tc64_starts<<<(unsigned)((n + 127) / 128), 128>>>(L, s, P->d_t6_lg0[s], np, g ? P->d_cc_x : P->d_gl_x,
                                                               P->d_t6_lsc[g], P->d_t6_ag[s], P->d_t6_stv[g][s],
                                                               P->d_t6_ste[g][s]);
            CU_LAUNCH_CHECK();
        }
    }
    return CUNUSHT_OK;
}

// One request's synthesis: the pole pair in closed form, every other pair on the
// tensor cores.  A last block with few rings costs less than the same rings on
// the CUDA cores, where one warp per order waits on the FP64 pipe for every l
// (fewer than 32 pairs there: spin 0, 514 pairs, lmax 1026 2.34 ms instead of 1.27,
// 1540 pairs 27.8 instead of 20.5; spin 2, 258 pairs 1.26 instead of 0.41, 1026
// pairs 21.0 instead of 12.1).
int leg_synth_tc64(const cunusht_plan_s *P, int npairs, const double *x, const int *rn, const int *rs, int ld,
                   int pole, int pole_rn, int pole_rs, bool cc, int spin, const double2 *G, const double2 *C,
                   const double *lf, double2 *H, cudaStream_t st) {
    const double2 *stv = P->d_t6_stv[cc ? 1 : 0][spin];
    const short2 *ste = P->d_t6_ste[cc ? 1 : 0][spin];
    const RingLog *lsc = P->d_t6_lsc[cc ? 1 : 0];
    const int st_ld = npairs, L = P->lmax;
    if (pole == 0 && npairs > 1) {
        RC_TRY(leg_synth_pole_pair(P, 1, spin, G, C, 0, lf, pole_rn, pole_rs, H, 0, ld, st));
        ++x, ++rn, ++rs, ++lsc;
        if (stv) ++stv, ++ste;
        --npairs;
    }
    const int per = spin == 0 ? T6_T : T6_T / 2;
    k_tc64_records<<<dim3((L - spin + T6_W) / T6_W, P->mmax + 1), T6_W, 0, st>>>(
        L, spin, G, C, lf, P->d_t6_ag[spin], P->d_t6_cl[spin], P->d_t6_woff[spin], P->d_t6_rec);
    CU_LAUNCH_CHECK();
    auto launch = [&](auto kern) {
        CU_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, T6_BYTES));
        kern<<<dim3((npairs + per - 1) / per, P->mmax + 1), T6_BLOCK, T6_BYTES, st>>>(
            L, spin, P->d_t6_rec, P->d_t6_woff[spin], P->d_t6_lg0[spin], npairs, x, lsc, rn, rs, stv, ste, st_ld,
            P->d_t6_es[spin], H, ld, P->wait_limit, P->d_status);
        CU_LAUNCH_CHECK();
        return CUNUSHT_OK;
    };
    return spin == 0 ? launch(k_leg_synth_tc64<true>) : launch(k_leg_synth_tc64<false>);
}

}  // namespace cunusht
