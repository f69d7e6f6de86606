// Adjoint Legendre transform of the FP64 plans on the tensor cores (tcgen05):
// the contraction of nusht2d1 and of the SHT analysis (the reference's SHTns
// analys, cunusht/sht/GPU_sht_transformer.py:65-73), FP64 recursion on the CUDA
// cores, exact integer digit products.
//
// For one order m and the ring columns X (spin s: (h+m re, h+m im, h-m re,
// h-m im), the -m column from the mirror ring; spin 0: the even / odd sums (E
// re, E im, O re, O im) of a ring pair)
//     D(l, col) = sum_ring lambda_l(theta_ring) X(ring, col),
// lambda_l = c_l mu_l with the rescaled recursion of legendre_tc64.cu (2 FP64
// instructions per step and ring; the CUDA-core kernel spends 14 to 22 per
// ring pair and l, its warp sums included, on a pipe of 2 lanes per SM and
// clock).  mu and X are split into seven 8-bit digits (rec64.cuh), exact in
// fp16: per chunk of 16 l one accumulator holds sum_ring t_j(ring, col)
// d_i(ring, l) in row (j, col) and column (i, l) -- M = 128 (28 rows used), N
// = 7 x 16, K = the block's 256 rings -- integers below 2^22, exact in FP32.
// The epilogue adds the pairs i + j <= 6 (the rest is below 2^-56) in 64-bit
// integers, and the block's part of D goes to the alm by FP64 atomics, one per
// (l, component) and block as in the CUDA-core kernel.
//
// Roles of the 11 warps: 8 ring warps (one ring per thread: recursion, digit
// split, the 16-byte rows of the B tile), one MMA warp (16 MMAs of 128 x 112 x
// 16 per chunk) and two epilogue warps, 8 l each (warps 0 and 4: a warp reads
// the tensor-memory lanes 32 (warp mod 4) .. + 31, and the used rows are lanes
// 0 .. 27).  Two B buffers and four tensor-memory buffers with full / empty
// mbarriers.  Every wait is bounded; on a timeout the block sets bit 0 of the
// plan's status word, makes the order's alm NaN (no caller polls that word) and
// returns.  The ring warps bound it (lmax 1023 spin 2, 2.21 ms: issue slots 41
// %, ALU pipe 47 %, FP64 pipe 26 %, tensor pipe 15 %, one block of 11 warps per SM).
#include "common.cuh"
#include "kernels.cuh"
#include "rec64.cuh"
#include "tcgen05.cuh"

namespace cunusht {

constexpr int A6_R = 256;                    // rings per block (K)
constexpr int A6_KC = 16;                    // l per chunk
constexpr int A6_ND = 7;
constexpr int A6_NN = A6_ND * A6_KC;         // 112 columns (digit, l)
constexpr int A6_NTB = 4;                    // tensor-memory chunk buffers, 128 columns apart
constexpr int A6_THREADS = 11 * 32;
constexpr int A6_MMA = 1;                    // the MMA warp; 0 and 4 are the epilogue warps
constexpr int A6_A_LBO = 16 * 128;           // A: [K-core 32][M-core 16][8 K-rows][16 B]
constexpr int A6_A_SBO = 128;
constexpr int A6_ABYTES = (A6_R / 8) * A6_A_LBO;
constexpr int A6_B_SBO = 128;                // B: [K-core 32][N-core 14 = (digit, l half)][8 K-rows][16 B]
constexpr int A6_B_LBO = 2 * A6_ND * A6_B_SBO;
constexpr int A6_BBUF = (A6_R / 8) * A6_B_LBO;
constexpr int A6_OFF_B = A6_ABYTES;
constexpr int A6_OFF_BAR = A6_OFF_B + 2 * A6_BBUF;   // bfull[2] bempty[2] tfull[4] tempty[4]
constexpr int A6_OFF_MISC = A6_OFF_BAR + 12 * 8;     // tmem base, bad flag, first chunk, pad, Ea[4], maxima[8][4]
constexpr int A6_BYTES = A6_OFF_MISC + 16 + 16 + 8 * 16;
static_assert(A6_BYTES <= 227 * 1024, "dynamic shared memory of one block");
static_assert(A6_BBUF % 1024 == 0 && A6_OFF_BAR % 8 == 0, "layout alignment");

__device__ __forceinline__ long long shfl_xor_ll(long long v, int mask) { return __shfl_xor_sync(0xffffffffu, v, mask); }

// n alm from entry i0 on become NaN, whatever other blocks add
__device__ __noinline__ void add_nan(double *G, double *C, long long i0, int n, int t, int nt) {
    for (int i = t; i < 2 * n; i += nt) {
        atomicAdd(G + 2 * i0 + i, nan(""));
        if (C) atomicAdd(C + 2 * i0 + i, nan(""));
    }
}

template <bool S0>
__global__ void __launch_bounds__(A6_THREADS, 1)
    k_leg_adj_tc64(int L, int spin, int ncomp, const double2 *__restrict__ H, int ldH, const double *__restrict__ lfac,
                   const double2 *__restrict__ ag, const FixCoef *__restrict__ fx, const double *__restrict__ cl,
                   const short *__restrict__ eb, const short *__restrict__ es,
                   const int *__restrict__ woff, const double2 *__restrict__ lg0, int npairs,
                   const double *__restrict__ px, const RingLog *__restrict__ lsc, const int *__restrict__ prn,
                   const int *__restrict__ prs, const double2 *__restrict__ stv, const short2 *__restrict__ ste,
                   int st_ld, double *__restrict__ Gout, double *__restrict__ Cout, int wlim, int *status) {
    extern __shared__ __align__(1024) unsigned char sm[];
    uint32_t *s_tm = reinterpret_cast<uint32_t *>(sm + A6_OFF_MISC);
    volatile int *s_bad = reinterpret_cast<volatile int *>(sm + A6_OFF_MISC + 4);
    int *s_c0 = reinterpret_cast<int *>(sm + A6_OFF_MISC + 8);
    int *s_ea = reinterpret_cast<int *>(sm + A6_OFF_MISC + 16);
    int *s_mx = reinterpret_cast<int *>(sm + A6_OFF_MISC + 32);  // [ring warp][col]
    const uint32_t sbase = smem_u32(sm);
    const uint32_t bfull0 = sbase + A6_OFF_BAR, bempty0 = bfull0 + 16, tfull0 = bfull0 + 32, tempty0 = bfull0 + 64;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool epi = (warp & 3) == 0 && warp < 8, ring_thread = !epi && warp != A6_MMA;
    const int rw = warp < 4 ? warp - 2 : warp - 3;  // ring warp index 0 .. 7 (warps 2, 3, 5 .. 10)
    const int rid = rw * 32 + lane;
    const int m = blockIdx.y;
    const int l0 = max(m, spin);
    const long long b = almidx(L, m, m) - m;  // (l, m) at b + l

    if (warp == A6_MMA) tmem_alloc(sbase + A6_OFF_MISC, 512);
    if (tid == 0) {
        mbar_init(bfull0, 8);
        mbar_init(bfull0 + 8, 8);
        mbar_init(bempty0, 1);
        mbar_init(bempty0 + 8, 1);
        for (int k = 0; k < A6_NTB; ++k) {
            mbar_init(tfull0 + 8 * k, 1);
            mbar_init(tempty0 + 8 * k, 2);
        }
        *s_bad = 0;
        *s_c0 = TC_NEVER;
        mbar_init_fence();
    }
    // A rows 28 .. 127 stay zero
    for (int i = tid; i < A6_ABYTES / 16; i += A6_THREADS) reinterpret_cast<uint4 *>(sm)[i] = make_uint4(0u, 0u, 0u, 0u);

    const int side = S0 ? 0 : rid / (A6_R / 2);  // 0: ring theta, 1: ring pi - theta
    const int p = S0 ? blockIdx.x * A6_R + rid : blockIdx.x * (A6_R / 2) + (rid & (A6_R / 2 - 1));
    const bool act = ring_thread && p < npairs;
    double cur = 0.0, prev = 0.0, X[4] = {0.0, 0.0, 0.0, 0.0};
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
        const int n = prn[p], s = prs[p];
        if (S0) {
            const double2 hn = H[(long long)m * ldH + n];
            X[0] = X[2] = hn.x;
            X[1] = X[3] = hn.y;
            if (s != n) {
                const double2 hs = H[(long long)m * ldH + s];
                X[0] += hs.x, X[1] += hs.y, X[2] -= hs.x, X[3] -= hs.y;
            }
        } else {
            // side 0: (h(+m) at n, h(-m) at s); side 1: (h(+m) at s, h(-m) at n); the S
            // ring of a self-paired ring carries no +m column and takes the -m one
            if (!(side && s == n)) {
                const double2 v = H[(long long)(L + m) * ldH + (side ? s : n)];
                X[0] = v.x, X[1] = v.y;
            }
            if (side || s != n) {
                const double2 v = H[(long long)(L - m) * ldH + (side ? n : s)];
                X[2] = v.x, X[3] = v.y;
            }
        }
    }
    const int c_warp = __reduce_min_sync(0xffffffffu, c_me);
    if (ring_thread) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int ex = __reduce_max_sync(0xffffffffu, (__double2hiint(X[c]) >> 20) & 0x7FF);
            if (lane == 0) s_mx[rw * 4 + c] = ex;
        }
    }
    __syncthreads();
    if (ring_thread && lane == 0 && c_warp < TC_NEVER) atomicMin(s_c0, c_warp);
    if (tid < 4) {
        int ex = 0;
        for (int w = 0; w < 8; ++w) ex = max(ex, s_mx[w * 4 + tid]);
        s_ea[tid] = max(ex, 64) - 1022;  // 2^Ea > |X| (zero columns: digits 0); 1025: a value that is not finite
    }
    __syncthreads();
    if (ring_thread) {
        // column digits t_j into A (MN-major: row j 4 + col, K = ring)
        unsigned char *aK = sm + (rid >> 3) * A6_A_LBO + (rid & 7) * 16;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const unsigned long long w = fix55_biased(X[c], 1030 + s_ea[c]);
            const uint32_t d[7] = {digit_pair<0>(w, w), digit_pair<1>(w, w), digit_pair<2>(w, w), digit_pair<3>(w, w),
                                   digit_pair<4>(w, w), digit_pair<5>(w, w), digit_pair<6>(w, w)};
#pragma unroll
            for (int j = 0; j < A6_ND; ++j) {
                const int row = j * 4 + c;
                *reinterpret_cast<unsigned short *>(aK + (row >> 3) * A6_A_SBO + (row & 7) * 2) = (unsigned short)d[j];
            }
        }
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = *s_tm;
    const int nchk = l0 <= L ? (L - l0 + A6_KC) / A6_KC : 0;
    const int cb = *s_c0;
    const int lstart = cb < nchk ? l0 + A6_KC * cb : L + 1;
    // the l before it get no digit products, but a column that is not finite makes them NaN as well
    if (lstart > l0 && max(max(s_ea[0], s_ea[1]), max(s_ea[2], s_ea[3])) == 1025)
        add_nan(Gout, !S0 && ncomp > 1 ? Cout : nullptr, b + l0, lstart - l0, tid, A6_THREADS);
    const short *ebm = eb + 8 * (long long)woff[m];  // El per chunk

    int issued = 0;  // chunks whose MMAs the MMA warp has issued
    if (warp == A6_MMA) {
        constexpr uint32_t IDESC = idesc_f16_f32(128, A6_NN) | (1u << 15) | (1u << 16);  // A, B MN-major
        int gc = 0;
        for (int lb = lstart; lb <= L; lb += A6_KC, ++gc) {
            const int buf = gc & 1, tb = gc % A6_NTB;
            bool got = !*s_bad && mbar_wait(bfull0 + 8 * buf, (gc >> 1) & 1, wlim);
            if (got && gc >= A6_NTB) got = mbar_wait(tempty0 + 8 * tb, ((gc / A6_NTB) - 1) & 1, wlim);
            if (!__all_sync(0xffffffffu, got)) {
                *s_bad = 1;
                break;
            }
            if (lane == 0) {
                tc_fence_after();
                const uint32_t bb = sbase + A6_OFF_B + buf * A6_BBUF;
#pragma unroll 4
                for (int ks = 0; ks < A6_R / 16; ++ks)
                    tc_mma(tbase + tb * 128, sdesc(sbase + 2 * ks * A6_A_LBO, A6_A_LBO, A6_A_SBO),
                           sdesc(bb + 2 * ks * A6_B_LBO, A6_B_LBO, A6_B_SBO), IDESC, ks > 0 ? 1u : 0u);
                tc_commit(bempty0 + 8 * buf);
                tc_commit(tfull0 + 8 * tb);
            }
            __syncwarp();
        }
        issued = gc;
    } else if (epi) {
        // lane = row (digit j = lane / 4, column lane % 4); rows 28 .. 31 are zero
        const int eh = warp >> 2, j = lane >> 2, col = lane & 3;
        const int ea = s_ea[col];
        const double sgs = (spin & 1) ? -1.0 : 1.0;
        int gc = 0;
        for (int lb = lstart; lb <= L; lb += A6_KC, ++gc) {
            const int tb = gc % A6_NTB;
            const bool got = !*s_bad && mbar_wait(tfull0 + 8 * tb, (gc / A6_NTB) & 1, wlim);
            if (!__all_sync(0xffffffffu, got)) {
                *s_bad = 1;
                break;
            }
            tc_fence_after();
            // hi: pairs i + j <= 3 at weight 2^-24, lo: 4 <= i + j <= 6 at 2^-48
            long long hi[8], lo[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) hi[q] = lo[q] = 0;
            const uint32_t ta = tbase + tb * 128 + 8 * eh;
            float v[A6_ND][8];  // all loads in flight before the one wait
#pragma unroll
            for (int i = 0; i < A6_ND; ++i) tmem_ld8_async(ta + i * A6_KC, v[i]);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < A6_ND; ++i) {
                const bool ih = i + j <= 3, il = !ih && i + j <= 6;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int d = (int)tmem_keep(v[i][q]);
                    if (ih) hi[q] = (hi[q] << 8) + d;
                    if (il) lo[q] = (lo[q] << 8) + d;
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty0 + 8 * tb);
            // sum over j, scattering the eight l over the j lanes: bit 16 -> l bit 2, 8 -> 1, 4 -> 0
#pragma unroll
            for (int st = 0; st < 3; ++st) {
                const int mask = 16 >> st, half = 4 >> st;
                const bool up = lane & mask;
#pragma unroll
                for (int q = 0; q < half; ++q) {
                    const long long sh_ = up ? hi[q] : hi[q + half], kh = up ? hi[q + half] : hi[q];
                    hi[q] = kh + shfl_xor_ll(sh_, mask);
                    const long long sl_ = up ? lo[q] : lo[q + half], kl = up ? lo[q + half] : lo[q];
                    lo[q] = kl + shfl_xor_ll(sl_, mask);
                }
            }
            const int l = lb + 8 * eh + j;
            const int sc = ebm[(lb - l0) / A6_KC] + ea - 14;
            const bool in = l <= L;
            double D = fma((double)hi[0], scalbn(1.0, sc - 24), (double)lo[0] * scalbn(1.0, sc - 48));
            if (ea == 1025) D = nan("");
            if (in) D *= cl[b + l];
            if (in && lfac) D *= lfac[l];
            const int base = lane & ~3;
            if (S0) {
                const double v = __shfl_sync(0xffffffffu, D, base | (((l + m) & 1) ? 2 : 0) | (col & 1));
                if (in && col < 2) atomicAdd(Gout + 2 * (b + l) + col, v);
            } else {
                // P = (D0, D1), Q = sgs par (D2, -D3); G = -(P + Q) / 2, C = (-(P im - Q im), P re - Q re) / 2
                const bool im = col == 1 || col == 2;
                const double P = __shfl_sync(0xffffffffu, D, base | (im ? 1 : 0));
                double Q = __shfl_sync(0xffffffffu, D, base | (im ? 3 : 2));
                const double f = ((l + m) & 1) ? -sgs : sgs;
                Q *= im ? -f : f;
                const double v = col < 2 ? -0.5 * (P + Q) : col == 2 ? -0.5 * (P - Q) : 0.5 * (P - Q);
                if (in && (col < 2 || ncomp > 1)) atomicAdd((col < 2 ? Gout : Cout) + 2 * (b + l) + (col & 1), v);
            }
        }
    } else {
        // ---------------- ring warps
        const double xs = act ? (side ? -px[p] : px[p]) : 0.0;
        // fixed point once every ring of the warp is past its turning point (rec64.cuh)
        const int Es = es[m];
        const long long XQ = fix62(xs, 1);  // Q61
        const int xh = (int)(XQ >> 31), xl = (int)XQ & 0x7FFFFFFF;
        const bool idle = c_me == TC_NEVER;
        const long long rnd = idle ? 0 : FIX_ROUND;
        bool fixed = false;
        const bool may_fix = __any_sync(0xffffffffu, !idle);
        const uint32_t boff = (rid >> 3) * A6_B_LBO + (rid & 7) * 16;
        int gc = 0, bad = 0;
        for (int lb = lstart; lb <= L; lb += A6_KC, ++gc) {
            const int buf = gc & 1, ck = (lb - l0) / A6_KC;
            if (gc >= 2) bad |= !mbar_wait(bempty0 + 8 * buf, ((gc - 2) >> 1) & 1, wlim);
            bad = __any_sync(0xffffffffu, bad | *s_bad);
            if (bad) break;
            unsigned char *sB = sm + A6_OFF_B + buf * A6_BBUF + boff;
            const bool live = ck >= c_me;  // before its first chunk a ring holds its table state and writes zero digits
            const int El = ebm[ck];
            if (may_fix && !fixed) {
                const double2 a = __ldg(ag + b + lb);
                fixed = __all_sync(0xffffffffu, idle || (live && fix_ready(cur, prev, e, a.x, a.y, xs, Es, El)));
                if (fixed) {
                    cur = __longlong_as_double(idle ? 0 : fix62(cur, Es));
                    prev = __longlong_as_double(idle ? 0 : fix62(prev, Es));
                }
            }
            if (fixed) {
                const int sh = 7 + El - Es;
                long long U = __double_as_longlong(cur), V = __double_as_longlong(prev);
#pragma unroll
                for (int lh = 0; lh < 2; ++lh) {
                    uint32_t pk[A6_ND][4];
#pragma unroll
                    for (int j2 = 0; j2 < 4; ++j2) {
                        const int l = lb + 8 * lh + 2 * j2;
                        const FixCoef q0 = fix_load(fx + b + min(l, L)), q1 = fix_load(fx + b + min(l + 1, L));
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
#pragma unroll
                    for (int k = 0; k < A6_ND; ++k)
                        *reinterpret_cast<uint4 *>(sB + (2 * k + lh) * A6_B_SBO) =
                            make_uint4(pk[k][0], pk[k][1], pk[k][2], pk[k][3]);
                }
                cur = __longlong_as_double(U);
                prev = __longlong_as_double(V);
            } else if (live) {
#pragma unroll
                for (int lh = 0; lh < 2; ++lh) {
                    const int nb = 1030 + El - e;  // e < 0: every digit 0
                    uint32_t pk[A6_ND][4];
#pragma unroll
                    for (int j2 = 0; j2 < 4; ++j2) {
                        unsigned long long w2[2];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            // a_L = 0: values past lmax stay bounded, and the epilogue ignores them
                            const double2 a = __ldg(ag + b + min(lb + 8 * lh + 2 * j2 + h, L));
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
                    for (int k = 0; k < A6_ND; ++k)
                        *reinterpret_cast<uint4 *>(sB + (2 * k + lh) * A6_B_SBO) =
                            make_uint4(pk[k][0], pk[k][1], pk[k][2], pk[k][3]);
                    if (e < 0 && ((__double2hiint(cur) >> 20) & 0x7FF) > 1023 + 200) {
                        cur *= 0x1p-512;
                        prev *= 0x1p-512;
                        e += 512;
                    }
                }
            } else {
#pragma unroll
                for (int k = 0; k < 2 * A6_ND; ++k)
                    *reinterpret_cast<uint4 *>(sB + k * A6_B_SBO) = make_uint4(0u, 0u, 0u, 0u);
            }
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(bfull0 + 8 * buf);
        }
        if (bad) *s_bad = 1;
    }
    tc_fence_before();
    __syncthreads();
    if (*s_bad) {  // the block's part of the sums is missing
        if (tid == 0 && status) atomicOr(status, 1);
        add_nan(Gout, !S0 && ncomp > 1 ? Cout : nullptr, b + l0, L + 1 - l0, tid, A6_THREADS);
    }
    if (warp == A6_MMA) {
        // after a wait that ran out, wherever it did, the MMAs issued may still be in flight
        if (*s_bad && issued > 0) mbar_wait(bempty0 + 8 * ((issued - 1) & 1), ((issued - 1) >> 1) & 1);
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tbase, 512);
    }
}

// One request's adjoint into G (and C), zeroed by the caller: the pole pair in
// closed form, every other pair on the tensor cores (a last block with few rings
// costs less than these on the CUDA cores: spin 0, 257 pairs, lmax 512 0.78 ms with
// them there, 0.42 without, 1300 pairs 24.8 and 19.1; spin 2, 129 pairs 0.52 and
// 0.15, 898 pairs 21.6 and 12.4).
int leg_adjoint_tc64(const cunusht_plan_s *P, int npairs, const double *x, const int *rn, const int *rs, int ld,
                     int pole, int pole_rn, int pole_rs, bool cc, int spin, int ncomp, const double2 *H,
                     const double *lf, double2 *G, double2 *C, cudaStream_t st) {
    const double2 *stv = P->d_t6_stv[cc ? 1 : 0][spin];
    const short2 *ste = P->d_t6_ste[cc ? 1 : 0][spin];
    const RingLog *lsc = P->d_t6_lsc[cc ? 1 : 0];
    const int st_ld = npairs, L = P->lmax;
    const bool has_pole = pole == 0 && npairs > 1;
    if (has_pole) {
        ++x, ++rn, ++rs, ++lsc;
        if (stv) ++stv, ++ste;
        --npairs;
    }
    const int per = spin == 0 ? A6_R : A6_R / 2;
    auto launch = [&](auto kern) {
        CU_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, A6_BYTES));
        kern<<<dim3((npairs + per - 1) / per, P->mmax + 1), A6_THREADS, A6_BYTES, st>>>(
            L, spin, ncomp, H, ld, lf, P->d_t6_ag[spin], P->d_t6_fx[spin], P->d_t6_cl[spin], P->d_t6_eb[spin],
            P->d_t6_es[spin], P->d_t6_woff[spin], P->d_t6_lg0[spin], npairs, x, lsc, rn, rs, stv, ste, st_ld, (double *)G, (double *)C, P->wait_limit, P->d_status);
        CU_LAUNCH_CHECK();
        return CUNUSHT_OK;
    };
    RC_TRY(spin == 0 ? launch(k_leg_adj_tc64<true>) : launch(k_leg_adj_tc64<false>));
    if (has_pole) RC_TRY(leg_adj_pole_pair(P, 1, spin, ncomp, H, 0, ld, lf, pole_rn, pole_rs, G, C, 0, st));
    return CUNUSHT_OK;
}

}  // namespace cunusht
