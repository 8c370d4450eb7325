// Double-double GEMV: y := alpha*op(A)*x + beta*y (mgemv.cpp:237-275).
//
// beta pre-pass first (mf_kernels.h:63-68: beta == 0 zeroes y, beta == 1
// leaves it), then nothing more when alpha == 0, as in the reference.
//
// mgemv_ forms the products of base-256 limbs on the tensor cores
// (k_gemv_limb below; limbmma.cuh), exact sums per output and chunk of the
// reduction, combined as extended floats in a fixed order; y := y + alpha*s is
// rounded once to double-double. The FP64 pipe, which would bound a
// double-double multiply-add at a fraction of HBM speed, is not used in the
// loop.
// mgemv_n_noalloc keeps the FP64 accumulation (TwoProduct + TwoSum into a
// (sum, error) pair, renormalised every 32 terms, the lo*lo product dropped as
// in mdot.cpp:60-64) so that its partial sums fit its fixed scratch array.
#include <cuda_fp16.h>

#include <algorithm>
#include <mutex>

#include "dd.cuh"
#include "fixacc.cuh"
#include "limbmma.cuh"
#include "level3.h"
#include "runtime.h"

namespace mw {

namespace {

__device__ __forceinline__ int64_t vidx(int64_t i, int64_t n, int64_t inc)
{
    return inc >= 0 ? i * inc : (n - 1 - i) * (-inc);
}

__device__ __forceinline__ void acc_prod(double &s, double &e, double2 a, double2 b)
{
    double p, pe, t;
    dd::two_prod(a.x, b.x, p, pe);
    e = __fma_rn(a.x, b.y, e);
    e = __fma_rn(a.y, b.x, e);
    e = __dadd_rn(e, pe);
    dd::two_sum(s, p, s, t);
    e = __dadd_rn(e, t);
}

__global__ void k_scale_vec(int64_t n, dd::real beta, int beta_kind, double2 *y, int64_t incy)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double2 *p = y + vidx(i, n, incy);
        if (beta_kind == 0) *p = make_double2(0.0, 0.0);
        else dd::store(p, dd::mul_exact(beta, dd::load(p)));
    }
}

__global__ void k_gemv_n_partial(int64_t m, int64_t n, const double2 *A, int64_t lda, const double2 *x, int64_t incx,
                                 int64_t chunk, double2 *part)
{
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= m) return;
    int64_t j0 = blockIdx.y * chunk, j1 = min(n, j0 + chunk);
    double s = 0.0, e = 0.0;
    int cnt = 0;
    for (int64_t j = j0; j < j1; ++j) {
        acc_prod(s, e, A[i + j * lda], x[vidx(j, n, incx)]);
        if (++cnt == 32) {
            dd::fast_two_sum(s, e, s, e);
            cnt = 0;
        }
    }
    double h, l;
    dd::two_sum(s, e, h, l);
    part[blockIdx.y * m + i] = make_double2(h, l);
}

__global__ void k_gemv_n_final(int64_t m, int nchunks, const double2 *part, dd::real alpha, double2 *y,
                               int64_t incy)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        dd::real s = dd::load(part + i);
        for (int c = 1; c < nchunks; ++c) s = dd::add_fast(s, dd::load(part + (int64_t)c * m + i));
        double2 *py = y + vidx(i, m, incy);
        dd::store(py, dd::add_exact(dd::load(py), dd::mul_exact(alpha, s)));
    }
}

// ---- byte-limb kernel (mgemv_) ----------------------------------------------------------
//
// One kernel for both directions: output r = 0..rows-1, reduction index
// c = 0..len-1, element (r, c) at A[r * rs + c * cs]. A warp takes 32 outputs
// in two MMA tiles; lane (g, t) = (lane / 4, lane % 4) owns the elements of
// outputs g, g + 8, g + 16, g + 24 at every fourth reduction index, and their
// aligned limbs (limbmma.cuh) are directly its share of the MMA operand A: the
// K slots of lane t in MMA u are limbs 4u..4u+3 of its element. Operand B holds
// the limbs of x as a Toeplitz band: slot (t, q) of result column s is limb
// s - q of x at t's index, so column s collects every product of weight
// 2^(8s), s = 7..30 in three N tiles (lower ones are below 2^-160 of the
// block). 10 of the 12 (u, tile) products are not identically zero. A lane's
// six distinct B pairs are 24 consecutive limbs of x from an offset that
// depends only on g: they are laid out once per window of 32 indices in shared
// memory and read with three 16-byte loads.
//
// Exactness: x's limbs are balanced (|.| <= 128), 15 of them, A's are bytes, at
// most 16, so a column grows by at most 16 * 255 * 128 per index and stays below
// 2^24 units for a window's 32; then it moves to an int32 (at most 64 windows
// per block). Each output keeps a block exponent: a product of exponent ep is
// aligned by B - ep bits, rounded to nearest where that cuts it. The first one
// above the block folds the sums into an extended float in shared memory and
// moves B to three bits above that product (with one bit of margin the moves
// cost 8 % on uniform and 50 % on normally distributed entries). So a product is
// off by at most half of 2^-113 of the largest of its output and chunk. Cut to
// four bits of margin, one dominating product among 2000 equal-signed ones made
// it 1.1 units of 2^-104 sum |a x|, now 0.1, at the same speed.
//
// Zeros, alignments beyond a word and products up to nine bits above their block
// go through a loop of their own, which shifts any way (the block moves at the
// window's end), and groups of zeros leave it early. 8192^2 N, us, with the
// general decode for each such group, as the digit form was, and now: 1 % zeros
// 538, 729 and 485; 90 % 755, 569 and 530; every fourth x zero 567, 492 and 488;
// a triangle 535, 383 and 335; exponents over 2^40 876, 519 and 540; dense 301,
// 493 and 301.
//
// Bound: HBM (16 B per element) in principle, instruction issue in practice:
// about 80 per element, where the 24-bit digit form with 19 IMAD.WIDE per
// product and a thread per row (N) or a block per column (T) took 151.
// Measured on one GB300, whole call: 16384^2 N 1.67 -> 1.01 ms (2.57 ->
// 4.27 TB/s), T 1.01 ms (2.12 -> 4.26 TB/s), 7001 x 5003 T 0.45 -> 0.19 ms;
// without the decode and alignment the same loads take 0.69 ms. Also measured
// at 16384^2 N: one 16-output tile per warp with two or three blocks per SM
// 1.11 ms (more shared-memory reads and set-up per element), loads into
// registers one group ahead in place of the cp.async ring 1.29 ms.

constexpr int kShort = 32;                // reductions up to this take a thread per output
constexpr int kWin = 32;                  // reduction indices per window
constexpr int kMaxChunk = 64 * kWin;      // per block: int32 column sums stay below 2^30
constexpr int kColWords = 104;            // B entry of one index: 8 x 12 words, its exponent, pad (8 mod 32 words:
                                          // the 8 lanes of a 16-byte phase read distinct banks)
constexpr int kR = 2, kE = 2 * kR;        // 16-output tiles per warp, elements per lane and group
constexpr int kStages = 4;                // groups of four indices in flight per thread (cp.async)
constexpr int kZeroE = -(1 << 20), kBadE = 1 << 20;   // exponent marks: zero (or past the end), non-finite
constexpr int kOver = 9;                  // bits a product may lie above its block
constexpr int kNoBlock = -(1 << 22);                  // an output that has seen no nonzero product yet

struct GemvArgs {
    const double2 *A;
    const double2 *x;
    double2 *y;
    fx::XFPod *part;      // [chunk][output]; null: one chunk, y updated here
    int64_t rows, len, rs, cs, incx, incy;
    int64_t rowblocks, chunk;
    dd::real alpha, beta;
    int beta_kind;
};

// y(i) := y(i) + alpha * sum_c part(c, i), one rounding to double-double.
__device__ __forceinline__ void fx_update_y(double2 *py, const xfp::XF &xa, xfp::XF s, bool bad)
{
    const double2 y0 = *py;
    if (bad) {
        *py = make_double2(__longlong_as_double(0x7ff8000000000000ll), __longlong_as_double(0x7ff8000000000000ll));
        return;
    }
    xfp::XF t = xfp::xf_mul(xa, s);
    if (!fx::finite_dd(y0)) {
        double h, l;
        xfp::xf_to_dd(t, h, l);
        dd::store(py, dd::add_exact(dd::make(y0.x, y0.y), dd::make(h, l)));
        return;
    }
    t = xfp::xf_add(xfp::xf_from_dd(y0.x, y0.y), t);
    double h, l;
    xfp::xf_to_dd(t, h, l);
    *py = make_double2(h, l);
}

// y := beta * y, then y := y + alpha * s
__device__ __forceinline__ void gemv_store(const GemvArgs &g, int64_t r, const xfp::XF &xa, const xfp::XF &s, bool bad)
{
    double2 *py = g.y + vidx(r, g.rows, g.incy);
    if (g.beta_kind == 0) *py = make_double2(0.0, 0.0);
    else if (g.beta_kind == 2) dd::store(py, dd::mul_exact(g.beta, dd::load(py)));
    fx_update_y(py, xa, s, bad);
}

__global__ void __launch_bounds__(256, 2) k_gemv_limb(const GemvArgs g)
{
    __shared__ __align__(16) uint32_t s_b[2][kWin * kColWords];
    __shared__ __align__(16) uint32_t s_x[2][kWin][36];   // limbs in descending order, two alignments
    __shared__ int s_e[2][kWin];
    __shared__ fx::XFPod s_tot[8][16 * kR];
    extern __shared__ __align__(16) unsigned char s_stage[];   // [stage][element][thread] 16 bytes
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int lg = lane >> 2, lt = lane & 3;
    const int64_t rb = blockIdx.x % g.rowblocks, ch = blockIdx.x / g.rowblocks;
    const int64_t k0 = ch * g.chunk;
    const int kn = (int)min(g.chunk, g.len - k0);
    const int nwin = (kn + kWin - 1) / kWin;
    const int64_t r0 = (rb * nw + wid) * (16 * kR);

    for (int i = threadIdx.x; i < 2 * kWin * 36; i += blockDim.x) (&s_x[0][0][0])[i] = 0u;
    if (lane < 16 * kR) s_tot[wid][lane] = fx::XFPod{0ull, 0ull, 0, 2};

    // x: lane per index of a window, windows dealt to the warps in turn
    const double2 *xbase = g.x;
    auto load_x = [&](int win) {
        const int c = win * kWin + lane;
        return c < kn ? xbase[vidx(k0 + c, g.len, g.incx)] : make_double2(0.0, 0.0);
    };
    double2 xnext = load_x(wid);
    auto split_x = [&](int win) {
        const fx::Op o = fx::decode(xnext);
        xnext = load_x(win + nw);
        // balanced base-256 digits of W: the bytes of W + 0x80..80, less 128 each
        uint32_t w[4];
        asm("add.cc.u32 %0, %4, 0x80808080;\n\t"
            "addc.cc.u32 %1, %5, 0x80808080;\n\t"
            "addc.cc.u32 %2, %6, 0x80808080;\n\t"
            "addc.u32 %3, %7, 0x80808080;"
            : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
            : "r"(o.w[0]), "r"(o.w[1]), "r"(o.w[2]), "r"(o.w[3]));
        const __half2 sg = __float2half2_rn((o.flags & fx::kNeg) ? -1.0f : 1.0f);
        const __half2 off = __float2half2_rn((o.flags & fx::kNeg) ? 1152.0f : -1152.0f);
        // limbs q (high half) and q + 1 (low half): 1024 + byte, times the sign, minus 1152
        uint32_t ev[8], od[8];
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            const uint32_t raw = __byte_perm(w[p >> 1], 0x64646464u, (p & 1) ? 0x4243 : 0x4041);
            const __half2 h = __hfma2(*reinterpret_cast<const __half2 *>(&raw), sg, off);
            ev[p] = *reinterpret_cast<const uint32_t *>(&h);
        }
#pragma unroll
        for (int p = 0; p < 8; ++p)   // limbs 2p - 1 (high half) and 2p (low half)
            od[p] = __byte_perm(ev[p], p ? ev[p > 0 ? p - 1 : 0] : 0u, 0x5432);
        // limb q at position 22 - q: pairs from even positions in words 0.., from odd ones in words 17..
        uint32_t *sx = s_x[win & 1][lane];
#pragma unroll
        for (int p = 0; p < 8; p += 4) {
            *reinterpret_cast<uint4 *>(sx + 8 - p) = make_uint4(od[p + 3], od[p + 2], od[p + 1], od[p]);
            *reinterpret_cast<uint4 *>(sx + 24 - p) = make_uint4(ev[p + 3], ev[p + 2], ev[p + 1], ev[p]);
        }
        s_e[win & 1][lane] = (o.flags & fx::kBad) ? kBadE : ((o.flags & fx::kZero) ? kZeroE : o.e - lmb::kExpBias);
    };
    auto expand = [&](int win) {
        const int buf = win & 1;
        for (int idx = threadIdx.x; idx < kWin * 8; idx += blockDim.x) {
            const int c = idx >> 3, q = idx & 7;
            const uint32_t *src = &s_x[buf][c][((q & 1) ? 0 : 17) + ((7 - q) >> 1)];
            uint32_t *dst = &s_b[buf][c * kColWords + q * 12];
#pragma unroll
            for (int v = 0; v < 3; ++v)
                *reinterpret_cast<uint4 *>(dst + 4 * v) =
                    make_uint4(src[4 * v], src[4 * v + 1], src[4 * v + 2], src[4 * v + 3]);
            if (q == 0) s_b[buf][c * kColWords + 96] = (uint32_t)s_e[buf][c];
        }
    };
    __syncthreads();
    for (int w = 0; w < 2 && w < nwin; ++w)
        if (wid == w % nw) split_x(w);
    __syncthreads();
    expand(0);
    __syncthreads();

    const bool active = r0 < g.rows;
    // lane (g, t): outputs r0 + g + 8e, e = 0..3 (past the last one its
    // elements again, their sums are not stored), indices t, t + 4, ..
    const int64_t row0 = min(r0 + lg, g.rows - 1);
    const double2 *pn = g.A + row0 * g.rs + (k0 + lt) * g.cs;
    int64_t dr[kE - 1];
#pragma unroll
    for (int e = 0; e < kE - 1; ++e) dr[e] = (min(r0 + lg + 8 * (e + 1), g.rows - 1) - row0) * g.rs;
    const int64_t step = 4 * g.cs;
    // a lane's slot in its warp's 512 bytes: what is contiguous in memory (over
    // t for A^T, over g else) stays contiguous, as cp.async writes 32-byte
    // sectors; g is xored with 2t so that the reads are free of bank conflicts
    const uint32_t slot = wid * 512u + (g.cs == 1 ? lane * 16u : lt * 128u + ((lg ^ (2 * lt)) * 16u));
    const uint32_t st0 = (uint32_t)__cvta_generic_to_shared(s_stage) + slot, st_e = blockDim.x * 16u;
    const int nit = (kn + 3) >> 2;
    // the four elements of group it into its stage of the thread's own ring
    auto load_a = [&](int it) {
        if (it < nit) {
            const double2 *q = pn;
            const int past = 4 * it + lt - (kn - 1);
            if (past > 0) q -= past * g.cs;   // past the end: the last index again (its limbs of x are zero there)
            const uint32_t d = st0 + (uint32_t)(it & (kStages - 1)) * kE * st_e;
            lmb::cp_async16(d, q);
#pragma unroll
            for (int e = 0; e < kE - 1; ++e) lmb::cp_async16(d + (e + 1) * st_e, q + dr[e]);
            pn += step;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int blk[kE];
    uint32_t bad = 0;
    float acc[kR][3][4];
    int sum[kR][3][4];
#pragma unroll
    for (int h = 0; h < kR; ++h)
#pragma unroll
        for (int v = 0; v < 3; ++v)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                blk[i % kE] = kNoBlock;
                acc[h][v][i] = 0.0f;
                sum[h][v][i] = 0;
            }
    auto flush = [&]() {
#pragma unroll
        for (int h = 0; h < kR; ++h)
#pragma unroll
            for (int v = 0; v < 3; ++v)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    sum[h][v][i] += __float2int_rn(acc[h][v][i] * 16777216.0f);
                    acc[h][v][i] = 0.0f;
                }
    };
    // the column sums into the outputs' extended floats: outputs r0 + g + 8e of the set bits e
    auto fold = [&](uint32_t which) {
        flush();
#pragma unroll
        for (int e = 0; e < kE; ++e) {
            if (!(which >> e & 1u)) continue;
            uint64_t W[4] = {0, 0, 0, 0};
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                int *c = &sum[e >> 1][v][2 * (e & 1)];
                lmb::add_at(W, (int64_t)c[0] + ((int64_t)c[1] << 8), 64 * v + 16 * lt);
                c[0] = c[1] = 0;
            }
            lmb::lane_sum256(W, 4);
            if (lt == 0 && blk[e] != kNoBlock) {
                fx::XFPod *tot = &s_tot[wid][lg + 8 * e];
                *tot = fx::to_pod(xfp::xf_add(fx::from_pod(*tot), fx::w256_to_xf(W, 56 + blk[e])), false);
            }
        }
        __syncwarp();
    };

    // += the aligned elements' limbs times x's
    auto products = [&](const uint32_t (&w)[kE][4], const uint32_t (&sgn)[kE], const uint32_t *sb) {
        uint32_t f[12];
#pragma unroll
        for (int v = 0; v < 3; ++v) {
            const uint4 q = *reinterpret_cast<const uint4 *>(sb + lg * 12 + 4 * v);
            f[4 * v] = q.x; f[4 * v + 1] = q.y; f[4 * v + 2] = q.z; f[4 * v + 3] = q.w;
        }
#pragma unroll
        for (int h = 0; h < kR; ++h)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t a0 = lmb::limbs_lo(w[2 * h][u], sgn[2 * h]);
                const uint32_t a1 = lmb::limbs_lo(w[2 * h + 1][u], sgn[2 * h + 1]);
                const uint32_t a2 = lmb::limbs_hi(w[2 * h][u], sgn[2 * h]);
                const uint32_t a3 = lmb::limbs_hi(w[2 * h + 1][u], sgn[2 * h + 1]);
#pragma unroll
                for (int v = 0; v < 3; ++v) {
                    if (v == 2 && u < 2) continue;        // limbs 16 and up of x: zero
                    const int b = 2 * (2 - (2 * v - u));   // pair of window 2v - u
                    lmb::mma16816(acc[h][v], a0, a1, a2, a3, f[b], f[b + 1]);
                }
            }
    };

    if (active)
        for (int it = 0; it < kStages - 1; ++it) load_a(it);
    bool any_shift = false, idle = false, far = false;
    uint32_t over = 0u;   // byte e: bits by which output r0 + g + 8e has gone above its block in this window
    for (int win = 0; win < nwin; ++win) {
        if (win + 1 < nwin) expand(win + 1);
        if (win + 2 < nwin && wid == (win + 2) % nw) split_x(win + 2);
        if (active) {
            const uint32_t *sb = s_b[win & 1] + lt * kColWords;
            const int it1 = min(8 * win + 8, nit);
            int it = 8 * win;
            while (it < it1) {
                // groups whose elements are all on the straight line, within a word of their block
#pragma unroll 1
                for (; it < it1 && !any_shift; ++it, sb += 4 * kColWords) {
                    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
                    const unsigned char *cur = s_stage + slot + (size_t)(it & (kStages - 1)) * kE * st_e;
                    uint32_t w[kE][4], sgn[kE];
                    int sh[kE];
                    const int xe = (int)sb[96];
                    bool fast = true;
#pragma unroll
                    for (int e = 0; e < kE; ++e) {
                        const double2 v = *reinterpret_cast<const double2 *>(cur + e * st_e);
                        int eh;
                        sh[e] = blk[e] - xe - lmb::hi_exp(v);
                        const bool ok = lmb::split_fast(v, w[e], eh, lmb::half_unit(sh[e]));
                        fast = fast && ok && (uint32_t)sh[e] < 32u;
                        sgn[e] = (uint32_t)__double2hiint(v.x) & 0x80000000u;
                    }
                    if (!__all_sync(0xffffffffu, fast)) {
                        any_shift = true;
                        break;
                    }
#pragma unroll
                    for (int e = 0; e < kE; ++e) lmb::shr_short(w[e], sh[e]);
                    load_a(it + kStages - 1);   // into the stage read in the previous turn
                    products(w, sgn, sb);
                }
                // the others, in a loop of their own (in the same one they cost it 5 to 15 %), until
                // a group that the first loop takes
#pragma unroll 1
                for (; it < it1 && any_shift; ++it, sb += 4 * kColWords) {
                    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
                    const unsigned char *cur = s_stage + slot + (size_t)(it & (kStages - 1)) * kE * st_e;
                    uint32_t w[kE][4], sgn[kE];
                    int sh[kE];
                    const int xe = (int)sb[96];
                    if (idle) {   // after a group of zeros, another one costs a look
                        bool dead = xe != kBadE;
#pragma unroll
                        for (int e = 0; e < kE; ++e) {
                            const double2 v = *reinterpret_cast<const double2 *>(cur + e * st_e);
                            dead = dead && (lmb::all_zero(v) || (xe == kZeroE && lmb::is_fast(v)));
                        }
                        if (__all_sync(0xffffffffu, dead)) {
                            load_a(it + kStages - 1);
                            continue;
                        }
                    }
                    // zeros, long alignments and products up to 2^kOver above their block (A's 16
                    // limbs hold 128 bits, W has 118; the block moves at the end of the window):
                    // the same decode, any shift
                    bool plain = xe != kBadE, live = false, fast = true, near = true;
                    uint32_t above = 0u;
#pragma unroll
                    for (int e = 0; e < kE; ++e) {
                        const double2 v = *reinterpret_cast<const double2 *>(cur + e * st_e);
                        int eh;
                        const bool ok = lmb::split_fast(v, w[e], eh), zero = lmb::all_zero(v);
                        const bool none = zero || xe == kZeroE;
                        sh[e] = blk[e] - xe - eh;
                        fast = fast && ok && (uint32_t)sh[e] < 32u;
                        near = near && ok && sh[e] < 32;
                        plain = plain && (ok || zero) && (sh[e] >= -kOver || none);
                        live = live || !none;
                        if (sh[e] < 0 && !none) above |= (uint32_t)min(-sh[e], kOver) << (8 * e);
                        sh[e] = none ? 127 : min(sh[e] + kOver, 127);   // at 127 nothing is left of a zero's W
                        sgn[e] = (uint32_t)__double2hiint(v.x) & 0x80000000u;
                    }
                    any_shift = !__all_sync(0xffffffffu, fast);
                    if (__all_sync(0xffffffffu, plain)) {
                        over = __vmaxu4(over, above);
                        idle = !__any_sync(0xffffffffu, live);
                        far = !__all_sync(0xffffffffu, near);
#pragma unroll
                        for (int e = 0; e < kE; ++e) {
                            uint32_t sv[4];
#pragma unroll
                            for (int i = 3; i > 0; --i) w[e][i] = __funnelshift_l(w[e][i - 1], w[e][i], kOver);
                            w[e][0] <<= kOver;
                            lmb::shr_round(w[e], sh[e], sv);
#pragma unroll
                            for (int i = 0; i < 4; ++i) w[e][i] = sv[i];
                        }
                    } else {
                        // operands off the straight-line path, a larger block
                        idle = false;
                        int ep[kE], top[kE];
                        uint32_t raise = 0u, move = 0u;   // blocks that go up, those of them with sums to fold
#pragma unroll
                        for (int e = 0; e < kE; ++e) {
                            const fx::Op o = fx::decode(*reinterpret_cast<const double2 *>(cur + e * st_e));
#pragma unroll
                            for (int i = 0; i < 4; ++i) w[e][i] = o.w[i];
                            const bool no = xe == kBadE || (o.flags & fx::kBad);
                            if (no) bad |= 1u << e;
                            ep[e] = (no || xe == kZeroE || (o.flags & fx::kZero)) ? kNoBlock : o.e + lmb::kExpBias + xe;
                            const int o8 = (int)(over >> (8 * e)) & 255;
                            top[e] = max(ep[e], o8 ? blk[e] + o8 : kNoBlock);
                            top[e] = max(top[e], __shfl_xor_sync(0xffffffffu, top[e], 1));
                            top[e] = max(top[e], __shfl_xor_sync(0xffffffffu, top[e], 2));
                            if (top[e] != kNoBlock && top[e] > blk[e]) {
                                raise |= 1u << e;
                                if (blk[e] != kNoBlock) move |= 1u << e;
                            }
                        }
                        over = 0u;
                        move = __reduce_or_sync(0xffffffffu, move);
                        if (move) fold(move);
#pragma unroll
                        for (int e = 0; e < kE; ++e) {
                            if (raise >> e & 1u) blk[e] = top[e] + 3;
                            const int d = ep[e] == kNoBlock ? 127 : min(blk[e] - ep[e], 127);
                            uint32_t sv[4];
                            lmb::shr_round(w[e], d, sv);
#pragma unroll
                            for (int i = 0; i < 4; ++i) w[e][i] = ep[e] == kNoBlock ? 0u : sv[i];
                        }
                    }
                    load_a(it + kStages - 1);   // into the stage read in the previous turn
                    if (!idle) products(w, sgn, sb);
                }
            }
            flush();
            // blocks that products went above go up, three bits above those, where that is what keeps
            // the groups in the second loop
            if (!far && __any_sync(0xffffffffu, over != 0u)) {
                over = __vmaxu4(over, __shfl_xor_sync(0xffffffffu, over, 1));
                over = __vmaxu4(over, __shfl_xor_sync(0xffffffffu, over, 2));
                uint32_t move = 0u;
#pragma unroll
                for (int e = 0; e < kE; ++e) move |= (over >> (8 * e) & 255u) ? 1u << e : 0u;
                fold(__reduce_or_sync(0xffffffffu, move));
#pragma unroll
                for (int e = 0; e < kE; ++e) {
                    const int o8 = (int)(over >> (8 * e)) & 255;
                    if (o8) blk[e] += o8 + 3;
                }
                over = 0u;
            }
        }
        __syncthreads();
    }
    if (!active) return;
    fold((1u << kE) - 1u);
    uint32_t mine = 0;   // lane r: whether output r saw a non-finite operand
#pragma unroll
    for (int e = 0; e < kE; ++e) {
        const uint32_t m = __ballot_sync(0xffffffffu, (bad >> e) & 1u);
        if ((lane >> 3) == e) mine = (m >> (4 * (lane & 7))) & 15u;
    }
    const int64_t r = r0 + lane;
    if (lane < 16 * kR && r < g.rows) {
        fx::XFPod p = s_tot[wid][lane];
        if (g.part) {
            if (mine) p.flags |= 4;
            g.part[ch * g.rows + r] = p;
        } else {
            gemv_store(g, r, xfp::xf_from_dd(g.alpha.hi, g.alpha.lo), fx::from_pod(p), mine != 0);
        }
    }
}

// Short reductions (len <= kShort): a thread per output, its products added in fixed
// point (fixacc.cuh) against x's digits in shared memory, y updated in the same
// launch. The limb kernel works in windows of 32 indices and sets up shared memory
// per 256 outputs. Whole call, us, limb kernel and this one: 2,000,000 outputs N,
// len 1 329 and 99, 8 369 and 187, 24 456 and 365, 32 577 and 459, 48 606 and 635;
// 5000 outputs, len 4 38 and 34, 24 41 and 39, 32 42 and 44.
__global__ void __launch_bounds__(256) k_gemv_short(const GemvArgs g)
{
    __shared__ fx::Dig s_d[kShort];
    bool mine = true;   // x holds neither zeros nor non-finite values
    if (threadIdx.x < (unsigned)g.len) {
        s_d[threadIdx.x] = fx::to_dig(fx::decode(g.x[vidx(threadIdx.x, g.len, g.incx)]));
        mine = (s_d[threadIdx.x].flags & (fx::kZero | fx::kBad)) == 0;
    }
    const bool plain = __syncthreads_and(mine) != 0;
    const xfp::XF xa = xfp::xf_from_dd(g.alpha.hi, g.alpha.lo);
    for (int64_t r = blockIdx.x * 256ll + threadIdx.x; r < g.rows; r += gridDim.x * 256ll) {
        const double2 *a = g.A + r * g.rs;
        fx::Acc acc;
        acc.reset();
        int c = 0;
        for (; c + 4 <= (int)g.len; c += 4) {   // four in flight, one block-exponent test for normal operands
            double2 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u, a += g.cs) v[u] = __ldcs(a);
            if (fx::decode_is_fast(v[0]) && fx::decode_is_fast(v[1]) && fx::decode_is_fast(v[2]) &&
                fx::decode_is_fast(v[3]) && plain) {
                fx::Op o[4];
                int e[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    o[u] = fx::decode_fast(v[u]);
                    e[u] = o[u].e + s_d[c + u].e;
                }
                acc.admit(max(max(e[0], e[1]), max(e[2], e[3])));
#pragma unroll
                for (int u = 0; u < 4; ++u) acc.mul_fast(o[u], s_d[c + u], acc.B - e[u]);
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u) acc.add_core(fx::decode(v[u]), s_d[c + u]);
            }
        }
        for (; c < (int)g.len; ++c, a += g.cs) acc.add_core(fx::decode(__ldcs(a)), s_d[c]);
        gemv_store(g, r, xa, acc.finish(), acc.bad);
    }
}

// The chunks' sums of each output, LANES lanes per output in a fixed order,
// then the update of y.
template <int LANES>
__global__ void __launch_bounds__(256) k_gemv_fold(const GemvArgs g, int nchunks)
{
    const xfp::XF xa = xfp::xf_from_dd(g.alpha.hi, g.alpha.lo);
    const int sub = threadIdx.x % LANES;
    const int64_t r = (int64_t)blockIdx.x * (256 / LANES) + threadIdx.x / LANES;
    xfp::XF s;
    s.zero = true; s.neg = false; s.m = 0; s.e = 0;
    bool bad = false;
    if (r < g.rows) {
        for (int c = sub; c < nchunks; c += LANES) {
            const fx::XFPod p = g.part[(int64_t)c * g.rows + r];
            bad |= (p.flags & 4) != 0;
            s = xfp::xf_add(s, fx::from_pod(p));
        }
    }
    for (int off = LANES / 2; off > 0; off >>= 1) {
        s = xfp::xf_add(s, fx::xf_shfl_down(s, off));
        bad |= __shfl_down_sync(0xffffffffu, bad ? 1 : 0, off) != 0;
    }
    if (sub == 0 && r < g.rows) gemv_store(g, r, xa, s, bad);
}

}  // namespace

bool gemv_device(bool trans, int64_t m, int64_t n, dd_host alpha, const void *A, int64_t lda, const void *x,
                 int64_t incx, dd_host beta, int beta_kind, void *y, int64_t incy, const char *routine)
{
    const int64_t rows = trans ? n : m, len = trans ? m : n;
    const int sms = device_sm_count();
    const dd::real be = dd::make(beta.hi, beta.lo);
    if ((alpha.hi == 0.0 && alpha.lo == 0.0) || len <= 0) {
        if (beta_kind != 1) {
            int64_t blocks = (rows + 255) / 256;
            if (blocks > sms * 8) blocks = sms * 8;
            k_scale_vec<<<(unsigned)blocks, 256, 0, stream()>>>(rows, be, beta_kind, (double2 *)y, incy);
            count_launch();
        }
        return true;
    }
    GemvArgs g;
    g.A = (const double2 *)A;
    g.x = (const double2 *)x;
    g.y = (double2 *)y;
    g.rows = rows;
    g.len = len;
    g.rs = trans ? lda : 1;
    g.cs = trans ? 1 : lda;
    g.incx = incx;
    g.incy = incy;
    g.alpha = dd::make(alpha.hi, alpha.lo);
    g.beta = be;
    g.beta_kind = beta_kind;
    if (len <= kShort) {
        const int64_t blocks = std::min<int64_t>((rows + 255) / 256, 8ll * sms);
        g.part = nullptr;
        k_gemv_short<<<(unsigned)blocks, 256, 0, stream()>>>(g);
        count_launch();
        return true;
    }
    // 16 kR outputs per warp, up to eight warps per block: fewer where eight
    // would leave SMs without a block (a small product is bound by the latency
    // of its windows in turn, about 2 us each), and four where the last block
    // would hold mostly idle warps (268 outputs in 3 x 128, not 2 x 256:
    // 268 x 16000 N 107 -> 92 us)
    const int64_t units = ((rows + 16 * kR - 1) / (16 * kR)) * ((len + 2 * kWin - 1) / (2 * kWin));
    int nw = rows > 64 * kR ? 8 : (rows > 32 * kR ? 4 : (rows > 16 * kR ? 2 : 1));
    if (nw == 8 && (rows + 127) / 128 * 128 * 8 <= (rows + 255) / 256 * 256 * 7) nw = 4;
    while (nw > 1 && units < (int64_t)nw * sms) nw >>= 1;
    g.rowblocks = (rows + 16 * kR * nw - 1) / (16 * kR * nw);
    // the reduction in chunks of whole windows, in whole waves of the
    // resident blocks (two of eight warps per SM, three of fewer), at about
    // 640 indices (a block's set-up and final sums cost about 60)
    const int64_t wave = (nw == 8 ? 2ll : 3ll) * sms;
    int64_t waves = (len * g.rowblocks + 640 * wave - 1) / (640 * wave);
    int64_t nchunks = waves * wave / g.rowblocks;
    if (nchunks < 1) nchunks = 1;
    int64_t chunk = (len + nchunks - 1) / nchunks;
    chunk = (chunk + kWin - 1) / kWin * kWin;
    if (chunk > kMaxChunk) chunk = kMaxChunk;
    nchunks = (len + chunk - 1) / chunk;
    g.chunk = chunk;
    if (nchunks * g.rowblocks > INT32_MAX) {
        set_error(routine, MWBLAS_ERR_UNSUPPORTED, "matrix too large for the GEMV grid");
        return false;
    }
    fx::XFPod *part = nullptr;
    if (nchunks > 1) {
        part = (fx::XFPod *)dev_alloc(sizeof(fx::XFPod) * (size_t)(nchunks * rows), routine);
        if (!part) return false;
    }
    g.part = part;
    const size_t smem = (size_t)kStages * kE * 16 * 32 * nw;
    cudaFuncSetAttribute(k_gemv_limb, cudaFuncAttributeMaxDynamicSharedMemorySize, kStages * kE * 16 * 256);
    k_gemv_limb<<<(unsigned)(nchunks * g.rowblocks), 32 * nw, smem, stream()>>>(g);
    count_launch();
    if (part) {
        // eight lanes per output (27 chunks of 16384 outputs: 15 us, a warp each 31),
        // a warp for many chunks (a few outputs, a long reduction)
        if (nchunks <= 64) k_gemv_fold<8><<<(unsigned)((rows + 31) / 32), 256, 0, stream()>>>(g, (int)nchunks);
        else k_gemv_fold<32><<<(unsigned)((rows + 7) / 8), 256, 0, stream()>>>(g, (int)nchunks);
        count_launch();
        dev_free(part);
    }
    return true;
}

}  // namespace mw

// ---- GEMV without device allocation ----------------------------------------------------
//
// For callers that must not allocate device memory on the call path: code whose
// device memory is owned by its own allocator under a fixed budget (cudaMalloc
// there would bypass the budget), and code that cannot afford the driver
// allocator's locking or cudaFree's device-wide synchronisation while other
// work is in flight. mgemv_ itself allocates the per-chunk partial sums of
// the no-transpose kernel (and staging copies of host arrays); this variant
// keeps the partial sums in a file-scope device array instead.
//
// The array below is the only scratch. It is 1 MiB (65536 double-double
// partial sums), every GPU that loads the library holds it until the process
// exits, and all calls share it: two calls whose kernels overlap on the GPU
// (different streams, or different host threads) race on it. Nothing in it
// needs to start at zero: every entry a call reads was written earlier by the
// same call. The host learns its device address once per device, with that
// device current, on the first call made on that device; that first call
// should therefore come before any stream capture. The address is cached
// together with the CUDA context it was looked up in and looked up again
// when the calling thread's current context differs (after cudaDeviceReset,
// or on a context other than the device's primary one).

namespace mw {
namespace {

constexpr int64_t kNoAllocScratch = 65536;   // double2 entries (1 MiB)
static __device__ __align__(256) double2 g_gemv_noalloc_scratch[kNoAllocScratch];

std::mutex g_noalloc_mu;
double2 *g_noalloc_addr[64] = {};
void *g_noalloc_ctx[64] = {};

// The calling thread's current CUDA context (driver entry point, looked up once).
void *current_context()
{
    using Fn = int (*)(void **);
    static Fn fn = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return (Fn)f;
    }();
    void *ctx = nullptr;
    if (!fn || fn(&ctx) != 0) return nullptr;
    return ctx;
}

}  // namespace
}  // namespace mw

extern "C" int mgemv_n_noalloc(int64_t m, int64_t n, const mwblas_real64x2 *alpha, const mwblas_real64x2 *a,
                               int64_t lda, const mwblas_real64x2 *x, int64_t incx, const mwblas_real64x2 *beta,
                               mwblas_real64x2 *y, int64_t incy, void *cuda_stream)
{
    using namespace mw;
    const char *routine = "mgemv_n_noalloc";
    clear_error();
    if (!alpha || !beta) { set_error(routine, 3, "null alpha or beta"); return 3; }
    if (m < 0) { set_error(routine, 1, "m < 0"); return 1; }
    if (n < 0) { set_error(routine, 2, "n < 0"); return 2; }
    if (lda < (m > 1 ? m : 1)) { set_error(routine, 5, "lda too small"); return 5; }
    if (incx == 0) { set_error(routine, 7, "incx == 0"); return 7; }
    if (incy == 0) { set_error(routine, 10, "incy == 0"); return 10; }
    if (m > kNoAllocScratch) {
        set_error(routine, 1, "m exceeds the 65536-row limit of the fixed 1 MiB scratch array");
        return 1;
    }
    if (m == 0 || n == 0) return 0;
    const dd_host al{alpha->limbs[0], alpha->limbs[1]}, be{beta->limbs[0], beta->limbs[1]};
    const bool alpha0 = (al.hi == 0.0 && al.lo == 0.0);
    const int bk = (be.hi == 0.0 && be.lo == 0.0) ? 0 : ((be.hi == 1.0 && be.lo == 0.0) ? 1 : 2);
    if (alpha0 && bk == 1) return 0;
    if (!y || !is_dd_device_pointer(y) ||
        (!alpha0 && (!a || !x || !is_dd_device_pointer(a) || !is_dd_device_pointer(x)))) {
        set_error(routine, 9, "A, x and y must be 16-byte aligned device or managed memory (this entry point stages nothing)");
        return 9;
    }
    int dev = 0;
    if (!cuda_ok(cudaGetDevice(&dev), routine, "cudaGetDevice")) return MWBLAS_ERR_CUDA;
    if (dev < 0 || dev >= 64) { set_error(routine, MWBLAS_ERR_DEVICE, "device ordinal out of range"); return MWBLAS_ERR_DEVICE; }
    double2 *scratch;
    {
        // null before the runtime has initialised a context on this thread; the
        // lookup below initialises it, and the context is read again after it
        void *ctx = current_context();
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        if (!g_noalloc_addr[dev] || g_noalloc_ctx[dev] != ctx) {
            void *p = nullptr;
            cudaError_t st = cudaGetSymbolAddress(&p, g_gemv_noalloc_scratch);
            if (st != cudaSuccess) {
                g_noalloc_addr[dev] = nullptr;
                cuda_ok(st, routine, "cudaGetSymbolAddress(scratch)");
                return MWBLAS_ERR_CUDA;
            }
            g_noalloc_addr[dev] = (double2 *)p;
            g_noalloc_ctx[dev] = current_context();
        }
        scratch = g_noalloc_addr[dev];
    }
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
    cudaStream_t s = cuda_stream ? (cudaStream_t)cuda_stream : stream();
    if (bk != 1) {
        int64_t blocks = (m + 255) / 256;
        if (blocks > (int64_t)sms * 8) blocks = (int64_t)sms * 8;
        k_scale_vec<<<(unsigned)blocks, 256, 0, s>>>(m, dd::make(be.hi, be.lo), bk, (double2 *)y, incy);
        count_launch();
    }
    if (!alpha0) {
        int64_t rowblocks = (m + 255) / 256;
        int64_t nchunks = (4 * (int64_t)sms + rowblocks - 1) / rowblocks;
        if (nchunks > kNoAllocScratch / m) nchunks = kNoAllocScratch / m;
        if (nchunks > n) nchunks = n;
        if (nchunks < 1) nchunks = 1;
        int64_t chunk = (n + nchunks - 1) / nchunks;
        nchunks = (n + chunk - 1) / chunk;
        dim3 grid((unsigned)rowblocks, (unsigned)nchunks);
        k_gemv_n_partial<<<grid, 256, 0, s>>>(m, n, (const double2 *)a, lda, (const double2 *)x, incx, chunk, scratch);
        int64_t fb = (m + 255) / 256;
        if (fb > (int64_t)sms * 8) fb = (int64_t)sms * 8;
        k_gemv_n_final<<<(unsigned)fb, 256, 0, s>>>(m, (int)nchunks, scratch, dd::make(al.hi, al.lo), (double2 *)y,
                                                     incy);
        count_launch(2);
    }
    cudaError_t st = cudaGetLastError();
    if (st != cudaSuccess) {
        cuda_ok(st, routine, "kernel launch");
        return MWBLAS_ERR_CUDA;
    }
    return 0;
}
