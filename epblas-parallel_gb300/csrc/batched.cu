// Batched uneven-size double-double GEMM and TRSM (no reference counterpart:
// the reference's CPU baseline for this workload is an OpenMP loop over
// instances calling mgemm_/mtrsm_, whose nested calls run serially,
// mgemm_parallel.cpp:53-60).
//
// mgemm_grouped: one persistent kernel over all instances. The work list is
// every (instance, 32x32 output tile, K split); CTAs of 256 threads pull items
// from an atomic counter, so thousands of uneven instances keep all SMs busy.
// Each item runs the fixed-point arithmetic of the integer-pipe engine
// (gemm_fixed.cu, fixgemm.cuh): its A rows / B columns are scaled from an
// exponent scan over the item's own K range (no pre-pass, no extra scratch),
// converted to balanced 24-bit digits while staged, and multiplied with
// exact 64-bit column sums. Items of a split instance write partial tiles as
// extended floats; the CTA that completes a tile's last split sums the
// partials in split order (deterministic) and applies alpha/beta with one
// rounding. The per-call state (descriptors, work counter, split counters,
// partial tiles) is uploaded and the kernel launched from a CUDA graph that is
// captured once per batch layout and replayed.
//
// The split-K policy (how many K elements a split must keep, and below how
// many tiles an instance is split) is chosen by mgemm_grouped_tune, which
// times the candidates on the caller's batch (writing to scratch copies of C)
// and caches the winner for batches of the same shape class.
//
// mtrsm_grouped: one persistent kernel; a work item is (instance, 32 right-hand
// sides), pulled by a warp from an atomic counter (longest triangles first);
// the warp solves them by substitution, one lane per right-hand side, each
// row's sum exact in fixed point, using the double-double reciprocal of the
// diagonal as the reference does (mtrsm_serial.cpp:144). Descriptors and
// scratch are kept per batch layout and the launch is replayed from a CUDA
// graph, as for the grouped GEMM.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <map>
#include <mutex>
#include <type_traits>
#include <vector>

#include "dd.cuh"
#include "fixgemm.cuh"
#include "fixbeta.cuh"
#include "fixround.cuh"
#include "limbmma.cuh"
#include "xword.cuh"
#include "level3.h"
#include "runtime.h"

namespace mw {

namespace {

using fxg::exp_bound;
using fxg::kNoExp;

constexpr int GTHREADS = 256;  // 16 x 16 threads
constexpr int GBK = 8;         // k-slab

struct GemmDesc {
    const double2 *A, *B;
    double2 *C;
    int64_t lda, ldb, ldc;
    int m, n, k;
    int ta, tb;
    double2 alpha, beta;
    int beta_kind;
    int tiles_m, tiles_n, splitk, klen;
    int64_t work_begin;   // first work item of this instance
    int64_t tile_begin;   // first tile counter (split instances only)
    int64_t part_begin;   // first partial-tile slot: earlier split instances
                          // hold tiles * splitk slots each
    // tensor-core tiles only: the operands as limb bytes in the wave's scratch
    int64_t conv_begin;   // first group of 32 lines (rows of op(A), then columns of op(B)) in the wave
    int64_t a_off, b_off; // [line][kp] entries of 16 bytes
    int64_t ea_off, eb_off;   // exponent bounds of the lines
    int kp, pad;          // k rounded up to 16
    xw::XW xa, xb;        // alpha, beta
};
static_assert(sizeof(xw::XW) == 24, "extended float size");

__device__ __forceinline__ double2 opA_at(const GemmDesc &d, int64_t i, int64_t p)
{
    return d.ta ? d.A[p + i * d.lda] : d.A[i + p * d.lda];
}
__device__ __forceinline__ double2 opB_at(const GemmDesc &d, int64_t p, int64_t j)
{
    return d.tb ? d.B[j + p * d.ldb] : d.B[p + j * d.ldb];
}

// R consecutive digits of a staged row (R = 1, 2 or 4 ints, one vector load).
template <int R>
__device__ __forceinline__ void load_digits(const int *src, int (&dst)[R])
{
    if constexpr (R == 4) {
        const int4 v = *reinterpret_cast<const int4 *>(src);
        dst[0] = v.x; dst[1] = v.y; dst[2] = v.z; dst[3] = v.w;
    } else {
        const int2 v = *reinterpret_cast<const int2 *>(src);
        dst[0] = v.x; dst[1] = v.y;
    }
}

// ---- 16 x 16 output tiles on the tensor cores (byte limbs) -----------------------------
//
// Operands are scaled to integers N below 2^116 of their row's (column's) bound,
// as in the digit kernel below, and held as 16 bytes each in two's complement:
// limbs 0..14 of N mod 2^120 and limb 15 = 1 where N < 0, of weight -2^120. A
// first kernel writes them once per operand (k_grp_limbs), [line][k], so that
// the tiles that share an operand do not convert it again (a batch of sizes
// log-uniform in [8, 512] has four tiles per operand line on average; with the
// conversion in the tiles the batch took as long as with the digit kernel).
//
// A warp takes two rows and 16 columns; for each output the 16 x 16 limb products
// summed over k are two m16n8k16 MMAs per 16 k (rows and columns in the order
// even limbs, odd limbs): one ldmatrix of 16-bit units per operand and 32 k,
// whose masked halves are fp16 subnormals (limbmma.cuh). The FP32 sums start at
// 2^-25 and stay, after 64 k at most 255 * 255 * 64 units of 2^-48 above it, in
// [2^-25, 2^-24): exact, their words are 0x33000000 + sum. Each lane joins its
// eight limb products of an output into one 64-bit integer (it holds limbs 2g,
// 2g + 1 of the row and 4t .. 4t + 3 of the column) and adds it to the output's
// row of 32 such sums in shared memory (64 chunks of 64 k at most per item). At
// the end every lane takes one output: the 32 sums at weights 2^(16 (g + 2t)) are
// one carry chain to a 256-bit integer, updated and rounded as in fixround.cuh.
//
// Bound: the legacy tensor path (1024 multiply-adds/clk/SM, 256 per limb-wise
// multiply-add) against 15 IMAD.WIDE (26 lanes/clk/SM) in the digit kernels: 0.25
// against 0.58 clk/SM; rows past m and columns past n cost nothing. Measured on
// 4000 products of sizes log-uniform in [8, 512] (those with m or n below 128 or
// k below 64): 9.8 ms and 0.84 for the limbs, 14.9 on 32 x 32 digit tiles; the
// tensor pipe is a third busy, latency (16 warps per SM) takes the rest.
constexpr int LT = 16;                              // tile edge
constexpr int LT_KC = 64;                           // k per chunk
constexpr int LT_OP = 2 * LT * LT_KC * 16;          // operand bytes of a chunk
constexpr int LT_ROW = 33;                          // 64-bit sums per output (32 and a pad)
constexpr int LT_SMEM = LT_OP + (GTHREADS / 32) * 32 * LT_ROW * 8;
constexpr int64_t LT_WAVE = 1ll << 26;              // scratch entries (1 GiB) from which a batch is cut into waves

// v * 2^sh (|.| < 2^116) rounded to an integer, as the 16 bytes described above.
__device__ __forceinline__ uint4 limb_bytes(double2 v, int sh)
{
    uint32_t w[4];
    int eh;
    const bool ok = lmb::split_fast(v, w, eh);
    const int r = lmb::kExpBias - sh - eh;
    const uint32_t m = (uint32_t)(__double2hiint(v.x) >> 31);
    uint32_t rb;
    if (ok && (uint32_t)(r - 1) < 31u) {
        rb = (w[0] >> (r - 1)) & 1u;
        lmb::shr_short(w, r);
    } else {
        const fx::Op o = fx::decode(v);
        const int q = -(o.e + sh);
        w[0] = w[1] = w[2] = w[3] = rb = 0u;
        if (!(o.flags & (fx::kZero | fx::kBad)) && q >= 1 && q < 118) {
            uint32_t h[4];
            fx::shr128(o.w, q, w);
            fx::shr128(o.w, q - 1, h);   // rounding bit
            rb = h[0] & 1u;
        }
    }
    asm("add.cc.u32 %0, %0, %4;\n\t"
        "addc.cc.u32 %1, %1, 0;\n\t"
        "addc.cc.u32 %2, %2, 0;\n\t"
        "addc.u32 %3, %3, 0;"
        : "+r"(w[0]), "+r"(w[1]), "+r"(w[2]), "+r"(w[3])
        : "r"(rb));
    uint4 b;
    asm("{\n\t.reg .u32 t;\n\t"
        "add.cc.u32 t, %4, 0xFFFFFFFF;\n\t"   // the carry in: m & 1
        "addc.cc.u32 %0, %5, 0;\n\t"
        "addc.cc.u32 %1, %6, 0;\n\t"
        "addc.cc.u32 %2, %7, 0;\n\t"
        "addc.u32 %3, %8, 0;\n\t}"
        : "=&r"(b.x), "=&r"(b.y), "=&r"(b.z), "=&r"(b.w)
        : "r"(m & 1u), "r"(w[0] ^ m), "r"(w[1] ^ m), "r"(w[2] ^ m), "r"(w[3] ^ m));
    b.w &= 0x01FFFFFFu;
    return b;
}

// The last descriptor whose `begin` is at most w.
template <typename F>
__device__ __forceinline__ int grp_search(int count, int64_t w, F begin)
{
    int lo = 0, hi = count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (begin(mid) <= w) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Exponent bounds and limb bytes of 32 lines (rows of op(A) or columns of op(B))
// of an instance per block; the second pass reads what the first left in the
// caches.
__global__ void __launch_bounds__(GTHREADS) k_grp_limbs(const GemmDesc *__restrict__ descs, int count, uint4 *out,
                                                        int *ex)
{
    __shared__ int s_e[32];
    const int tid = threadIdx.x;
    const GemmDesc &d =
        descs[grp_search(count, (int64_t)blockIdx.x, [&](int q) { return descs[q].conv_begin; })];
    int grp = (int)((int64_t)blockIdx.x - d.conv_begin);
    const int ga = (d.m + 31) / 32;
    const bool isA = grp < ga;
    if (!isA) grp -= ga;
    const int line0 = grp * 32, nl = min(32, (isA ? d.m : d.n) - line0), k = d.k, kp = d.kp;
    const bool along_k = isA ? d.ta != 0 : d.tb == 0;   // a line's entries are neighbours in memory
    const int64_t ld = isA ? d.lda : d.ldb;
    const double2 *X = (isA ? d.A : d.B) + (along_k ? line0 * ld : line0);
    const int64_t sl = along_k ? ld : 1, sk = along_k ? 1 : ld;
    if (tid < 32) s_e[tid] = kNoExp;
    __syncthreads();
    {
        const int l = along_k ? tid >> 3 : tid & 31, q = along_k ? tid & 7 : tid >> 5;
        if (l < nl) {
            const double2 *x = X + l * sl + q * sk;
            int e = kNoExp;
#pragma unroll 4
            for (int p = q; p < k; p += 8, x += 8 * sk) e = max(e, exp_bound(x->x));
            atomicMax(&s_e[l], e);
        }
    }
    __syncthreads();
    if (tid < nl) ex[(isA ? d.ea_off : d.eb_off) + line0 + tid] = s_e[tid];
    // 8 neighbours along k, or 8 lines x 4 k per warp: whole 64 bytes either way
    const int l = along_k ? tid >> 3 : (tid & 7) + 8 * ((tid >> 5) & 3);
    const int q = along_k ? tid & 7 : ((tid >> 3) & 3) + 4 * (tid >> 7);
    if (l >= nl) return;
    const int e = s_e[l];
    const bool live = e > kNoExp / 2 && e < 1024;
    const double2 *x = X + l * sl + q * sk;
    uint4 *o = out + (isA ? d.a_off : d.b_off) + (int64_t)(line0 + l) * kp;
#pragma unroll 2
    for (int p = q; p < kp; p += 8, x += 8 * sk)
        o[p] = live && p < k ? limb_bytes(*x, fxg::FX_S - e) : make_uint4(0u, 0u, 0u, 0u);
}

// Even and odd limbs of an ldmatrix word (16-bit units of two elements).
__device__ __forceinline__ uint32_t limbs_even(uint32_t v) { return v & 0x00FF00FFu; }
__device__ __forceinline__ uint32_t limbs_odd(uint32_t v) { return __byte_perm(v, 0u, 0x4341); }

__global__ void __launch_bounds__(GTHREADS, 2) k_gemm_grouped_limb(const GemmDesc *__restrict__ descs, int count,
                                                                  int total, unsigned long long *work_counter,
                                                                  int *tile_counters, fx::XFPod *partials,
                                                                  const uint4 *__restrict__ limbs,
                                                                  const int *__restrict__ ex)
{
    extern __shared__ __align__(16) unsigned char s_dyn[];   // [operand row 0..31][64 k] 16 bytes, then the sums
    __shared__ int s_item, s_last;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    unsigned long long *sums = reinterpret_cast<unsigned long long *>(s_dyn + LT_OP) + wid * (32 * LT_ROW);
    const uint32_t op = (uint32_t)__cvta_generic_to_shared(s_dyn);
    const uint32_t n15 = t == 3 ? 0u - 256u : 256u;
    const int m15 = g == 7 ? -256 : 256;
    // the 0x33000000 of each accumulator word (those times 256 vanish mod 2^32)
    const unsigned long long off = (unsigned long long)(0x33000000ll * 65537 * (1 + m15));
    for (;;) {
        if (tid == 0) s_item = (int)min(atomicAdd(work_counter, 1ull), (unsigned long long)total);
        __syncthreads();
        const int w = s_item;
        if (w >= total) return;
        const GemmDesc &d = descs[grp_search(count, (int64_t)w, [&](int q) { return descs[q].work_begin; })];
        const uint32_t local = (uint32_t)(w - d.work_begin), tile = local / (uint32_t)d.splitk;
        const int split = (int)(local % (uint32_t)d.splitk);
        const int i0 = (int)(tile % (uint32_t)d.tiles_m) * LT, j0 = (int)(tile / (uint32_t)d.tiles_m) * LT;
        const int k0 = split * d.klen, kn = min(d.kp, k0 + d.klen) - k0;   // klen: multiples of 16 where split
        const int mr = min(LT, d.m - i0), nc = min(LT, d.n - j0);
        const uint4 *pA = limbs + d.a_off + (int64_t)i0 * d.kp + k0, *pB = limbs + d.b_off + (int64_t)j0 * d.kp + k0;
        const bool rows = 2 * wid < mr;   // this warp has rows of the output
        const uint32_t a_at = op + (2 * wid) * (LT_KC * 16);
        const bool some = d.k > 0;
        for (int c0 = 0; some && c0 < kn; c0 += LT_KC) {
            if (c0 > 0) __syncthreads();   // the previous chunk's operands have been read
            const int kc = min(LT_KC, kn - c0), p = tid & 63;
            // rows 0..15 of op(A), 16..31 columns of op(B), four per turn; k goes to
            // place k ^ (row % 8), so that ldmatrix is free of bank conflicts
            if (p < kc) {
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int r = (tid >> 6) + 4 * (u & 3);
                    const uint4 *src = (u < 4 ? pA : pB) + (int64_t)r * d.kp + c0 + p;
                    if (r < (u < 4 ? mr : nc))
                        lmb::cp_async16(op + ((((u < 4 ? 0 : LT) + r) * LT_KC + (p ^ (r & 7))) << 4), src);
                }
            }
            asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            if (!rows) continue;
            const int nks = kc >> 4;   // steps of 16 k
#pragma unroll 1
            for (int r = 0; r < 2; ++r) {
                uint32_t a[4][4];   // the row's operands of every step
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t x[4];
                    lmb::ldmatrix_x4_trans(x, a_at + r * (LT_KC * 16) + (((32 * h + lane) ^ ((2 * wid + r) & 7)) << 4));
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        a[2 * h + q][0] = limbs_even(x[2 * q]);
                        a[2 * h + q][1] = limbs_odd(x[2 * q]);
                        a[2 * h + q][2] = limbs_even(x[2 * q + 1]);
                        a[2 * h + q][3] = limbs_odd(x[2 * q + 1]);
                    }
                }
                // four columns at a time, so that their products and sums overlap
                auto columns = [&](int c, auto width) {
                    constexpr int NC = decltype(width)::value;
                    float acc[NC][2][4];
                    uint32_t x[NC][4];
#pragma unroll
                    for (int s = 0; s < 4; ++s) {
                        if (s >= nks) break;
                        if ((s & 1) == 0)
#pragma unroll
                            for (int u = 0; u < NC; ++u)
                                lmb::ldmatrix_x4_trans(x[u], op + (LT + c + u) * (LT_KC * 16) +
                                                                 (((16 * s + lane) ^ ((c + u) & 7)) << 4));
#pragma unroll
                        for (int u = 0; u < NC; ++u) {
                            const uint32_t x0 = x[u][2 * (s & 1)], x1 = x[u][2 * (s & 1) + 1];
                            const uint32_t e0 = limbs_even(x0), e1 = limbs_even(x1);
                            const uint32_t o0 = limbs_odd(x0), o1 = limbs_odd(x1);
                            if (s == 0) {
                                lmb::mma16816_from(acc[u][0], a[s][0], a[s][1], a[s][2], a[s][3], e0, e1, 0x1p-25f);
                                lmb::mma16816_from(acc[u][1], a[s][0], a[s][1], a[s][2], a[s][3], o0, o1, 0x1p-25f);
                            } else {
                                lmb::mma16816(acc[u][0], a[s][0], a[s][1], a[s][2], a[s][3], e0, e1);
                                lmb::mma16816(acc[u][1], a[s][0], a[s][1], a[s][2], a[s][3], o0, o1);
                            }
                        }
                    }
#pragma unroll
                    for (int u = 0; u < NC; ++u) {
                        // limbs 4t .. 4t + 3 of the column for each of the row's two limbs;
                        // limb 15 (t = 3) and the row's limb 15 (g = 7) have negative weight
                        auto word = [&](int b, int i) { return __float_as_uint(acc[u][b][i]); };
                        const int lo0 = (int)(word(0, 0) + 256u * word(1, 0)), hi0 = (int)(word(0, 1) + n15 * word(1, 1));
                        const int lo1 = (int)(word(0, 2) + 256u * word(1, 2)), hi1 = (int)(word(0, 3) + n15 * word(1, 3));
                        const long long lo = (long long)lo1 * m15 + lo0, hi = (long long)hi1 * m15 + hi0;
                        unsigned long long *at = sums + ((c + u) * 2 + r) * LT_ROW + lane;
                        const unsigned long long q = (unsigned long long)(lo + hi * 65536) - off;
                        *at = c0 == 0 ? q : *at + q;
                    }
                };
                int c = 0;
                for (; c + 4 <= nc; c += 4) columns(c, std::integral_constant<int, 4>{});
                for (; c < nc; ++c) columns(c, std::integral_constant<int, 1>{});
            }
        }
        __syncwarp();

        // each lane one output: row 2 wid + (lane & 1), column lane / 2
        const int orow = 2 * wid + (lane & 1), ocol = lane >> 1;
        const bool in = orow < mr && ocol < nc;
        const int ei = in && some ? ex[d.ea_off + i0 + orow] : kNoExp, ej = in && some ? ex[d.eb_off + j0 + ocol] : kNoExp;
        bool bad = ei >= 1024 || ej >= 1024;
        const bool live = !bad && ei > kNoExp / 2 && ej > kNoExp / 2;
        double2 *pc = d.C + i0 + orow + (int64_t)(j0 + ocol) * d.ldc;
        const double2 c_in = in && d.beta_kind != 0 && d.splitk == 1 ? *pc : make_double2(0.0, 0.0);
        uint64_t W[4] = {0, 0, 0, 0};
        if (live) {
            const unsigned long long *at = sums + lane * LT_ROW;
            long long carry = 0;   // sum at weight 2^(16 s), its low 16 bits to the result
#pragma unroll
            for (int s = 0; s < 14; ++s) {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (s - 2 * q >= 0 && s - 2 * q < 8) carry += (long long)at[4 * (s - 2 * q) + q];
                W[s >> 2] |= (uint64_t)((uint32_t)carry & 0xFFFFu) << (16 * (s & 3));
                carry >>= 16;
            }
            W[3] |= (uint64_t)carry << 32;
        }
        const int e0 = ei + ej - 2 * fxg::FX_S;
        bool done = false;
        if (in && live && d.splitk == 1) {
            // the top 160 bits of |W| (2^-134 of the largest product is cut), alpha, beta C, one rounding
            const uint32_t m = (uint32_t)((int64_t)W[3] >> 63);
            uint32_t x[8];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                x[2 * q] = (uint32_t)W[q];
                x[2 * q + 1] = (uint32_t)(W[q] >> 32);
            }
            fxr::cond_neg<8>(x, m);
            fxr::Fix a;
            a.neg = m & 1u;
            if (d.alpha.x == 1.0 && d.alpha.y == 0.0) {
#pragma unroll
                for (int q = 0; q < 5; ++q) a.w[q] = x[3 + q];
                a.e = e0 + 96;
            } else {
                fxr::mul54(x + 3, d.xa.w, a.w);
                a.neg ^= d.xa.neg;
                a.e = e0 + 96 + 128 + d.xa.e;
            }
            a.w[5] = 0u;
            if (d.beta_kind == 0 || add_beta_c(a, c_in, d.xb, d.beta_kind == 1, 0u)) {
                double h, l;
                fxr::to_dd(a, h, l);
                *pc = make_double2(h, l);
                done = true;
            }
        }
        xfp::XF v;
        v.zero = true; v.neg = false; v.m = 0; v.e = 0;
        if (live && !done) v = fx::w256_to_xf(W, e0);
        if (d.splitk > 1) {
            // this split's sums, then the last split of the tile finishes it
            fx::XFPod *pt = partials + (d.part_begin + (int64_t)tile * d.splitk + split) * (LT * LT);
            pt[ocol * LT + orow] = fx::to_pod(v, bad);
            __threadfence();
            __syncthreads();
            if (tid == 0) s_last = atomicAdd(&tile_counters[d.tile_begin + tile], 1) == d.splitk - 1;
            __syncthreads();
            if (!s_last) continue;
            __threadfence();
            const fx::XFPod *base = partials + (d.part_begin + (int64_t)tile * d.splitk) * (LT * LT) + ocol * LT + orow;
            v.zero = true; v.neg = false; v.m = 0; v.e = 0;
            bad = false;
            for (int s2 = 0; s2 < d.splitk; ++s2) {
                // partials written by other CTAs: read through L2
                const fx::XFPod *q = base + (int64_t)s2 * (LT * LT);
                fx::XFPod pv;
                pv.hi = __ldcg(&q->hi);
                pv.lo = __ldcg(&q->lo);
                pv.e = __ldcg(&q->e);
                pv.flags = __ldcg(&q->flags);
                bad |= (pv.flags & 4) != 0;
                v = xfp::xf_add(v, fx::from_pod(pv));
            }
            if (tid == 0) tile_counters[d.tile_begin + tile] = 0;   // ready for the next replay
        }
        if (in && !done) {
            if (bad) {
                const double qnan = __longlong_as_double(0x7ff8000000000000ll);
                *pc = make_double2(qnan, qnan);
            } else {
                fxg::store_axpby(pc, v, xfp::xf_from_dd(d.alpha.x, d.alpha.y), d.alpha.x == 1.0 && d.alpha.y == 0.0,
                                 xfp::xf_from_dd(d.beta.x, d.beta.y), dd::make(d.beta.x, d.beta.y), d.beta_kind);
            }
        }
        __syncthreads();   // s_item and the operands are reused
    }
}

// GT x GT output tiles (GT = 32 or 64) on the integer pipes, 256 threads as 16 x 16, each with R x R outputs (R = GT / 16): rows R tx ..,
// columns R ty ...
template <int GT>
__global__ void __launch_bounds__(GTHREADS) k_gemm_grouped(const GemmDesc *__restrict__ descs, int count,
                                                          int64_t total, unsigned long long *work_counter,
                                                          int *tile_counters, fx::XFPod *partials)
{
    constexpr int R = GT / 16;
    __shared__ __align__(16) int sA[GBK][5][GT], sB[GBK][5][GT];
    __shared__ int s_ea[GT], s_eb[GT];
    __shared__ long long s_item;
    __shared__ int s_last;
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    for (;;) {
        if (tid == 0) s_item = (long long)atomicAdd(work_counter, 1ull);
        __syncthreads();
        const long long w = s_item;
        __syncthreads();
        if (w >= total) return;
        // locate the instance (descs sorted by work_begin)
        const GemmDesc d = descs[grp_search(count, w, [&](int q) { return descs[q].work_begin; })];
        const int64_t local = w - d.work_begin;
        const int split = (int)(local % d.splitk);
        const int64_t tile = local / d.splitk;
        const int tm = (int)(tile % d.tiles_m), tn = (int)(tile / d.tiles_m);
        const int64_t i0 = (int64_t)tm * GT, j0 = (int64_t)tn * GT;
        const int64_t k0 = (int64_t)split * d.klen, k1 = min((int64_t)d.k, k0 + d.klen);

        // exponent bounds of the tile's rows / columns over [k0, k1)
        if (tid < GT) {
            int e = kNoExp;
            const int64_t i = i0 + tid;
            if (i < d.m)
                for (int64_t p = k0; p < k1; ++p) e = max(e, exp_bound(opA_at(d, i, p).x));
            s_ea[tid] = e;
        } else if (tid < 2 * GT) {
            int e = kNoExp;
            const int64_t j = j0 + (tid - GT);
            if (j < d.n)
                for (int64_t p = k0; p < k1; ++p) e = max(e, exp_bound(opB_at(d, p, j).x));
            s_eb[tid - GT] = e;
        }
        __syncthreads();

        long long acc[R][R][5];
#pragma unroll
        for (int a = 0; a < R; ++a)
#pragma unroll
            for (int b = 0; b < R; ++b)
#pragma unroll
                for (int q = 0; q < 5; ++q) acc[a][b][q] = 0;

        for (int64_t kk = k0; kk < k1; kk += GBK) {
            // stage the A and B tiles (GT x GBK elements each) as digits
            for (int idx = tid; idx < GT * GBK; idx += GTHREADS) {
                int dg[5];
                {
                    int r, p;
                    if (!d.ta) { r = idx % GT; p = idx / GT; }
                    else       { p = idx % GBK; r = idx / GBK; }
                    const int64_t gi = i0 + r, gp = kk + p;
                    const double2 v = (gp < k1 && gi < d.m) ? opA_at(d, gi, gp) : make_double2(0.0, 0.0);
                    const int e = s_ea[r];
                    fxg::dd_digits(v, (e <= kNoExp / 2 || e >= 1024) ? -100000 : fxg::FX_S - e, dg);
#pragma unroll
                    for (int t = 0; t < 5; ++t) sA[p][t][r] = dg[t];
                }
                {
                    int c, p;
                    if (!d.tb) { p = idx % GBK; c = idx / GBK; }
                    else       { c = idx % GT; p = idx / GT; }
                    const int64_t gj = j0 + c, gp = kk + p;
                    const double2 v = (gp < k1 && gj < d.n) ? opB_at(d, gp, gj) : make_double2(0.0, 0.0);
                    const int e = s_eb[c];
                    fxg::dd_digits(v, (e <= kNoExp / 2 || e >= 1024) ? -100000 : fxg::FX_S - e, dg);
#pragma unroll
                    for (int t = 0; t < 5; ++t) sB[p][t][c] = dg[t];
                }
            }
            __syncthreads();
#pragma unroll 2
            for (int p = 0; p < GBK; ++p) {
                int da[R][5], db[R][5];
#pragma unroll
                for (int t = 0; t < 5; ++t) {
                    int va[R], vb[R];
                    load_digits<R>(&sA[p][t][R * tx], va);
                    load_digits<R>(&sB[p][t][R * ty], vb);
#pragma unroll
                    for (int u = 0; u < R; ++u) {
                        da[u][t] = va[u];
                        db[u][t] = vb[u];
                    }
                }
#pragma unroll
                for (int a = 0; a < R; ++a)
#pragma unroll
                    for (int b = 0; b < R; ++b) fxg::mac_digits(acc[a][b], da[a], db[b]);
            }
            __syncthreads();
        }

        // the R x R outputs as extended floats (non-finite rows/columns flagged)
        xfp::XF v[R][R];
        bool badv[R][R];
#pragma unroll
        for (int a = 0; a < R; ++a)
#pragma unroll
            for (int b = 0; b < R; ++b) {
                const int ei = s_ea[R * tx + a], ej = s_eb[R * ty + b];
                badv[a][b] = ei >= 1024 || ej >= 1024;
                if (badv[a][b] || ei <= kNoExp / 2 || ej <= kNoExp / 2) {
                    v[a][b].zero = true; v[a][b].neg = false; v[a][b].m = 0; v[a][b].e = 0;
                } else {
                    v[a][b] = fxg::sums_to_xf(acc[a][b], ei, ej);
                }
            }

        if (d.splitk > 1) {
            // write this split's partial tile, then let the last split finish
            fx::XFPod *pt = partials + (d.part_begin + tile * d.splitk + split) * (GT * GT);
#pragma unroll
            for (int a = 0; a < R; ++a)
#pragma unroll
                for (int b = 0; b < R; ++b) pt[(R * ty + b) * GT + R * tx + a] = fx::to_pod(v[a][b], badv[a][b]);
            __threadfence();
            __syncthreads();
            if (tid == 0) {
                int old = atomicAdd(&tile_counters[d.tile_begin + tile], 1);
                s_last = (old == d.splitk - 1);
            }
            __syncthreads();
            if (!s_last) continue;
            __threadfence();
            const fx::XFPod *base = partials + (d.part_begin + tile * d.splitk) * (GT * GT);
#pragma unroll
            for (int a = 0; a < R; ++a)
#pragma unroll
                for (int b = 0; b < R; ++b) {
                    xfp::XF sum;
                    sum.zero = true; sum.neg = false; sum.m = 0; sum.e = 0;
                    bool bad = false;
                    for (int s2 = 0; s2 < d.splitk; ++s2) {
                        // partials written by other CTAs: read through L2
                        const fx::XFPod *q = base + (int64_t)s2 * GT * GT + (R * ty + b) * GT + R * tx + a;
                        fx::XFPod pv;
                        pv.hi = __ldcg(&q->hi);
                        pv.lo = __ldcg(&q->lo);
                        pv.e = __ldcg(&q->e);
                        pv.flags = __ldcg(&q->flags);
                        bad |= (pv.flags & 4) != 0;
                        sum = xfp::xf_add(sum, fx::from_pod(pv));
                    }
                    v[a][b] = sum;
                    badv[a][b] = bad;
                }
            if (tid == 0) tile_counters[d.tile_begin + tile] = 0;   // ready for the next replay
        }
        const dd::real beta = dd::make(d.beta.x, d.beta.y);
        const xfp::XF xa = xfp::xf_from_dd(d.alpha.x, d.alpha.y), xb = xfp::xf_from_dd(d.beta.x, d.beta.y);
        const bool alpha_one = d.alpha.x == 1.0 && d.alpha.y == 0.0;
#pragma unroll
        for (int b = 0; b < R; ++b) {
            const int64_t j = j0 + R * ty + b;
            if (j >= d.n) continue;
#pragma unroll
            for (int a = 0; a < R; ++a) {
                const int64_t i = i0 + R * tx + a;
                if (i >= d.m) continue;
                double2 *pc = d.C + i + j * d.ldc;
                if (badv[a][b]) {
                    const double qnan = __longlong_as_double(0x7ff8000000000000ll);
                    *pc = make_double2(qnan, qnan);
                    continue;
                }
                fxg::store_axpby(pc, v[a][b], xa, alpha_one, xb, beta, d.beta_kind);
            }
        }
    }
}

// ---- grouped TRSM ----------------------------------------------------------------

struct TrsmDesc {
    const double2 *A;
    double2 *B;
    int64_t lda, ldb;
    int m, n;
    double2 alpha;
    int nchunks;          // groups of 32 right-hand sides
    int64_t work_begin;
    int64_t xop_begin;    // this instance's decoded solutions in the scratch array (na * 32 per chunk)
};

constexpr int kTrsmTile = 256;   // entries of a row of op(A) split into digits at a time

__device__ __forceinline__ dd::real dd_recip(dd::real b)
{
    // Hida-Li-Bailey accurate division 1 / b
    double q1 = __ddiv_rn(1.0, b.hi);
    dd::real r = dd::sub_exact(dd::make(1.0, 0.0), dd::mul_exact(dd::make(q1, 0.0), b));
    double q2 = __ddiv_rn(r.hi, b.hi);
    r = dd::sub_exact(r, dd::mul_exact(dd::make(q2, 0.0), b));
    double q3 = __ddiv_rn(r.hi, b.hi);
    dd::real q;
    dd::fast_two_sum(q1, q2, q.hi, q.lo);
    return dd::add_exact(q, dd::make(q3, 0.0));
}

// One work item of the grouped TRSM: instance descs[*] (found by binary
// search on work_begin), right-hand sides [32 chunk, 32 chunk + 32).
__device__ __forceinline__ void trsm_item(const TrsmDesc *__restrict__ descs, int count, int64_t w, int side,
                                          int lower, int trans, int unit, fx::Op *xops, fx::Dig *arow, int lane)
{
    int lo = 0, hi = count - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (descs[mid].work_begin <= w) lo = mid;
        else hi = mid - 1;
    }
    const TrsmDesc d = descs[lo];
    const int chunk = (int)(w - d.work_begin);
    const dd::real alpha = dd::make(d.alpha.x, d.alpha.y);
    const bool alpha1 = (d.alpha.x == 1.0 && d.alpha.y == 0.0);
    const int na = side == 0 ? d.m : d.n;                 // order of the triangle
    const int64_t nr = side == 0 ? d.n : d.m;             // right-hand sides
    const int64_t rhs = (int64_t)chunk * 32 + lane;
    const bool active = rhs < nr;
    fx::Op *xw = xops + d.xop_begin + (int64_t)chunk * na * 32;   // [row][lane]
    const int64_t my = active ? rhs : nr - 1;             // clamped: loads stay in bounds
    // element t of this lane's right-hand side (a column of B for side L, a row for R)
    auto bptr = [&](int t) -> double2 * {
        return side == 0 ? d.B + my * d.ldb + t : d.B + my + (int64_t)t * d.ldb;
    };
#define OPA(i, j) (trans ? d.A[(j) + (int64_t)(i) * d.lda] : d.A[(i) + (int64_t)(j) * d.lda])
    // side L: op(A) X = alpha B, forward if op(A) is lower;
    // side R: X op(A) = alpha B, forward if op(A) is upper.
    const bool forward = side == 0 ? lower : !lower;
    fx::Dig one;
    {
        const fx::Op o = fx::decode(make_double2(1.0, 0.0));
        one = fx::to_dig(o);
    }
    dd::real inv = dd::make(1.0, 0.0);
    for (int s = 0; s < na; ++s) {
        const int r = forward ? s : na - 1 - s;
        if (!unit && (s & 31) == 0) {
            // reciprocals of the next 32 diagonal entries, one per lane
            const int sl = s + lane;
            if (sl < na) {
                const int rl = forward ? sl : na - 1 - sl;
                inv = dd_recip(dd::load(&OPA(rl, rl)));
            }
        }
        fx::Acc acc;
        acc.reset();
        dd::real b0 = dd::load(bptr(r));
        if (!alpha1) b0 = dd::mul_fast(b0, alpha);
        acc.add_dig(fx::decode(make_double2(b0.hi, b0.lo)), one);
        const int p0 = forward ? 0 : r + 1, p1 = forward ? r : na;
        for (int t0 = p0; t0 < p1; t0 += kTrsmTile) {
            const int tl = min(kTrsmTile, p1 - t0);
            // side L: sum_p op(A)(r, p) x_p; side R: sum_p x_p op(A)(p, r)
            for (int q = lane; q < tl; q += 32) {
                const int p = t0 + q;
                arow[q] = fx::to_dig(fx::decode(side == 0 ? OPA(r, p) : OPA(p, r)));
            }
            __syncwarp();
            const fx::Op *xp = xw + (int64_t)t0 * 32 + lane;
            int q = 0;
            // four solutions loaded ahead of their products, so the loads overlap
            for (; q + 4 <= tl; q += 4, xp += 128) {
                fx::Op xo[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) xo[u] = xp[32 * u];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    xo[u].flags ^= fx::kNeg;
                    acc.add_dig(xo[u], arow[q + u]);
                }
            }
            for (; q < tl; ++q, xp += 32) {
                fx::Op xo = *xp;
                xo.flags ^= fx::kNeg;
                acc.add_dig(xo, arow[q]);
            }
            __syncwarp();
        }
        double h, l;
        xfp::xf_to_dd(acc.finish(), h, l);
        dd::real v = dd::make(h, l);
        if (acc.bad) v = dd::make(__longlong_as_double(0x7ff8000000000000ll), 0.0);
        if (!unit) {
            const double ih = __shfl_sync(0xffffffffu, inv.hi, s & 31);
            const double il = __shfl_sync(0xffffffffu, inv.lo, s & 31);
            v = dd::mul_fast(v, dd::make(ih, il));
        }
        if (active) dd::store(bptr(r), v);
        xw[(int64_t)r * 32 + lane] = fx::decode(make_double2(v.hi, v.lo));
        __syncwarp();
    }
#undef OPA
}

// side: 0 left, 1 right; lower: op(A) lower triangular; trans: op = A^T.
// Warp per (instance, 32 right-hand sides), lane per right-hand side. The
// reciprocals of the diagonal are computed 32 rows at a time, one row per
// lane, and broadcast with shuffles; each row's sum alpha*b - sum_p A x is
// accumulated exactly in fixed point (fixacc.cuh) and rounded once before the
// multiplication by the reciprocal. All lanes stay in the loop (lanes past
// the last right-hand side do the work on a clamped column and store
// nothing) so that the shuffles see the whole warp.
// Persistent: every warp pulls work items (instance, 32 right-hand sides) from
// an atomic counter until none is left; descriptors are sorted longest
// triangle first, so the long solves start first and the short ones fill the
// tail.
__global__ void __launch_bounds__(128, 4) k_trsm_grouped(const TrsmDesc *__restrict__ descs, int count, int64_t total,
                                                     int side, int lower, int trans, int unit, fx::Op *xops,
                                                     unsigned long long *work_counter)
{
    // per warp: a tile of the current row of op(A), split into digits once
    // for all 32 right-hand sides
    __shared__ fx::Dig s_arow[4][kTrsmTile];
    fx::Dig *arow = s_arow[(threadIdx.x >> 5) & 3];
    const int lane = threadIdx.x & 31;
    for (;;) {
        unsigned long long wl = 0;
        if (lane == 0) wl = atomicAdd(work_counter, 1ull);
        const int64_t w = (int64_t)__shfl_sync(0xffffffffu, wl, 0);
        if (w >= total) return;   // whole warp leaves together
        trsm_item(descs, count, w, side, lower, trans, unit, xops, arow, lane);
    }
}

// ---- host: plans, graphs, autotuner ----------------------------------------------

struct Policy {
    int min_k_per_split = 0;   // 0: never split
    int max_tiles_split = 4;   // split only instances with at most this many tiles
    int tile = 32;             // output tile edge: 16, 32 or 64
    int oz_min = 0;            // instances with m, n >= oz_min and k >= 64 run on the tensor cores (0: none)
    int pack_k = 0;            // the other instances with k >= pack_k share tensor-core slots, in pieces of <= 256 x 256 (0: none)
};

struct Plan {
    std::vector<GemmDesc> descs;
    std::vector<OzGroupItem> oz_items;   // instances routed to the tensor-core engine
    OzGroupPlan *oz = nullptr;
    int tile = 32;
    int64_t total = 0, split_tiles = 0, partial_elems = 0;
    // tensor-core tiles: descriptors [first, first + count) share the limb scratch
    struct Wave {
        int first, count;
        int64_t work, groups, entries, lines;
    };
    std::vector<Wave> waves;
    int64_t wave_entries = 0, wave_lines = 0;   // largest of any wave
    // device state
    void *dev = nullptr;
    size_t dev_bytes = 0;
    cudaGraphExec_t exec = nullptr;
    uint64_t key = 0;
};

std::mutex g_batched_mu;
std::map<uint64_t, Policy> g_policy_cache;   // shape class -> tuned policy
Policy g_default_policy{512, 4, 16, 128, 0};
thread_local int t_tuned_tile = 0;   // tile chosen by this thread's most recent tuning
thread_local int t_tuned_oz = -1;    // tensor-core threshold chosen by it (0: none)
std::atomic<int> g_forced_tile{0};   // mwblas_set_grouped_tile: 0 = tuned or default
std::atomic<int> g_forced_oz{-1};    // mwblas_set_grouped_tensor_min: -1 = tuned or default
std::atomic<int> g_forced_pack{-1};  // mwblas_set_grouped_tensor_pack: -1 = tuned or default
thread_local int t_tuned_pack = -1;  // shared-slot depth chosen by this thread's most recent tuning
thread_local Plan t_plan;

uint64_t mix(uint64_t h, uint64_t v)
{
    h ^= v + 0x9e3779b97f4a7c15ull + (h << 6) + (h >> 2);
    return h;
}

// Shape class: count and log-size histogram (the policy depends on shapes, not data).
uint64_t shape_class(int64_t count, const int64_t *m, const int64_t *n, const int64_t *k)
{
    int hist[3][12] = {};
    for (int64_t i = 0; i < count; ++i) {
        int64_t v[3] = {m[i], n[i], k[i]};
        for (int t = 0; t < 3; ++t) {
            int b = 0;
            while (b < 11 && ((int64_t)1 << (b + 1)) <= v[t]) ++b;
            hist[t][b]++;
        }
    }
    uint64_t h = (uint64_t)count;
    for (int t = 0; t < 3; ++t)
        for (int b = 0; b < 12; ++b) h = mix(h, (uint64_t)(hist[t][b] * 16 / (count > 0 ? count : 1)));
    return h;
}

void build_descs(Plan &pl, int64_t count, const char *ta, const char *tb, const int64_t *m, const int64_t *n,
                 const int64_t *k, const mwblas_real64x2 *alpha, const mwblas_real64x2 *const *a, const int64_t *lda,
                 const mwblas_real64x2 *const *b, const int64_t *ldb, const mwblas_real64x2 *beta,
                 mwblas_real64x2 *const *c, const int64_t *ldc, const Policy &pol)
{
    pl.descs.clear();
    pl.descs.reserve((size_t)count);
    pl.oz_items.clear();
    const int oz_min = (pol.oz_min > 0 && ozaki_available()) ? pol.oz_min : 0;
    const int pack_k = (pol.pack_k > 0 && ozaki_available()) ? pol.pack_k : 0;
    const int GT = pol.tile;
    pl.tile = GT;
    int64_t work = 0, stiles = 0, pslots = 0;
    pl.waves.clear();
    pl.wave_entries = pl.wave_lines = 0;
    for (int64_t i = 0; i < count; ++i) {
        if (m[i] <= 0 || n[i] <= 0) continue;
        GemmDesc d;
        memset(&d, 0, sizeof(d));   // the plan key hashes the bytes, padding included
        d.A = (const double2 *)a[i];
        d.B = (const double2 *)b[i];
        d.C = (double2 *)c[i];
        d.lda = lda[i];
        d.ldb = ldb[i];
        d.ldc = ldc[i];
        d.m = (int)m[i];
        d.n = (int)n[i];
        d.k = (int)k[i];
        char TA = (char)toupper(ta[i]), TB = (char)toupper(tb[i]);
        d.ta = (TA != 'N');
        d.tb = (TB != 'N');
        d.alpha = make_double2(alpha[i].limbs[0], alpha[i].limbs[1]);
        d.beta = make_double2(beta[i].limbs[0], beta[i].limbs[1]);
        const bool alpha0 = (d.alpha.x == 0.0 && d.alpha.y == 0.0);
        d.beta_kind = (d.beta.x == 0.0 && d.beta.y == 0.0) ? 0 : ((d.beta.x == 1.0 && d.beta.y == 0.0) ? 1 : 2);
        const bool own_slot = oz_min > 0 && d.m >= oz_min && d.n >= oz_min && d.k >= 64;
        // the other instances of depth >= pack_k share slots; those with m or
        // n above 256 (the skinny ones) as pieces of at most 256 x 256
        const bool shared_slot = pack_k > 0 && d.k >= pack_k;
        if (!alpha0 && (own_slot || shared_slot) && d.k <= 16384 && d.m <= 8192 && d.n <= 8192) {
            OzGroupItem it;
            memset(&it, 0, sizeof(it));   // the plan key hashes the bytes, padding included
            it.lda = d.lda; it.ldb = d.ldb; it.ldc = d.ldc;
            it.k = d.k;
            it.ta = d.ta != 0; it.tb = d.tb != 0;
            it.alpha = dd_host{d.alpha.x, d.alpha.y};
            it.beta = dd_host{d.beta.x, d.beta.y};
            it.beta_kind = d.beta_kind;
            it.pack = own_slot ? 0 : 1;
            const int pm = own_slot ? d.m : 256, pn = own_slot ? d.n : 256;
            for (int r0 = 0; r0 < d.m; r0 += pm) {
                for (int c0 = 0; c0 < d.n; c0 += pn) {
                    // rows r0.. of op(A), columns c0.. of op(B) and C
                    it.A = d.A + (d.ta ? (int64_t)r0 * d.lda : r0);
                    it.B = d.B + (d.tb ? c0 : (int64_t)c0 * d.ldb);
                    it.C = d.C + r0 + (int64_t)c0 * d.ldc;
                    it.m = std::min(pm, d.m - r0);
                    it.n = std::min(pn, d.n - c0);
                    pl.oz_items.push_back(it);
                }
            }
            continue;
        }
        if (alpha0 || d.k == 0) {
            // only the beta pass: run as a k = 0 product (sigma irrelevant)
            d.k = 0;
        }
        d.tiles_m = (d.m + GT - 1) / GT;
        d.tiles_n = (d.n + GT - 1) / GT;
        const int tiles = d.tiles_m * d.tiles_n;
        d.splitk = 1;
        if (pol.min_k_per_split > 0 && tiles <= pol.max_tiles_split && d.k >= 2 * pol.min_k_per_split)
            d.splitk = std::min(16, d.k / pol.min_k_per_split);
        // the digit column sums hold at most 16384 multiply-adds per split, the
        // limb sums 4096 (64 chunks below 2^54 each, four of them added)
        const int kmax = GT == LT ? 4096 : 16384;
        const int need_splits = (d.k + kmax - 1) / kmax;
        if (d.splitk < need_splits) d.splitk = need_splits;
        d.kp = (d.k + 15) / 16 * 16;
        const int kstep = GT == LT ? 16 : GBK;
        d.klen = d.splitk > 1 ? ((d.k + d.splitk - 1) / d.splitk + kstep - 1) / kstep * kstep
                              : std::max(GT == LT ? d.kp : d.k, 1);
        if (d.k == 0) d.klen = 1;
        if (GT == LT) {
            // splits past k would be empty: as many as klen needs
            if (d.splitk > 1) d.splitk = (d.k + d.klen - 1) / d.klen;
            d.xa = xw::from_dd(d.alpha.x, d.alpha.y);
            d.xb = xw::from_dd(d.beta.x, d.beta.y);
            const int64_t entries = ((int64_t)d.m + d.n) * d.kp, lines = d.k > 0 ? (int64_t)d.m + d.n : 0;
            const int64_t tw = (int64_t)tiles * d.splitk;
            if (pl.waves.empty() || pl.waves.back().entries + entries > LT_WAVE ||
                pl.waves.back().work + tw > INT32_MAX)
                pl.waves.push_back(Plan::Wave{(int)pl.descs.size(), 0, 0, 0, 0, 0});
            Plan::Wave &wv = pl.waves.back();
            work = wv.work;   // work items are numbered within the wave
            d.conv_begin = wv.groups;
            d.a_off = wv.entries;
            d.b_off = wv.entries + (int64_t)d.m * d.kp;
            d.ea_off = wv.lines;
            d.eb_off = wv.lines + d.m;
            wv.groups += d.k > 0 ? (d.m + 31) / 32 + (d.n + 31) / 32 : 0;
            wv.entries += entries;
            wv.lines += lines;
            wv.work += tw;
            wv.count++;
            pl.wave_entries = std::max(pl.wave_entries, wv.entries);
            pl.wave_lines = std::max(pl.wave_lines, wv.lines);
        }
        d.work_begin = work;
        d.tile_begin = d.splitk > 1 ? stiles : 0;
        d.part_begin = d.splitk > 1 ? pslots : 0;
        if (d.splitk > 1) {
            stiles += tiles;
            pslots += (int64_t)tiles * d.splitk;
        }
        work += (int64_t)tiles * d.splitk;
        pl.descs.push_back(d);
    }
    pl.total = work;
    for (const Plan::Wave &wv : pl.waves) pl.total = std::max(pl.total, wv.work);
    pl.split_tiles = stiles;
    pl.partial_elems = pslots * GT * GT;   // extended-float partials
}

uint64_t plan_key(const Plan &pl)
{
    // FNV-1a over 64-bit words (GemmDesc is a multiple of 8 bytes)
    static_assert(sizeof(GemmDesc) % 8 == 0, "descriptor size");
    uint64_t h = 1469598103934665603ull;
    const uint64_t *p = (const uint64_t *)pl.descs.data();
    const size_t nw = pl.descs.size() * sizeof(GemmDesc) / 8;
    for (size_t i = 0; i < nw; ++i) h = (h ^ p[i]) * 1099511628211ull;
    static_assert(sizeof(OzGroupItem) % 8 == 0, "item size");
    const uint64_t *q = (const uint64_t *)pl.oz_items.data();
    const size_t nq = pl.oz_items.size() * sizeof(OzGroupItem) / 8;
    for (size_t i = 0; i < nq; ++i) h = (h ^ q[i]) * 1099511628211ull;
    return mix(mix(h, (uint64_t)pl.tile), (uint64_t)pl.oz_items.size());
}

// (Re)creates the device buffers and the graph when the batch layout changed.
// use_graph = false (the library's own calls, whose layouts change from call
// to call): the kernels are enqueued directly instead of capturing a graph.
bool prepare_and_launch(Plan &pl, const char *routine, bool use_graph = true)
{
    if ((pl.descs.empty() || pl.total == 0) && pl.oz_items.empty()) return true;
    const size_t d_bytes = pl.descs.size() * sizeof(GemmDesc);
    const size_t cnt_bytes = 256 + (size_t)(pl.split_tiles + 1) * sizeof(int);
    const size_t part_bytes = (size_t)pl.partial_elems * sizeof(fx::XFPod);
    const size_t limb_bytes_ = (size_t)pl.wave_entries * 16, ex_bytes = (size_t)pl.wave_lines * sizeof(int);
    const size_t need = d_bytes + cnt_bytes + part_bytes + limb_bytes_ + ex_bytes + 1024;
    const uint64_t key = plan_key(pl);
    cudaStream_t s = stream();
    if (pl.dev_bytes < need) {
        if (pl.exec) {
            cudaGraphExecDestroy(pl.exec);
            pl.exec = nullptr;
        }
        if (pl.dev) cudaFree(pl.dev);
        pl.dev = nullptr;
        pl.dev_bytes = 0;
        if (!cuda_ok(cudaMalloc(&pl.dev, need), routine, "grouped plan buffer")) return false;
        pl.dev_bytes = need;
        // the tile counters start at zero (each replay leaves them so)
        if (!cuda_ok(cudaMemset(pl.dev, 0, d_bytes + cnt_bytes + 512), routine, "grouped plan clear")) return false;
    }
    // layout: [descriptors][work counter (256 B) | tile counters][partials],
    // each region starting on a 256-byte boundary
    char *base = (char *)pl.dev;
    const size_t cnt_off = (d_bytes + 255) / 256 * 256;
    const size_t part_off = (cnt_off + cnt_bytes + 255) / 256 * 256;
    GemmDesc *ddesc = (GemmDesc *)base;
    unsigned long long *counter = (unsigned long long *)(base + cnt_off);
    int *tile_counters = (int *)(counter + 32);
    fx::XFPod *partials = (fx::XFPod *)(base + part_off);
    const size_t limb_off = (part_off + part_bytes + 255) / 256 * 256;
    uint4 *limbs = (uint4 *)(base + limb_off);
    int *ex = (int *)(base + (limb_off + limb_bytes_ + 255) / 256 * 256);
    const int sms = device_sm_count();
    const int grid = (int)std::min<int64_t>(pl.total, (int64_t)sms * 16);
    if (pl.key != key) {
        // descriptors change only with the batch layout; upload outside the graph
        if (!pl.descs.empty() &&
            !cuda_ok(cudaMemcpyAsync(ddesc, pl.descs.data(), d_bytes, cudaMemcpyHostToDevice, s), routine,
                     "descriptor upload"))
            return false;
        if (!pl.oz_items.empty() || pl.oz) {
            if (!pl.oz) pl.oz = ozgroup_create();
            if (!ozgroup_prepare(pl.oz, pl.oz_items, routine)) return false;
        }
    }
    // the integer-pipe or limb-tile part on stream q; its counters start at zero
    auto enqueue = [&](cudaStream_t q) {
        cudaMemsetAsync(counter, 0, cnt_bytes, q);
        if (pl.tile != LT) {
            auto kern = pl.tile == 64 ? k_gemm_grouped<64> : k_gemm_grouped<32>;
            kern<<<grid, GTHREADS, 0, q>>>(ddesc, (int)pl.descs.size(), pl.total, counter, tile_counters, partials);
            return;
        }
        cudaFuncSetAttribute(k_gemm_grouped_limb, cudaFuncAttributeMaxDynamicSharedMemorySize, LT_SMEM);
        bool first = true;
        for (const Plan::Wave &wv : pl.waves) {
            if (!first) cudaMemsetAsync(counter, 0, sizeof(*counter), q);
            first = false;
            if (wv.groups > 0) k_grp_limbs<<<(unsigned)wv.groups, GTHREADS, 0, q>>>(ddesc + wv.first, wv.count, limbs, ex);
            const int wgrid = (int)std::min<int64_t>(wv.work, (int64_t)sms * 2);
            k_gemm_grouped_limb<<<wgrid, GTHREADS, LT_SMEM, q>>>(ddesc + wv.first, wv.count, (int)wv.work, counter,
                                                                tile_counters, partials, limbs, ex);
        }
    };
    if (!use_graph) {
        pl.key = key;
        if (pl.total > 0) {
            enqueue(s);
            count_launch(pl.tile == LT ? 2 * (int64_t)pl.waves.size() : 1);
        }
        if (pl.oz && ozgroup_count(pl.oz) > 0) ozgroup_launch(pl.oz, s);
        return cuda_ok(cudaGetLastError(), routine, "grouped launch");
    }
    if (!pl.exec || pl.key != key) {
        if (pl.exec) {
            cudaGraphExecDestroy(pl.exec);
            pl.exec = nullptr;
        }
        cudaStream_t cap;
        if (!cuda_ok(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking), routine, "capture stream")) return false;
        cudaGraph_t graph;
        bool ok = cuda_ok(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal), routine, "begin capture");
        if (ok) {
            // counters start at zero on every replay
            if (pl.total > 0) enqueue(cap);
            // the large instances on the tensor cores, in the same graph
            if (pl.oz && ozgroup_count(pl.oz) > 0) ozgroup_launch(pl.oz, cap);
            ok = cuda_ok(cudaStreamEndCapture(cap, &graph), routine, "end capture");
        }
        if (ok) {
            ok = cuda_ok(cudaGraphInstantiate(&pl.exec, graph, 0), routine, "graph instantiate");
            cudaGraphDestroy(graph);
        }
        cudaStreamDestroy(cap);
        if (!ok) return false;
        pl.key = key;
    }
    count_launch();
    return cuda_ok(cudaGraphLaunch(pl.exec, s), routine, "graph launch");
}

// The grouped TRSM's per-thread plan: descriptors, work counter and decoded
// solutions in one device buffer, kept while the batch layout is unchanged,
// and a CUDA graph (counter reset + the persistent kernel) replayed per call.
struct TrsmPlan {
    std::vector<TrsmDesc> descs;
    int64_t total = 0, xop_elems = 0;
    int side = 0, lower = 0, trans = 0, unit = 0;
    void *dev = nullptr;
    size_t dev_bytes = 0;
    cudaGraphExec_t exec = nullptr;
    uint64_t key = 0;
};
thread_local TrsmPlan t_tplan;

bool trsm_prepare_and_launch(TrsmPlan &pl, const char *routine)
{
    if (pl.descs.empty() || pl.total == 0) return true;
    const size_t d_bytes = (pl.descs.size() * sizeof(TrsmDesc) + 255) / 256 * 256;
    const size_t need = d_bytes + 256 + (size_t)pl.xop_elems * sizeof(fx::Op);
    static_assert(sizeof(TrsmDesc) % 8 == 0, "descriptor size");
    uint64_t key = 1469598103934665603ull;
    const uint64_t *w = (const uint64_t *)pl.descs.data();
    for (size_t i = 0; i < pl.descs.size() * sizeof(TrsmDesc) / 8; ++i) key = (key ^ w[i]) * 1099511628211ull;
    key = mix(key, (uint64_t)(pl.side | pl.lower << 1 | pl.trans << 2 | pl.unit << 3));
    cudaStream_t s = stream();
    if (pl.dev_bytes < need) {
        if (pl.exec) {
            cudaGraphExecDestroy(pl.exec);
            pl.exec = nullptr;
        }
        if (pl.dev) cudaFree(pl.dev);
        pl.dev = nullptr;
        pl.dev_bytes = 0;
        pl.key = 0;
        if (!cuda_ok(cudaMalloc(&pl.dev, need), routine, "grouped TRSM plan buffer")) return false;
        pl.dev_bytes = need;
    }
    // layout: [descriptors][work counter (256 B)][decoded solutions]
    TrsmDesc *ddesc = (TrsmDesc *)pl.dev;
    unsigned long long *counter = (unsigned long long *)((char *)pl.dev + d_bytes);
    fx::Op *xops = (fx::Op *)((char *)pl.dev + d_bytes + 256);
    if (pl.key != key) {
        if (pl.exec) {
            cudaGraphExecDestroy(pl.exec);
            pl.exec = nullptr;
        }
        if (!cuda_ok(cudaMemcpyAsync(ddesc, pl.descs.data(), pl.descs.size() * sizeof(TrsmDesc),
                                     cudaMemcpyHostToDevice, s),
                     routine, "descriptor upload"))
            return false;
        // resident blocks: four 4-warp blocks per SM (the kernel's launch bounds)
        const int warps = 4;
        const int64_t grid = std::min<int64_t>((pl.total + warps - 1) / warps, (int64_t)device_sm_count() * 4);
        cudaStream_t cap;
        if (!cuda_ok(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking), routine, "capture stream")) return false;
        cudaGraph_t graph;
        bool ok = cuda_ok(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal), routine, "begin capture");
        if (ok) {
            cudaMemsetAsync(counter, 0, sizeof(unsigned long long), cap);
            k_trsm_grouped<<<(unsigned)grid, warps * 32, 0, cap>>>(ddesc, (int)pl.descs.size(), pl.total, pl.side,
                                                                 pl.lower, pl.trans, pl.unit, xops, counter);
            ok = cuda_ok(cudaStreamEndCapture(cap, &graph), routine, "end capture");
        }
        if (ok) {
            ok = cuda_ok(cudaGraphInstantiate(&pl.exec, graph, 0), routine, "graph instantiate");
            cudaGraphDestroy(graph);
        }
        cudaStreamDestroy(cap);
        if (!ok) return false;
        pl.key = key;
    }
    count_launch();
    return cuda_ok(cudaGraphLaunch(pl.exec, s), routine, "graph launch");
}

bool grouped_validate(const char *routine, int64_t count, const char *ta, const char *tb, const int64_t *m,
                      const int64_t *n, const int64_t *k, const mwblas_real64x2 *alpha,
                      const mwblas_real64x2 *const *a, const int64_t *lda, const mwblas_real64x2 *const *b,
                      const int64_t *ldb, const mwblas_real64x2 *beta, mwblas_real64x2 *const *c, const int64_t *ldc)
{
    if (count < 0) { set_error(routine, 1, "count < 0"); return false; }
    if (count == 0) return true;
    if (!ta || !tb || !m || !n || !k || !alpha || !a || !lda || !b || !ldb || !beta || !c || !ldc) {
        set_error(routine, 2, "null argument array");
        return false;
    }
    for (int64_t i = 0; i < count; ++i) {
        char TA = (char)toupper(ta[i]), TB = (char)toupper(tb[i]);
        if (TA != 'N' && TA != 'T' && TA != 'C') { set_error(routine, 2, "invalid transa in instance " + std::to_string(i)); return false; }
        if (TB != 'N' && TB != 'T' && TB != 'C') { set_error(routine, 3, "invalid transb in instance " + std::to_string(i)); return false; }
        if (m[i] < 0 || n[i] < 0 || k[i] < 0) { set_error(routine, 4, "negative size in instance " + std::to_string(i)); return false; }
        if (m[i] > (1 << 30) || n[i] > (1 << 30) || k[i] > (1 << 30)) { set_error(routine, 4, "size too large"); return false; }
        int64_t nra = (TA == 'N') ? m[i] : k[i], nrb = (TB == 'N') ? k[i] : n[i];
        if (lda[i] < std::max<int64_t>(1, nra)) { set_error(routine, 9, "lda too small in instance " + std::to_string(i)); return false; }
        if (ldb[i] < std::max<int64_t>(1, nrb)) { set_error(routine, 11, "ldb too small in instance " + std::to_string(i)); return false; }
        if (ldc[i] < std::max<int64_t>(1, m[i])) { set_error(routine, 14, "ldc too small in instance " + std::to_string(i)); return false; }
        if (m[i] > 0 && n[i] > 0 && !is_dd_device_pointer(c[i])) {
            set_error(routine, 13, "grouped calls take 16-byte aligned device (or managed) arrays; C of instance " +
                                       std::to_string(i));
            return false;
        }
        if (m[i] > 0 && n[i] > 0 && k[i] > 0 && !(is_dd_device_pointer(a[i]) && is_dd_device_pointer(b[i]))) {
            set_error(routine, 8, "grouped calls take 16-byte aligned device (or managed) arrays; A or B of instance " +
                                      std::to_string(i));
            return false;
        }
    }
    return true;
}

}  // namespace

// Grouped GEMM for the library's own use (device arrays, arguments already
// valid): its own plan, default split policy, stream-ordered (no sync).
bool grouped_gemm_device(int64_t count, const char *ta, const char *tb, const int64_t *m, const int64_t *n,
                         const int64_t *k, const mwblas_real64x2 *alpha, const mwblas_real64x2 *const *a,
                         const int64_t *lda, const mwblas_real64x2 *const *b, const int64_t *ldb,
                         const mwblas_real64x2 *beta, mwblas_real64x2 *const *c, const int64_t *ldc,
                         int tensor_min, const char *routine)
{
    if (count == 0) return true;
    static thread_local Plan internal;
    Policy pol = g_default_policy;
    pol.oz_min = tensor_min;
    build_descs(internal, count, ta, tb, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, pol);
    return prepare_and_launch(internal, routine, false);
}

}  // namespace mw

using mw::Plan;
using mw::Policy;

extern "C" int mgemm_grouped(int64_t count, const char *transa, const char *transb, const int64_t *m,
                             const int64_t *n, const int64_t *k, const mwblas_real64x2 *alpha,
                             const mwblas_real64x2 *const *a, const int64_t *lda, const mwblas_real64x2 *const *b,
                             const int64_t *ldb, const mwblas_real64x2 *beta, mwblas_real64x2 *const *c,
                             const int64_t *ldc)
{
    using namespace mw;
    const char *routine = "mgemm_grouped";
    clear_error();
    if (!grouped_validate(routine, count, transa, transb, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc))
        return mwblas_last_error();
    if (count == 0) return 0;
    if (!ensure_device(routine)) return mwblas_last_error();
    Policy pol = g_default_policy;
    {
        std::lock_guard<std::mutex> lk(g_batched_mu);
        auto it = g_policy_cache.find(shape_class(count, m, n, k));
        if (it != g_policy_cache.end()) pol = it->second;
    }
    if (g_forced_tile.load() > 0) pol.tile = g_forced_tile.load();
    if (g_forced_oz.load() >= 0) pol.oz_min = g_forced_oz.load();
    if (g_forced_pack.load() >= 0) pol.pack_k = g_forced_pack.load();
    Plan &pl = t_plan;
    build_descs(pl, count, transa, transb, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, pol);
    if (!prepare_and_launch(pl, routine)) return mwblas_last_error();
    if (!finish(routine)) return mwblas_last_error();
    return 0;
}

// Times the tensor-core size threshold (none, 64, 128, 256), the depth from
// which the remaining small instances share tensor-core slots (none, 16, 32,
// 64), then tile edges (16, 32, 64) and split-K policies for the rest, on the
// caller's batch
// (outputs go to scratch copies of C, the caller's C is not modified)
// and caches the fastest for batches of the same shape class. Returns 0 and
// the chosen minimum K per split in *chosen (0 = no split); the chosen tile
// edge is returned by mwblas_grouped_tuned_tile().
extern "C" int mgemm_grouped_tune(int64_t count, const char *transa, const char *transb, const int64_t *m,
                                  const int64_t *n, const int64_t *k, const mwblas_real64x2 *alpha,
                                  const mwblas_real64x2 *const *a, const int64_t *lda,
                                  const mwblas_real64x2 *const *b, const int64_t *ldb, const mwblas_real64x2 *beta,
                                  mwblas_real64x2 *const *c, const int64_t *ldc, int *chosen)
{
    using namespace mw;
    const char *routine = "mgemm_grouped_tune";
    clear_error();
    if (!grouped_validate(routine, count, transa, transb, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc))
        return mwblas_last_error();
    if (count == 0) return 0;
    if (!ensure_device(routine)) return mwblas_last_error();
    // scratch copies of every C
    std::vector<int64_t> off((size_t)count);
    int64_t tot = 0;
    for (int64_t i = 0; i < count; ++i) {
        off[(size_t)i] = tot;
        tot += (m[i] > 0 && n[i] > 0) ? ldc[i] * n[i] : 0;
    }
    double2 *scratch = nullptr;
    if (!cuda_ok(cudaMalloc(&scratch, sizeof(double2) * (size_t)std::max<int64_t>(tot, 1)), routine, "tune scratch"))
        return mwblas_last_error();
    std::vector<mwblas_real64x2 *> cs((size_t)count);
    for (int64_t i = 0; i < count; ++i) {
        cs[(size_t)i] = (mwblas_real64x2 *)(scratch + off[(size_t)i]);
        if (m[i] > 0 && n[i] > 0)
            cudaMemcpyAsync(cs[(size_t)i], c[i], sizeof(double2) * (size_t)(ldc[i] * n[i]), cudaMemcpyDeviceToDevice,
                            stream());
    }
    // two stages: the tile edge at the default split policy, then the split
    // policy at that tile
    const int tiles[] = {16, 32, 64};
    const int cands[] = {0, 2048, 1024, 512, 256, 128};
    Plan pl;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    auto time_policy = [&](const Policy &pol) -> float {
        build_descs(pl, count, transa, transb, m, n, k, alpha, a, lda, b, ldb, beta, cs.data(), ldc, pol);
        if (!prepare_and_launch(pl, routine)) return 1e30f;   // warm + capture
        cudaEventRecord(e0, stream());
        const int reps = 3;
        for (int r = 0; r < reps; ++r) prepare_and_launch(pl, routine);
        cudaEventRecord(e1, stream());
        cudaEventSynchronize(e1);
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, e0, e1);
        return ms;
    };
    // stages: the size from which instances run on the tensor cores, the
    // depth from which the smaller ones share slots there, then the tile edge
    // of the rest (integer pipes), then its split policy
    float best = 1e30f;
    int best_tile = g_default_policy.tile, best_k = g_default_policy.min_k_per_split, best_oz = 0;
    const int ozc[] = {0, 64, 128, 256};
    for (int oz : ozc) {
        if (oz > 0 && !ozaki_available()) break;
        const float ms = time_policy(Policy{best_k, 4, best_tile, oz, 0});
        if (ms < best) {
            best = ms;
            best_oz = oz;
        }
    }
    int best_pack = 0;
    const int packc[] = {16, 32, 64};
    for (int pk : packc) {
        if (!ozaki_available()) break;
        const float ms = time_policy(Policy{best_k, 4, best_tile, best_oz, pk});
        if (ms < best) {
            best = ms;
            best_pack = pk;
        }
    }
    for (int t : tiles) {
        if (t == best_tile) continue;   // timed above
        const float ms = time_policy(Policy{best_k, 4, t, best_oz, best_pack});
        if (ms < best) {
            best = ms;
            best_tile = t;
        }
    }
    for (int cand : cands) {
        if (cand == best_k) continue;   // timed above
        const float ms = time_policy(Policy{cand, 4, best_tile, best_oz, best_pack});
        if (ms < best) {
            best = ms;
            best_k = cand;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (pl.exec) cudaGraphExecDestroy(pl.exec);
    if (pl.dev) cudaFree(pl.dev);
    ozgroup_destroy(pl.oz);
    cudaFree(scratch);
    {
        std::lock_guard<std::mutex> lk(g_batched_mu);
        g_policy_cache[shape_class(count, m, n, k)] = Policy{best_k, 4, best_tile, best_oz, best_pack};
    }
    t_tuned_oz = best_oz;
    t_tuned_pack = best_pack;
    t_tuned_tile = best_tile;
    if (chosen) *chosen = best_k;
    return finish(routine) ? 0 : mwblas_last_error();
}

extern "C" int mtrsm_grouped(int64_t count, char side, char uplo, char transa, char diag, const int64_t *m,
                             const int64_t *n, const mwblas_real64x2 *alpha, const mwblas_real64x2 *const *a,
                             const int64_t *lda, mwblas_real64x2 *const *b, const int64_t *ldb)
{
    using namespace mw;
    const char *routine = "mtrsm_grouped";
    clear_error();
    char S = (char)toupper(side), U = (char)toupper(uplo), T = (char)toupper(transa), D = (char)toupper(diag);
    if (T == 'C') T = 'T';
    if (count < 0) { set_error(routine, 1, "count < 0"); return 1; }
    if (S != 'L' && S != 'R') { set_error(routine, 2, "invalid side"); return 2; }
    if (U != 'U' && U != 'L') { set_error(routine, 3, "invalid uplo"); return 3; }
    if (T != 'N' && T != 'T') { set_error(routine, 4, "invalid transa"); return 4; }
    if (D != 'N' && D != 'U') { set_error(routine, 5, "invalid diag"); return 5; }
    if (count == 0) return 0;
    if (!m || !n || !alpha || !a || !lda || !b || !ldb) { set_error(routine, 6, "null argument array"); return 6; }
    std::vector<TrsmDesc> descs;
    descs.reserve((size_t)count);
    int64_t work = 0;
    for (int64_t i = 0; i < count; ++i) {
        if (m[i] < 0 || n[i] < 0) { set_error(routine, 6, "negative size in instance " + std::to_string(i)); return 6; }
        if (m[i] == 0 || n[i] == 0) continue;
        int64_t na = (S == 'L') ? m[i] : n[i];
        if (lda[i] < std::max<int64_t>(1, na)) { set_error(routine, 10, "lda too small in instance " + std::to_string(i)); return 10; }
        if (ldb[i] < std::max<int64_t>(1, m[i])) { set_error(routine, 12, "ldb too small in instance " + std::to_string(i)); return 12; }
        if (!is_dd_device_pointer(b[i])) {
            set_error(routine, 11, "grouped calls take 16-byte aligned device (or managed) arrays; B of instance " +
                                       std::to_string(i));
            return 11;
        }
        if (!is_dd_device_pointer(a[i])) {
            set_error(routine, 9, "grouped calls take 16-byte aligned device (or managed) arrays; A of instance " +
                                      std::to_string(i));
            return 9;
        }
        TrsmDesc d{};
        d.A = (const double2 *)a[i];
        d.B = (double2 *)b[i];
        d.lda = lda[i];
        d.ldb = ldb[i];
        d.m = (int)m[i];
        d.n = (int)n[i];
        d.alpha = make_double2(alpha[i].limbs[0], alpha[i].limbs[1]);
        const int64_t rhs = (S == 'L') ? n[i] : m[i];
        d.nchunks = (int)((rhs + 31) / 32);
        descs.push_back(d);
    }
    if (descs.empty()) return 0;
    // the longest triangles first, so that they do not form the tail
    std::stable_sort(descs.begin(), descs.end(), [S](const TrsmDesc &x, const TrsmDesc &y) {
        return (S == 'L' ? x.m : x.n) > (S == 'L' ? y.m : y.n);
    });
    int64_t xop_elems = 0;
    for (TrsmDesc &d : descs) {
        d.work_begin = work;
        work += d.nchunks;
        d.xop_begin = xop_elems;
        xop_elems += (int64_t)d.nchunks * (S == 'L' ? d.m : d.n) * 32;
    }
    if (!ensure_device(routine)) return mwblas_last_error();
    const bool trans = (T != 'N');
    const bool lower = ((U == 'L') != trans);
    TrsmPlan &pl = t_tplan;
    pl.descs.swap(descs);
    pl.total = work;
    pl.xop_elems = xop_elems;
    pl.side = S == 'L' ? 0 : 1;
    pl.lower = lower ? 1 : 0;
    pl.trans = trans ? 1 : 0;
    pl.unit = D == 'U' ? 1 : 0;
    if (!trsm_prepare_and_launch(pl, routine)) return mwblas_last_error();
    if (!finish(routine)) return mwblas_last_error();
    return 0;
}

extern "C" int mwblas_grouped_tuned_tile(void) { return mw::t_tuned_tile; }
extern "C" int mwblas_grouped_tuned_tensor_min(void) { return mw::t_tuned_oz; }
extern "C" int mwblas_grouped_tuned_tensor_pack(void) { return mw::t_tuned_pack; }

extern "C" int mwblas_set_grouped_tensor_pack(int kmin)
{
    return mw::g_forced_pack.exchange(kmin < 0 ? -1 : kmin);
}

extern "C" int mwblas_set_grouped_tensor_min(int size)
{
    return mw::g_forced_oz.exchange(size < 0 ? -1 : size);
}

extern "C" int mwblas_set_grouped_tile(int tile)
{
    const int t = (tile == 16 || tile == 32 || tile == 64) ? tile : 0;
    return mw::g_forced_tile.exchange(t);
}
