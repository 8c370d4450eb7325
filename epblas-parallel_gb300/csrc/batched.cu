// Batched uneven-size double-double GEMM and TRSM (no reference counterpart:
// the reference's CPU baseline for this workload is an OpenMP loop over
// instances calling mgemm_/mtrsm_, whose nested calls run serially,
// mgemm_parallel.cpp:53-60).
//
// mgemm_grouped: the large instances go to the residue engine (ozaki.cu), the rest
// to tiles of one kernel over all of them, so that thousands of uneven instances
// keep all SMs busy. By default these are limb tiles on the tensor cores (their
// section below). Square tiles (32 x 32 beside the limb tiles where build_descs says
// so, 32 x 32 or 64 x 64 for all where forced or tuned) run the fixed-point
// arithmetic of the integer-pipe engine (gemm_fixed.cu, fixgemm.cuh): CTAs of 256
// threads pull (instance, tile, K split) items from an atomic counter, and the
// item's A rows / B columns are scaled from an exponent scan over its own K range
// (no pre-pass, no extra scratch), converted to balanced 24-bit digits while
// staged, and multiplied with exact 64-bit column sums. Items of a split instance
// write partial tiles as extended floats; the CTA that completes a tile's last
// split sums the partials in split order (deterministic) and applies alpha/beta
// with one rounding. The per-call state (descriptors, work counter, split counters,
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
#include <vector>

#include "dd.cuh"
#include "fixgemm.cuh"
#include "fixbeta.cuh"
#include "fixround.cuh"
#include "limbmma.cuh"
#include "xword.cuh"
#include "level3.h"
#include "runtime.h"
#include "sm100.cuh"

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
    // tensor-core tiles only: the operands as limbs in the wave's scratch
    int64_t conv_begin;   // first (32 lines of op(A), then op(B); K split) of the conversion in the wave
    int64_t a_off, b_off; // [64 k][line] blocks of LT_BLOCK bytes
    int64_t ea_off, eb_off;   // exponent bounds of the lines, split after split
    int kp, kc;           // k rounded up to 16, blocks along k
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

// ---- 8 x 16 output tiles on the tensor cores (byte limbs) -------------------------------
//
// Operands are scaled to integers N below 2^116 of their row's (column's) bound over
// the tile's K split, as in the digit kernel below, and held as 15 digits d_i in [-128, 127] of base
// 256, fp16 each, and a zero. A first kernel writes them once per operand
// (k_grp_limbs) in blocks of 16 digits x 64 k per line, as the shared-memory image
// of a K-major operand with 128-byte swizzle; the blocks of neighbouring lines are
// neighbours, so the operands of a tile and 64 k are two bulk copies.
//
// A tile is one tcgen05 accumulator: rows are the digits of 8 rows of op(A),
// columns the digits of 16 columns of op(B), 128 x 256. Over 256 k its entries are
// integers of at most 2^22, exact in FP32. Warps by role, one block per SM:
//   0      finds the tiles' instances, 32 tiles at a time
//   1      issues the MMAs; two accumulators, one filling while the other is read
//   2..9   join the 256 digit products of an output to 32 64-bit sums at weights
//          2^(16 (g + 2 t)) in shared memory: a lane holds one digit of a row and
//          joins it with the 16 of a column (one tcgen05.ld) to words of 16, then
//          32 bits, and with its neighbour's digit to its half of those
//   10..17 two groups that take turns: a lane takes one output; the 32 sums are
//          one carry chain to a 256-bit integer, updated and rounded as in
//          fixround.cuh
//   18     issues the tiles' copies, three stages ahead
//
// Bound: the chain of its stages. On 1000 products of sizes log-uniform in [8, 512]
// (those with m or n below 128 or k below 64) it takes 1.03 ms; the copies alone,
// 7.7 GB from L2, take 0.46, with the MMAs 0.65, without the joining 0.78, without
// the finishing 0.93; the tensor pipe is 20 % busy, issue 55 %. 16 joining or 12
// finishing warps change nothing; with the search for a tile's instance in the
// copying warp it took 1.2. On 4000 such products 9.8 ms on 16 x 16 tiles of the
// legacy MMA (mma.sync, a third busy), 14.9 on 32 x 32 digit tiles, now 4.6, with
// 1.26 for the digits (0.84 as bytes).
constexpr int LT = 16;                              // the policy's name for these tiles
constexpr int LT_M = 8, LT_N = 16;                  // rows and columns of a tile
constexpr int LT_BLOCK = 16 * 64 * 2;               // bytes of a line's digits over 64 k
constexpr int LT_A = LT_M * LT_BLOCK, LT_STAGE = (LT_M + LT_N) * LT_BLOCK, LT_STAGES = 3;
constexpr int LT_ACC_K = 256;                       // k per accumulator
constexpr int LT_ROW = 33;                          // 64-bit sums per output (32 and a pad)
constexpr int LT_SUMS = LT_M * LT_N * LT_ROW;       // of a tile
constexpr int LT_BATCH = 32;                        // tiles announced together, two batches at a time
constexpr int LT_EXT = 8, LT_FIN = 8;              // extracting and finishing warps
constexpr int LT_GROUPS = LT_FIN / 4;               // of finishing warps, taking turns
constexpr int LT_EXTN = LT_N / (LT_EXT / 4);        // columns of an extracting warp
constexpr int LT_THREADS = 32 * (3 + LT_EXT + LT_FIN);
constexpr int LT_SMEM = 1024 + LT_STAGES * LT_STAGE + 2 * LT_SUMS * 8;
constexpr int64_t LT_WAVE = 1ll << 19;              // blocks (1 GiB) of a wave at most

// v * 2^sh (|.| < 2^116) rounded to an integer N, as the bytes of N + 128 (1 + 256 +
// .. + 256^14): byte i holds d_i + 128.
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
        "addc.u32 %3, %8, 0;\n\t"
        "add.cc.u32 %0, %0, 0x80808080;\n\t"
        "addc.cc.u32 %1, %1, 0x80808080;\n\t"
        "addc.cc.u32 %2, %2, 0x80808080;\n\t"
        "addc.u32 %3, %3, 0x00808080;\n\t}"
        : "=&r"(b.x), "=&r"(b.y), "=&r"(b.z), "=&r"(b.w)
        : "r"(m & 1u), "r"(w[0] ^ m), "r"(w[1] ^ m), "r"(w[2] ^ m), "r"(w[3] ^ m));
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

// Exponent bounds and digits of 32 lines (rows of op(A) or columns of op(B)) of
// one K split of an instance per block; the second pass reads what the first left
// in the caches. A thread converts 8 k of a line: 16 bytes in each of the block's
// rows. (A block per 32 lines for all of k left 3 products of 64 x 64 x 16384 to 12
// blocks: 1039 us the call, now 244.)
__global__ void __launch_bounds__(GTHREADS) k_grp_limbs(const GemmDesc *__restrict__ descs, int count,
                                                        unsigned char *out, int *ex)
{
    __shared__ int s_e[32];
    const int tid = threadIdx.x;
    const GemmDesc &d =
        descs[grp_search(count, (int64_t)blockIdx.x, [&](int q) { return descs[q].conv_begin; })];
    const uint32_t at = (uint32_t)((int64_t)blockIdx.x - d.conv_begin);
    int grp = (int)(d.splitk == 1 ? at : at / (uint32_t)d.splitk);
    const int sp = (int)(at - (uint32_t)grp * (uint32_t)d.splitk), k0 = sp * d.klen;
    const int ga = (d.m + 31) / 32;
    const bool isA = grp < ga;
    if (!isA) grp -= ga;
    const int lines = isA ? d.m : d.n, line0 = grp * 32, nl = min(32, lines - line0);
    const int k = min(d.k - k0, d.klen), kp = min(d.kp - k0, d.klen);
    const bool along_k = isA ? d.ta != 0 : d.tb == 0;   // a line's entries are neighbours in memory
    const int64_t ld = isA ? d.lda : d.ldb;
    const int64_t sl = along_k ? ld : 1, sk = along_k ? 1 : ld;
    const double2 *X = (isA ? d.A : d.B) + line0 * sl + k0 * sk;
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
    if (tid < nl) ex[(isA ? d.ea_off : d.eb_off) + (int64_t)sp * lines + line0 + tid] = s_e[tid];
    // 8 neighbours along k, or 8 lines x 4 k per warp: whole 64 bytes either way
    const int l = along_k ? tid >> 3 : (tid & 7) + 8 * ((tid >> 5) & 3);
    const int q = along_k ? tid & 7 : ((tid >> 3) & 3) + 4 * (tid >> 7);
    if (l >= nl) return;
    const int e = s_e[l];
    const bool live = e > kNoExp / 2 && e < 1024;
    const double2 *x = X + l * sl + (int64_t)(8 * q) * sk;
    unsigned char *o = out + ((isA ? d.a_off : d.b_off) + (int64_t)(k0 / 64) * lines + line0 + l) * LT_BLOCK;
    const int64_t next = (int64_t)lines * LT_BLOCK;
    for (int p0 = 8 * q; p0 < kp; p0 += 64, x += 64 * sk, o += next) {
        double2 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = live && p0 + u < k ? x[u * sk] : make_double2(0.0, 0.0);
        uint4 b[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
            b[u] = live ? limb_bytes(v[u], fxg::FX_S - e)
                        : make_uint4(0x80808080u, 0x80808080u, 0x80808080u, 0x808080u);
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            uint32_t h[4] = {0u, 0u, 0u, 0u};
            if (r < 15) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    auto word = [&](const uint4 &y) { return r < 4 ? y.x : r < 8 ? y.y : r < 12 ? y.z : y.w; };
                    // 1024 + byte in both halves, less 1152
                    const uint32_t t = __byte_perm(word(b[2 * u]), word(b[2 * u + 1]), (r & 3) | (4 + (r & 3)) << 8);
                    asm("sub.f16x2 %0, %1, %2;" : "=r"(h[u]) : "r"((t & 0x00FF00FFu) | 0x64006400u), "r"(0x64806480u));
                }
            }
            *reinterpret_cast<uint4 *>(o + r * 128 + ((q ^ (r & 7)) << 4)) = make_uint4(h[0], h[1], h[2], h[3]);
        }
    }
}

// A tile as announced to the roles.
struct LtItem {
    int64_t a, b;                // first blocks of its operands
    int64_t ea, eb;              // first of its lines' exponent bounds
    int desc, i0, j0, mr, nc, kn, tile, split;
    int lines_a, lines_b;        // blocks from one 64 k to the next
};

__global__ void __launch_bounds__(LT_THREADS, 1) k_gemm_grouped_limb(const GemmDesc *__restrict__ descs, int count,
                                                                    int total, int *tile_counters,
                                                                    fx::XFPod *partials,
                                                                    const unsigned char *__restrict__ limbs,
                                                                    const int *__restrict__ ex, int *status,
                                                                    int lose_loads)
{
    extern __shared__ unsigned char s_dyn[];   // stages, then the sums of two tiles
    __shared__ uint64_t full[LT_STAGES], empty[LT_STAGES], accf[2], acce[2], sumf[LT_GROUPS], sume[2];
    __shared__ uint64_t itemf[2], iteme[2], drain;
    __shared__ uint64_t partf[LT_GROUPS], lastf[LT_GROUPS];   // a group's partial sums are out; s_last is set
    __shared__ LtItem items[2 * LT_BATCH];
    __shared__ uint32_t s_tmem;
    __shared__ int s_last[LT_GROUPS];
    unsigned char *stages = (unsigned char *)(((uintptr_t)s_dyn + 1023) & ~(uintptr_t)1023);
    unsigned long long *sums = reinterpret_cast<unsigned long long *>(stages + LT_STAGES * LT_STAGE);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_items = (total - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;

    if (threadIdx.x == 0) {
        for (int q = 0; q < LT_STAGES; ++q) {
            sm100::mbar_init(&full[q], 1);
            sm100::mbar_init(&empty[q], 1);
        }
        for (int q = 0; q < 2; ++q) {
            sm100::mbar_init(&accf[q], 1);
            sm100::mbar_init(&acce[q], LT_EXT);
            sm100::mbar_init(&sume[q], 4);
        }
        for (int q = 0; q < LT_GROUPS; ++q) {
            sm100::mbar_init(&sumf[q], LT_EXT);
            sm100::mbar_init(&partf[q], 4);
            sm100::mbar_init(&lastf[q], 1);
        }
        for (int q = 0; q < 2; ++q) {
            sm100::mbar_init(&itemf[q], 1);
            sm100::mbar_init(&iteme[q], 2 + LT_EXT + LT_FIN);
        }
        sm100::mbar_init(&drain, 1);
        sm100::fence_mbar_init();
    }
    if (warp == 1) {
        sm100::tmem_alloc(&s_tmem, 512);
        sm100::tmem_relinquish();
    }
    sm100::tc_fence_before();
    __syncthreads();
    sm100::tc_fence_after();
    const uint32_t tmem = s_tmem;

    // Tile `it` of this block, once its batch is announced; `last` is the caller's
    // previous tile (-1: none), whose batch it gives back with the step to another.
    auto item = [&](int it, int last, int code) -> bool {
        const int n = it / LT_BATCH;
        if (last >= 0 && last / LT_BATCH == n) return true;
        if (last >= 0) {
            __syncwarp();
            if (lane == 0) sm100::mbar_arrive(&iteme[(n - 1) & 1]);
        }
        return __all_sync(0xffffffffu, sm100::mbar_wait(&itemf[n & 1], (n >> 1) & 1, status, code));
    };
    if (warp == 0) {
        for (int n = 0; n * LT_BATCH < n_items; ++n) {
            if (n >= 2 &&
                !__all_sync(0xffffffffu, sm100::mbar_wait(&iteme[n & 1], ((n >> 1) - 1) & 1, status, 1)))
                break;
            const int it = n * LT_BATCH + lane, w = (int)blockIdx.x + it * (int)gridDim.x;
            if (it < n_items) {   // a lane's binary search beside the others'
                LtItem x;
                x.desc = grp_search(count, (int64_t)w, [&](int q) { return descs[q].work_begin; });
                const GemmDesc &d = descs[x.desc];
                const uint32_t local = (uint32_t)(w - d.work_begin), tile = local / (uint32_t)d.splitk;
                x.tile = (int)tile;
                x.split = (int)(local % (uint32_t)d.splitk);
                x.i0 = (int)(tile % (uint32_t)d.tiles_m) * LT_M;
                x.j0 = (int)(tile / (uint32_t)d.tiles_m) * LT_N;
                const int k0 = x.split * d.klen;   // klen: multiples of 64 where split
                x.kn = d.k > 0 ? min(d.kp, k0 + d.klen) - k0 : 0;
                x.mr = min(LT_M, d.m - x.i0);
                x.nc = min(LT_N, d.n - x.j0);
                x.lines_a = d.m;
                x.lines_b = d.n;
                x.a = d.a_off + (int64_t)(k0 / 64) * d.m + x.i0;
                x.b = d.b_off + (int64_t)(k0 / 64) * d.n + x.j0;
                x.ea = d.ea_off + (int64_t)x.split * d.m + x.i0;
                x.eb = d.eb_off + (int64_t)x.split * d.n + x.j0;
                items[it % (2 * LT_BATCH)] = x;
            }
            __syncwarp();
            if (lane == 0) sm100::mbar_arrive(&itemf[n & 1]);
        }
    } else if (warp == 2 + LT_EXT + LT_FIN) {
        uint32_t gs = 0;   // stages filled
        bool ok = true;
        // lose_loads (a failure-injection hook): no copy at all, so that nothing is in
        // flight and the MMA warp's first wait runs out
        for (int it = 0; it < n_items && ok && !lose_loads; ++it) {
            if (!item(it, it - 1, 1)) break;
            const LtItem &x = items[it % (2 * LT_BATCH)];
            const unsigned char *pA = limbs + x.a * LT_BLOCK, *pB = limbs + x.b * LT_BLOCK;
            for (int c0 = 0; c0 < x.kn; c0 += 64, ++gs) {
                const int st = gs % LT_STAGES;
                ok = gs < LT_STAGES ||
                     __all_sync(0xffffffffu, sm100::mbar_wait(&empty[st], (gs / LT_STAGES - 1) & 1, status, 1));
                if (!ok) break;
                if (lane == 0) {
                    unsigned char *at = stages + st * LT_STAGE;
                    sm100::mbar_arrive_expect_tx(&full[st], (uint32_t)(x.mr + x.nc) * LT_BLOCK);
                    sm100::bulk_load(at, pA, (uint32_t)x.mr * LT_BLOCK, &full[st]);
                    sm100::bulk_load(at + LT_A, pB, (uint32_t)x.nc * LT_BLOCK, &full[st]);
                }
                pA += (int64_t)x.lines_a * LT_BLOCK;
                pB += (int64_t)x.lines_b * LT_BLOCK;
            }
        }
        // never leave with copies in flight: wait (bounded) for the last use of every stage
        for (uint32_t t = gs > LT_STAGES ? gs - LT_STAGES : 0; t < gs; ++t)
            sm100::mbar_wait(&full[t % LT_STAGES], (t / LT_STAGES) & 1, nullptr, 0);
    } else if (warp == 1) {
        uint32_t gs = 0, cg = 0;   // stages used, accumulators filled
        bool ok = true;
        for (int it = 0; it < n_items && ok; ++it) {
            if (!item(it, it - 1, 2)) break;
            const LtItem &x = items[it % (2 * LT_BATCH)];
            const int kn = x.kn;
            const uint32_t idesc = sm100::idesc_f16_f32(128, 16 * x.nc);
            for (int c0 = 0; c0 < kn && ok; c0 += LT_ACC_K, ++cg) {
                const int b = cg & 1;
                if (cg >= 2) {
                    ok = __all_sync(0xffffffffu, sm100::mbar_wait(&acce[b], (cg / 2 - 1) & 1, status, 2));
                    if (!ok) break;
                    sm100::tc_fence_after();
                }
                const int c1 = min(kn, c0 + LT_ACC_K);
                for (int c = c0; c < c1; c += 64, ++gs) {
                    const int st = gs % LT_STAGES;
                    ok = __all_sync(0xffffffffu, sm100::mbar_wait(&full[st], (gs / LT_STAGES) & 1, status, 3));
                    if (!ok) break;
                    sm100::tc_fence_after();
                    if (lane == 0) {
                        const uint64_t ad = sm100::smem_desc_sw128(sm100::smem_u32(stages + st * LT_STAGE));
                        const uint64_t bd = sm100::smem_desc_sw128(sm100::smem_u32(stages + st * LT_STAGE + LT_A));
                        const int steps = min(4, (c1 - c) / 16);
                        for (int q = 0; q < steps; ++q)
                            sm100::mma_f16(tmem + b * 256, ad + 2 * q, bd + 2 * q, idesc, c > c0 || q > 0 ? 1u : 0u);
                        sm100::mma_commit(&empty[st]);
                        if (c + 64 >= c1) sm100::mma_commit(&accf[b]);
                    }
                    __syncwarp();
                }
            }
        }
        // no MMA may still be writing TMEM when it is freed
        if (lane == 0) {
            sm100::mma_commit(&drain);
            sm100::mbar_wait(&drain, 0, nullptr, 0);
        }
    } else if (warp < 2 + LT_EXT) {
        // rows 2 quad, 2 quad + 1 of the tile (lane: digit lane % 16 of one), columns LT_EXTN part ..
        const int quad = warp & 3, part = (warp - 2) >> 2, odd = lane & 1;
        const int row = 2 * quad + (lane >> 4);
        const uint32_t at0 = tmem + ((uint32_t)(quad * 32) << 16) + part * (16 * LT_EXTN);
        // weights of this lane's digit and its neighbour's
        const uint32_t own = odd ? 256u : 1u, other = odd ? 1u : 256u;
        const unsigned long long off = 0x8B400000ull * 257u * 65537u;
        uint32_t cg = 0;
        bool ok = true;
        for (int it = 0; it < n_items && ok; ++it) {
            const int sb = it & 1;
            if (!item(it, it - 1, 4)) break;
            const LtItem &x = items[it % (2 * LT_BATCH)];
            const int nc = min(LT_EXTN, x.nc - LT_EXTN * part);
            if (it >= 2) {
                ok = __all_sync(0xffffffffu, sm100::mbar_wait(&sume[sb], (it / 2 - 1) & 1, status, 4));
                if (!ok) break;
            }
            unsigned long long *to = sums + sb * LT_SUMS + ((LT_EXTN * part) * LT_M + row) * LT_ROW +
                                     4 * ((lane & 15) >> 1) + 2 * odd;
            for (int c0 = 0; c0 < x.kn; c0 += LT_ACC_K, ++cg) {
                const int b = cg & 1;
                ok = __all_sync(0xffffffffu, sm100::mbar_wait(&accf[b], (cg / 2) & 1, status, 4));
                if (!ok) break;
                sm100::tc_fence_after();
                if (2 * quad < x.mr) {
#pragma unroll 1
                    for (int j = 0; j < nc; j += 2) {   // (a column past nc is stored too: nobody reads it)
                        uint32_t r[32];
                        sm100::tmem_ld32(at0 + b * 256 + j * 16, r);
                        sm100::tmem_wait_ld();
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            uint32_t p[8];
#pragma unroll
                            for (int q = 0; q < 8; ++q) {
                                float2 f = make_float2(__uint_as_float(r[16 * u + 2 * q]),
                                                       __uint_as_float(r[16 * u + 2 * q + 1]));
                                f = __fadd2_rn(f, make_float2(12582912.0f, 12582912.0f));   // 0x4B400000 + integer
                                p[q] = __float_as_uint(f.x) + 256u * __float_as_uint(f.y);   // 0x8B400000 + integer
                            }
                            uint32_t keep[4], got[4];
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                keep[q] = odd ? p[4 + q] : p[q];
                                got[q] = __shfl_xor_sync(0xffffffffu, odd ? p[q] : p[4 + q], 1);
                            }
                            unsigned long long *dst = to + (j + u) * (LT_M * LT_ROW);
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                unsigned long long y = (c0 == 0 ? 0ull : dst[h]) - off;
                                y += (unsigned long long)keep[2 * h] * own;
                                y += (unsigned long long)got[2 * h] * other;
                                y += (unsigned long long)keep[2 * h + 1] * (own << 16);
                                y += (unsigned long long)got[2 * h + 1] * (other << 16);
                                dst[h] = y;
                            }
                        }
                    }
                }
                sm100::tc_fence_before();
                __syncwarp();
                if (lane == 0) sm100::mbar_arrive(&acce[b]);
            }
            __syncwarp();
            if (ok && lane == 0) sm100::mbar_arrive(&sumf[it % LT_GROUPS]);
        }
    } else {
        const int group = (warp - 2 - LT_EXT) >> 2, part = (warp - 2 - LT_EXT) & 3;
        const int orow = lane & 7, ocol = 4 * part + (lane >> 3), out = ocol * LT_M + orow;
        uint32_t splits = 0;   // split tiles of this group so far
        for (int it = group; it < n_items; it += LT_GROUPS) {
            const int sb = it & 1;
            const unsigned long long *at = sums + sb * LT_SUMS + out * LT_ROW;
            if (!item(it, it >= LT_GROUPS ? it - LT_GROUPS : -1, 5)) break;
            const LtItem &x = items[it % (2 * LT_BATCH)];
            const GemmDesc &d = descs[x.desc];
            const bool in = orow < x.mr && ocol < x.nc, some = d.k > 0;
            const int ei = in && some ? ex[x.ea + orow] : kNoExp;
            const int ej = in && some ? ex[x.eb + ocol] : kNoExp;
            bool bad = ei >= 1024 || ej >= 1024;
            const bool live = !bad && ei > kNoExp / 2 && ej > kNoExp / 2;
            double2 *pc = d.C + x.i0 + orow + (int64_t)(x.j0 + ocol) * d.ldc;
            const double2 c_in = in && d.beta_kind != 0 && d.splitk == 1 ? *pc : make_double2(0.0, 0.0);
            if (!__all_sync(0xffffffffu, sm100::mbar_wait(&sumf[group], (it / LT_GROUPS) & 1, status, 5))) break;
            uint64_t W[4] = {0, 0, 0, 0};
            if (live) {
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
            __syncwarp();
            if (lane == 0) sm100::mbar_arrive(&sume[sb]);
            const int e0 = ei + ej - 2 * fxg::FX_S;
            bool done = false;
            if (in && live && d.splitk == 1) {
                // the top 160 bits of |W| (2^-134 of the largest product is cut), alpha, beta C, one rounding
                const uint32_t m = (uint32_t)((int64_t)W[3] >> 63);
                uint32_t x8[8];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    x8[2 * q] = (uint32_t)W[q];
                    x8[2 * q + 1] = (uint32_t)(W[q] >> 32);
                }
                fxr::cond_neg<8>(x8, m);
                fxr::Fix a;
                a.neg = m & 1u;
                if (d.alpha.x == 1.0 && d.alpha.y == 0.0) {
#pragma unroll
                    for (int q = 0; q < 5; ++q) a.w[q] = x8[3 + q];
                    a.e = e0 + 96;
                } else {
                    fxr::mul54(x8 + 3, d.xa.w, a.w);
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
                fx::XFPod *base = partials + (d.part_begin + (int64_t)x.tile * d.splitk) * (LT_M * LT_N) + out;
                base[x.split * (LT_M * LT_N)] = fx::to_pod(v, bad);
                __threadfence();
                __syncwarp();
                // the group's warps meet at barriers with a limit (not at a named barrier): one
                // of them may have left after a wait that gave up
                const uint32_t phase = splits++ & 1;
                if (lane == 0) sm100::mbar_arrive(&partf[group]);
                if (part == 0) {
                    if (!__all_sync(0xffffffffu, sm100::mbar_wait(&partf[group], phase, status, 6))) break;
                    if (lane == 0) {
                        s_last[group] = atomicAdd(&tile_counters[d.tile_begin + x.tile], 1) == d.splitk - 1;
                        sm100::mbar_arrive(&lastf[group]);
                    }
                }
                if (!__all_sync(0xffffffffu, sm100::mbar_wait(&lastf[group], phase, status, 6))) break;
                const bool finish = s_last[group] != 0;
                __syncwarp();
                if (!finish) continue;
                __threadfence();
                v.zero = true; v.neg = false; v.m = 0; v.e = 0;
                bad = false;
                for (int s2 = 0; s2 < d.splitk; ++s2) {
                    // partials written by other CTAs: read through L2
                    const fx::XFPod *q = base + s2 * (LT_M * LT_N);
                    fx::XFPod pv;
                    pv.hi = __ldcg(&q->hi);
                    pv.lo = __ldcg(&q->lo);
                    pv.e = __ldcg(&q->e);
                    pv.flags = __ldcg(&q->flags);
                    bad |= (pv.flags & 4) != 0;
                    v = xfp::xf_add(v, fx::from_pod(pv));
                }
                if (part == 0 && lane == 0) tile_counters[d.tile_begin + x.tile] = 0;   // ready for the next replay
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
        }
    }

    sm100::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        sm100::tc_fence_after();
        sm100::tmem_dealloc(tmem, 512);
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
    bool by_cost = true;       // limb tiles: not for a short k that the 32 x 32 tiles finish sooner
};

struct Plan {
    std::vector<GemmDesc> descs;
    std::vector<OzGroupItem> oz_items;   // instances routed to the tensor-core engine
    OzGroupPlan *oz = nullptr;
    int tile = 32;
    int64_t split_tiles = 0, partial_elems = 0;
    // square tiles: the descriptors from `square` on, their work items and the place of
    // their partial tiles
    int64_t square = 0, square_work = 0, square_partials = 0;
    // limb tiles: descriptors [first, first + count) share the limb scratch
    struct Wave {
        int first, count;
        int64_t work, groups, blocks, lines;
    };
    std::vector<Wave> waves;
    int64_t wave_blocks = 0, wave_lines = 0;   // largest of any wave
    // device state
    void *dev = nullptr;
    size_t dev_bytes = 0;
    cudaGraphExec_t exec = nullptr;
    uint64_t key = 0;

    Plan() = default;
    Plan(const Plan &) = delete;
    Plan &operator=(const Plan &) = delete;
    ~Plan()   // at the end of its thread (or of a tuner call)
    {
        if (exec) cudaGraphExecDestroy(exec);
        if (dev) cudaFree(dev);
        ozgroup_destroy(oz);
    }
};

// Device time of an m x n x k product on the limb and on the 32 x 32 digit tiles, in
// ns of a full GPU. The limb tiles' digit products are joined whatever k is (us of
// 2000 products, limb and digit tiles: 127 x 127 x 8 3650 and 2625, x 16 3660 and
// 3210, x 32 3700 and 4400; 48 x 48 x 8 1155 and 1080, x 16 1160 and 1250).
double limb_ns(int64_t m, int64_t n, int64_t k)
{
    return (double)((m + LT_M - 1) / LT_M) * (double)((n + LT_N - 1) / LT_N) * (12.0 + 0.085 * (k > 64 ? k - 64 : 0));
}
double digit_ns(int64_t m, int64_t n, int64_t k)
{
    return (double)((m + 31) / 32) * (double)((n + 31) / 32) * (50.0 + 19.0 * (k <= 8 ? 0 : (k - 1) / 8));
}

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
    pl.tile = pol.tile;
    std::vector<GemmDesc> squares;
    int64_t stiles = 0, pslots = 0, sq_work = 0, sq_pslots = 0;
    pl.waves.clear();
    pl.wave_blocks = pl.wave_lines = 0;
    // Instances with a short k on the digit tiles, in a launch of their own, where that
    // saves a sixth of the limb tiles' time (4000 products in [8, 512], a quarter of them
    // of k <= 24: 40 us slower with two launches; 127 x 127 x 8: a quarter faster).
    bool short_k = false;
    if (pol.tile == LT && pol.by_cost) {
        double all = 0.0, saved = 0.0;
        for (int64_t i = 0; i < count; ++i) {
            if (m[i] <= 0 || n[i] <= 0) continue;
            const double l = limb_ns(m[i], n[i], k[i]);
            if (!(oz_min > 0 && m[i] >= oz_min && n[i] >= oz_min && k[i] >= 64)) all += l;
            if (k[i] <= 24) saved += std::max(0.0, l - digit_ns(m[i], n[i], k[i]));
        }
        short_k = saved > all / 6.0;
    }
    // d on tiles of GT: its tiles, splits and places
    auto place = [&](GemmDesc &d, const int GT) {
        d.tiles_m = GT == LT ? (d.m + LT_M - 1) / LT_M : (d.m + GT - 1) / GT;
        d.tiles_n = (d.n + GT - 1) / GT;
        const int tiles = d.tiles_m * d.tiles_n;
        d.splitk = 1;
        // (limb tiles: counted as 32 x 32 ones, so that the same products split)
        const int64_t count_as = GT == LT ? ((int64_t)d.m + 31) / 32 * (((int64_t)d.n + 31) / 32) : tiles;
        if (pol.min_k_per_split > 0 && count_as <= pol.max_tiles_split && d.k >= 2 * pol.min_k_per_split)
            d.splitk = std::min(16, d.k / pol.min_k_per_split);
        // the digit column sums hold at most 16384 multiply-adds per split, the
        // limb sums 4096 (16 accumulators' sums below 2^56 each, four of them added)
        const int kmax = GT == LT ? 4096 : 16384;
        const int need_splits = (d.k + kmax - 1) / kmax;
        if (d.splitk < need_splits) d.splitk = need_splits;
        d.kp = (d.k + 15) / 16 * 16;
        const int kstep = GT == LT ? 64 : GBK;
        d.klen = d.splitk > 1 ? ((d.k + d.splitk - 1) / d.splitk + kstep - 1) / kstep * kstep
                              : std::max(GT == LT ? d.kp : d.k, 1);
        if (d.k == 0) d.klen = 1;
        int64_t *work = &sq_work, *slots = &sq_pslots;
        if (GT == LT) {
            // splits past k would be empty: as many as klen needs
            if (d.splitk > 1) d.splitk = (d.k + d.klen - 1) / d.klen;
            d.xa = xw::from_dd(d.alpha.x, d.alpha.y);
            d.xb = xw::from_dd(d.beta.x, d.beta.y);
            d.kc = (d.k + 63) / 64;
            const int64_t blocks = ((int64_t)d.m + d.n) * d.kc;
            const int64_t lines = d.k > 0 ? ((int64_t)d.m + d.n) * d.splitk : 0;   // bounds: one per line and split
            const int64_t tw = (int64_t)tiles * d.splitk;
            if (pl.waves.empty() || pl.waves.back().blocks + blocks > LT_WAVE ||
                pl.waves.back().work + tw > INT32_MAX)
                pl.waves.push_back(Plan::Wave{(int)pl.descs.size(), 0, 0, 0, 0, 0});
            Plan::Wave &wv = pl.waves.back();
            d.conv_begin = wv.groups;
            d.a_off = wv.blocks;
            d.b_off = wv.blocks + (int64_t)d.m * d.kc;
            d.ea_off = wv.lines;
            d.eb_off = wv.lines + (int64_t)d.m * d.splitk;
            wv.groups += d.k > 0 ? ((int64_t)(d.m + 31) / 32 + (d.n + 31) / 32) * d.splitk : 0;
            wv.blocks += blocks;
            wv.lines += lines;
            wv.count++;
            pl.wave_blocks = std::max(pl.wave_blocks, wv.blocks);
            pl.wave_lines = std::max(pl.wave_lines, wv.lines);
            work = &wv.work;   // work items are numbered within the wave
            slots = &pslots;
        }
        d.work_begin = *work;
        d.tile_begin = d.splitk > 1 ? stiles : 0;
        d.part_begin = d.splitk > 1 ? *slots : 0;
        if (d.splitk > 1) {
            stiles += tiles;
            *slots += (int64_t)tiles * d.splitk;
        }
        *work += (int64_t)tiles * d.splitk;
        (GT == LT ? pl.descs : squares).push_back(d);
    };
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
        // An instance of many lines goes in pieces that a wave holds. On the square tiles,
        // which need no scratch: one with a k so long that its pieces would be thin, and one
        // whose splits (every 4096 k here, 16384 there) would leave partial tiles of more than
        // a wave and an eighth of its operands.
        const int64_t kc = std::max<int64_t>(1, ((int64_t)d.k + 63) / 64), lines = LT_WAVE / kc;
        const double partial = d.k > 4096 ? 32.0 * d.m * d.n * ((d.k + 4095) / 4096) : 0.0;
        if (pol.tile != LT) {
            place(d, pol.tile);
        } else if ((short_k && digit_ns(d.m, d.n, d.k) < limb_ns(d.m, d.n, d.k)) || ((int64_t)d.m + d.n > lines && lines < 512) ||
                   (partial > (double)LT_WAVE * LT_BLOCK && partial > 2.0 * ((double)d.m + d.n) * d.k)) {
            place(d, 32);
        } else {
            if ((int64_t)d.m + d.n <= lines) {
                place(d, LT);
                continue;
            }
            const int half = (int)(lines / 2 / 16 * 16);
            const int pm = d.m <= half ? d.m : (d.n <= half ? (int)((lines - d.n) / 16 * 16) : half);
            const int pn = d.n <= half ? d.n : (d.m <= half ? (int)((lines - d.m) / 16 * 16) : half);
            for (int r0 = 0; r0 < d.m; r0 += pm) {
                for (int c0 = 0; c0 < d.n; c0 += pn) {
                    GemmDesc q = d;
                    q.A = d.A + (d.ta ? (int64_t)r0 * d.lda : r0);
                    q.B = d.B + (d.tb ? c0 : (int64_t)c0 * d.ldb);
                    q.C = d.C + r0 + (int64_t)c0 * d.ldc;
                    q.m = std::min(pm, d.m - r0);
                    q.n = std::min(pn, d.n - c0);
                    place(q, LT);
                }
            }
        }
    }
    pl.square = (int64_t)pl.descs.size();
    pl.square_work = sq_work;
    pl.descs.insert(pl.descs.end(), squares.begin(), squares.end());
    pl.split_tiles = stiles;
    // extended-float partials
    const int sq = pl.tile == LT ? 32 : pl.tile;
    pl.square_partials = pslots * (LT_M * LT_N);
    pl.partial_elems = pl.square_partials + sq_pslots * sq * sq;
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
    return mix(mix(mix(h, (uint64_t)pl.tile), (uint64_t)pl.square), (uint64_t)pl.oz_items.size());
}

// (Re)creates the device buffers and the graph when the batch layout changed.
// use_graph = false (the library's own calls, whose layouts change from call
// to call): the kernels are enqueued directly instead of capturing a graph.
bool prepare_and_launch(Plan &pl, const char *routine, bool use_graph = true)
{
    if (pl.descs.empty() && pl.oz_items.empty()) return true;
    const size_t d_bytes = pl.descs.size() * sizeof(GemmDesc);
    const size_t cnt_bytes = 256 + (size_t)(pl.split_tiles + 1) * sizeof(int);
    const size_t part_bytes = (size_t)pl.partial_elems * sizeof(fx::XFPod);
    const size_t limb_bytes_ = (size_t)pl.wave_blocks * LT_BLOCK, ex_bytes = (size_t)pl.wave_lines * sizeof(int);
    const size_t need = d_bytes + cnt_bytes + part_bytes + limb_bytes_ + ex_bytes + 1024;
    const uint64_t key = plan_key(pl);
    cudaStream_t s = stream();
    // The key names the layout whose descriptors the buffers hold: none from here
    // until every step for a new one has succeeded, so that a call that fails half
    // way cannot leave the old key over memory that is gone or rewritten.
    const bool same = pl.key == key && pl.dev_bytes >= need;
    if (!same) pl.key = 0;
    if (pl.dev_bytes < need) {
        if (pl.exec) {
            cudaGraphExecDestroy(pl.exec);
            pl.exec = nullptr;
        }
        if (pl.dev) cudaFree(pl.dev);
        pl.dev = nullptr;
        pl.dev_bytes = 0;
        if (!(pl.dev = plan_alloc(need, routine))) return false;
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
    unsigned char *limbs = (unsigned char *)(base + limb_off);
    int *ex = (int *)(base + (limb_off + limb_bytes_ + 255) / 256 * 256);
    const int sms = device_sm_count();
    if (!same) {
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
    // a launch with lost copies (test hook) is not kept in a graph
    const int lose = !pl.waves.empty() ? take_lost_load_injection() : 0;
    if (lose) use_graph = false;
    // the square-tile and limb-tile parts on stream q; the counters start at zero
    auto enqueue = [&](cudaStream_t q) {
        if (pl.descs.empty()) return;
        cudaMemsetAsync(counter, 0, cnt_bytes, q);
        if (pl.square_work > 0) {
            auto kern = pl.tile == 64 ? k_gemm_grouped<64> : k_gemm_grouped<32>;
            const int grid = (int)std::min<int64_t>(pl.square_work, (int64_t)sms * 16);
            kern<<<grid, GTHREADS, 0, q>>>(ddesc + pl.square, (int)((int64_t)pl.descs.size() - pl.square),
                                           pl.square_work, counter, tile_counters, partials + pl.square_partials);
        }
        if (pl.waves.empty()) return;
        cudaFuncSetAttribute(k_gemm_grouped_limb, cudaFuncAttributeMaxDynamicSharedMemorySize, LT_SMEM);
        for (const Plan::Wave &wv : pl.waves) {
            if (wv.groups > 0)
                k_grp_limbs<<<(unsigned)wv.groups, GTHREADS, 0, q>>>(ddesc + wv.first, wv.count, limbs, ex);
            const int wgrid = (int)std::min<int64_t>(wv.work, sms);
            k_gemm_grouped_limb<<<wgrid, LT_THREADS, LT_SMEM, q>>>(ddesc + wv.first, wv.count, (int)wv.work,
                                                                  tile_counters, partials, limbs, ex,
                                                                  device_status_word(), lose);
        }
    };
    if (!use_graph) {
        pl.key = lose ? 0 : key;
        enqueue(s);
        count_launch(2 * (int64_t)pl.waves.size() + (pl.square_work > 0 ? 1 : 0));
        if (pl.oz && ozgroup_count(pl.oz) > 0) ozgroup_launch(pl.oz, s);
        return cuda_ok(cudaGetLastError(), routine, "grouped launch");
    }
    if (!pl.exec || !same) {
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
            enqueue(cap);
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
        if (!(pl.dev = plan_alloc(need, routine))) return false;
        pl.dev_bytes = need;
    }
    // layout: [descriptors][work counter (256 B)][decoded solutions]
    TrsmDesc *ddesc = (TrsmDesc *)pl.dev;
    unsigned long long *counter = (unsigned long long *)((char *)pl.dev + d_bytes);
    fx::Op *xops = (fx::Op *)((char *)pl.dev + d_bytes + 256);
    if (pl.key != key) {
        pl.key = 0;   // until the new layout's steps have all succeeded
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

void set_grouped_wait_limit(uint64_t ns)
{
    cudaMemcpyToSymbol(sm100::g_wait_limit_ns, &ns, sizeof(ns));
}

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
    if (g_forced_tile.load() > 0) {
        pol.tile = g_forced_tile.load();
        pol.by_cost = false;
    }
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
