// Byte-limb products of double-double operands on the tensor cores, for the
// bandwidth-bound reductions (GEMV, DOT).
//
// An operand's aligned magnitude (the 118-bit integer W of fixacc.cuh, shifted
// right to its block) lies in four 32-bit words, so its base-256 limbs are the
// words' bytes. A byte c with a zero byte above it is the fp16 subnormal
// c * 2^-24, and with the sign bit in that upper byte -c * 2^-24: one PRMT
// makes the signed fp16 pair of two limbs, without a conversion. Tensor-core
// products of fp16 subnormals are exact, and the FP32 accumulator holds every
// sum of limb products below 2^24 units (of 2^-24) exactly; it is moved to
// integers before it could grow past that.
//
// Against the digit form of fixacc.cuh (19 IMAD.WIDE per product, which issue
// at 26 lanes/clk/SM with register operands) the CUDA cores keep only the
// decode, the alignment and 8 PRMT per operand, all at 64 lanes/clk/SM.
// (Shifts and sums rewritten as multiply-adds for the FP32 pipe, to relieve
// the integer ALU pipe, made the GEMV slower, 3.9 against 4.3 TB/s: the count
// of instructions decides, not one pipe.)
#pragma once
#include "fixacc.cuh"

namespace lmb {

using fx::XF;

// The 118-bit magnitude of a double-double on the straight-line path:
// W = hi's mantissa * 2^64 +- lo's mantissa shifted to its place (what falls
// below bit 0, under 2^-117 of hi, is cut), v = +-W * 2^(eh - 1139). False for
// the operands that need fixacc.cuh's general decode: hi zero, non-finite or
// below 2^-895, lo non-finite or less than 53 binades below hi (not
// normalised). A zero or subnormal lo needs no test: its biased exponent 0
// makes the shift at least 75, which leaves nothing of it (a subnormal lo is
// then below 2^-127 of hi).
// `half`: added to W's lowest word, 2^(sh - 1) for a W that is then shifted right
// by sh, which rounds it to nearest.
__device__ __forceinline__ bool is_fast(double2 v)
{
    const uint32_t uh = ((uint32_t)__double2hiint(v.x) << 1) >> 21, ul = ((uint32_t)__double2hiint(v.y) << 1) >> 21;
    return (uh - 128u) < 0x77Fu && (int)(uh - ul - 53u) >= 0;
}
__device__ __forceinline__ bool split_fast(double2 v, uint32_t w[4], int &eh, uint32_t half = 0u)
{
    const uint32_t hl = (uint32_t)__double2loint(v.x), hh = (uint32_t)__double2hiint(v.x);
    const uint32_t ll = (uint32_t)__double2loint(v.y), lh = (uint32_t)__double2hiint(v.y);
    const uint32_t uh = (hh << 1) >> 21, ul = (lh << 1) >> 21;
    // lo's mantissa with its top bit at bit 63, shifted right by r = gap - 53
    const uint32_t l1 = __funnelshift_l(ll, (lh & 0xFFFFFu) | 0x100000u, 11), l0 = ll << 11;
    const uint32_t r = uh - ul - 53u;
    const uint32_t t1 = __funnelshift_rc(l1, 0u, r);
    const uint32_t t0 = r < 32u ? __funnelshift_r(l0, l1, r) : __funnelshift_rc(l1, 0u, r - 32u);
    const uint32_t mask = (uint32_t)((int)(hh ^ lh) >> 31);
    asm("add.cc.u32 %0, %4, %8;\n\t"
        "addc.cc.u32 %1, %5, 0;\n\t"
        "addc.cc.u32 %2, %6, %9;\n\t"
        "addc.u32 %3, %7, %9;"
        : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
        : "r"(t0 ^ mask), "r"(t1 ^ mask), "r"(hl), "r"((hh & 0xFFFFFu) | 0x100000u), "r"(half - mask), "r"(mask));
    eh = (int)uh;
    return is_fast(v);
}

// fixacc.cuh's exponent (v = +-W * 2^e) of a biased hi exponent
constexpr int kExpBias = 1139;

// split_fast's eh
__device__ __forceinline__ int hi_exp(double2 v) { return (int)(((uint32_t)__double2hiint(v.x) << 1) >> 21); }

// hi and lo both zero, of either sign (split_fast's W is 2^116 then)
__device__ __forceinline__ bool all_zero(double2 v)
{
    return ((((uint32_t)__double2hiint(v.x) | (uint32_t)__double2hiint(v.y)) << 1) | (uint32_t)__double2loint(v.x) |
            (uint32_t)__double2loint(v.y)) == 0u;
}

// 2^(sh - 1) for 0 < sh < 32, 0 for sh = 0
__device__ __forceinline__ uint32_t half_unit(int sh) { return __funnelshift_l(0x80000000u, 0u, sh); }

// W / 2^sh rounded to nearest, 0 <= sh < 128
__device__ __forceinline__ void shr_round(const uint32_t w[4], int sh, uint32_t y[4])
{
    uint32_t t[4];
    fx::shr128(w, sh > 0 ? sh - 1 : 0, t);
    const uint32_t one = sh > 0 ? 1u : 0u;
    asm("add.cc.u32 %0, %0, %4;\n\t"
        "addc.cc.u32 %1, %1, 0;\n\t"
        "addc.cc.u32 %2, %2, 0;\n\t"
        "addc.u32 %3, %3, 0;"
        : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3])
        : "r"(one));
    y[0] = __funnelshift_r(t[0], t[1], one);
    y[1] = __funnelshift_r(t[1], t[2], one);
    y[2] = __funnelshift_r(t[2], t[3], one);
    y[3] = t[3] >> one;
}

// W >> sh for 0 <= sh < 32
__device__ __forceinline__ void shr_short(uint32_t w[4], int sh)
{
    w[0] = __funnelshift_r(w[0], w[1], sh);
    w[1] = __funnelshift_r(w[1], w[2], sh);
    w[2] = __funnelshift_r(w[2], w[3], sh);
    w[3] >>= sh & 31;
}

// Limbs 4u..4u+3 (one word) as two fp16 pairs; sgn: the sign in bit 31, the
// bits of its top byte below it zero.
__device__ __forceinline__ uint32_t limbs_lo(uint32_t word, uint32_t sgn) { return __byte_perm(word, sgn, 0x7170); }
__device__ __forceinline__ uint32_t limbs_hi(uint32_t word, uint32_t sgn) { return __byte_perm(word, sgn, 0x7372); }

// D += A * B, 16 x 8 x 16, fp16 operands and FP32 sums
__device__ __forceinline__ void mma16816(float d[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// 16 bytes from global to shared memory, in the thread's open group of copies
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// Four 8 x 8 fp16 tiles transposed: lane l gives the address of row l % 8 of
// tile l / 8 (16 bytes) and receives entries (2t, g), (2t + 1, g) of each tile.
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t r[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}

// 256-bit two's complement helpers (four 64-bit words, least significant first)
__device__ __forceinline__ void add256(uint64_t a[4], const uint64_t b[4])
{
    asm("add.cc.u64 %0, %0, %4;\n\t"
        "addc.cc.u64 %1, %1, %5;\n\t"
        "addc.cc.u64 %2, %2, %6;\n\t"
        "addc.u64 %3, %3, %7;"
        : "+l"(a[0]), "+l"(a[1]), "+l"(a[2]), "+l"(a[3])
        : "l"(b[0]), "l"(b[1]), "l"(b[2]), "l"(b[3]));
}
// += x * 2^s, 0 <= s < 256
__device__ __forceinline__ void add_at(uint64_t W[4], int64_t x, int s)
{
    const uint64_t ext = x < 0 ? ~0ull : 0ull;
    const int b = s & 63, q = s >> 6;
    const uint64_t lo = (uint64_t)x << b, hi = b ? (((uint64_t)x >> (64 - b)) | (ext << b)) : ext;
    uint64_t v[4];
    v[0] = q == 0 ? lo : 0ull;
    v[1] = q == 0 ? hi : (q == 1 ? lo : 0ull);
    v[2] = q == 0 ? ext : (q == 1 ? hi : (q == 2 ? lo : 0ull));
    v[3] = q <= 1 ? ext : (q == 2 ? hi : lo);
    add256(W, v);
}
// sum over the groups of `span` neighbouring lanes (a power of two), in all of them
__device__ __forceinline__ void lane_sum256(uint64_t W[4], int span)
{
    for (int off = 1; off < span; off <<= 1) {
        uint64_t o[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) o[t] = __shfl_xor_sync(0xffffffffu, (unsigned long long)W[t], off);
        add256(W, o);
    }
}

}  // namespace lmb
