// Fixed-point update and rounding of the CRT reconstruction: products and sums
// as integers of up to six 32-bit words with one binary exponent, normalised
// only once, when the result is rounded to double-double.
//
// The extended-float form (xword.cuh) normalises after every step, with word
// selects and branches each time: about 730 instructions per output for the
// fraction, alpha M, beta C, the sum and the rounding. Here the 160-bit fraction
// times the 128-bit alpha M keeps its top 160 bits whatever its leading zeros
// (its own error is about 2^-148 of a unit), beta C's 256 bits keep 160, and the
// sum is formed in the coarser of the two frames: about 240 instructions.
//
// __host__ __device__: the host build is unit-tested.
#pragma once
#include "xword.cuh"

namespace fxr {

// value = (neg ? -1 : 1) * W * 2^e, W in six words (the top one is headroom)
struct Fix {
    uint32_t w[6];
    int e;
    uint32_t neg;
};

// w := m ? -w : w over N words (m all ones or zero)
template <int N>
XW_HD void cond_neg(uint32_t *w, uint32_t m)
{
    uint32_t c = m & 1u;
    for (int t = 0; t < N; ++t) {
        const uint64_t v = (uint64_t)(w[t] ^ m) + c;
        w[t] = (uint32_t)v;
        c = (uint32_t)(v >> 32);
    }
}

// a += (m ? -b : b) over six words, two's complement
XW_HD void add6(uint32_t a[6], const uint32_t b[6], uint32_t m)
{
#ifdef __CUDA_ARCH__
    uint32_t t;
    asm("add.cc.u32 %6, %13, 0xFFFFFFFF;\n\t"   // the carry in: m & 1
        "addc.cc.u32 %0, %0, %7;\n\t"
        "addc.cc.u32 %1, %1, %8;\n\t"
        "addc.cc.u32 %2, %2, %9;\n\t"
        "addc.cc.u32 %3, %3, %10;\n\t"
        "addc.cc.u32 %4, %4, %11;\n\t"
        "addc.u32 %5, %5, %12;"
        : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "=&r"(t)
        : "r"(b[0] ^ m), "r"(b[1] ^ m), "r"(b[2] ^ m), "r"(b[3] ^ m), "r"(b[4] ^ m), "r"(b[5] ^ m), "r"(m & 1u));
#else
    uint64_t c = m & 1u;
    for (int t = 0; t < 6; ++t) {
        c += (uint64_t)a[t] + (b[t] ^ m);
        a[t] = (uint32_t)c;
        c >>= 32;
    }
#endif
}

// Words 4..8 of the 288-bit product t * a (the partial products of columns 0..2
// are dropped: the result is at most 4 units low).
XW_HD void mul54(const uint32_t t[5], const uint32_t a[4], uint32_t p[5])
{
#ifdef __CUDA_ARCH__
    uint32_t c3;
    asm("mul.lo.u32 %0, %6, %14;\n\t"
        "mul.lo.u32 %1, %7, %14;\n\t"
        "mul.lo.u32 %2, %8, %14;\n\t"
        "mul.lo.u32 %3, %9, %14;\n\t"
        "mul.lo.u32 %4, %10, %14;\n\t"
        "mad.hi.cc.u32 %1, %6, %14, %1;\n\t"
        "madc.hi.cc.u32 %2, %7, %14, %2;\n\t"
        "madc.hi.cc.u32 %3, %8, %14, %3;\n\t"
        "madc.hi.cc.u32 %4, %9, %14, %4;\n\t"
        "madc.hi.u32 %5, %10, %14, 0;\n\t"
        // a2: t1 .. t4 at columns 3 .. 6
        "mad.lo.cc.u32 %0, %7, %13, %0;\n\t"
        "madc.lo.cc.u32 %1, %8, %13, %1;\n\t"
        "madc.lo.cc.u32 %2, %9, %13, %2;\n\t"
        "madc.lo.cc.u32 %3, %10, %13, %3;\n\t"
        "addc.cc.u32 %4, %4, 0;\n\t"
        "addc.u32 %5, %5, 0;\n\t"
        "mad.hi.cc.u32 %1, %7, %13, %1;\n\t"
        "madc.hi.cc.u32 %2, %8, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, %9, %13, %3;\n\t"
        "madc.hi.cc.u32 %4, %10, %13, %4;\n\t"
        "addc.u32 %5, %5, 0;\n\t"
        // a1: t2 .. t4 at columns 3 .. 5
        "mad.lo.cc.u32 %0, %8, %12, %0;\n\t"
        "madc.lo.cc.u32 %1, %9, %12, %1;\n\t"
        "madc.lo.cc.u32 %2, %10, %12, %2;\n\t"
        "addc.cc.u32 %3, %3, 0;\n\t"
        "addc.cc.u32 %4, %4, 0;\n\t"
        "addc.u32 %5, %5, 0;\n\t"
        "mad.hi.cc.u32 %1, %8, %12, %1;\n\t"
        "madc.hi.cc.u32 %2, %9, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, %10, %12, %3;\n\t"
        "addc.cc.u32 %4, %4, 0;\n\t"
        "addc.u32 %5, %5, 0;\n\t"
        // a0: t3, t4 at columns 3, 4
        "mad.lo.cc.u32 %0, %9, %11, %0;\n\t"
        "madc.lo.cc.u32 %1, %10, %11, %1;\n\t"
        "addc.cc.u32 %2, %2, 0;\n\t"
        "addc.cc.u32 %3, %3, 0;\n\t"
        "addc.cc.u32 %4, %4, 0;\n\t"
        "addc.u32 %5, %5, 0;\n\t"
        "mad.hi.cc.u32 %1, %9, %11, %1;\n\t"
        "madc.hi.cc.u32 %2, %10, %11, %2;\n\t"
        "addc.cc.u32 %3, %3, 0;\n\t"
        "addc.cc.u32 %4, %4, 0;\n\t"
        "addc.u32 %5, %5, 0;"
        : "=&r"(c3), "=&r"(p[0]), "=&r"(p[1]), "=&r"(p[2]), "=&r"(p[3]), "=&r"(p[4])
        : "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]));
#else
    uint64_t col[10] = {};   // 32-bit digits with room for the carries
    for (int i = 0; i < 5; ++i)
        for (int j = 0; j < 4; ++j)
            if (i + j >= 3) {
                const uint64_t v = (uint64_t)t[i] * a[j];
                col[i + j] += (uint32_t)v;
                col[i + j + 1] += v >> 32;
            }
    uint64_t c = 0;
    for (int q = 3; q < 9; ++q) {
        c += col[q];
        if (q >= 4) p[q - 4] = (uint32_t)c;
        c >>= 32;
    }
#endif
}

// Words 3..7 of the 256-bit product a * b (the partial products of columns 0..2
// are dropped: less than 2^130, 2^34 units).
XW_HD void mul44(const uint32_t a[4], const uint32_t b[4], uint32_t p[5])
{
#ifdef __CUDA_ARCH__
    asm("mul.lo.u32 %0, %5, %12;\n\t"
        "mul.lo.u32 %1, %6, %12;\n\t"
        "mul.lo.u32 %2, %7, %12;\n\t"
        "mul.lo.u32 %3, %8, %12;\n\t"
        "mad.hi.cc.u32 %1, %5, %12, %1;\n\t"
        "madc.hi.cc.u32 %2, %6, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, %7, %12, %3;\n\t"
        "madc.hi.u32 %4, %8, %12, 0;\n\t"
        "mad.lo.cc.u32 %0, %6, %11, %0;\n\t"
        "madc.lo.cc.u32 %1, %7, %11, %1;\n\t"
        "madc.lo.cc.u32 %2, %8, %11, %2;\n\t"
        "addc.cc.u32 %3, %3, 0;\n\t"
        "addc.u32 %4, %4, 0;\n\t"
        "mad.hi.cc.u32 %1, %6, %11, %1;\n\t"
        "madc.hi.cc.u32 %2, %7, %11, %2;\n\t"
        "madc.hi.cc.u32 %3, %8, %11, %3;\n\t"
        "addc.u32 %4, %4, 0;\n\t"
        "mad.lo.cc.u32 %0, %7, %10, %0;\n\t"
        "madc.lo.cc.u32 %1, %8, %10, %1;\n\t"
        "addc.cc.u32 %2, %2, 0;\n\t"
        "addc.cc.u32 %3, %3, 0;\n\t"
        "addc.u32 %4, %4, 0;\n\t"
        "mad.hi.cc.u32 %1, %7, %10, %1;\n\t"
        "madc.hi.cc.u32 %2, %8, %10, %2;\n\t"
        "addc.cc.u32 %3, %3, 0;\n\t"
        "addc.u32 %4, %4, 0;\n\t"
        "mad.lo.cc.u32 %0, %8, %9, %0;\n\t"
        "addc.cc.u32 %1, %1, 0;\n\t"
        "addc.cc.u32 %2, %2, 0;\n\t"
        "addc.cc.u32 %3, %3, 0;\n\t"
        "addc.u32 %4, %4, 0;\n\t"
        "mad.hi.cc.u32 %1, %8, %9, %1;\n\t"
        "addc.cc.u32 %2, %2, 0;\n\t"
        "addc.cc.u32 %3, %3, 0;\n\t"
        "addc.u32 %4, %4, 0;"
        : "=&r"(p[0]), "=&r"(p[1]), "=&r"(p[2]), "=&r"(p[3]), "=&r"(p[4])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]));
#else
    uint64_t col[9] = {};
    for (int i = 0; i < 4; ++i)
        for (int j = 0; j < 4; ++j)
            if (i + j >= 3) {
                const uint64_t v = (uint64_t)a[i] * b[j];
                col[i + j] += (uint32_t)v;
                col[i + j + 1] += v >> 32;
            }
    uint64_t c = 0;
    for (int q = 3; q < 8; ++q) {
        c += col[q];
        p[q - 3] = (uint32_t)c;
        c >>= 32;
    }
#endif
}

// w >> d over six words, 0 <= d < 192
XW_HD void shr6(uint32_t w[6], int d)
{
    if (d & 32) {
        for (int t = 0; t < 5; ++t) w[t] = w[t + 1];
        w[5] = 0u;
    }
    if (d & 64) {
        for (int t = 0; t < 4; ++t) w[t] = w[t + 2];
        w[4] = w[5] = 0u;
    }
    if (d & 128) {
        w[0] = w[4];
        w[1] = w[5];
        w[2] = w[3] = w[4] = w[5] = 0u;
    }
    const int r = d & 31;
    for (int t = 0; t < 5; ++t) w[t] = xw::fshr(w[t], w[t + 1], r);
    w[5] = w[5] >> r;
}

XW_HD bool is_zero(const Fix &a) { return (a.w[0] | a.w[1] | a.w[2] | a.w[3] | a.w[4] | a.w[5]) == 0u; }

// a += (neg ? -q : q) * 2^eq, cut below the unit of the coarser operand
// (a zero a takes q's frame). q's frame counts even where q is zero: sums
// whose terms can be zero use add_term.
XW_HD void add(Fix &a, const uint32_t q[5], int eq, uint32_t neg)
{
    const int d = is_zero(a) ? -192 : a.e - eq;
    // the finer operand is shifted into the frame of the coarser one
    const bool sq = d >= 0;
    uint32_t s[6], k[6];
    for (int t = 0; t < 5; ++t) {
        s[t] = sq ? q[t] : a.w[t];
        k[t] = sq ? a.w[t] : q[t];
    }
    s[5] = sq ? 0u : a.w[5];
    k[5] = sq ? a.w[5] : 0u;
    const uint32_t nk = sq ? a.neg : neg;
    const int ad = sq ? d : -d;
    shr6(s, ad < 191 ? ad : 191);
    add6(k, s, 0u - (a.neg ^ neg));
    const uint32_t m = 0u - (k[5] >> 31);   // the subtraction went below zero
    cond_neg<6>(k, m);
    for (int t = 0; t < 6; ++t) a.w[t] = k[t];
    a.e = sq ? a.e : eq;
    a.neg = nk ^ (m & 1u);
}

// add for a term that may be zero: a zero has no frame, so a stays as it is
// (beta = (0, b) on a complex C: a zero product of exponent -31 would cut the
// sum, held to 2^-139, at 2^-31).
XW_HD void add_term(Fix &a, const uint32_t q[5], int eq, uint32_t neg)
{
    if ((q[0] | q[1] | q[2] | q[3] | q[4]) != 0u) add(a, q, eq, neg);
}

// Round to double-double as xword.cuh's to_dd: hi the top 53 bits, rounded half
// up, lo the rest rounded to 53 bits.
XW_HD void to_dd(const Fix &a, double &out_hi, double &out_lo)
{
    uint32_t n4 = a.w[4], n3 = a.w[3], n2 = a.w[2], n1 = a.w[1], n0 = a.w[0];
    int e = a.e + 32;
    if (a.w[5] != 0u) {
        n0 = n1; n1 = n2; n2 = n3; n3 = n4; n4 = a.w[5];
        e += 32;
    }
    for (int t = 0; t < 4 && n4 == 0u; ++t) {
        n4 = n3; n3 = n2; n2 = n1; n1 = n0; n0 = 0u;
        e -= 32;
    }
    if (n4 == 0u) {
        out_hi = out_lo = 0.0;
        return;
    }
    const int z = xw::clz32(n4);
    xw::XW v;
    v.w[3] = xw::fshl(n3, n4, z);
    v.w[2] = xw::fshl(n2, n3, z);
    v.w[1] = xw::fshl(n1, n2, z);
    v.w[0] = xw::fshl(n0, n1, z);
    v.e = e - z;
    v.neg = a.neg;
    const int ex = v.e + 127 + 1023;   // biased exponent of hi
    if ((uint32_t)(ex - 200) > 1840u) {   // near either end of the range
        xw::to_dd(v, out_hi, out_lo);
        return;
    }
    // hi: a carry out of the mantissa raises the exponent field by itself
    const uint32_t up = (v.w[2] >> 10) & 1u;
    const uint64_t hb = (((uint64_t)(((uint32_t)(ex - 1) << 20) + (v.w[3] >> 11)) << 32) |
                         xw::fshl(v.w[2], v.w[3], 21)) + up;
    // the rest, less 2^75 where hi went up: its low 75 bits as a signed integer
    uint32_t r[3] = {v.w[0], v.w[1], (uint32_t)((int32_t)(v.w[2] << 21) >> 21)};
    const uint32_t m = 0u - (r[2] >> 31);
    cond_neg<3>(r, m);
    int le = v.e + 95;   // exponent of bit 31 of r[2]
    for (int t = 0; t < 2 && r[2] == 0u; ++t) {
        r[2] = r[1]; r[1] = r[0]; r[0] = 0u;
        le -= 32;
    }
    const int lz = xw::clz32(r[2]);
    uint64_t lb = 0;
    if (r[2] != 0u) {
        const uint32_t l3 = xw::fshl(r[1], r[2], lz), l2 = xw::fshl(r[0], r[1], lz);
        lb = (((uint64_t)(((uint32_t)(le - lz + 1022) << 20) + (l3 >> 11)) << 32) | xw::fshl(l2, l3, 21)) +
             ((l2 >> 10) & 1u);
        lb |= (uint64_t)(a.neg ^ (m & 1u)) << 63;
    }
    out_hi = xw::dbl_make((uint32_t)(hb >> 32) | (a.neg << 31), (uint32_t)hb);
    out_lo = xw::dbl_make((uint32_t)(lb >> 32), (uint32_t)lb);
}

}  // namespace fxr
