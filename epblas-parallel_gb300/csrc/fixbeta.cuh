// beta C in the fixed-point update (fixround.cuh) of the CRT reconstruction and
// the grouped limb tiles. __host__ __device__: the host build is unit-tested.
#pragma once
#include "fixround.cuh"

namespace mw {

// The double-double hi + lo as +-W * 2^e with W < 2^128, to 2^-127 of it as
// xword.cuh's from_dd (hi's mantissa 74 bits up, lo's in its place below). False
// for what needs the general path: hi zero, non-finite or below 2^-895, lo
// non-finite or less than 53 binades below hi. A zero or subnormal lo needs no
// test: its biased exponent 0 shifts all of it away (a subnormal one is below
// 2^-127 of hi).
XW_HD bool split_c(double hi, double lo, uint32_t w[4], int &e)
{
    const uint32_t hl = xw::dbl_lo(hi), hh = xw::dbl_hi(hi), ll = xw::dbl_lo(lo), lh = xw::dbl_hi(lo);
    const uint32_t uh = (hh << 1) >> 21, ul = (lh << 1) >> 21;
    const uint32_t mh = (hh & 0xFFFFFu) | 0x100000u, ml = (lh & 0xFFFFFu) | 0x100000u;
    // lo's mantissa with its top bit at bit 73, shifted right by r = gap - 53
    const uint32_t r = uh - ul - 53u, q = r >> 5, s = r & 31u;
    const uint32_t a0 = ll << 21, a1 = xw::fshl(ll, ml, 21), a2 = ml >> 11;
    const uint32_t b0 = q == 0u ? a0 : (q == 1u ? a1 : (q == 2u ? a2 : 0u));
    const uint32_t b1 = q == 0u ? a1 : (q == 1u ? a2 : 0u), b2 = q == 0u ? a2 : 0u;
    const uint32_t m = 0u - ((hh ^ lh) >> 31);
    uint32_t t[4] = {xw::fshr(b0, b1, (int)s) ^ m, xw::fshr(b1, b2, (int)s) ^ m, (b2 >> s) ^ m, m};
    w[0] = m & 1u;
    w[1] = 0u;
    w[2] = hl << 10;
    w[3] = xw::fshl(hl, mh, 10);
    xw::add4(w, t);
    e = (int)uh - 1149;
    return (uh - 128u) < 0x77Fu && (int)r >= 0;
}

// a += (neg ? -1 : 1) * beta part b (which may be zero; one: b is one) times the
// double-double hi + lo; false where that needs the general path (a is unchanged
// then).
XW_HD bool add_beta_c(fxr::Fix &a, double hi, double lo, const xw::XW &b, bool one, uint32_t neg)
{
    const uint32_t hh = xw::dbl_hi(hi);
    if (((hh << 1) | xw::dbl_lo(hi)) == 0u)   // zero: nothing to add, unless lo is not finite
        return ((xw::dbl_hi(lo) >> 20) & 0x7FFu) != 0x7FFu;
    uint32_t w[4], q[5];
    int e;
    if (!split_c(hi, lo, w, e)) return false;
    if (one) {
        // a word below C's bits: a sum in this frame keeps its other term to 2^-158 of C
        q[0] = 0u; q[1] = w[0]; q[2] = w[1]; q[3] = w[2]; q[4] = w[3];
        e -= 32;
    } else {
        // (W has its top bit at 126 or 127, so the columns the product drops stay below 2^-123 of it)
        fxr::mul44(w, b.w, q);
        e += b.e + 96;
        neg ^= b.neg;
    }
    fxr::add_term(a, q, e, neg ^ (hh >> 31));
    return true;
}

#ifdef __CUDACC__
__device__ __forceinline__ bool add_beta_c(fxr::Fix &a, double2 c, const xw::XW &b, bool one, uint32_t neg)
{
    return add_beta_c(a, c.x, c.y, b, one, neg);
}
#endif

}  // namespace mw
