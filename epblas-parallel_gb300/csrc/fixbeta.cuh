// beta C in the fixed-point update (fixround.cuh) of the CRT reconstruction and
// the grouped limb tiles. __host__ __device__: the host build is unit-tested.
#pragma once
#include "fixround.cuh"

namespace mw {

// A double-double as +-W * 2^e with W < 2^128, to 2^-127 of it as xword.cuh's
// from_dd (hi's mantissa 74 bits up, lo's in its place below).
struct ImageC {
    uint32_t w[4];
    int e;
    uint32_t neg, zero;
};

// The image of hi + lo. False for what needs the general path: hi zero with lo not
// finite, hi non-finite or below 2^-895, lo non-finite or less than 53 binades below
// hi. A zero or subnormal lo needs no test: its biased exponent 0 shifts all of it
// away (a subnormal one is below 2^-127 of hi).
XW_HD bool image_c(double hi, double lo, ImageC &c)
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
    const uint32_t t[4] = {xw::fshr(b0, b1, (int)s) ^ m, xw::fshr(b1, b2, (int)s) ^ m, (b2 >> s) ^ m, m};
    c.w[0] = m & 1u;
    c.w[1] = 0u;
    c.w[2] = hl << 10;
    c.w[3] = xw::fshl(hl, mh, 10);
    xw::add4(c.w, t);
    c.e = (int)uh - 1149;
    c.neg = hh >> 31;
    c.zero = ((hh << 1) | hl) == 0u;
    return c.zero ? ul != 0x7FFu : (uh - 128u) < 0x77Fu && (int)r >= 0;
}

// a += (neg ? -1 : 1) * beta part b (which may be zero; one: b is one) times c
XW_HD void add_image(fxr::Fix &a, const ImageC &c, const xw::XW &b, bool one, uint32_t neg)
{
    if (c.zero) return;
    uint32_t q[5];
    int e = c.e;
    if (one) {
        // a word below C's bits: a sum in this frame keeps its other term to 2^-158 of C
        q[0] = 0u; q[1] = c.w[0]; q[2] = c.w[1]; q[3] = c.w[2]; q[4] = c.w[3];
        e -= 32;
    } else {
        // (W has its top bit at 126 or 127, so the columns the product drops stay below 2^-123 of it)
        fxr::mul44(c.w, b.w, q);
        e += b.e + 96;
        neg ^= b.neg;
    }
    fxr::add_term(a, q, e, neg ^ c.neg);
}

// The same for the double-double hi + lo; false where that needs the general path
// (a is unchanged then).
XW_HD bool add_beta_c(fxr::Fix &a, double hi, double lo, const xw::XW &b, bool one, uint32_t neg)
{
    ImageC c;
    if (!image_c(hi, lo, c)) return false;
    add_image(a, c, b, one, neg);
    return true;
}

#ifdef __CUDACC__
__device__ __forceinline__ bool add_beta_c(fxr::Fix &a, double2 c, const xw::XW &b, bool one, uint32_t neg)
{
    return add_beta_c(a, c.x, c.y, b, one, neg);
}
#endif

}  // namespace mw
