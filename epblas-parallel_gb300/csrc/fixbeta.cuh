// beta C in the fixed-point update (fixround.cuh) of the CRT reconstruction and
// the grouped limb tiles.
#pragma once
#include "fixround.cuh"
#include "limbmma.cuh"

namespace mw {

// a += (neg ? -1 : 1) * beta part b (which may be zero; kind 1: one) times the
// double-double c; false where c needs the general path (a is unchanged then).
__device__ __forceinline__ bool add_beta_c(fxr::Fix &a, double2 c, const xw::XW &b, bool one, uint32_t neg)
{
    const uint32_t hh = (uint32_t)__double2hiint(c.x);
    if (((hh << 1) | (uint32_t)__double2loint(c.x)) == 0u)   // zero: nothing to add, unless lo is not finite
        return ((__double2hiint(c.y) >> 20) & 0x7FF) != 0x7FF;
    uint32_t w[4], q[5];
    int eh;
    if (!lmb::split_fast(c, w, eh)) return false;
    int e = eh - lmb::kExpBias;
    if (one) {
        q[0] = w[0]; q[1] = w[1]; q[2] = w[2]; q[3] = w[3]; q[4] = 0u;
    } else {
        // W < 2^118 up to the top of its words first, so that the columns the
        // product drops stay below 2^-123 of it
        w[3] = __funnelshift_l(w[2], w[3], 10);
        w[2] = __funnelshift_l(w[1], w[2], 10);
        w[1] = __funnelshift_l(w[0], w[1], 10);
        w[0] <<= 10;
        fxr::mul44(w, b.w, q);
        e += b.e + 86;
        neg ^= b.neg;
    }
    fxr::add_term(a, q, e, neg ^ (hh >> 31));
    return true;
}

}  // namespace mw
