// Host-side harness for epblas-parallel_gb300/csrc/fixbeta.cuh, compiled with
// g++ by tests/test_fixbeta.py.
#include "../epblas-parallel_gb300/csrc/fixbeta.cuh"

// (w, e, neg) += (bhi + blo) * (hi + lo); 0 where that needs the general path
extern "C" int fb_add(uint32_t *w, int *e, uint32_t *neg, double hi, double lo, double bhi, double blo, int one)
{
    fxr::Fix a;
    for (int t = 0; t < 6; ++t) a.w[t] = w[t];
    a.e = *e;
    a.neg = *neg;
    const bool ok = mw::add_beta_c(a, hi, lo, xw::from_dd(bhi, blo), one != 0, 0u);
    for (int t = 0; t < 6; ++t) w[t] = a.w[t];
    *e = a.e;
    *neg = a.neg;
    return ok ? 1 : 0;
}
