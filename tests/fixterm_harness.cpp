// Host-side harness for the sums of epblas-parallel_gb300/csrc/fixround.cuh
// whose terms may be zero, compiled with g++ by tests/test_fixterm.py.
#include "../epblas-parallel_gb300/csrc/fixround.cuh"

extern "C" void fr_add_term(uint32_t *w, int *e, uint32_t *neg, const uint32_t *q, int eq, uint32_t negq)
{
    fxr::Fix a;
    for (int t = 0; t < 6; ++t) a.w[t] = w[t];
    a.e = *e;
    a.neg = *neg;
    fxr::add_term(a, q, eq, negq);
    for (int t = 0; t < 6; ++t) w[t] = a.w[t];
    *e = a.e;
    *neg = a.neg;
}
