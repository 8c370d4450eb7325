// Host-side harness for epblas-parallel_gb300/csrc/fixround.cuh, compiled with
// g++ by tests/test_fixround.py.
#include "../epblas-parallel_gb300/csrc/fixround.cuh"

extern "C" {

void fr_mul54(const uint32_t *t, const uint32_t *a, uint32_t *p) { fxr::mul54(t, a, p); }
void fr_mul44(const uint32_t *a, const uint32_t *b, uint32_t *p) { fxr::mul44(a, b, p); }

// (a.w, a.e, a.neg) += (q, eq, negq); w, e and neg are updated
void fr_add(uint32_t *w, int *e, uint32_t *neg, const uint32_t *q, int eq, uint32_t negq)
{
    fxr::Fix a;
    for (int t = 0; t < 6; ++t) a.w[t] = w[t];
    a.e = *e;
    a.neg = *neg;
    fxr::add(a, q, eq, negq);
    for (int t = 0; t < 6; ++t) w[t] = a.w[t];
    *e = a.e;
    *neg = a.neg;
}

void fr_to_dd(const uint32_t *w, int e, uint32_t neg, double *hi, double *lo)
{
    fxr::Fix a;
    for (int t = 0; t < 6; ++t) a.w[t] = w[t];
    a.e = e;
    a.neg = neg;
    fxr::to_dd(a, *hi, *lo);
}

}
