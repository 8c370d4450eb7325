// Fixed-point double-double GEMM on the integer pipes ("fixed" engine).
//
// The FP64 pipe of this part issues ~1.6 lane-operations per clock per SM,
// the integer multiply-add pipe ~40x more. This engine therefore forms the
// double-double products in integers:
//
//  * op(A)'s rows and op(B)'s columns are scaled by powers of two from their
//    exponent bounds (as the tensor-core engine does): a(i,p) * 2^(S - ea_i)
//    is rounded to an integer below 2^116 (S = 115), the exact image of the
//    106-bit hi + lo; likewise b(p,j) * 2^(S - eb_j).
//  * Each integer is held as five signed ("balanced") 24-bit digits,
//    d_0 + d_1 2^24 + ... + d_4 2^96 with |d_t| <= 2^23, converted on the fly
//    when the tile is staged in shared memory.
//  * A multiply-add is 15 IMAD.WIDE: the digit products d_s e_t with
//    s + t >= 4, accumulated exactly in five signed 64-bit column sums (one per
//    weight 2^(24w), w = 4..8). The 10 dropped products with s + t <= 3 are
//    below 2^-110 of |a|max |b|max per term.
//  * The epilogue assembles the column sums into one 256-bit integer, scales
//    it back by 2^(ea_i + eb_j - 2S + 96) and computes alpha*X + beta*C in
//    128-bit extended floats with a single rounding to double-double.
//
// Column sums stay below 2^63 for up to 16384 multiply-adds (5 products of
// at most 2^46 per step), so longer K runs in chunks of 16384 with beta = 1
// for all but the first. Rows or columns with a non-finite entry give NaN
// outputs, as the reference's double-double products of an infinity do (the
// TwoProduct error term is inf - inf). Accuracy is normwise, like the tensor-
// core engine's: entries far below their row/column maximum keep fewer bits.
#include <cmath>

#include "dd.cuh"
#include "fixacc.cuh"
#include "fixgemm.cuh"
#include "gemm.h"
#include "runtime.h"
#include "xfloat.cuh"

namespace mw {

namespace {

using xfp::XF;
using namespace fxg;

constexpr int FX_BM = 64, FX_BN = 64, FX_BK = 8;
constexpr int FX_THREADS = 256;      // 16 x 16 threads, 4 x 4 outputs each
constexpr int64_t FX_MAX_K = 16384;  // per launch (column-sum headroom)

template <bool TA, bool TB>
__global__ void __launch_bounds__(FX_THREADS, 1)
    k_gemm_fixed(int64_t m, int64_t n, int64_t k, const double2 *__restrict__ A, int64_t lda,
                 const double2 *__restrict__ B, int64_t ldb, const int *__restrict__ ea, const int *__restrict__ eb,
                 dd::real alpha, int alpha_one, dd::real beta, int beta_kind, double2 *C, int64_t ldc, int uplo)
{
    __shared__ __align__(16) int sA[FX_BK][5][FX_BM];   // digit planes, rows contiguous
    __shared__ __align__(16) int sB[FX_BK][5][FX_BN];
    __shared__ int s_sa[FX_BM], s_sb[FX_BN];

    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;   // rows 4tx..4tx+3, columns 4ty..4ty+3
    const int64_t i0 = (int64_t)blockIdx.x * FX_BM, j0 = (int64_t)blockIdx.y * FX_BN;
    if ((uplo == 1 && i0 > j0 + FX_BN - 1) || (uplo == 2 && i0 + FX_BM - 1 < j0)) return;

    if (tid < FX_BM) {
        const int64_t i = i0 + tid;
        const int e = (i < m) ? ea[i] : kNoExp;
        s_sa[tid] = (e <= kNoExp / 2) ? -100000 : FX_S - e;
    } else if (tid < FX_BM + FX_BN) {
        const int64_t j = j0 + (tid - FX_BM);
        const int e = (j < n) ? eb[j] : kNoExp;
        s_sb[tid - FX_BM] = (e <= kNoExp / 2) ? -100000 : FX_S - e;
    }
    __syncthreads();

    long long acc[4][4][5];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int w = 0; w < 5; ++w) acc[a][b][w] = 0;

    // each thread stages 2 elements of the A tile and 2 of the B tile per slab
    double2 ra[2], rb[2];
    auto load = [&](int64_t kk) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int idx = tid + u * FX_THREADS;
            int r, p;
            if (!TA) { r = idx % FX_BM; p = idx / FX_BM; }
            else     { p = idx % FX_BK; r = idx / FX_BK; }
            const int64_t gi = i0 + r, gp = kk + p;
            ra[u] = (gi < m && gp < k) ? (TA ? A[gp + gi * lda] : A[gi + gp * lda]) : make_double2(0.0, 0.0);
            int c;
            if (!TB) { p = idx % FX_BK; c = idx / FX_BK; }
            else     { c = idx % FX_BN; p = idx / FX_BN; }
            const int64_t gj = j0 + c, gq = kk + p;
            rb[u] = (gj < n && gq < k) ? (TB ? B[gj + gq * ldb] : B[gq + gj * ldb]) : make_double2(0.0, 0.0);
        }
    };
    auto stage = [&]() {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int idx = tid + u * FX_THREADS;
            int r, p, d[5];
            if (!TA) { r = idx % FX_BM; p = idx / FX_BM; }
            else     { p = idx % FX_BK; r = idx / FX_BK; }
            dd_digits(ra[u], s_sa[r], d);
#pragma unroll
            for (int t = 0; t < 5; ++t) sA[p][t][r] = d[t];
            int c;
            if (!TB) { p = idx % FX_BK; c = idx / FX_BK; }
            else     { c = idx % FX_BN; p = idx / FX_BN; }
            dd_digits(rb[u], s_sb[c], d);
#pragma unroll
            for (int t = 0; t < 5; ++t) sB[p][t][c] = d[t];
        }
    };

    load(0);
    for (int64_t kk = 0; kk < k; kk += FX_BK) {
        stage();
        __syncthreads();
        if (kk + FX_BK < k) load(kk + FX_BK);   // next slab in flight during the products
#pragma unroll 2
        for (int p = 0; p < FX_BK; ++p) {
            int da[5][4], db[5][4];
#pragma unroll
            for (int t = 0; t < 5; ++t) {
                const int4 va = *reinterpret_cast<const int4 *>(&sA[p][t][4 * tx]);
                const int4 vb = *reinterpret_cast<const int4 *>(&sB[p][t][4 * ty]);
                da[t][0] = va.x; da[t][1] = va.y; da[t][2] = va.z; da[t][3] = va.w;
                db[t][0] = vb.x; db[t][1] = vb.y; db[t][2] = vb.z; db[t][3] = vb.w;
            }
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    long long *c = acc[a][b];
                    c[0] += (long long)da[0][a] * db[4][b] + (long long)da[1][a] * db[3][b] +
                            (long long)da[2][a] * db[2][b] + (long long)da[3][a] * db[1][b] +
                            (long long)da[4][a] * db[0][b];
                    c[1] += (long long)da[1][a] * db[4][b] + (long long)da[2][a] * db[3][b] +
                            (long long)da[3][a] * db[2][b] + (long long)da[4][a] * db[1][b];
                    c[2] += (long long)da[2][a] * db[4][b] + (long long)da[3][a] * db[3][b] +
                            (long long)da[4][a] * db[2][b];
                    c[3] += (long long)da[3][a] * db[4][b] + (long long)da[4][a] * db[3][b];
                    c[4] += (long long)da[4][a] * db[4][b];
                }
        }
        __syncthreads();
    }

    const XF xa = xfp::xf_from_dd(alpha.hi, alpha.lo), xb = xfp::xf_from_dd(beta.hi, beta.lo);
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const int64_t j = j0 + 4 * ty + b;
        if (j >= n) continue;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int64_t i = i0 + 4 * tx + a;
            if (i >= m) continue;
            if ((uplo == 1 && i > j) || (uplo == 2 && i < j)) continue;
            const int ei = ea[i], ej = eb[j];
            double2 *pc = C + i + j * ldc;
            if (ei >= 1024 || ej >= 1024) {   // a non-finite entry in row i of op(A) or column j of op(B)
                const double qnan = __longlong_as_double(0x7ff8000000000000ll);
                *pc = make_double2(qnan, qnan);
                continue;
            }
            XF v;
            if (ei <= kNoExp / 2 || ej <= kNoExp / 2) {
                v.zero = true; v.neg = false; v.m = 0; v.e = 0;
            } else {
                v = sums_to_xf(acc[a][b], ei, ej);
            }
            store_axpby(pc, v, xa, alpha_one != 0, xb, beta, beta_kind);
        }
    }
}

// Small products: tiles of T x T outputs (16 or 8), one output per thread
// (T = 8: four threads, every fourth k each), and K in chunks of 64 over
// grid.z, so that a product of a few thousand outputs spreads over the SMs.
// A block holds its whole chunk, so it finds the row and column exponent bounds
// itself: the elements are loaded once into registers, the bounds reduced in
// shared memory, then the digits staged there. One chunk: C is updated here
// (one launch, no scratch). Several: the chunks' sums go out as extended floats
// and k_fixed_small_fold adds them in order; each chunk has its own bounds,
// never above those of the whole rows, so nothing is lost against one scan.
//
// Bound: latency. 48 x 33 x 40 took 174 us as one 64 x 64 block behind two
// exponent scans, now 8;
// whole calls: 16^3 118 -> 27 us, 48 x 33 x 40 148 -> 27, 100^3 226 -> 46,
// 16 x 16 x 8000 10.0 ms -> 55 us, 256^3 422 -> 100 us.
constexpr int SM_KC = 64;

template <int T, bool TA, bool TB>
__global__ void __launch_bounds__(FX_THREADS)
    k_gemm_fixed_small(int64_t m, int64_t n, int64_t k, const double2 *__restrict__ A, int64_t lda,
                       const double2 *__restrict__ B, int64_t ldb, dd::real alpha, int alpha_one, dd::real beta,
                       int beta_kind, double2 *C, int64_t ldc, int uplo, fx::XFPod *part)
{
    constexpr int G = FX_THREADS / (T * T);          // threads per output
    constexpr int NU = T * SM_KC / FX_THREADS;       // elements per thread and operand
    constexpr int S = 5 * T + 1;                     // digits of one k: odd stride for transposed staging
    __shared__ __align__(8) int sA[SM_KC * S], sB[SM_KC * S];
    __shared__ int s_ea[T], s_eb[T];
    const int tid = threadIdx.x;
    const int64_t i0 = (int64_t)blockIdx.x * T, j0 = (int64_t)blockIdx.y * T, k0 = (int64_t)blockIdx.z * SM_KC;
    if ((uplo == 1 && i0 > j0 + T - 1) || (uplo == 2 && i0 + T - 1 < j0)) return;
    const int kc = (int)min((int64_t)SM_KC, k - k0);
    if (tid < T) s_ea[tid] = kNoExp;
    else if (tid < 2 * T) s_eb[tid - T] = kNoExp;

    double2 ra[NU], rb[NU];
    int ia[NU], ib[NU];   // row (column) of the tile and k of each element
#pragma unroll
    for (int u = 0; u < NU; ++u) {
        const int idx = tid + u * FX_THREADS;
        const int r = TA ? idx / SM_KC : idx % T, pa = TA ? idx % SM_KC : idx / T;
        const int c = TB ? idx % T : idx / SM_KC, pb = TB ? idx / T : idx % SM_KC;
        ia[u] = r | pa << 8;
        ib[u] = c | pb << 8;
        ra[u] = (i0 + r < m && pa < kc) ? (TA ? A[k0 + pa + (i0 + r) * lda] : A[i0 + r + (k0 + pa) * lda])
                                        : make_double2(0.0, 0.0);
        rb[u] = (j0 + c < n && pb < kc) ? (TB ? B[j0 + c + (k0 + pb) * ldb] : B[k0 + pb + (j0 + c) * ldb])
                                        : make_double2(0.0, 0.0);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < NU; ++u) {
        atomicMax(&s_ea[ia[u] & 255], exp_bound(ra[u].x));
        atomicMax(&s_eb[ib[u] & 255], exp_bound(rb[u].x));
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < NU; ++u) {
        int d[5];
        const int ea = s_ea[ia[u] & 255], eb = s_eb[ib[u] & 255];
        dd_digits(ra[u], ea <= kNoExp / 2 ? -100000 : FX_S - ea, d);
#pragma unroll
        for (int t = 0; t < 5; ++t) sA[(ia[u] >> 8) * S + t * T + (ia[u] & 255)] = d[t];
        dd_digits(rb[u], eb <= kNoExp / 2 ? -100000 : FX_S - eb, d);
#pragma unroll
        for (int t = 0; t < 5; ++t) sB[(ib[u] >> 8) * S + t * T + (ib[u] & 255)] = d[t];
    }
    __syncthreads();

    const int r = tid % T, c = (tid / T) % T, kg = tid / (T * T);
    long long acc[5] = {0, 0, 0, 0, 0};
#pragma unroll 4
    for (int p = kg; p < kc; p += G) {
        int da[5], db[5];
#pragma unroll
        for (int t = 0; t < 5; ++t) {
            da[t] = sA[p * S + t * T + r];
            db[t] = sB[p * S + t * T + c];
        }
        mac_digits(acc, da, db);
    }
    if (G > 1) {   // the output's shares, exact integers, into its first thread
        __syncthreads();
        long long *red = reinterpret_cast<long long *>(sA);
        if (kg > 0)
#pragma unroll
            for (int w = 0; w < 5; ++w) red[((kg - 1) * 5 + w) * (T * T) + tid % (T * T)] = acc[w];
        __syncthreads();
        if (kg > 0) return;
#pragma unroll
        for (int q = 0; q < G - 1; ++q)
#pragma unroll
            for (int w = 0; w < 5; ++w) acc[w] += red[(q * 5 + w) * (T * T) + tid];
    }
    const int64_t i = i0 + r, j = j0 + c;
    if (i >= m || j >= n || (uplo == 1 && i > j) || (uplo == 2 && i < j)) return;
    const int ei = s_ea[r], ej = s_eb[c];
    const bool bad = ei >= 1024 || ej >= 1024;   // a non-finite entry in row i of op(A) or column j of op(B)
    XF v;
    if (bad || ei <= kNoExp / 2 || ej <= kNoExp / 2) {
        v.zero = true; v.neg = false; v.m = 0; v.e = 0;
    } else {
        v = sums_to_xf(acc, ei, ej);
    }
    if (part) {
        part[blockIdx.z * (m * n) + i + j * m] = fx::to_pod(v, bad);
        return;
    }
    double2 *pc = C + i + j * ldc;
    if (bad) {
        const double qnan = __longlong_as_double(0x7ff8000000000000ll);
        *pc = make_double2(qnan, qnan);
        return;
    }
    store_axpby(pc, v, xfp::xf_from_dd(alpha.hi, alpha.lo), alpha_one != 0, xfp::xf_from_dd(beta.hi, beta.lo), beta,
                beta_kind);
}

// The chunks' sums of each output, eight lanes per output in a fixed order,
// then C := alpha * sum + beta * C.
__global__ void __launch_bounds__(256)
    k_fixed_small_fold(int64_t m, int64_t n, int chunks, const fx::XFPod *__restrict__ part, dd::real alpha,
                       int alpha_one, dd::real beta, int beta_kind, double2 *C, int64_t ldc, int uplo)
{
    const int sub = threadIdx.x & 7;
    const int64_t o = (int64_t)blockIdx.x * 32 + (threadIdx.x >> 3), i = o % m, j = o / m;
    const bool in = o < m * n && !(uplo == 1 && i > j) && !(uplo == 2 && i < j);
    XF s;
    s.zero = true; s.neg = false; s.m = 0; s.e = 0;
    int bad = 0;
    if (in) {
        for (int c = sub; c < chunks; c += 8) {
            const fx::XFPod p = part[(int64_t)c * (m * n) + o];
            bad |= p.flags & 4;
            s = xfp::xf_add(s, fx::from_pod(p));
        }
    }
    for (int off = 4; off > 0; off >>= 1) {
        s = xfp::xf_add(s, fx::xf_shfl_down(s, off));
        bad |= __shfl_down_sync(0xffffffffu, bad, off);
    }
    if (sub != 0 || !in) return;
    double2 *pc = C + i + j * ldc;
    if (bad) {
        const double qnan = __longlong_as_double(0x7ff8000000000000ll);
        *pc = make_double2(qnan, qnan);
        return;
    }
    store_axpby(pc, s, xfp::xf_from_dd(alpha.hi, alpha.lo), alpha_one != 0, xfp::xf_from_dd(beta.hi, beta.lo), beta,
                beta_kind);
}

// Device time of the small-tile path in us (fitted, +-20 %: 256^3 75, 500 x 500
// x 8 20): blocks of 16 x 16 outputs x 64 k over the SMs, 6000 clocks each for
// staging and epilogue and 236 per k for the products; < 0 where it does not
// apply (grid and scratch limits).
double small_us(int64_t m, int64_t n, int64_t k)
{
    const double chunks = std::ceil(k / (double)SM_KC);
    if (n > 8 * 65535 || chunks > 65535.0 || chunks * (double)m * (double)n * sizeof(fx::XFPod) > 64.0 * 1048576.0)
        return -1.0;
    const double blocks = std::ceil(m / 16.0) * std::ceil(n / 16.0) * chunks;
    return std::ceil(blocks / device_sm_count()) * (6000.0 + 236.0 * (k < SM_KC ? k : SM_KC)) / 1900.0;
}

// Whether the product goes to the small tiles: the 64 x 64 ones cost a wave of
// 100,000 clocks (scans, the serial epilogue of 16 outputs per thread) and
// 2363 per k, whether or not it fills the SMs.
bool small_tiles(const GemmArgs &g)
{
    const double us = small_us(g.m, g.n, g.k);
    const double waves = std::ceil(std::ceil(g.m / 64.0) * std::ceil(g.n / 64.0) / device_sm_count());
    return us >= 0.0 && us < waves * (100000.0 + 2363.0 * g.k) / 1900.0;
}

template <int T>
bool launch_small(const GemmArgs &g, const char *routine)
{
    const int64_t chunks = (g.k + SM_KC - 1) / SM_KC;
    fx::XFPod *part = nullptr;
    if (chunks > 1) {
        part = (fx::XFPod *)dev_alloc(sizeof(fx::XFPod) * (size_t)(chunks * g.m * g.n), routine);
        if (!part) return false;
    }
    const dim3 grid((unsigned)((g.m + T - 1) / T), (unsigned)((g.n + T - 1) / T), (unsigned)chunks);
    const dd::real al = dd::make(g.alpha.hi, g.alpha.lo), be = dd::make(g.beta.hi, g.beta.lo);
    const int alpha_one = (g.alpha.hi == 1.0 && g.alpha.lo == 0.0);
#define MW_FXS(TA, TB)                                                                                             \
    k_gemm_fixed_small<T, TA, TB><<<grid, FX_THREADS, 0, stream()>>>(g.m, g.n, g.k, (const double2 *)g.A, g.lda,   \
                                                                     (const double2 *)g.B, g.ldb, al, alpha_one,  \
                                                                     be, g.beta_kind, (double2 *)g.C, g.ldc,      \
                                                                     g.uplo, part)
    if (!g.ta && !g.tb) MW_FXS(false, false);
    else if (!g.ta && g.tb) MW_FXS(false, true);
    else if (g.ta && !g.tb) MW_FXS(true, false);
    else MW_FXS(true, true);
#undef MW_FXS
    count_launch();
    if (part) {
        k_fixed_small_fold<<<(unsigned)((g.m * g.n + 31) / 32), 256, 0, stream()>>>(
            g.m, g.n, (int)chunks, part, al, alpha_one, be, g.beta_kind, (double2 *)g.C, g.ldc, g.uplo);
        count_launch();
        dev_free(part);
    }
    return true;
}

}  // namespace

double gemm_fixed_small_us(int64_t m, int64_t n, int64_t k) { return small_us(m, n, k); }

bool gemm_fixed_real(const GemmArgs &g0, const char *routine)
{
    GemmArgs g = g0;
    if (!std::isfinite(g.alpha.hi) || !std::isfinite(g.beta.hi)) return gemm_plain_real(g, routine);
    if (g.k == 0) {
        launch_scale_matrix(g.m, g.n, g.beta, g.beta_kind, g.C, g.ldc, g.uplo);
        return true;
    }
    if (small_tiles(g)) {
        // 8 x 8 tiles where 16 x 16 ones would still leave half of the SMs idle
        const int64_t t16 = ((g.m + 15) / 16) * ((g.n + 15) / 16) * ((g.k + SM_KC - 1) / SM_KC);
        return 2 * t16 <= device_sm_count() ? launch_small<8>(g, routine) : launch_small<16>(g, routine);
    }
    int *ex = (int *)dev_alloc(sizeof(int) * (size_t)(g.m + g.n), routine);
    if (!ex) return false;
    int *ea = ex, *eb = ex + g.m;
    dim3 grid((unsigned)((g.m + FX_BM - 1) / FX_BM), (unsigned)((g.n + FX_BN - 1) / FX_BN));
    const dd::real al = dd::make(g.alpha.hi, g.alpha.lo);
    const int alpha_one = (g.alpha.hi == 1.0 && g.alpha.lo == 0.0);
    for (int64_t k0 = 0; k0 < g.k; k0 += FX_MAX_K) {
        const int64_t kc = (g.k - k0 < FX_MAX_K) ? g.k - k0 : FX_MAX_K;
        const double2 *A = (const double2 *)g.A + (g.ta ? k0 : k0 * g.lda);
        const double2 *B = (const double2 *)g.B + (g.tb ? k0 * g.ldb : k0);
        // exponent bounds of this chunk's rows of op(A) and columns of op(B)
        launch_exp_operands(g, kc, A, B, 1, ex, g.m + g.n, eb, nullptr, nullptr);
        const dd::real be = (k0 == 0) ? dd::make(g.beta.hi, g.beta.lo) : dd::make(1.0, 0.0);
        const int bk = (k0 == 0) ? g.beta_kind : 1;
#define MW_FX(TA, TB)                                                                                         \
    k_gemm_fixed<TA, TB><<<grid, FX_THREADS, 0, stream()>>>(g.m, g.n, kc, A, g.lda, B, g.ldb, ea, eb, al,    \
                                                            alpha_one, be, bk, (double2 *)g.C, g.ldc, g.uplo)
        if (!g.ta && !g.tb) MW_FX(false, false);
        else if (!g.ta && g.tb) MW_FX(false, true);
        else if (g.ta && !g.tb) MW_FX(true, false);
        else MW_FX(true, true);
#undef MW_FX
        count_launch();
    }
    dev_free(ex);
    return true;
}

}  // namespace mw
