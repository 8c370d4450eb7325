// Level-1 double-double kernels: SCAL, AXPY, COPY, SWAP, I*AMAX, DOT and the
// complex twins.
//
// Bit-exactness. The reference's unit-stride SCAL/AXPY run the FMA-fused
// "fast" product on the first (len & ~3) elements of each OpenMP slice and the
// scalar-operator product on the remaining 0..3 (mscal.cpp:42-58,
// maxpy.cpp:42-58, wscal.cpp, wmscal.cpp), where the slices are the balanced
// front-loaded partition of blas_part_bound (common/blas_omp.h:79-84). Every
// element is independent, so a kernel that knows the team size T reproduces
// the same per-element operation sequence on any grid: element i is a "tail"
// element iff its offset inside its slice is >= (slice length & ~3).
// Strided calls use the scalar operators for every element (mscal.cpp:96-100).
// A zero increment on an output makes the reference's loop sequential
// (the same element is updated n times in order); those calls run a
// single-thread kernel that repeats the loop literally.
#include "dd.cuh"
#include "fixacc.cuh"
#include "l1.h"
#include "limbmma.cuh"
#include "runtime.h"

namespace mw {

namespace {

constexpr int kThreads = 256;

// Offset of logical element i for a BLAS vector (negative inc starts at the
// far end).
__device__ __forceinline__ int64_t vidx(int64_t i, int64_t n, int64_t inc)
{
    return inc >= 0 ? i * inc : (n - 1 - i) * (-inc);
}

// Position of a thread's elements in the T-way blas_part_bound partition of
// [0, n) (blas_omp.h:79-84): slice t has base + 1 elements for t < rem and
// base after that. An element is in the scalar tail when it lies in the last
// len % 4 elements of its slice. The slice of the thread's first element is
// found with divisions once; after that the grid-stride walk only advances
// the slice (the strided index moves forward), so the per-element test is
// two compares instead of 64-bit divisions.
struct SliceWalk {
    int64_t base, rem, t, lo, len, tmax;

    __device__ __forceinline__ void start(int64_t i, int64_t n, int64_t T)
    {
        tmax = T - 1;
        base = n / T;
        rem = n % T;
        const int64_t big = rem * (base + 1);
        if (i < big) {
            t = i / (base + 1);
            lo = t * (base + 1);
            len = base + 1;
        } else {
            t = rem + (base ? (i - big) / base : 0);
            lo = t * base + rem;
            len = base;
        }
    }
    // i must not decrease between calls
    __device__ __forceinline__ bool tail(int64_t i)
    {
        while (i >= lo + len && t < tmax) {   // every slice before the last is non-empty
            lo += len;
            ++t;
            len = (t < rem) ? base + 1 : base;
        }
        return (i - lo) >= (len & ~(int64_t)3);
    }
};

int grid_for(int64_t n)
{
    int64_t blocks = (n + kThreads - 1) / kThreads;
    int64_t cap = (int64_t)device_sm_count() * 8;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    return (int)blocks;
}

// ---- SCAL ----------------------------------------------------------------

__global__ void k_mscal_unit(int64_t n, dd::real alpha, double2 *x, int64_t T)
{
    const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    SliceWalk sw;
    if (i0 < n) sw.start(i0, n, T);
    for (int64_t i = i0; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        dd::real v = dd::load(x + i);
        v = sw.tail(i) ? dd::mul_exact(v, alpha) : dd::mul_fast(v, alpha);
        dd::store(x + i, v);
    }
}

__global__ void k_mscal_strided(int64_t n, dd::real alpha, double2 *x, int64_t inc)
{
    if (inc == 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            dd::real v = dd::load(x);
            for (int64_t i = 0; i < n; ++i) v = dd::mul_exact(v, alpha);
            dd::store(x, v);
        }
        return;
    }
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double2 *p = x + vidx(i, n, inc);
        dd::store(p, dd::mul_exact(dd::load(p), alpha));
    }
}

__global__ void k_wscal_unit(int64_t n, dd::cplx alpha, double2 *x, int64_t T)
{
    const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    SliceWalk sw;
    if (i0 < n) sw.start(i0, n, T);
    for (int64_t i = i0; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        dd::cplx v = dd::cload(x + 2 * i);
        v = sw.tail(i) ? dd::cmul_exact(v, alpha) : dd::cmul_fast(v, alpha);
        dd::cstore(x + 2 * i, v);
    }
}

__global__ void k_wscal_strided(int64_t n, dd::cplx alpha, double2 *x, int64_t inc)
{
    if (inc == 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            dd::cplx v = dd::cload(x);
            for (int64_t i = 0; i < n; ++i) v = dd::cmul_exact(v, alpha);
            dd::cstore(x, v);
        }
        return;
    }
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double2 *p = x + 2 * vidx(i, n, inc);
        dd::cstore(p, dd::cmul_exact(dd::cload(p), alpha));
    }
}

__global__ void k_wmscal_unit(int64_t n, dd::real alpha, double2 *x, int64_t T)
{
    const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    SliceWalk sw;
    if (i0 < n) sw.start(i0, n, T);
    for (int64_t i = i0; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        dd::cplx v = dd::cload(x + 2 * i);
        if (sw.tail(i)) {
            v.re = dd::mul_exact(v.re, alpha);
            v.im = dd::mul_exact(v.im, alpha);
        } else {
            v.re = dd::mul_fast(v.re, alpha);
            v.im = dd::mul_fast(v.im, alpha);
        }
        dd::cstore(x + 2 * i, v);
    }
}

__global__ void k_wmscal_strided(int64_t n, dd::real alpha, double2 *x, int64_t inc)
{
    if (inc == 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            dd::cplx v = dd::cload(x);
            for (int64_t i = 0; i < n; ++i) {
                v.re = dd::mul_exact(v.re, alpha);
                v.im = dd::mul_exact(v.im, alpha);
            }
            dd::cstore(x, v);
        }
        return;
    }
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double2 *p = x + 2 * vidx(i, n, inc);
        dd::cplx v = dd::cload(p);
        v.re = dd::mul_exact(v.re, alpha);
        v.im = dd::mul_exact(v.im, alpha);
        dd::cstore(p, v);
    }
}

// ---- AXPY ------------------------------------------------------------------

__global__ void k_maxpy_unit(int64_t n, dd::real alpha, const double2 *x, double2 *y, int64_t T)
{
    const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    SliceWalk sw;
    if (i0 < n) sw.start(i0, n, T);
    for (int64_t i = i0; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        dd::real xv = dd::load(x + i), yv = dd::load(y + i);
        dd::real r;
        if (sw.tail(i))
            r = dd::add_exact(yv, dd::mul_exact(alpha, xv));
        else
            r = dd::add_fast(yv, dd::mul_fast(alpha, xv));
        dd::store(y + i, r);
    }
}

__global__ void k_maxpy_strided(int64_t n, dd::real alpha, const double2 *x, int64_t incx, double2 *y,
                                int64_t incy)
{
    if (incy == 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            dd::real yv = dd::load(y);
            for (int64_t i = 0; i < n; ++i)
                yv = dd::add_exact(yv, dd::mul_exact(alpha, dd::load(x + vidx(i, n, incx))));
            dd::store(y, yv);
        }
        return;
    }
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double2 *py = y + vidx(i, n, incy);
        dd::real xv = dd::load(x + vidx(i, n, incx));
        dd::store(py, dd::add_exact(dd::load(py), dd::mul_exact(alpha, xv)));
    }
}

// ---- COPY / SWAP -----------------------------------------------------------

// elem2 = number of double2 words per element (1 real, 2 complex).
__global__ void k_copy(int64_t n, const double2 *x, int64_t incx, double2 *y, int64_t incy, int elem2)
{
    if (incy == 0) {
        // Sequential reference loop: the last logical element wins.
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            const double2 *src = x + elem2 * vidx(n - 1, n, incx);
            for (int w = 0; w < elem2; ++w) y[w] = src[w];
        }
        return;
    }
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double2 *src = x + elem2 * vidx(i, n, incx);
        double2 *dst = y + elem2 * vidx(i, n, incy);
        for (int w = 0; w < elem2; ++w) dst[w] = src[w];
    }
}

__global__ void k_swap(int64_t n, double2 *x, int64_t incx, double2 *y, int64_t incy, int elem2)
{
    if (incx == 0 || incy == 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            for (int64_t i = 0; i < n; ++i) {
                double2 *px = x + elem2 * vidx(i, n, incx);
                double2 *py = y + elem2 * vidx(i, n, incy);
                for (int w = 0; w < elem2; ++w) {
                    double2 t = px[w];
                    px[w] = py[w];
                    py[w] = t;
                }
            }
        }
        return;
    }
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double2 *px = x + elem2 * vidx(i, n, incx);
        double2 *py = y + elem2 * vidx(i, n, incy);
        for (int w = 0; w < elem2; ++w) {
            double2 t = px[w];
            px[w] = py[w];
            py[w] = t;
        }
    }
}

// ---- I*AMAX ------------------------------------------------------------------
// Order: lexicographic (|hi|, sign-adjusted lo) maximum, lowest index on ties
// (imamax.cpp:43-72, mf_pred.h:60-63). Complex magnitude |re|+|im| uses the
// scalar-operator add (iwamax.cpp:36-76).
//
// The comparison runs on the integer pipe: each magnitude becomes a 128-bit
// unsigned key whose order is the FP64 order of (|hi|, lo). Word 0..1 hold the
// bits of |hi| (monotone for non-negative doubles), words 2..3 the usual
// orderable image of lo (negative: all bits inverted; positive: sign bit set),
// with -0 mapped to +0 so the two zeros tie as they do under FP64 '=='. A NaN
// hi gives the all-zero key and a NaN lo the zero low half, so a NaN never
// beats a number, as with the reference's -inf-seeded vector scan in which
// 'NaN > best' is false; among all-NaN inputs the lowest index wins.

struct AmaxKey {
    uint32_t k[4];   // k[0] most significant
    int64_t idx;     // 0-based; -1 = empty
};

__device__ __forceinline__ AmaxKey amax_key(uint4 v, int64_t idx)
{
    // v = {hi.lo32, hi.hi32, lo.lo32, lo.hi32}
    AmaxKey r;
    const uint32_t ah = v.y & 0x7fffffffu;
    const bool hnan = ah > 0x7ff00000u || (ah == 0x7ff00000u && v.x != 0u);
    const uint32_t lh = v.w ^ (v.y & 0x80000000u);   // lo, sign flipped when hi < 0
    const uint32_t al = lh & 0x7fffffffu;
    const bool lnan = al > 0x7ff00000u || (al == 0x7ff00000u && v.z != 0u);
    const bool lzero = (al | v.z) == 0u;
    const uint32_t m = (uint32_t)((int32_t)lh >> 31);
    uint32_t k2 = lh ^ (m | 0x80000000u), k3 = v.z ^ m;
    if (lzero) { k2 = 0x80000000u; k3 = 0u; }
    if (lnan) { k2 = 0u; k3 = 0u; }
    r.k[0] = hnan ? 0u : ah;
    r.k[1] = hnan ? 0u : v.x;
    r.k[2] = hnan ? 0u : k2;
    r.k[3] = hnan ? 0u : k3;
    r.idx = idx;
    return r;
}

// a.k > b.k as 128-bit unsigned numbers: the borrow out of b - a.
__device__ __forceinline__ bool key_gt(const AmaxKey &a, const AmaxKey &b)
{
    uint32_t borrow;
    asm("{\n\t"
        ".reg .u32 t;\n\t"
        "sub.cc.u32 t, %4, %8;\n\t"
        "subc.cc.u32 t, %3, %7;\n\t"
        "subc.cc.u32 t, %2, %6;\n\t"
        "subc.cc.u32 t, %1, %5;\n\t"
        "subc.u32 %0, 0, 0;\n\t"
        "}"
        : "=r"(borrow)
        : "r"(b.k[0]), "r"(b.k[1]), "r"(b.k[2]), "r"(b.k[3]), "r"(a.k[0]), "r"(a.k[1]), "r"(a.k[2]),
          "r"(a.k[3]));
    return borrow != 0u;
}

__device__ __forceinline__ bool key_eq(const AmaxKey &a, const AmaxKey &b)
{
    return ((a.k[0] ^ b.k[0]) | (a.k[1] ^ b.k[1]) | (a.k[2] ^ b.k[2]) | (a.k[3] ^ b.k[3])) == 0u;
}

// Merge order of two partial results (either may be empty).
__device__ __forceinline__ bool amax_better(const AmaxKey &a, const AmaxKey &b)
{
    if (a.idx < 0) return false;
    if (b.idx < 0) return true;
    return key_gt(a, b) || (key_eq(a, b) && a.idx < b.idx);
}

__device__ __forceinline__ AmaxKey amax_shfl(const AmaxKey &k, int off)
{
    AmaxKey r;
#pragma unroll
    for (int w = 0; w < 4; ++w) r.k[w] = __shfl_down_sync(0xffffffffu, k.k[w], off);
    r.idx = __shfl_down_sync(0xffffffffu, k.idx, off);
    return r;
}

__device__ __forceinline__ AmaxKey amax_empty()
{
    AmaxKey r;
    r.k[0] = r.k[1] = r.k[2] = r.k[3] = 0u;
    r.idx = -1;
    return r;
}

__device__ AmaxKey amax_block_reduce(AmaxKey k)
{
    __shared__ AmaxKey sh[kThreads / 32];
    for (int off = 16; off > 0; off >>= 1) {
        AmaxKey o = amax_shfl(k, off);
        if (amax_better(o, k)) k = o;
    }
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) sh[wid] = k;
    __syncthreads();
    if (wid == 0) {
        k = (lane < (int)(blockDim.x >> 5)) ? sh[lane] : amax_empty();
        for (int off = 16; off > 0; off >>= 1) {
            AmaxKey o = amax_shfl(k, off);
            if (amax_better(o, k)) k = o;
        }
    }
    return k;
}

__device__ __forceinline__ uint4 dd_bits(dd::real m)
{
    const unsigned long long h = (unsigned long long)__double_as_longlong(m.hi);
    const unsigned long long l = (unsigned long long)__double_as_longlong(m.lo);
    return make_uint4((uint32_t)h, (uint32_t)(h >> 32), (uint32_t)l, (uint32_t)(l >> 32));
}

// Within one thread the candidates arrive in increasing index order, so a
// strict '>' keeps the lowest index among equal keys.
template <bool CPLX>
__global__ void k_iamax_partial(int64_t n, const double2 *x, int64_t inc, AmaxKey *part)
{
    AmaxKey best = amax_empty();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (!CPLX && inc == 1) {
        // unit stride: two adjacent elements (32 bytes) per thread and step
        const uint4 *v = (const uint4 *)x;
        const int64_t npair = n >> 1;
        for (int64_t p = i0; p < npair; p += stride) {
            const uint4 a = __ldcs(v + 2 * p), b = __ldcs(v + 2 * p + 1);
            const AmaxKey ka = amax_key(a, 2 * p), kb = amax_key(b, 2 * p + 1);
            if (best.idx < 0 || key_gt(ka, best)) best = ka;
            if (key_gt(kb, best)) best = kb;
        }
        if ((n & 1) && i0 == 0) {
            const AmaxKey kl = amax_key(__ldcs(v + n - 1), n - 1);
            if (best.idx < 0 || key_gt(kl, best)) best = kl;   // highest index: strict '>'
        }
    } else {
        for (int64_t i = i0; i < n; i += stride) {
            uint4 bits;
            if (CPLX) {
                const double2 *p = x + 2 * vidx(i, n, inc);
                bits = dd_bits(dd::add_exact(dd::mag(dd::load(p)), dd::mag(dd::load(p + 1))));
            } else {
                bits = __ldcs((const uint4 *)(x + vidx(i, n, inc)));
            }
            const AmaxKey c = amax_key(bits, i);
            if (best.idx < 0 || key_gt(c, best)) best = c;
        }
    }
    best = amax_block_reduce(best);
    if (threadIdx.x == 0) part[blockIdx.x] = best;
}

__global__ void k_iamax_final(int nparts, const AmaxKey *part, int64_t *out)
{
    AmaxKey best = amax_empty();
    for (int i = threadIdx.x; i < nparts; i += blockDim.x)
        if (amax_better(part[i], best)) best = part[i];
    best = amax_block_reduce(best);
    if (threadIdx.x == 0) *out = best.idx;
}

// ---- DOT ---------------------------------------------------------------------
// mdot.cpp:48-87 accumulates TwoProduct + Bailey three-limb sums on the FP64
// pipe. Here each product, one factor rounded to 2^-115 of the largest of its
// warp's block of at most 4096 products, is accumulated exactly as limb products
// on the tensor cores, the warps' sums are added as 128-bit extended floats in a
// fixed order (block, then the grid's block partials), and the result is rounded
// once to double-double. It is deterministic for a given n and device, and off by
// at most 2^-104 sum |x y| beyond that rounding.

__device__ fx::XF xf_block_sum(fx::XF v)
{
    __shared__ fx::XFPod sh[kThreads / 32];
    v = fx::xf_warp_sum(v);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) sh[wid] = fx::to_pod(v, false);
    __syncthreads();
    if (wid == 0) {
        if (lane < (int)(blockDim.x >> 5)) {
            v = fx::from_pod(sh[lane]);
        } else {
            v.zero = true; v.neg = false; v.m = 0; v.e = 0;
        }
        v = fx::xf_warp_sum(v);
    }
    return v;
}

__device__ bool block_any(bool b)
{
    return __syncthreads_or(b ? 1 : 0) != 0;
}

// The tensor-core form (limbmma.cuh): of a warp's 32 pairs (x_i, y_i), x_i is
// aligned by the product's exponent to the warp's block, both are written as
// 16 bytes to warp-private shared memory, and one ldmatrix of 16-bit units per
// operand transposes them: lane (g, t) gets limbs 2g and 2g + 1 of elements
// 2t, 2t + 1 of each eight, which two masks turn into fp16 subnormal pairs.
// D[q][r] += sum_i X_iq Y_ir is then a 16 x 16 outer-product sum over K = 32 in
// four MMAs (rows and columns in the order even limbs, odd limbs), all limb
// products kept, and the dot product is sum D[q][r] 2^(8(q+r)).
// Where the product is negative, X's limbs 0..14 are complemented, which
// stands for 2^120 - 1 - X, and limb 15 is 1: D[15][r] sums the Y that
// 2^120 - 1 has to be taken off for.
// Two groups of 32 pairs per turn hide each other's latency; four turns of
// pairs are in flight per lane (cp.async).
//
// Exactness: D grows by at most 255 * 255 per pair and stays below 2^24 units
// for 4 turns of 64; then it moves to int32 sums, and after 16 of those (or
// when a product above the block moves it up) to the warp's extended float.
//
// Accuracy: x_i is rounded where its alignment cuts it (for free: the half unit
// enters the decode's carry chain), and every 4096 pairs the warp starts from
// the block of the next products again. Cut to one block for the whole run with
// three bits more of margin, a dominating product among equal-signed small ones
// made it 8 units of 2^-104 sum |x y| off at n = 10^7 and 80 at 10^8 (per-thread
// blocks of some 330 products: 0.1 and 0.7); now below 0.1 at any n.
//
// Bound: HBM (32 B per pair) and instruction issue, both about two thirds busy.
// Measured at n = 10^8: 867 -> 598 us (3.69 -> 5.35 TB/s) before the rounding and
// the restarts; 149 instructions per pair, where 19 IMAD.WIDE
// digit products and their digit splits took 223. Turns with zeros or alignments
// beyond a word have a loop of their own, which shifts any way, and pass without
// products where all are zero: whole call at n = 10^8, with the general decode for
// each such turn, as the digit form was, and now: a zero in 64 1268, 949 and 866 us;
// the second half zero 897, 691 and 675; exponents over 2^40 1245, 957 and 888;
// dense 642, 907 and 641.
constexpr int kDotFlush = 4;            // turns of 64 pairs per move to the int32 sums
constexpr int kDotFold = 16;            // moves per fold into the extended float
constexpr int kDotStages = 4;           // turns in flight
constexpr int kNoBlock = -(1 << 22);    // no nonzero product yet
constexpr int kDotSmem = kDotStages * 4 * 16 * kThreads + 2 * 1024 * (kThreads / 32);

__global__ void __launch_bounds__(kThreads, 2) k_mdot_limb(int64_t n, const double2 *__restrict__ x, int64_t incx,
                                                          const double2 *__restrict__ y, int64_t incy,
                                                          fx::XFPod *part)
{
    // [stage][pair 0 x, y, pair 1 x, y][thread] 16 bytes, then per warp [pair][operand][element] 16 bytes
    extern __shared__ __align__(16) unsigned char s_dot[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t nwarps = (int64_t)gridDim.x * (kThreads / 32), warp = (int64_t)blockIdx.x * (kThreads / 32) + wid;
    const int64_t total = (n + 63) / 64;
    const int64_t turns = warp < total ? (total - warp + nwarps - 1) / nwarps : 0;
    // the lane's next pair (and the one 32 further), as addresses: either order
    // of a BLAS increment is a start and a step
    const int64_t i00 = warp * 64 + lane, sx = nwarps * 64 * incx, sy = nwarps * 64 * incy;
    const double2 *px = x + vidx(i00, n, incx), *py = y + vidx(i00, n, incy);
    int64_t room = n - i00;   // > 0: px, py are pairs of the vectors
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(s_dot) + threadIdx.x * 16u;
    constexpr uint32_t kPlane = 16u * kThreads;
    auto load = [&](int64_t turn) {   // turns in order; past the end nothing is read
        const uint32_t d = ring + ((uint32_t)turn & (kDotStages - 1)) * (4 * kPlane);
        if (room > 0) {
            lmb::cp_async16(d, px);
            lmb::cp_async16(d + kPlane, py);
        }
        if (room > 32) {
            lmb::cp_async16(d + 2 * kPlane, px + 32 * incx);
            lmb::cp_async16(d + 3 * kPlane, py + 32 * incy);
        }
        px += sx;
        py += sy;
        room -= nwarps * 64;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int blk = kNoBlock;
    bool bad = false;
    float acc[2][4];
    int sum[2][4];
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            acc[b][i] = 0.0f;
            sum[b][i] = 0;
        }
    fx::XF tot;
    tot.zero = true; tot.neg = false; tot.m = 0; tot.e = 0;
    auto flush = [&]() {
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                sum[b][i] += __float2int_rn(acc[b][i] * 0x1p48f);
                acc[b][i] = 0.0f;
            }
    };
    // the warp's sums into its extended float (the same in every lane)
    auto fold = [&]() {
        flush();
        // the lane's entries: limb 2g + a of x, 2(2t + c) + b of y
        const int g = lane >> 2, t = lane & 3;
        uint64_t W[4] = {0, 0, 0, 0};
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            int64_t p = 0;   // over the lane's limbs 4t .. 4t + 3 of y
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int c = 0; c < 2; ++c) p += (int64_t)sum[b][2 * a + c] << (8 * (2 * c + b));
            const bool last = a == 1 && g == 7;   // limb 15: - (2^120 - 1)
            lmb::add_at(W, last ? -p : p, 8 * (last ? 15 : 2 * g + a) + 32 * t);
            lmb::add_at(W, last ? p : 0, 32 * t);
        }
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int i = 0; i < 4; ++i) sum[b][i] = 0;
        lmb::lane_sum256(W, 32);
        if (blk != kNoBlock) tot = xfp::xf_add(tot, fx::w256_to_xf(W, blk - 2 * lmb::kExpBias));
    };

    for (int u = 0; u < kDotStages - 1; ++u) load(u);
    unsigned char *limbs = s_dot + kDotStages * 4 * kPlane + wid * 2048;
    const uint32_t lrow = (uint32_t)__cvta_generic_to_shared(limbs) + lane * 16u;
    bool any_shift = true;   // (the first turn has no block)
    // the turn's aligned limbs into the sums, and what is due after it
    auto products = [&](int64_t turn, const uint32_t (&wx)[2][4], const uint32_t (&wy)[2][4], const uint32_t (&neg)[2],
                        bool go) {
        load(turn + kDotStages - 1);   // into the stage read in the previous turn
        if (go) {
            __syncwarp();   // the previous turn's limbs have been read
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                uint4 *st = reinterpret_cast<uint4 *>(limbs + 1024 * p) + lane;
                st[0] = make_uint4(wx[p][0] ^ neg[p], wx[p][1] ^ neg[p], wx[p][2] ^ neg[p],
                                   (wx[p][3] ^ (neg[p] & 0xFFFFFFu)) | (neg[p] & 0x1000000u));
                st[32] = make_uint4(wy[p][0], wy[p][1], wy[p][2], wy[p][3]);
            }
            __syncwarp();
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                uint32_t a[4], b[4];   // elements 8j .. 8j + 7 in [j]
                lmb::ldmatrix_x4_trans(a, lrow + 1024u * p);
                lmb::ldmatrix_x4_trans(b, lrow + 1024u * p + 512u);
#pragma unroll
                for (int h = 0; h < 4; h += 2) {
                    const uint32_t a0 = a[h] & 0xFF00FFu, a1 = __byte_perm(a[h], 0u, 0x4341);
                    const uint32_t a2 = a[h + 1] & 0xFF00FFu, a3 = __byte_perm(a[h + 1], 0u, 0x4341);
                    lmb::mma16816(acc[0], a0, a1, a2, a3, b[h] & 0xFF00FFu, b[h + 1] & 0xFF00FFu);
                    lmb::mma16816(acc[1], a0, a1, a2, a3, __byte_perm(b[h], 0u, 0x4341),
                                  __byte_perm(b[h + 1], 0u, 0x4341));
                }
            }
        }
        if ((turn & (kDotFlush - 1)) == kDotFlush - 1) {
            flush();
            if ((turn & (kDotFlush * kDotFold - 1)) == kDotFlush * kDotFold - 1) {
                fold();
                blk = kNoBlock;   // the next products find their own block
                any_shift = true;
            }
        }
    };
    int64_t turn = 0;
    while (turn < turns) {
        // turns whose operands are all on the straight line, within a word of the block
#pragma unroll 1
        for (; turn < turns && !any_shift; ++turn) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kDotStages - 2) : "memory");
            const unsigned char *cur = s_dot + ((uint32_t)turn & (kDotStages - 1)) * (4 * kPlane) + threadIdx.x * 16u;
            uint32_t wx[2][4], wy[2][4], neg[2];
            int sh[2];
            bool fast = (warp + turn * nwarps) * 64 + 64 <= n;
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                const double2 vx = *reinterpret_cast<const double2 *>(cur + 2 * p * kPlane);
                const double2 vy = *reinterpret_cast<const double2 *>(cur + (2 * p + 1) * kPlane);
                int ehx, ehy;
                const bool oky = lmb::split_fast(vy, wy[p], ehy);
                sh[p] = blk - lmb::hi_exp(vx) - ehy;
                const bool okx = lmb::split_fast(vx, wx[p], ehx, lmb::half_unit(sh[p]));
                fast = fast && okx && oky && (uint32_t)sh[p] < 32u;
                neg[p] = (uint32_t)((__double2hiint(vx.x) ^ __double2hiint(vy.x)) >> 31);
            }
            if (!__all_sync(0xffffffffu, fast)) {
                any_shift = true;
                break;
            }
#pragma unroll
            for (int p = 0; p < 2; ++p) lmb::shr_short(wx[p], sh[p]);
            products(turn, wx, wy, neg, true);
        }
        // the others, in a loop of their own (in the same one they cost it 2 to 5 %), until a turn
        // that the first loop takes
#pragma unroll 1
        for (; turn < turns && any_shift; ++turn) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kDotStages - 2) : "memory");
            const unsigned char *cur = s_dot + ((uint32_t)turn & (kDotStages - 1)) * (4 * kPlane) + threadIdx.x * 16u;
            const int64_t i0 = (warp + turn * nwarps) * 64;
            uint32_t wx[2][4], wy[2][4], neg[2];
            int sh[2];
            // zeros and long alignments at the block there is: the same decode, any shift
            bool plain = i0 + 64 <= n, live = false, fast = plain;
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                const double2 vx = *reinterpret_cast<const double2 *>(cur + 2 * p * kPlane);
                const double2 vy = *reinterpret_cast<const double2 *>(cur + (2 * p + 1) * kPlane);
                int ehx, ehy;
                const bool okx = lmb::split_fast(vx, wx[p], ehx), oky = lmb::split_fast(vy, wy[p], ehy);
                const bool zx = lmb::all_zero(vx), zy = lmb::all_zero(vy), none = zx || zy;
                sh[p] = blk - ehx - ehy;
                fast = fast && okx && oky && (uint32_t)sh[p] < 32u;
                plain = plain && (okx || zx) && (oky || zy) && (sh[p] >= 0 || none);
                live = live || !none;
                sh[p] = none ? 127 : min(sh[p], 127);   // W < 2^118: nothing is left of it at 127
                neg[p] = (uint32_t)((__double2hiint(vx.x) ^ __double2hiint(vy.x)) >> 31);
            }
            any_shift = !__all_sync(0xffffffffu, fast);
            bool go = true;
            if (__all_sync(0xffffffffu, plain)) {
                go = __any_sync(0xffffffffu, live);
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    uint32_t sv[4];
                    lmb::shr_round(wx[p], sh[p], sv);
#pragma unroll
                    for (int i = 0; i < 4; ++i) wx[p][i] = sv[i];
                }
            } else {
                // the end, operands off the straight-line path, a larger block
                any_shift = false;   // the next turn may well be dense
                int ep[2], top = kNoBlock;
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    const fx::Op ox = fx::decode(*reinterpret_cast<const double2 *>(cur + 2 * p * kPlane));
                    const fx::Op oy = fx::decode(*reinterpret_cast<const double2 *>(cur + (2 * p + 1) * kPlane));
                    const bool no = ((ox.flags | oy.flags) & fx::kBad) != 0;
                    const bool in = i0 + lane + 32 * p < n;   // else the stage holds an older pair or nothing
                    bad = bad || (no && in);
                    ep[p] = (no || !in || ((ox.flags | oy.flags) & fx::kZero))
                                ? kNoBlock
                                : ox.e + oy.e + 2 * lmb::kExpBias;
                    // (an x that is not normalised may have more than 118 bits)
                    if (ep[p] != kNoBlock) top = max(top, ep[p] + max(0, 10 - __clz((int)ox.w[3])));
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        wx[p][i] = ox.w[i];
                        wy[p][i] = oy.w[i];
                    }
                }
                top = __reduce_max_sync(0xffffffffu, top);
                if (top != kNoBlock && top > blk) {
                    if (blk != kNoBlock) fold();
                    blk = top + 1;
                }
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    uint32_t sv[4];
                    lmb::shr_round(wx[p], ep[p] == kNoBlock ? 127 : min(blk - ep[p], 127), sv);
#pragma unroll
                    for (int i = 0; i < 4; ++i) wx[p][i] = ep[p] == kNoBlock ? 0u : sv[i];
                }
            }
            products(turn, wx, wy, neg, go);
        }
    }
    fold();
    bad = block_any(bad);
    __shared__ fx::XFPod sh_tot[kThreads / 32];
    if (lane == 0) sh_tot[wid] = fx::to_pod(tot, false);
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kThreads / 32; ++w) tot = xfp::xf_add(tot, fx::from_pod(sh_tot[w]));
        part[blockIdx.x] = fx::to_pod(tot, bad);
    }
}

__global__ void __launch_bounds__(kThreads) k_mdot_final(int nparts, const fx::XFPod *part, double2 *out)
{
    fx::XF acc;
    acc.zero = true; acc.neg = false; acc.m = 0; acc.e = 0;
    bool bad = false;
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
        const fx::XFPod p = part[i];
        bad |= (p.flags & 4) != 0;
        acc = xfp::xf_add(acc, fx::from_pod(p));
    }
    bad = block_any(bad);
    acc = xf_block_sum(acc);
    if (threadIdx.x == 0) {
        double h, l;
        xfp::xf_to_dd(acc, h, l);
        if (bad) h = l = __longlong_as_double(0x7ff8000000000000ll);
        *out = make_double2(h, l);
    }
}

}  // namespace

// ---- launchers ---------------------------------------------------------------

void launch_mscal(int64_t n, dd_host alpha, void *x, int64_t inc, bool unit, int64_t team)
{
    dd::real a = dd::make(alpha.hi, alpha.lo);
    if (unit)
        k_mscal_unit<<<grid_for(n), kThreads, 0, stream()>>>(n, a, (double2 *)x, team);
    else
        k_mscal_strided<<<inc == 0 ? 1 : grid_for(n), kThreads, 0, stream()>>>(n, a, (double2 *)x, inc);
    count_launch();
}

void launch_wscal(int64_t n, cdd_host alpha, void *x, int64_t inc, bool unit, int64_t team)
{
    dd::cplx a;
    a.re = dd::make(alpha.re.hi, alpha.re.lo);
    a.im = dd::make(alpha.im.hi, alpha.im.lo);
    if (unit)
        k_wscal_unit<<<grid_for(n), kThreads, 0, stream()>>>(n, a, (double2 *)x, team);
    else
        k_wscal_strided<<<inc == 0 ? 1 : grid_for(n), kThreads, 0, stream()>>>(n, a, (double2 *)x, inc);
    count_launch();
}

void launch_wmscal(int64_t n, dd_host alpha, void *x, int64_t inc, bool unit, int64_t team)
{
    dd::real a = dd::make(alpha.hi, alpha.lo);
    if (unit)
        k_wmscal_unit<<<grid_for(n), kThreads, 0, stream()>>>(n, a, (double2 *)x, team);
    else
        k_wmscal_strided<<<inc == 0 ? 1 : grid_for(n), kThreads, 0, stream()>>>(n, a, (double2 *)x, inc);
    count_launch();
}

void launch_maxpy(int64_t n, dd_host alpha, const void *x, int64_t incx, void *y, int64_t incy, bool unit,
                  int64_t team)
{
    dd::real a = dd::make(alpha.hi, alpha.lo);
    if (unit)
        k_maxpy_unit<<<grid_for(n), kThreads, 0, stream()>>>(n, a, (const double2 *)x, (double2 *)y, team);
    else
        k_maxpy_strided<<<incy == 0 ? 1 : grid_for(n), kThreads, 0, stream()>>>(n, a, (const double2 *)x, incx,
                                                                               (double2 *)y, incy);
    count_launch();
}

void launch_copy(int64_t n, const void *x, int64_t incx, void *y, int64_t incy, int elem2)
{
    k_copy<<<incy == 0 ? 1 : grid_for(n), kThreads, 0, stream()>>>(n, (const double2 *)x, incx, (double2 *)y,
                                                                  incy, elem2);
    count_launch();
}

void launch_swap(int64_t n, void *x, int64_t incx, void *y, int64_t incy, int elem2)
{
    bool seq = (incx == 0 || incy == 0);
    k_swap<<<seq ? 1 : grid_for(n), kThreads, 0, stream()>>>(n, (double2 *)x, incx, (double2 *)y, incy, elem2);
    count_launch();
}

bool launch_iamax(int64_t n, const void *x, int64_t inc, bool cplx, int64_t *result_host, const char *routine)
{
    int g = grid_for(n);
    size_t bytes = (size_t)g * sizeof(AmaxKey) + 64;
    char *scratch = (char *)dev_alloc(bytes, routine);
    if (!scratch) return false;
    AmaxKey *part = (AmaxKey *)scratch;
    int64_t *out = (int64_t *)(scratch + (((size_t)g * sizeof(AmaxKey) + 15) / 16) * 16);
    if (cplx)
        k_iamax_partial<true><<<g, kThreads, 0, stream()>>>(n, (const double2 *)x, inc, part);
    else
        k_iamax_partial<false><<<g, kThreads, 0, stream()>>>(n, (const double2 *)x, inc, part);
    k_iamax_final<<<1, kThreads, 0, stream()>>>(g, part, out);
    count_launch(2);
    bool ok = cuda_ok(cudaMemcpyAsync(result_host, out, sizeof(int64_t), cudaMemcpyDeviceToHost, stream()), routine,
                      "iamax result readback");
    dev_free(scratch);
    if (!ok) return false;
    return cuda_ok(cudaStreamSynchronize(stream()), routine, "iamax sync");
}

bool launch_mdot(int64_t n, const void *x, int64_t incx, const void *y, int64_t incy, dd_host *result_host,
                 const char *routine)
{
    // one wave of resident blocks (two per SM), a turn of 64 pairs per warp at least
    const int64_t wave = 2ll * device_sm_count(), need = (n + 2 * kThreads - 1) / (2 * kThreads);
    const int g = (int)(need < wave ? need : wave);
    size_t bytes = (size_t)g * sizeof(fx::XFPod) + 256;
    char *buf = (char *)dev_alloc(bytes, routine);
    if (!buf) return false;
    fx::XFPod *part = (fx::XFPod *)buf;
    double2 *res = (double2 *)(buf + ((size_t)g * sizeof(fx::XFPod) + 15) / 16 * 16);
    cudaFuncSetAttribute(k_mdot_limb, cudaFuncAttributeMaxDynamicSharedMemorySize, kDotSmem);
    k_mdot_limb<<<g, kThreads, kDotSmem, stream()>>>(n, (const double2 *)x, incx, (const double2 *)y, incy, part);
    k_mdot_final<<<1, kThreads, 0, stream()>>>(g, part, res);
    count_launch(2);
    double2 r;
    bool ok = cuda_ok(cudaMemcpyAsync(&r, res, sizeof(double2), cudaMemcpyDeviceToHost, stream()), routine,
                      "dot result readback");
    dev_free(buf);
    if (!ok) return false;
    if (!cuda_ok(cudaStreamSynchronize(stream()), routine, "dot sync")) return false;
    result_host->hi = r.x;
    result_host->lo = r.y;
    return true;
}

}  // namespace mw
