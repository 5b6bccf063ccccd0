/*
 * udev_norm.cu - the reference's float L1 norm (a sequential sum of |v_i| in
 * memory order, ufo-ir-basic-ops.c:259-277), in parallel and bit for bit.
 *
 * While the running sum stays in one binade [2^e, 2^(e+1)) it is an integer m
 * of units u = 2^(e-23), and adding x >= 0 adds round(x / u) to m. That
 * increment does not depend on m, except in a tie, which goes to the even
 * neighbour and so depends on m's parity alone. An element is therefore a map
 * {m even -> d0, m odd -> d1}; maps compose ((a then b): m + a_p, then b of
 * the new parity), associatively, so any run of elements folds to one pair
 * (d0, d1), in parallel. Subnormal sums share the units of the first normal
 * binade. What is left of the chain is the places where the sum reaches the
 * next binade, a few dozen at most: m would pass 2^24 there.
 *
 *  1. l1_sums_kernel: float sums of up to 512 chunks of 512 elements or more (a
 *     prediction of where each chunk starts, and whether it holds a NaN);
 *  2. l1_steps_kernel: each chunk's (d0, d1) in the three binades around its
 *     predicted start;
 *  3. l1_walk_kernel, one CTA per slice: a warp scans 32 chunks at a time and
 *     takes those that end inside the binade; the chunk that does not is
 *     folded again by the whole CTA, segment by segment of one thread, and
 *     the one segment that crosses is added element by element.
 *
 * One thread adding in order waited for its loads, 13 ns an element: 3.36 ms for
 * 530^2 of them, 0.04 ms with the three kernels here (most of it the walk: a few
 * microseconds at each of the binades left after the first 1024 elements).
 * Those cost 30 us whatever the size, so up to 8192 elements one thread adds
 * from shared memory (l1_short_kernel, 2 ns an element). A call with 256 / 1024 /
 * 4096 / 8192 / 8200 / 65536 elements takes 16 / 18 / 27 / 39 / 42 / 42 us of
 * which 15 are the call; 18 / 26 / 65 / 115 / 114 / 800 element by element from
 * global memory, 47 / 54 / 54 / 54 / 54 / 46 with the three kernels and 512
 * chunks always. Chunks of at least 512 elements keep stacks of small slices from
 * launching mostly idle CTAs: ASD-POCS of 1000 slices of 64^2, two iterations,
 * 6.3 ms element by element, 86 with 512 chunks each, 3.3 now; 200 of 120^2
 * 12.1, 19.9 and 4.8.
 */
#include <cuda_runtime.h>

#include "udev_internal.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kChunks = 512;                 /* chunks per slice at most */
constexpr int kMinChunk = 512;               /* elements of a chunk at least */
constexpr int kCand = 3;                     /* binades tried per chunk */
constexpr int kHead = 1024;                  /* elements added one by one at the start */
constexpr size_t kShort = 8192;              /* elements of a slice that one thread adds */
constexpr unsigned int kTop = 1u << 24;      /* units at the end of a binade */
constexpr unsigned int kMany = 1u << 25;     /* any increment past the binade */

struct Step {
    unsigned int d0, d1;
};

/* One chunk's record in the scratch. */
struct __align__(8) ChunkRec {
    float sum;
    int e0;                  /* first of its kCand binades */
    Step s[kCand];
};
static_assert(sizeof(ChunkRec) == 4 * sizeof(double), "udev_l1_partials counts four doubles a chunk");

/* a, then b */
__device__ __forceinline__ Step compose(Step a, Step b)
{
    Step r;
    r.d0 = min(a.d0 + ((a.d0 & 1u) ? b.d1 : b.d0), kMany);
    r.d1 = min(a.d1 + ((a.d1 & 1u) ? b.d0 : b.d1), kMany);
    return r;
}

/* What adding |v| (bits) does to a sum in binade e >= -126. */
__device__ __forceinline__ Step element(unsigned int bits, int e)
{
    const unsigned int ab = bits & 0x7fffffffu, ex = ab >> 23;
    const unsigned int m = (ab & 0x7fffffu) | (ex ? 0x800000u : 0u);
    const int sh = e + 127 - (int) max(ex, 1u);
    Step r;
    if (sh <= 0) {
        r.d0 = r.d1 = sh == 0 ? m : (m ? kMany : 0u);
    } else if (sh > 24) {
        r.d0 = r.d1 = 0u;
    } else {
        const unsigned int k = m >> sh, rem = m & ((1u << sh) - 1u), half = 1u << (sh - 1);
        const unsigned int up = rem > half ? 1u : 0u, tie = rem == half ? 1u : 0u;
        r.d0 = k + up + (tie & k);
        r.d1 = k + up + (tie & ~k & 1u);
    }
    return r;
}

__device__ __forceinline__ Step shfl_up_step(Step s, int o)
{
    Step r;
    r.d0 = __shfl_up_sync(0xffffffffu, s.d0, o);
    r.d1 = __shfl_up_sync(0xffffffffu, s.d1, o);
    return r;
}

/* Inclusive composition over the lanes of a warp, in lane order. */
__device__ __forceinline__ Step warp_scan(Step s, int lane)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const Step p = shfl_up_step(s, o);
        if (lane >= o)
            s = compose(p, s);
    }
    return s;
}

/* Binade and units of a sum (finite, >= 0). */
__device__ __forceinline__ void split(unsigned int bits, int &e, unsigned int &m)
{
    const unsigned int ex = bits >> 23;
    e = (int) max(ex, 1u) - 127;
    m = (bits & 0x7fffffu) | (ex ? 0x800000u : 0u);
}

/* The sum of m <= 2^24 units in binade e. */
__device__ __forceinline__ unsigned int join(int e, unsigned int m)
{
    if (m >= kTop)
        return (unsigned int) (e + 128) << 23;
    return m >= 0x800000u ? ((unsigned int) (e + 127) << 23) | (m & 0x7fffffu) : m;
}

/* Elements of chunk c of len. */
__device__ __forceinline__ void chunk_range(size_t count, size_t len, int c, size_t &lo, size_t &hi)
{
    lo = min((size_t) c * len, count);
    hi = min(lo + len, count);
}

__global__ void __launch_bounds__(kThreads) l1_sums_kernel(const float *__restrict__ v, size_t count, size_t len,
                                                           ChunkRec *__restrict__ recs)
{
    __shared__ float part[kWarps];
    const float *p = v + (size_t) blockIdx.y * count;
    size_t lo, hi;
    chunk_range(count, len, (int) blockIdx.x, lo, hi);
    float s = 0.0f;
    for (size_t i = lo + threadIdx.x; i < hi; i += kThreads)
        s += fabsf(p[i]);
    for (int o = 16; o > 0; o >>= 1)
        s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0)
        part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kWarps; ++w)
            s += part[w];
        recs[(size_t) blockIdx.y * kChunks + blockIdx.x].sum = s;
    }
}

__global__ void __launch_bounds__(kThreads) l1_steps_kernel(const float *__restrict__ v, size_t count, size_t len,
                                                            ChunkRec *__restrict__ recs)
{
    __shared__ float part[kWarps];
    __shared__ Step steps[kWarps][kCand];
    const int lane = (int) (threadIdx.x & 31), warp = (int) (threadIdx.x >> 5);
    const int c = (int) blockIdx.x;
    ChunkRec *rs = recs + (size_t) blockIdx.y * kChunks;
    const float *p = v + (size_t) blockIdx.y * count;
    /* the predicted start: the sums of the chunks before */
    float s = 0.0f;
    for (int k = (int) threadIdx.x; k < c; k += kThreads)
        s += rs[k].sum;
    for (int o = 16; o > 0; o >>= 1)
        s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0)
        part[warp] = s;
    __syncthreads();
    s = 0.0f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w)
        s += part[w];
    const int ex = (int) ((__float_as_uint(s) & 0x7fffffffu) >> 23);
    const int e0 = max(max(ex, 1) - 127 - 1, -126);
    size_t lo, hi;
    chunk_range(count, len, c, lo, hi);
    /* a warp folds a run of whole 32-element rows, each lane 4 adjacent
     * elements of a 128-element step */
    const size_t per = (hi - lo + 128 * kWarps - 1) / (128 * kWarps) * 128;
    const size_t w0 = min(lo + (size_t) warp * per, hi), w1 = min(w0 + per, hi);
    Step acc[kCand];
#pragma unroll
    for (int k = 0; k < kCand; ++k)
        acc[k].d0 = acc[k].d1 = 0u;
    for (size_t i = w0; i < w1; i += 128) {
        unsigned int b[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const size_t j = i + 4 * (size_t) lane + q;
            b[q] = j < w1 ? __float_as_uint(p[j]) : 0u;
        }
#pragma unroll
        for (int k = 0; k < kCand; ++k) {
            Step t = element(b[0], e0 + k);
#pragma unroll
            for (int q = 1; q < 4; ++q)
                t = compose(t, element(b[q], e0 + k));
            /* ordered fold of the 32 lanes: lane l takes [l, l + 2o) */
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                Step n;
                n.d0 = __shfl_down_sync(0xffffffffu, t.d0, o);
                n.d1 = __shfl_down_sync(0xffffffffu, t.d1, o);
                t = compose(t, n);
            }
            acc[k] = compose(acc[k], t);      /* lane 0's is the row's */
        }
    }
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < kCand; ++k)
            steps[warp][k] = acc[k];
    __syncthreads();
    if (threadIdx.x < kCand) {
        Step t = steps[0][threadIdx.x];
        for (int w = 1; w < kWarps; ++w)
            t = compose(t, steps[w][threadIdx.x]);
        rs[c].s[threadIdx.x] = t;
        if (threadIdx.x == 0)
            rs[c].e0 = e0;
    }
}

/* The sum after elements [lo, hi), from `bits` before them; all threads. */
__device__ unsigned int walk_chunk(const float *__restrict__ p, size_t lo, size_t hi, unsigned int bits,
                                   Step (&tot)[kWarps], unsigned int (&share)[2])
{
    const int t = (int) threadIdx.x, lane = t & 31, warp = t >> 5;
    const size_t seg = (hi - lo + kThreads - 1) / kThreads;
    const size_t a = min(lo + (size_t) t * seg, hi), b = min(a + seg, hi);
    int from = 0;      /* threads before this one have been added */
    while (from < kThreads && bits < 0x7f800000u) {
        int e;
        unsigned int m;
        split(bits, e, m);
        Step own;
        own.d0 = own.d1 = 0u;
        if (t >= from)
            for (size_t i = a; i < b; ++i)
                own = compose(own, element(__float_as_uint(p[i]), e));
        Step inc = warp_scan(own, lane);
        if (lane == 31)
            tot[warp] = inc;
        if (t == 0)
            share[0] = kThreads;
        __syncthreads();
        Step before;
        before.d0 = before.d1 = 0u;
        for (int w = 0; w < warp; ++w)
            before = compose(before, tot[w]);
        inc = compose(before, inc);
        const unsigned int end = m + ((m & 1u) ? inc.d1 : inc.d0);
        const unsigned int fail = __ballot_sync(0xffffffffu, end > kTop);
        if (fail && lane == 0)
            atomicMin(&share[0], (unsigned int) (32 * warp + __ffs((int) fail) - 1));
        __syncthreads();
        const int bad = (int) share[0];
        Step prev = shfl_up_step(inc, 1);
        if (lane == 0)
            prev = before;
        if (t == bad) {
            /* this segment leaves the binade: element by element */
            float sum = __uint_as_float(join(e, m + ((m & 1u) ? prev.d1 : prev.d0)));
            for (size_t i = a; i < b; ++i)
                sum = __fadd_rn(sum, fabsf(p[i]));
            share[1] = __float_as_uint(sum);
        }
        if (bad == kThreads && t == kThreads - 1)
            share[1] = join(e, end);
        __syncthreads();
        bits = share[1];
        from = bad + 1;
        __syncthreads();
    }
    return bits;
}

/* FULL: kChunks of them, known to the code generator (3 % of the walk). */
template <bool FULL>
__global__ void __launch_bounds__(kThreads) l1_walk_kernel(const float *__restrict__ v, size_t count, size_t any_len,
                                                           int any_chunks, const ChunkRec *__restrict__ recs, float *out)
{
    const int chunks = FULL ? kChunks : any_chunks;
    const size_t len = FULL ? (count + kChunks - 1) / kChunks : any_len;
    __shared__ ChunkRec rs[kChunks];
    __shared__ float head[kHead];
    __shared__ Step tot[kWarps];
    __shared__ unsigned int share[2];
    __shared__ int next;
    const float *p = v + (size_t) blockIdx.x * count;
    const int lane = (int) (threadIdx.x & 31), warp = (int) (threadIdx.x >> 5);
    bool nan = false;
    for (int c = (int) threadIdx.x; c < chunks; c += kThreads) {
        rs[c] = recs[(size_t) blockIdx.x * kChunks + c];
        nan = nan || rs[c].sum != rs[c].sum;
    }
    if (__syncthreads_or(nan)) {        /* a sum of magnitudes is NaN only through a NaN */
        if (threadIdx.x == 0)
            out[blockIdx.x] = __uint_as_float(0x7fffffffu);
        return;
    }
    /* the first elements, where a binade lasts a few of them, one by one */
    unsigned int bits = 0u;
    int c = 0;
    {
        size_t lo, hi;
        chunk_range(count, len, 0, lo, hi);
        const int n_head = (int) min(hi, (size_t) kHead);
        for (int i = (int) threadIdx.x; i < kHead; i += kThreads)
            head[i] = i < n_head ? fabsf(p[i]) : 0.0f;
        __syncthreads();
        if (threadIdx.x == 0) {
            float sum = 0.0f;
            for (int i = 0; i < n_head; i += 16) {
#pragma unroll
                for (int q = 0; q < 16; ++q)
                    sum = __fadd_rn(sum, head[i + q]);
            }
            share[1] = __float_as_uint(sum);
        }
        __syncthreads();
        bits = share[1];
        __syncthreads();
        if ((size_t) n_head < hi)
            bits = walk_chunk(p, (size_t) n_head, hi, bits, tot, share);
        c = 1;
    }
    while (c < chunks && bits < 0x7f800000u) {
        if (warp == 0) {
            for (;;) {
                int e;
                unsigned int m;
                split(bits, e, m);
                Step s;
                s.d0 = s.d1 = 0u;
                if (c + lane < chunks) {
                    const int k = e - rs[c + lane].e0;
                    if (k >= 0 && k < kCand)
                        s = rs[c + lane].s[k];
                    else
                        s.d0 = s.d1 = kMany;
                }
                s = warp_scan(s, lane);
                const unsigned int end = m + ((m & 1u) ? s.d1 : s.d0);
                const unsigned int fail = __ballot_sync(0xffffffffu, end > kTop);
                const int good = fail ? __ffs((int) fail) - 1 : 32;
                if (good > 0)
                    bits = join(e, __shfl_sync(0xffffffffu, end, max(good, 1) - 1));
                c += good;
                if (good < 32 || c >= chunks || bits >= 0x7f800000u)
                    break;
            }
            if (lane == 0) {
                share[1] = bits;
                next = min(c, chunks);
            }
        }
        __syncthreads();
        bits = share[1];
        c = next;
        __syncthreads();
        if (c >= chunks || bits >= 0x7f800000u)
            break;
        size_t lo, hi;
        chunk_range(count, len, c, lo, hi);
        bits = walk_chunk(p, lo, hi, bits, tot, share);
        ++c;
    }
    if (threadIdx.x == 0)
        out[blockIdx.x] = __uint_as_float(bits);
}

/* The plain sum of a short slice: one thread adds from shared memory (4 cycles
 * an element) while the next elements are on their way. */
__global__ void __launch_bounds__(kThreads) l1_short_kernel(const float *__restrict__ v, int count, float *out)
{
    __shared__ __align__(16) float part[kHead];
    const float *p = v + (size_t) blockIdx.x * count;
    constexpr int kEach = kHead / kThreads;
    float next[kEach];
    auto load = [&](int i0) {
#pragma unroll
        for (int q = 0; q < kEach; ++q) {
            const int i = i0 + q * kThreads + (int) threadIdx.x;
            next[q] = i < count ? fabsf(p[i]) : 0.0f;
        }
    };
    float sum = 0.0f;
    load(0);
    for (int i0 = 0; i0 < count; i0 += kHead) {
#pragma unroll
        for (int q = 0; q < kEach; ++q)
            part[q * kThreads + threadIdx.x] = next[q];
        __syncthreads();
        load(i0 + kHead);
        if (threadIdx.x == 0) {
            const int n = min(kHead, count - i0);
            for (int i = 0; i < n; i += 16) {      /* zeros after the end */
#pragma unroll
                for (int q = 0; q < 16; ++q)
                    sum = __fadd_rn(sum, part[i + q]);
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
        out[blockIdx.x] = sum;
}

}  // namespace

extern "C" size_t udev_l1_partials(int n_slices)
{
    return 4 * (size_t) kChunks * (size_t) (n_slices > 0 ? n_slices : 0);
}

int udev_l1_compat(udev *d, const float *v, size_t count, int n_slices, double *scratch, float *d_out)
{
    ChunkRec *recs = reinterpret_cast<ChunkRec *>(scratch);
    int rc;
    if (count <= kShort) {
        l1_short_kernel<<<(unsigned int) n_slices, kThreads, 0, d->stream>>>(v, (int) count, d_out);
        return udev_after_launch(d, "l1_short_kernel");
    }
    const size_t fit = count / kMinChunk;
    const int chunks = fit < (size_t) kChunks ? (int) fit : kChunks;
    const size_t len = (count + chunks - 1) / chunks;
    const dim3 grid((unsigned int) chunks, (unsigned int) n_slices);
    l1_sums_kernel<<<grid, kThreads, 0, d->stream>>>(v, count, len, recs);
    if ((rc = udev_after_launch(d, "l1_sums_kernel")))
        return rc;
    l1_steps_kernel<<<grid, kThreads, 0, d->stream>>>(v, count, len, recs);
    if ((rc = udev_after_launch(d, "l1_steps_kernel")))
        return rc;
    if (chunks == kChunks)
        l1_walk_kernel<true><<<(unsigned int) n_slices, kThreads, 0, d->stream>>>(v, count, len, chunks, recs, d_out);
    else
        l1_walk_kernel<false><<<(unsigned int) n_slices, kThreads, 0, d->stream>>>(v, count, len, chunks, recs, d_out);
    return udev_after_launch(d, "l1_walk_kernel");
}
