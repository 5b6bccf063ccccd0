/*
 * udev_ops.cu - element-wise ops, TV subgradient, periodic differences and
 * the deterministic reductions used by the methods.
 *
 * Element-wise ops replace ufo-ir-basic-ops.cl:4-171,255-273 and the host
 * loops of ufo-ir-basic-ops-processor.c:324-430,544-604; every operation
 * rounds as the reference's (IEEE float, no contraction).
 * l1_grad replaces ufo-math-tvstd-method.cl:5-57, Dx/Dxt/Dy/Dyt replace
 * ufo-ir-gradient-processor.cl:1-51.
 *
 * Reductions (replacing the reference's host loops, ufo-ir-basic-ops.c:259-277
 * and ufo-ir-basic-ops-processor.c:148-247):
 *   COMPAT mode reproduces the float sequential sums bit for bit (the L1
 *   norm in udev_norm.cu);
 *   FP64 mode sums the same terms in double with a fixed-shape tree (the
 *   same result on every run), then rounds to float.
 */
#include <cuda_runtime.h>

#include "udev_internal.cuh"

namespace {

__global__ void fill_kernel(float *p, size_t n, float v)
{
    for (size_t i = blockIdx.x * (size_t) blockDim.x + threadIdx.x; i < n;
         i += (size_t) gridDim.x * blockDim.x)
        p[i] = v;
}

template <int OP>
__device__ __forceinline__ float binop(float a, float b, float m)
{
    if (OP == UDEV_MUL)
        return __fmul_rn(a, b);
    if (OP == UDEV_ADD)
        return __fadd_rn(a, b);
    if (OP == UDEV_SUB)
        return __fsub_rn(a, b);
    if (OP == UDEV_SUB_SCALED)
        return __fsub_rn(a, __fmul_rn(m, b));
    if (OP == UDEV_ADD_SCALED)
        return __fadd_rn(a, __fmul_rn(m, b));
    if (OP == UDEV_MAX)
        return fmaxf(a, b);
    return __fdiv_rn(a, b);
}

template <int OP>
__global__ void binary_kernel(const float *a, const float *b, float m, float *out, size_t n)
{
    for (size_t i = blockIdx.x * (size_t) blockDim.x + threadIdx.x; i < n;
         i += (size_t) gridDim.x * blockDim.x)
        out[i] = binop<OP>(a[i], b[i], m);
}

template <int OP>
__device__ __forceinline__ float unop(float a, float m, float m2)
{
    if (OP == UDEV_INV)
        return a != 0.0f ? __fdiv_rn(1.0f, a) : 0.0f;
    if (OP == UDEV_POSC)
        return a > 0.0f ? a : 0.0f;
    if (OP == UDEV_SQRT)
        return __fsqrt_rn(a);
    if (OP == UDEV_SCALE)
        return __fmul_rn(a, m);
    if (OP == UDEV_ADDC)
        return __fadd_rn(m, a);
    if (OP == UDEV_MAXC)
        return fmaxf(a, m);
    /* UDEV_NORMALIZE: delta * v - min * delta (ufo-ir-basic-ops-processor.c:365) */
    return __fsub_rn(__fmul_rn(m, a), __fmul_rn(m2, m));
}

template <int OP>
__global__ void unary_kernel(const float *a, float m, float m2, float *out, size_t n)
{
    for (size_t i = blockIdx.x * (size_t) blockDim.x + threadIdx.x; i < n;
         i += (size_t) gridDim.x * blockDim.x)
        out[i] = unop<OP>(a[i], m, m2);
}

__device__ __forceinline__ float tex0(const float *img, int x, int y, int w, int h)
{
    return (x >= 0 && y >= 0 && x < w && y < h) ? img[(size_t) y * w + x] : 0.0f;
}

template <int WHICH>
__global__ void diff_kernel(const float *in, float *out, int w, int h, long long stride)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h)
        return;
    const size_t base = (size_t) blockIdx.z * stride;
    const long long idx = (long long) y * w + x;
    const long long last = (long long) w * h;
    long long j;
    if (WHICH == UDEV_DX)
        j = idx - 1 + (x == 0 ? w : 0);
    else if (WHICH == UDEV_DXT)
        j = idx + 1 - (x == w - 1 ? w : 0);
    else if (WHICH == UDEV_DY)
        j = idx - w + (y == 0 ? last : 0);
    else
        j = idx + w - (y == h - 1 ? last : 0);
    out[base + idx] = __fsub_rn(in[base + idx], in[base + j]);
}

/* ---------------- reductions ---------------- */

constexpr int kRedThreads = 256;
constexpr int kRedBlocks = 512;   /* partial sums per slice in FP64 mode */

__device__ __forceinline__ double block_sum_double(double v)
{
    __shared__ double warp_sums[kRedThreads / 32];
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_down_sync(0xffffffffu, v, o);
    const int tid = (int) (threadIdx.y * blockDim.x + threadIdx.x), lane = tid & 31, wid = tid >> 5;
    if (lane == 0)
        warp_sums[wid] = v;
    __syncthreads();
    double r = 0.0;
    if (wid == 0) {
        r = lane < kRedThreads / 32 ? warp_sums[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1)
            r += __shfl_down_sync(0xffffffffu, r, o);
    }
    return r;   /* valid in thread 0 */
}

/* l1_grad: 7-point isotropic-TV subgradient with EPS 0.001 and zero border.
 * With NORM also the FP64 sum of its magnitudes, one partial per CTA.
 *
 * A CTA takes 32 x 32 tiles in turn, 4 rows per thread, from the tile and its
 * one-pixel halo staged in shared memory (zeros outside the image). Bound by
 * issue: three divisions and square roots per pixel. The root under the
 * second term is the first term's of the pixel to the right, taken from the
 * next lane; lanes 0 .. 3 compute those right of the tile, one row each. The
 * FP64 additions and conversions (2 per clock and SM) run beside it, so the
 * norm costs little: the gradient and its norm took 38 + 40 us at 2900^2 (11 +
 * 12 at 1448^2, 11 + 16 for four slices of 724^2) as two kernels, and take 55
 * (17, 21) here. */
constexpr int kGradTile = 32;
constexpr int kGradRows = kGradTile / 8;
/* CTAs and partial sums per slice at most: what 152 SMs run at once (the
 * reduction scratch holds 2048). Not by the number of slices or of SMs, as the
 * sum's grouping follows it and a slice is to have one norm in any stack.
 * (Gradient calls of 4 x 724^2 35 -> 31 us and 3 x 2900^2 212 -> 150 against
 * 1216 CTAs shared among the slices.) */
constexpr int kGradBlocks = 1216;

template <bool NORM>
__global__ void __launch_bounds__(256) l1_grad_kernel(const float *in, float *out, int w, int h, long long stride,
                                                      double *partials)
{
    __shared__ float t[kGradTile + 2][kGradTile + 3];
    const int tiles_x = (w + kGradTile - 1) / kGradTile, tiles = tiles_x * ((h + kGradTile - 1) / kGradTile);
    const float *img = in + (size_t) blockIdx.y * stride;
    float *dst = out + (size_t) blockIdx.y * stride;
    const int lane = (int) threadIdx.x, lx = lane + 1;
    const float eps = 0.001f;
    double acc = 0.0;
    for (int tile = (int) blockIdx.x; tile < tiles; tile += (int) gridDim.x) {
        const int x0 = tile % tiles_x * kGradTile, y0 = tile / tiles_x * kGradTile;
        /* a warp stages whole rows: its 32 columns, then lanes 0 and 1 the two at the end */
        for (int ty = (int) threadIdx.y; ty < kGradTile + 2; ty += 8) {
            t[ty][lane] = tex0(img, x0 - 1 + lane, y0 - 1 + ty, w, h);
            if (lane < 2)
                t[ty][kGradTile + lane] = tex0(img, x0 - 1 + kGradTile + lane, y0 - 1 + ty, w, h);
        }
        __syncthreads();
        /* sqrt(eps + (f(x, y) - f(x - 1, y))^2 + (f(x, y) - f(x, y + 1))^2) at the pixel right of the tile */
        const int er = (int) threadIdx.y + 8 * (lane & (kGradRows - 1)) + 1;
        const float ef = t[er][kGradTile + 1];
        const float eh = __fsub_rn(ef, t[er][kGradTile]), ev = __fsub_rn(ef, t[er + 1][kGradTile + 1]);
        const float edge = __fsqrt_rn(__fadd_rn(__fadd_rn(eps, __fmul_rn(eh, eh)), __fmul_rn(ev, ev)));
#pragma unroll 4
        for (int m = 0; m < kGradRows; ++m) {
            const int ly = (int) threadIdx.y + 8 * m + 1, y = y0 + ly - 1, x = x0 + lane;
            const float f3 = t[ly][lx];
            const float f1 = t[ly - 1][lx];
            const float f0 = t[ly - 1][lx - 1];
            const float f2 = t[ly][lx - 1];
            const float f4 = t[ly][lx + 1];
            const float f5 = t[ly + 1][lx];
            const float d32 = __fsub_rn(f3, f2), d35 = __fsub_rn(f3, f5);
            const float d43 = __fsub_rn(f4, f3);
            const float d13 = __fsub_rn(f1, f3), d10 = __fsub_rn(f1, f0);
            const float n1 = __fsqrt_rn(__fadd_rn(__fadd_rn(eps, __fmul_rn(d32, d32)), __fmul_rn(d35, d35)));
            const float n3 = __fsqrt_rn(__fadd_rn(__fadd_rn(eps, __fmul_rn(d13, d13)), __fmul_rn(d10, d10)));
            const float right = __shfl_down_sync(0xffffffffu, n1, 1), last = __shfl_sync(0xffffffffu, edge, m);
            const float n2 = lane == 31 ? last : right;
            const float t1 = __fdiv_rn(__fsub_rn(__fsub_rn(__fmul_rn(2.0f, f3), f2), f5), n1);
            const float t2 = __fdiv_rn(d43, n2);
            const float t3 = __fdiv_rn(d13, n3);
            const float g = __fsub_rn(__fsub_rn(t1, t2), t3);
            if (x < w && y < h) {
                dst[(size_t) y * w + x] = g;
                if (NORM)
                    acc += (double) fabsf(g);
            }
        }
        __syncthreads();
    }
    if (NORM) {
        acc = block_sum_double(acc);
        if (threadIdx.x == 0 && threadIdx.y == 0)
            partials[(size_t) blockIdx.y * gridDim.x + blockIdx.x] = acc;
    }
}

/* FP64 l1, pass 1: block b of slice s sums a fixed contiguous chunk. */
__global__ void __launch_bounds__(kRedThreads) l1_fp64_partial_kernel(const float *v, size_t count,
                                                                      long long stride, double *partials)
{
    const float *p = v + (size_t) blockIdx.y * stride;
    const size_t chunk = (count + gridDim.x - 1) / gridDim.x;
    const size_t lo = (size_t) blockIdx.x * chunk;
    const size_t hi = lo + chunk < count ? lo + chunk : count;
    double acc = 0.0;
    for (size_t i = lo + threadIdx.x; i < hi; i += kRedThreads)
        acc += (double) fabsf(p[i]);
    acc = block_sum_double(acc);
    if (threadIdx.x == 0)
        partials[(size_t) blockIdx.y * gridDim.x + blockIdx.x] = acc;
}

/* FP64 pass 2: one block per slice sums its partials in a fixed tree. */
__global__ void __launch_bounds__(kRedThreads) sum_partials_kernel(const double *partials, int per_slice,
                                                                   float *out)
{
    const double *p = partials + (size_t) blockIdx.x * per_slice;
    double acc = 0.0;
    for (int i = threadIdx.x; i < per_slice; i += kRedThreads)
        acc += p[i];
    acc = block_sum_double(acc);
    if (threadIdx.x == 0)
        out[blockIdx.x] = (float) acc;
}

/* dot product of ufo_ir_basic_ops_processor_dot_product: for part p < h,
 * partial[p] = sum_{i < w} a[p*i] * b[p*i]; the result sums the partials
 * in order. The reads of a part lie p elements apart, one 32-byte sector
 * each, so the time is how many of them are in flight. */

/* FP64: a warp per part, its lanes' sums folded by shuffles. (One thread per
 * part: 155 us for four slices of 724^2, this: 17 us.) */
__global__ void __launch_bounds__(128) dot_parts_fp64_kernel(const float *a, const float *b, unsigned int w,
                                                             unsigned int h, long long stride, double *parts)
{
    const unsigned int part = blockIdx.x * 4u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (part >= h)
        return;
    const float *pa = a + (size_t) blockIdx.y * stride;
    const float *pb = b + (size_t) blockIdx.y * stride;
    double acc = 0.0;
    unsigned int i = lane;
    for (; i + 224u < w; i += 256u) {
        float x[8], y[8];
#pragma unroll
        for (unsigned int k = 0; k < 8; ++k) {
            x[k] = pa[part * (i + 32u * k)];
            y[k] = pb[part * (i + 32u * k)];
        }
#pragma unroll
        for (int k = 0; k < 8; ++k)
            acc += (double) x[k] * (double) y[k];
    }
    for (; i < w; i += 32u)
        acc += (double) pa[part * i] * (double) pb[part * i];
    for (int o = 16; o > 0; o >>= 1)
        acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0)
        parts[(size_t) blockIdx.y * h + part] = acc;
}

/* COMPAT: a thread adds its part in order, 16 pairs of loads in flight. */
__global__ void __launch_bounds__(32) dot_parts_compat_kernel(const float *a, const float *b, unsigned int w,
                                                              unsigned int h, long long stride, double *parts)
{
    const unsigned int part = blockIdx.x * 32u + threadIdx.x;
    if (part >= h)
        return;
    const float *pa = a + (size_t) blockIdx.y * stride;
    const float *pb = b + (size_t) blockIdx.y * stride;
    float acc = 0.0f;
    unsigned int i = 0;
    for (; i + 16u <= w; i += 16u) {
        float x[16], y[16];
#pragma unroll
        for (unsigned int k = 0; k < 16; ++k) {
            x[k] = pa[part * (i + k)];
            y[k] = pb[part * (i + k)];
        }
#pragma unroll
        for (int k = 0; k < 16; ++k)
            acc = __fadd_rn(acc, __fmul_rn(x[k], y[k]));
    }
    for (; i < w; i++)
        acc = __fadd_rn(acc, __fmul_rn(pa[part * i], pb[part * i]));
    parts[(size_t) blockIdx.y * h + part] = (double) acc;
}

/* The parts in order: a warp loads 32 of them at a time and adds them one
 * after another from its lanes. */
__global__ void dot_compat_sum_kernel(const double *parts, unsigned int h, float *out)
{
    const double *p = parts + (size_t) blockIdx.x * h;
    float norm = 0.0f;
    float next = threadIdx.x < h ? (float) p[threadIdx.x] : 0.0f;
    for (unsigned int i = 0; i < h; i += 32) {
        const float v = next;
        if (i + 32 + threadIdx.x < h)
            next = (float) p[i + 32 + threadIdx.x];
        const int left = (int) min(32u, h - i);
        for (int k = 0; k < left; ++k)
            norm = __fadd_rn(norm, __shfl_sync(0xffffffffu, v, k));
    }
    if (threadIdx.x == 0)
        out[blockIdx.x] = norm;
}

constexpr int kMinMaxBlocks = 64;

__device__ __forceinline__ void block_minmax(float lo, float hi, float *out)
{
    __shared__ float smin[kRedThreads / 32], smax[kRedThreads / 32];
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_down_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_down_sync(0xffffffffu, hi, o));
    }
    if ((threadIdx.x & 31) == 0) {
        smin[threadIdx.x >> 5] = lo;
        smax[threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < kRedThreads / 32; ++k) {
            lo = fminf(lo, smin[k]);
            hi = fmaxf(hi, smax[k]);
        }
        out[0] = lo;
        out[1] = hi;
    }
}

/* Minimum and maximum of block b's share of slice s (one block per slice
 * took 31 us for 724 x 360). */
__global__ void __launch_bounds__(kRedThreads) minmax_kernel(const float *v, size_t count, long long stride,
                                                             float *out)
{
    const float *p = v + (size_t) blockIdx.y * stride;
    float lo = 3.402823466e38f, hi = -3.402823466e38f;
    for (size_t i = (size_t) blockIdx.x * kRedThreads + threadIdx.x; i < count;
         i += (size_t) gridDim.x * kRedThreads) {
        lo = fminf(lo, p[i]);
        hi = fmaxf(hi, p[i]);
    }
    block_minmax(lo, hi, out + 2 * ((size_t) blockIdx.y * gridDim.x + blockIdx.x));
}

__global__ void __launch_bounds__(kRedThreads) minmax_final_kernel(const float *parts, int n_parts, float *out)
{
    const float *p = parts + 2 * (size_t) blockIdx.x * n_parts;
    float lo = 3.402823466e38f, hi = -3.402823466e38f;
    for (int i = (int) threadIdx.x; i < n_parts; i += kRedThreads) {
        lo = fminf(lo, p[2 * i]);
        hi = fmaxf(hi, p[2 * i + 1]);
    }
    block_minmax(lo, hi, out + 2 * blockIdx.x);
}

unsigned int grid_for(udev *d, size_t n)
{
    size_t blocks = (n + 255) / 256;
    const size_t cap = (size_t) d->sm_count * 8;
    if (blocks > cap)
        blocks = cap;
    return (unsigned int) (blocks ? blocks : 1);
}

}  // namespace

extern "C" int udev_fill(udev *d, float *p, size_t n, float v)
{
    if (n == 0)
        return UFOIR_OK;
    UDEV_BIND(d);
    fill_kernel<<<grid_for(d, n), 256, 0, d->stream>>>(p, n, v);
    return udev_after_launch(d, "fill_kernel");
}

extern "C" int udev_binary(udev *d, int op, const float *a, const float *b, float m, float *out, size_t n)
{
    if (n == 0)
        return UFOIR_OK;
    UDEV_BIND(d);
    const unsigned int g = grid_for(d, n);
    switch (op) {
    case UDEV_MUL: binary_kernel<UDEV_MUL><<<g, 256, 0, d->stream>>>(a, b, m, out, n); break;
    case UDEV_ADD: binary_kernel<UDEV_ADD><<<g, 256, 0, d->stream>>>(a, b, m, out, n); break;
    case UDEV_SUB: binary_kernel<UDEV_SUB><<<g, 256, 0, d->stream>>>(a, b, m, out, n); break;
    case UDEV_SUB_SCALED: binary_kernel<UDEV_SUB_SCALED><<<g, 256, 0, d->stream>>>(a, b, m, out, n); break;
    case UDEV_ADD_SCALED: binary_kernel<UDEV_ADD_SCALED><<<g, 256, 0, d->stream>>>(a, b, m, out, n); break;
    case UDEV_MAX: binary_kernel<UDEV_MAX><<<g, 256, 0, d->stream>>>(a, b, m, out, n); break;
    case UDEV_DIV: binary_kernel<UDEV_DIV><<<g, 256, 0, d->stream>>>(a, b, m, out, n); break;
    default:
        udev_set_error(d, "unknown binary op %d", op);
        return UFOIR_ERR_INVALID;
    }
    return udev_after_launch(d, "binary_kernel");
}

extern "C" int udev_unary(udev *d, int op, const float *a, float m, float m2, float *out, size_t n)
{
    if (n == 0)
        return UFOIR_OK;
    UDEV_BIND(d);
    const unsigned int g = grid_for(d, n);
    switch (op) {
    case UDEV_INV: unary_kernel<UDEV_INV><<<g, 256, 0, d->stream>>>(a, m, m2, out, n); break;
    case UDEV_POSC: unary_kernel<UDEV_POSC><<<g, 256, 0, d->stream>>>(a, m, m2, out, n); break;
    case UDEV_SQRT: unary_kernel<UDEV_SQRT><<<g, 256, 0, d->stream>>>(a, m, m2, out, n); break;
    case UDEV_SCALE: unary_kernel<UDEV_SCALE><<<g, 256, 0, d->stream>>>(a, m, m2, out, n); break;
    case UDEV_ADDC: unary_kernel<UDEV_ADDC><<<g, 256, 0, d->stream>>>(a, m, m2, out, n); break;
    case UDEV_MAXC: unary_kernel<UDEV_MAXC><<<g, 256, 0, d->stream>>>(a, m, m2, out, n); break;
    case UDEV_NORMALIZE: unary_kernel<UDEV_NORMALIZE><<<g, 256, 0, d->stream>>>(a, m, m2, out, n); break;
    default:
        udev_set_error(d, "unknown unary op %d", op);
        return UFOIR_ERR_INVALID;
    }
    return udev_after_launch(d, "unary_kernel");
}

/* CTAs per slice for the gradient. */
static unsigned int grad_blocks(int w, int h)
{
    const long long tiles = (long long) udev_div_up(w, kGradTile) * udev_div_up(h, kGradTile);
    return (unsigned int) (tiles < kGradBlocks ? tiles : kGradBlocks);
}

extern "C" int udev_l1_grad(udev *d, const float *in, float *out, int w, int h, int n_slices)
{
    if (n_slices <= 0)
        return UFOIR_OK;
    UDEV_BIND(d);
    const dim3 grid(grad_blocks(w, h), (unsigned int) n_slices);
    l1_grad_kernel<false><<<grid, dim3(32, 8), 0, d->stream>>>(in, out, w, h, (long long) w * h, nullptr);
    return udev_after_launch(d, "l1_grad_kernel");
}

extern "C" int udev_l1_grad_norm(udev *d, const float *in, float *out, int w, int h, int n_slices, int mode,
                                 double *partials, float *d_out)
{
    int rc;
    if (n_slices <= 0)
        return UFOIR_OK;
    if (mode == UFOIR_NORM_COMPAT) {
        if ((rc = udev_l1_grad(d, in, out, w, h, n_slices)))
            return rc;
        return udev_l1_norm_to(d, out, (size_t) w, (size_t) h, n_slices, mode, partials, d_out);
    }
    UDEV_BIND(d);
    const dim3 grid(grad_blocks(w, h), (unsigned int) n_slices);
    l1_grad_kernel<true><<<grid, dim3(32, 8), 0, d->stream>>>(in, out, w, h, (long long) w * h, partials);
    if ((rc = udev_after_launch(d, "l1_grad_kernel")))
        return rc;
    sum_partials_kernel<<<n_slices, kRedThreads, 0, d->stream>>>(partials, (int) grid.x, d_out);
    return udev_after_launch(d, "sum_partials_kernel");
}

extern "C" int udev_diff(udev *d, int which, const float *in, float *out, int w, int h, int n_slices)
{
    if (n_slices <= 0)
        return UFOIR_OK;
    UDEV_BIND(d);
    dim3 grid(udev_div_up(w, 32), udev_div_up(h, 8), (unsigned int) n_slices);
    const long long stride = (long long) w * h;
    switch (which) {
    case UDEV_DX: diff_kernel<UDEV_DX><<<grid, dim3(32, 8), 0, d->stream>>>(in, out, w, h, stride); break;
    case UDEV_DXT: diff_kernel<UDEV_DXT><<<grid, dim3(32, 8), 0, d->stream>>>(in, out, w, h, stride); break;
    case UDEV_DY: diff_kernel<UDEV_DY><<<grid, dim3(32, 8), 0, d->stream>>>(in, out, w, h, stride); break;
    case UDEV_DYT: diff_kernel<UDEV_DYT><<<grid, dim3(32, 8), 0, d->stream>>>(in, out, w, h, stride); break;
    default:
        udev_set_error(d, "unknown difference %d", which);
        return UFOIR_ERR_INVALID;
    }
    return udev_after_launch(d, "diff_kernel");
}

extern "C" int udev_l1_norm(udev *d, const float *v, size_t w, size_t h, int n_slices, int mode,
                            float *host_out)
{
    if (n_slices <= 0)
        return UFOIR_OK;
    UDEV_BIND(d);
    int rc = udev_reduction_scratch(d, udev_l1_partials(n_slices), (size_t) n_slices);
    if (!rc)
        rc = udev_l1_norm_to(d, v, w, h, n_slices, mode, d->red_partials, d->red_out);
    if (rc)
        return rc;
    UDEV_CHECK(d, cudaMemcpyAsync(d->h_red, d->red_out, sizeof(float) * n_slices, cudaMemcpyDeviceToHost, d->stream));
    UDEV_CHECK(d, cudaStreamSynchronize(d->stream));
    for (int i = 0; i < n_slices; i++)
        host_out[i] = d->h_red[i];
    return UFOIR_OK;
}

extern "C" int udev_l1_norm_to(udev *d, const float *v, size_t w, size_t h, int n_slices, int mode, double *partials,
                               float *d_out)
{
    if (n_slices <= 0)
        return UFOIR_OK;
    UDEV_BIND(d);
    const size_t count = w * h;
    int rc;
    if (mode == UFOIR_NORM_COMPAT)
        return udev_l1_compat(d, v, count, n_slices, partials, d_out);
    l1_fp64_partial_kernel<<<dim3(kRedBlocks, n_slices), kRedThreads, 0, d->stream>>>(v, count, (long long) count,
                                                                                       partials);
    if ((rc = udev_after_launch(d, "l1_fp64_partial_kernel")))
        return rc;
    sum_partials_kernel<<<n_slices, kRedThreads, 0, d->stream>>>(partials, kRedBlocks, d_out);
    return udev_after_launch(d, "sum_partials_kernel");
}

extern "C" int udev_dots(udev *d, int pairs, const float *const *a, const float *const *b, size_t w, size_t h,
                         int n_slices, int mode, float *host_out)
{
    if (n_slices <= 0 || pairs <= 0)
        return UFOIR_OK;
    if (w * h > 0xffffffffull) {
        udev_set_error(d, "dot: %zu elements exceed the 32-bit index of the reference", w * h);
        return UFOIR_ERR_INVALID;
    }
    UDEV_BIND(d);
    const size_t outs = (size_t) pairs * n_slices;
    int rc = udev_reduction_scratch(d, h * outs, outs);
    if (rc)
        return rc;
    const long long stride = (long long) (w * h);
    for (int k = 0; k < pairs; ++k) {
        double *parts = d->red_partials + (size_t) k * h * n_slices;
        if (mode == UFOIR_NORM_COMPAT)
            dot_parts_compat_kernel<<<dim3(udev_div_up(h, 32), (unsigned int) n_slices), 32, 0, d->stream>>>(
                a[k], b[k], (unsigned int) w, (unsigned int) h, stride, parts);
        else
            dot_parts_fp64_kernel<<<dim3(udev_div_up(h, 4), (unsigned int) n_slices), 128, 0, d->stream>>>(
                a[k], b[k], (unsigned int) w, (unsigned int) h, stride, parts);
        if ((rc = udev_after_launch(d, "dot_parts_kernel")))
            return rc;
    }
    if (mode == UFOIR_NORM_COMPAT)
        dot_compat_sum_kernel<<<(unsigned int) outs, 32, 0, d->stream>>>(d->red_partials, (unsigned int) h, d->red_out);
    else
        sum_partials_kernel<<<(unsigned int) outs, kRedThreads, 0, d->stream>>>(d->red_partials, (int) h, d->red_out);
    if ((rc = udev_after_launch(d, "sum_partials_kernel")))
        return rc;
    UDEV_CHECK(d, cudaMemcpyAsync(d->h_red, d->red_out, sizeof(float) * outs, cudaMemcpyDeviceToHost, d->stream));
    UDEV_CHECK(d, cudaStreamSynchronize(d->stream));
    for (size_t i = 0; i < outs; i++)
        host_out[i] = d->h_red[i];
    return UFOIR_OK;
}

extern "C" int udev_minmax(udev *d, const float *v, size_t n, int n_slices, float *host_min, float *host_max)
{
    if (n_slices <= 0)
        return UFOIR_OK;
    UDEV_BIND(d);
    /* two floats a block fit the doubles of the scratch */
    int rc = udev_reduction_scratch(d, (size_t) kMinMaxBlocks * n_slices, (size_t) n_slices);
    if (rc)
        return rc;
    float *parts = reinterpret_cast<float *>(d->red_partials);
    minmax_kernel<<<dim3(kMinMaxBlocks, (unsigned int) n_slices), kRedThreads, 0, d->stream>>>(v, n, (long long) n,
                                                                                              parts);
    if ((rc = udev_after_launch(d, "minmax_kernel")))
        return rc;
    minmax_final_kernel<<<n_slices, kRedThreads, 0, d->stream>>>(parts, kMinMaxBlocks, d->red_out);
    if ((rc = udev_after_launch(d, "minmax_final_kernel")))
        return rc;
    UDEV_CHECK(d, cudaMemcpyAsync(d->h_red, d->red_out, 2 * sizeof(float) * n_slices, cudaMemcpyDeviceToHost, d->stream));
    UDEV_CHECK(d, cudaStreamSynchronize(d->stream));
    for (int i = 0; i < n_slices; i++) {
        host_min[i] = d->h_red[2 * i];
        host_max[i] = d->h_red[2 * i + 1];
    }
    return UFOIR_OK;
}
