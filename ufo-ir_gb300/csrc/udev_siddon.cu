/*
 * udev_siddon.cu - the "siddon" projector model: exact line integrals of the
 * pixel image (piecewise constant), and their exact adjoint.
 *
 * The reference ships only the Joseph model, but its projector exposes a
 * "model" property for others (parallel-projector-task.c:123-128). This
 * model keeps the geometry of the reference's backprojector
 * (projector-parallel-joseph.cl:174-195): pixel (i, j) covers
 * X in [i - n/2, i + 1 - n/2], Y in [j - n/2, j + 1 - n/2], and detector
 * bin k of angle theta is the line X cos - Y sin + axis = k + 0.5 (cos, sin
 * from the float LUT; lengths are measured with the line's normal scaled to
 * unit length, as sin^2 + cos^2 of the LUT is not exactly 1). The ray
 * of a bin meets pixel (i, j) over the chord of a line through a unit
 * square: with a = |cos|, b = |sin| and d the distance of the line from the
 * pixel centre, measured along the detector,
 *   L(d) = 1 / max(a, b)                 for |d| <= |a - b| / 2,
 *   L(d) = ((a + b) / 2 - |d|) / (a b)   up to |d| = (a + b) / 2, 0 beyond.
 *
 * Forward: a ray walks the slabs (rows for |cos| >= |sin|, columns
 * otherwise) of the zero-padded image or its padded transpose, the copies the
 * Joseph forward projector reads; in a slab it covers at most two pixels, and
 * its length in the slab (1 / max(a, b)) splits where it crosses the pixel
 * boundary. Whole angle sets run in the Joseph projector's tiles
 * (udev_fp_tiles.cu, 1.62 -> 1.03 ms for one slice of 1448^2 x 1200) where those
 * are many and full enough (siddon_tiles_pay); the kernel here, one thread per
 * ray, serves the other sets, subsets and sizes beyond the tiles'.
 * Backward: one register sum per pixel evaluates L for the (at most two) bins
 * whose lines cross the pixel, per angle. Both compute the same
 * chord lengths, so the backprojector is the adjoint of the forward one up
 * to rounding. Arithmetic is FP32; the sums are per ray in slab order and
 * per pixel in angle order, with the reference's contract for accumulation
 * (sino = src + scale * S; per subset v = v + relax * sum).
 */
#include <cuda_runtime.h>

#include "bp_shapes.cuh"
#include "joseph.cuh"
#include "udev_internal.cuh"

namespace {

struct SiddonFpArgs {
    const float *volP;      /* padded image rows (walked by row-mode rays) */
    const float *volTP;     /* padded transposed rows (column-mode rays) */
    const float *src;
    const float *w;
    float *out;
    const float *sinv;
    const float *cosv;
    int n;
    int a0;
    int na;
    int pitch;
    float axis;
    float scale;
    long long volp_stride;
    long long sino_stride;
    long long w_stride;
};

constexpr int kPadL = 2;                       /* zero columns left of a padded row */
constexpr float kFloorMagic = 12582912.0f;     /* 1.5 * 2^23 */
constexpr int kFloorMagicBits = 0x4B400000;

/*
 * Grid (ceil(n / 128), na, slices), 128 threads: thread = detector bin.
 * A ray walks the rows of the padded image (rows for |cos| >= |sin|, else
 * the rows of the padded transpose, i.e. the image's columns) with the
 * coordinate across the slab at its lower edge, x0 + j slope, formed by one
 * fma from the ray start (no drift). In slab j the ray spans [lo, hi]
 * (hi - lo = |slope| <= 1): pixel floor(lo), and where it crosses the next
 * boundary the fraction f = (floor(lo) + 1 - lo) / |slope| of the length
 * stays in that pixel and 1 - f goes to the next. floor() is a
 * round-toward-minus-infinity add of 1.5 * 2^23 (exact for |x| < 2^22);
 * the padded column floor(lo) + 2 is clamped (as unsigned) to n + 2, whose
 * two taps are pad zeros, so rays outside the image read zeros without
 * bounds checks.
 */
template <bool UP>
__device__ __forceinline__ float siddon_walk(const float *__restrict__ img, int n, int pitch, float x0, float slope,
                                             float inv)
{
    const uint32_t lim = (uint32_t) n + 2u;
    float sum = 0.0f, xa = x0, jf = 0.0f;
    uint32_t ro = 0;
#pragma unroll 4
    for (int j = 0; j < n; ++j) {
        jf += 1.0f;
        const float xb = fmaf(jf, slope, x0);
        const float lo = UP ? xa : xb;
        const float y = __fadd_rd(lo, kFloorMagic);
        const float c1 = (y - kFloorMagic) + 1.0f;        /* floor(lo) + 1 */
        const uint32_t p = min((uint32_t) (__float_as_int(y) - (kFloorMagicBits - kPadL)), lim);
        const float *row = img + ro + p;
        const float v0 = __ldg(row), v1 = __ldg(row + 1);
        /* the part of the slab's length left of the boundary c1: all of it
         * when the ray does not reach c1 ((c1 - lo) / |slope| >= 1) */
        const float f = fminf((c1 - lo) * inv, 1.0f);
        sum += f * v0 + (1.0f - f) * v1;
        xa = xb;
        ro += (uint32_t) pitch;
    }
    return sum;
}

__global__ void __launch_bounds__(128) siddon_fp_kernel(SiddonFpArgs P)
{
    const int k = (int) (blockIdx.x * blockDim.x + threadIdx.x);
    const int angle = P.a0 + (int) blockIdx.y;
    const int slice = (int) blockIdx.z;
    const int n = P.n;
    if (k >= n)
        return;
    const float sr = __ldg(P.sinv + angle), cr = __ldg(P.cosv + angle);
    const float r = sqrtf(sr * sr + cr * cr);
    const float sn = sr / r, cs = cr / r;
    const float half = 0.5f * (float) n;
    const float u0 = (((float) k + 0.5f) - P.axis) / r;   /* X cos - Y sin = u0, unit normal */
    const bool rows = fabsf(cs) >= fabsf(sn);
    /* rows: X(Y) = (u0 + Y sin) / cos; columns: Y(X) = (X cos - u0) / sin */
    const float len = rows ? 1.0f / fabsf(cs) : 1.0f / fabsf(sn);
    const float slope = rows ? sn / cs : cs / sn;
    const float x0 = (rows ? u0 / cs : (-u0) / sn) + (-half) * slope + half;
    const float inv = 1.0f / fabsf(slope);         /* inf for slope 0: never crosses */
    const float *img = (rows ? P.volP : P.volTP) + (size_t) slice * P.volp_stride;
    /* the slope's sign is the angle's (uniform per block), so each loop
     * knows which slab end is the lower one */
    const float sum = slope >= 0.0f ? siddon_walk<true>(img, n, P.pitch, x0, slope, inv)
                                    : siddon_walk<false>(img, n, P.pitch, x0, slope, inv);
    const size_t oidx = (size_t) slice * P.sino_stride + (size_t) angle * n + k;
    float result = P.src ? P.src[oidx] : 0.0f;
    result += P.scale * (sum * len);
    if (P.w)
        result *= P.w[(size_t) slice * P.w_stride + (size_t) angle * n + k];
    P.out[oidx] = result;
}

constexpr int kMaxSub = 16;

struct SiddonBpArgs {
    const float *sino;
    const float *base;
    float *dst;
    const float *sinv;
    const float *cosv;
    int n;
    int n_subsets;
    int total_angles;
    float axis;
    float relax;
    long long vol_stride;
    long long sino_stride;
    unsigned int sub_offset[kMaxSub];
    unsigned int sub_n[kMaxSub];
};

/*
 * Backprojection on the tiles of the Joseph one (bp_shapes.cuh): the CTA
 * stages, per angle, the detector window its pixels can reach, and a thread
 * keeps one register sum per pixel. With t the bin coordinate of a pixel's
 * centre (less 0.5), only bins floor(t) and floor(t) + 1 can cross it, at
 * distances f = frac(t) and 1 - f, and the trapezoid is its slope clamped:
 * L = h sat(q (w - f / r)) with q = 1 / min(a, b), as the slope reaches h at p.
 * So a pixel pair takes the coordinate (1 packed operation, with COLS / 2 + PR
 * products an angle), the floor (3), four saturating multiply-adds, two taps
 * and three multiply-adds.
 *
 * A pixel's t is the tile centre's bin coordinate C = Xc cos - Yc sin + axis -
 * 0.5, kept as an integer kb and a fraction, plus its offset (|dx| <= 63.5,
 * |dy| <= 31.5) times cos and sin: ~4e-6 bins of rounding.
 *
 * Bound by the FMA pipe. Global gathers for two pixels a thread, with the
 * trapezoid by comparison (64 instructions a pixel pair), took 2.39 ms for one
 * slice of 1448^2 x 1200; this takes 1.21.
 */
using namespace bp;

struct __align__(16) SiddonAngle {
    float2 cs, sn;
    float2 h;            /* chord where the line misses both corners' slopes */
    float frac;
    float a, b, c;       /* L / h = sat(a - b f) and sat(c + b f) */
    uint32_t base;       /* shared address of bin kb, less the floor bits */
    int w0;
};

template <class T>
struct __align__(16) SiddonSmem {
    float win[2][kAC][T::Win];
    SiddonAngle ang[2][kAC];
    unsigned int aligned[2];     /* angles of a chunk that take siddon_aligned */
};

/* Bin coordinate of (Xc, Yc), Xc cos - Yc sin + axis - 0.5, as an integer
 * and a fraction: the products' rounding errors (exact by FMA) and both sums'
 * (TwoSum), with explicit rounding so that no contraction merges the steps;
 * the sum less its integer part is exact. */
__device__ __forceinline__ void siddon_centre(float Xc, float Yc, float cr, float sr, float axis, float &kbf,
                                              float &frac)
{
    const float pa = __fmul_rn(Xc, cr), pb = __fmul_rn(Yc, sr);
    const float ea = fmaf(Xc, cr, -pa), eb = fmaf(Yc, sr, -pb);
    const float s1 = __fsub_rn(pa, pb);
    const float b1 = __fsub_rn(s1, pa);
    const float e1 = __fadd_rn(__fsub_rn(pa, __fsub_rn(s1, b1)), __fsub_rn(-pb, b1));
    const float ax = axis - 0.5f;
    const float hi = __fadd_rn(s1, ax);
    const float b2 = __fsub_rn(hi, s1);
    const float e2 = __fadd_rn(__fsub_rn(s1, __fsub_rn(hi, b2)), __fsub_rn(ax, b2));
    kbf = floorf(hi);
    frac = __fadd_rn(__fsub_rn(hi, kbf), __fadd_rn(__fadd_rn(e1, __fsub_rn(ea, eb)), e2));
}

/*
 * Angles closer to an axis than kAligned: L falls from h to 0 within min(a, b)
 * bins, so where a scan's bins meet pixel boundaries (an axis half a bin off
 * the centre) the side a pixel falls on hangs on the coordinate's last bit.
 * These angles (0 and 90 degrees, as a rule) keep the coordinate of 64 x 8
 * pixel blocks and L by comparison.
 */
constexpr float kAligned = 1.0e-3f;

struct SiddonAligned {
    float cr, sr;
    float ir, iab, p, w_ab, h;
};

__device__ __forceinline__ SiddonAligned siddon_aligned_of(float cr, float sr)
{
    SiddonAligned A;
    A.cr = cr;
    A.sr = sr;
    A.ir = 1.0f / sqrtf(cr * cr + sr * sr);
    const float a = fabsf(cr) * A.ir, b = fabsf(sr) * A.ir, ab = a * b;
    A.iab = ab > 0.0f ? 1.0f / ab : 3.0e38f;
    A.p = 0.5f * fabsf(a - b);
    A.w_ab = 0.5f * (a + b) * A.iab;
    A.h = 1.0f / fmaxf(a, b);
    return A;
}

/* What pixels (x, y) and (x + 32, y), of one 64-column block, add to their
 * sums. One call for two pixels, the angle's constants outside: one angle of 0
 * degrees on 2900^2 took 35 of a 60 us call with a call a pixel that worked them
 * out again, and takes 11 of 36 (and 49 of 120, now 21 of 57, on 4096^2). */
__device__ __noinline__ float2 siddon_aligned(const float *win, int w0, int width, int x, int y, int n, float axis,
                                              const SiddonAligned A)
{
    const float half = 0.5f * (float) n;
    float kbf, frac;
    siddon_centre((float) ((x & ~63) + 32) - half, (float) ((y & ~7) + 4) - half, A.cr, A.sr, axis, kbf, frac);
    const float dx = ((float) (x & 63) + 0.5f) - 32.0f, dy = ((float) (y & 7) + 0.5f) - 4.0f;
    const float row = fmaf(-dy, A.sr, frac);
    const int kb = (int) kbf - w0 - kFloorMagicBits;
    float s[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const float t = fmaf(dx + 32.0f * (float) q, A.cr, row);
        const float v = __fadd_rd(t, kFloorMagic);
        const float f = t - (v - kFloorMagic);
        const int k = kb + __float_as_int(v);
        const float da = f * A.ir, db = A.ir - da;
        const float la = da <= A.p ? A.h : fmaxf(0.0f, fmaf(-da, A.iab, A.w_ab));
        const float lb = db <= A.p ? A.h : fmaxf(0.0f, fmaf(-db, A.iab, A.w_ab));
        const float va = (unsigned int) k < (unsigned int) width ? win[k] : 0.0f;
        const float vb = (unsigned int) (k + 1) < (unsigned int) width ? win[k + 1] : 0.0f;
        s[q] = fmaf(lb, vb, la * va);
    }
    return make_float2(s[0], s[1]);
}

__device__ __forceinline__ int siddon_angle_of(const SiddonBpArgs &P, int vi)
{
    for (int k = 0; k < P.n_subsets; ++k) {
        if (vi < (int) P.sub_n[k])
            return (int) P.sub_offset[k] + vi;
        vi -= (int) P.sub_n[k];
    }
    return 0;
}

template <class T>
__device__ void siddon_load_chunk(const SiddonBpArgs &P, SiddonSmem<T> &S, int buf, int first, int count,
                                  const float *sino, float Xc, float Yc)
{
    const int lane = (int) threadIdx.x, warp = (int) threadIdx.y;
    bool aligned = false;
    if (warp == 0 && lane < count) {
        const int angle = siddon_angle_of(P, first + lane);
        const float cr = __ldg(P.cosv + angle), sr = __ldg(P.sinv + angle);
        const float r = sqrtf(cr * cr + sr * sr), ir = 1.0f / r;
        const float a = fabsf(cr) * ir, b = fabsf(sr) * ir, lo_ab = fminf(a, b);
        float kbf, frac;
        siddon_centre(Xc, Yc, cr, sr, P.axis, kbf, frac);
        SiddonAngle A;
        int kb;
        if (fabsf(kbf) < 1.0e6f) {
            kb = (int) kbf;
            A.cs = joseph::splat(cr);
            A.sn = joseph::splat(sr);
            A.frac = frac;
            aligned = lo_ab < kAligned;
        } else {
            /* no bin near (an axis far outside, or no geometry): a window of zeros */
            kb = -1000000;
            A.cs = A.sn = joseph::splat(0.0f);
            A.frac = 0.0f;
        }
        /* axis-aligned: L = h up to half a bin and 0 beyond; the slope's q
         * stays finite and the half itself counts */
        const float q = lo_ab > 0.0f ? 1.0f / lo_ab : 3.0e38f, edge = lo_ab > 0.0f ? 0.0f : 1.0e-6f;
        const float w = 0.5f * (a + b) + edge;
        A.h = joseph::splat(1.0f / fmaxf(a, b));
        A.a = w * q;
        A.b = ir * q;
        A.c = (w - ir) * q;
        const float half_x = 0.5f * (float) (T::TileX - 1), half_y = 0.5f * (float) (T::TileY - 1);
        const float lo = A.frac - half_x * fabsf(A.cs.x) - half_y * fabsf(A.sn.x);
        A.w0 = align_window(kb + (int) floorf(lo) - 1, sino + (size_t) angle * P.n);
        A.base = (uint32_t) __cvta_generic_to_shared(&S.win[buf][lane][0]) + 4u * (uint32_t) (kb - A.w0) -
                 4u * (uint32_t) joseph::kFloorMagicBits;
        S.ang[buf][lane] = A;
    }
    if (warp == 0) {
        const unsigned int m = __ballot_sync(0xffffffffu, aligned);
        if (lane == 0)
            S.aligned[buf] = m;
    }
    __syncthreads();
    for (int slot = warp; slot < count; slot += T::TY) {
        const int w0 = S.ang[buf][slot].w0;
        copy_window<T>(S.win[buf][slot], sino + (ptrdiff_t) siddon_angle_of(P, first + slot) * P.n + w0, w0, P.n);
    }
}

template <class T>
__global__ void __launch_bounds__(T::Threads, T::CTAS) siddon_bp_kernel(const __grid_constant__ SiddonBpArgs P)
{
    __shared__ SiddonSmem<T> S;
    const int n = P.n;
    const int tiles_x = (n + T::TileX - 1) / T::TileX;
    const int x0 = ((int) blockIdx.x % tiles_x) * T::TileX, y0 = ((int) blockIdx.x / tiles_x) * T::TileY;
    const int slice = (int) blockIdx.y;
    const float *sino = P.sino + (size_t) slice * P.sino_stride;
    const float half = 0.5f * (float) n;
    /* tile centre and the pixels' offsets from it (all exact: half-integers) */
    const float Xc = (float) (x0 + T::TileX / 2) - half, Yc = (float) (y0 + T::TileY / 2) - half;
    const int x = x0 + (int) threadIdx.x;
    float2 dx[T::H], ndy[T::PR], sum[T::PR][T::H], v[T::PR][T::H];
#pragma unroll
    for (int h = 0; h < T::H; ++h) {
        const float d = ((float) ((int) threadIdx.x + 2 * kTX * h) + 0.5f) - (float) (T::TileX / 2);
        dx[h] = make_float2(d, d + (float) kTX);
    }
#pragma unroll
    for (int p = 0; p < T::PR; ++p) {
        const int y = y0 + (int) threadIdx.y + T::TY * p;
        ndy[p] = joseph::splat((float) (T::TileY / 2) - ((float) ((int) threadIdx.y + T::TY * p) + 0.5f));
        const size_t row = (size_t) slice * P.vol_stride + (size_t) y * n;
#pragma unroll
        for (int h = 0; h < T::H; ++h) {
            const int xa = x + 2 * kTX * h, xb = xa + kTX;
            v[p][h] = make_float2((P.base && xa < n && y < n) ? P.base[row + xa] : 0.0f,
                                  (P.base && xb < n && y < n) ? P.base[row + xb] : 0.0f);
            sum[p][h] = make_float2(0.0f, 0.0f);
        }
    }
    const int total = P.total_angles, nchunks = (total + kAC - 1) / kAC;
    const float2 relax = joseph::splat(P.relax);
    int sub = 0, sub_end = P.n_subsets > 0 ? (int) P.sub_n[0] : 0;
    if (nchunks > 0) {
        siddon_load_chunk<T>(P, S, 0, 0, min(kAC, total), sino, Xc, Yc);
        cp_async_commit();
    }
    for (int ch = 0; ch < nchunks; ++ch) {
        const int buf = ch & 1, first = ch * kAC, count = min(kAC, total - first);
        if (ch + 1 < nchunks) {
            siddon_load_chunk<T>(P, S, buf ^ 1, first + kAC, min(kAC, total - first - kAC), sino, Xc, Yc);
            cp_async_commit();
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        for (int i = 0; i < count;) {
            if (first + i == sub_end) {
                /* end of a subset: v = v + relax * sum */
#pragma unroll
                for (int p = 0; p < T::PR; ++p)
#pragma unroll
                    for (int h = 0; h < T::H; ++h) {
                        v[p][h] = joseph::fma2(relax, sum[p][h], v[p][h]);
                        sum[p][h] = make_float2(0.0f, 0.0f);
                    }
                ++sub;
                sub_end += (int) P.sub_n[sub];
                continue;
            }
            /* up to the next subset, or axis-aligned angle */
            const unsigned int al = S.aligned[buf] >> i;
            if (al & 1u) {
                const SiddonAligned A = siddon_aligned_of(S.ang[buf][i].cs.x, S.ang[buf][i].sn.x);
                const int w0 = S.ang[buf][i].w0;
#pragma unroll
                for (int p = 0; p < T::PR; ++p)
#pragma unroll
                    for (int h = 0; h < T::H; ++h) {
                        const int y = y0 + (int) threadIdx.y + T::TY * p;
                        sum[p][h] = joseph::add2(sum[p][h], siddon_aligned(S.win[buf][i], w0, T::Win, x + 2 * kTX * h,
                                                                           y, n, P.axis, A));
                    }
                ++i;
                continue;
            }
            const int end = min(min(count, sub_end - first), al ? i + __ffs((int) al) - 1 : count);
#pragma unroll 2
            for (; i < end; ++i) {
                const SiddonAngle A = S.ang[buf][i];
                float2 px[T::H];
#pragma unroll
                for (int h = 0; h < T::H; ++h)
                    px[h] = joseph::mul2(dx[h], A.cs);
#pragma unroll
                for (int p = 0; p < T::PR; ++p) {
                    const float2 py = joseph::fma2(ndy[p], A.sn, joseph::splat(A.frac));
#pragma unroll
                    for (int h = 0; h < T::H; ++h) {
                        float2 f;
                        const float2 y = joseph::floor2(joseph::add2(px[h], py), f);
                        const uint32_t a0 = A.base + 4u * (uint32_t) __float_as_int(y.x);
                        const uint32_t a1 = A.base + 4u * (uint32_t) __float_as_int(y.y);
                        const float2 va = make_float2(joseph::lds(a0), joseph::lds(a1));
                        const float2 vb = make_float2(joseph::lds(a0 + 4u), joseph::lds(a1 + 4u));
                        const float2 la = make_float2(joseph::fma_sat(-A.b, f.x, A.a), joseph::fma_sat(-A.b, f.y, A.a));
                        const float2 lb = make_float2(joseph::fma_sat(A.b, f.x, A.c), joseph::fma_sat(A.b, f.y, A.c));
                        const float2 s = joseph::fma2(lb, vb, joseph::mul2(la, va));
                        sum[p][h] = joseph::fma2(A.h, s, sum[p][h]);
                    }
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int p = 0; p < T::PR; ++p) {
        const int y = y0 + (int) threadIdx.y + T::TY * p;
#pragma unroll
        for (int c = 0; c < T::COLS; ++c) {
            const int xc = x + kTX * c;
            if (xc >= n || y >= n)
                continue;
            const float2 vv = joseph::fma2(relax, sum[p][c >> 1], v[p][c >> 1]);
            P.dst[(size_t) slice * P.vol_stride + (size_t) y * n + xc] = (c & 1) ? vv.y : vv.x;
        }
    }
}

template <class T>
int launch_siddon_bp(udev *d, const SiddonBpArgs &A, int n_slices)
{
    const dim3 grid(udev_div_up(A.n, T::TileX) * udev_div_up(A.n, T::TileY), (unsigned int) n_slices);
    siddon_bp_kernel<T><<<grid, dim3(kTX, T::TY), 0, d->stream>>>(A);
    return udev_after_launch(d, "siddon_bp_kernel");
}

}  // namespace

extern "C" int udev_siddon_fp(udev *d, const udev_geom *g, int a0, int na, const float *volP, const float *volTP,
                              const float *src, const float *w, int w_shared, float *out, float scale, int n_slices)
{
    if (n_slices <= 0 || na <= 0)
        return UFOIR_OK;
    const int n = g->n_dets;
    if (a0 < 0 || a0 + na > g->n_angles || n < 1 || n > 32768 || n_slices > UDEV_SIDDON_MOST || na > UDEV_SIDDON_MOST) {
        udev_set_error(d, "siddon_fp: angles [%d, %d) of %d, n = %d, %d slices out of range", a0, a0 + na,
                       g->n_angles, n, n_slices);
        return UFOIR_ERR_INVALID;
    }
    UDEV_BIND(d);
    SiddonFpArgs A;
    A.volP = volP;
    A.volTP = volTP;
    A.src = src;
    A.w = w;
    A.out = out;
    A.sinv = g->d_sin;
    A.cosv = g->d_cos;
    A.n = n;
    A.a0 = a0;
    A.na = na;
    A.pitch = udev_fp_pitch(n);
    A.axis = g->axis;
    A.scale = scale;
    A.volp_stride = (long long) n * A.pitch;
    A.sino_stride = (long long) g->n_angles * n;
    A.w_stride = w_shared ? 0 : A.sino_stride;
    dim3 grid(udev_div_up(n, 128), (unsigned int) na, (unsigned int) n_slices);
    siddon_fp_kernel<<<grid, 128, 0, d->stream>>>(A);
    return udev_after_launch(d, "siddon_fp_kernel");
}

extern "C" int udev_siddon_bp(udev *d, const udev_geom *g, const ufoir_subset *subsets, int n_subsets,
                              const float *sino, const float *base, float *dst, float relax, int n_slices)
{
    if (n_slices <= 0)
        return UFOIR_OK;
    const int n = g->n_dets;
    if (n_subsets < 0 || n_subsets > kMaxSub || n < 1 || n_slices > UDEV_SIDDON_MOST) {
        udev_set_error(d, "siddon_bp: %d subsets (at most %d), %d slices", n_subsets, kMaxSub, n_slices);
        return UFOIR_ERR_INVALID;
    }
    SiddonBpArgs A;
    A.total_angles = 0;
    for (int s = 0; s < n_subsets; ++s) {
        if (subsets[s].offset + subsets[s].n > (unsigned int) g->n_angles) {
            udev_set_error(d, "siddon_bp: subset %d [%u, %u) beyond %d angles", s, subsets[s].offset,
                           subsets[s].offset + subsets[s].n, g->n_angles);
            return UFOIR_ERR_INVALID;
        }
        A.sub_offset[s] = subsets[s].offset;
        A.sub_n[s] = subsets[s].n;
        A.total_angles += (int) subsets[s].n;
    }
    UDEV_BIND(d);
    A.sino = sino;
    A.base = base;
    A.dst = dst;
    A.sinv = g->d_sin;
    A.cosv = g->d_cos;
    A.n = n;
    A.n_subsets = n_subsets;
    A.axis = g->axis;
    A.relax = relax;
    A.vol_stride = (long long) n * n;
    A.sino_stride = (long long) g->n_angles * n;
    switch (bp_shape(d, n, n_slices)) {
    case 0: return launch_siddon_bp<ShapeL>(d, A, n_slices);
    case 1: return launch_siddon_bp<ShapeM>(d, A, n_slices);
    case 2: return launch_siddon_bp<ShapeS>(d, A, n_slices);
    default: return launch_siddon_bp<ShapeT>(d, A, n_slices);
    }
}
