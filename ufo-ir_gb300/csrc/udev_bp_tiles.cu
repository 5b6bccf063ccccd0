/*
 * udev_bp_tiles.cu - pixel-driven backprojection over many angles, with the
 * sinogram windows of a pixel tile staged in shared memory.
 *
 * One CTA owns a tile of pixels; thread (tx, ty) owns COLS columns
 * (x0 + tx + 32c) of PR rows (y0 + ty + TY p) and walks the angles with one
 * register sum per pixel. Two columns of a row form a packed pair, so an
 * angle costs COLS / 2 + PR packed products for COLS * PR pixels, and 32
 * lanes (adjacent x) touch adjacent words of the staged window (no bank
 * conflicts). For a chunk of 32 angles the CTA copies, per angle, the
 * detector values the tile can reach (cp.async, double buffered; detectors
 * outside [0, n) read 0), so every sample reads shared memory.
 *
 * Bound by the FMA pipe (a packed FP32 instruction takes two of its cycles)
 * and the instructions around it: ncu at 4 slices of 1448^2 x 1200 counts
 * 23.7 instructions and 13.5 on the FMA pipe per warp and 64 samples with 16
 * pixels of one column per thread and the row products staged in shared
 * memory, 19.1 and 11.2 with 4 columns x 8 rows and the products in
 * registers. What that and the forms below gave, 16 slices of 1448^2 x 1200:
 * 16.13 -> 13.69 ms; one slice 1.112 -> 1.005; six slices of 1001^2 x 451
 * off-centre in the fast arithmetic 1.096 -> 0.938; one of 367^2 x 180
 * 0.0424 -> 0.0300 (launch shapes below):
 *  - the filter's three-operation form (joseph::lerp2n) where a chunk's
 *    windows are finite, which every chunk checks as it lands (< 1 %);
 *  - per chunk, a bit per angle says whether the whole tile lies inside the
 *    detector edges (no clamp: before, whole tiles clamped, and every tile of
 *    an off-centre axis) or beyond one edge (every pixel adds one value);
 *  - the angle loop unrolled four times (16 slices: 14.40 -> 13.70 ms; eight
 *    times 15.33, past the instruction cache). Prefetching the next angle's
 *    record gained 4 % at two and nothing at four.
 *
 * Arithmetic is the reference's BP (projector-parallel-joseph.cl:158-218):
 * s = fX * cos - fY * sin + (os - ros), clamped to the active detector
 * edges, linear interpolation along s at the row centre, per-subset float
 * sums over the angles in order, then v = v + relax * sum per subset; the
 * epilogue optionally applies v * cw + add (SIRT update).
 */
#include <cuda_runtime.h>

#include <cstring>

#include "bp_shapes.cuh"
#include "joseph.cuh"
#include "udev_internal.cuh"

namespace {

using namespace bp;

constexpr int kMaxSub = 16;

struct BpTileArgs {
    const float *sino;
    const float *base;
    const float *cw;
    const float *add;
    float *dst;
    const float *sinv;
    const float *cosv;
    int n;
    float axis;
    float relax;
    long long vol_stride;
    long long sino_stride;
    long long cw_stride;
    int n_subsets;
    int total_angles;
    int contiguous;      /* subsets cover [first_angle, first_angle + total) in order */
    int first_angle;
    float neg_zero;      /* -0.0f: the addend of unfusable packed products */
    unsigned int sub_offset[kMaxSub];
    unsigned int sub_n[kMaxSub];
};

/* Per angle of a chunk: constants of packed operations twice, the shared
 * address of the window's detector 0 less the floor bits, the window's first
 * detector, and the clamped coordinate of a tile outside the detector edges. */
struct __align__(16) BpAngle {
    float2 cs, sn;
    uint32_t base;
    int w0;
    float edge;
    int pad_;
};

template <class T>
struct __align__(16) BpSmem {
    float win[2][kAC][T::Win];
    BpAngle ang[2][kAC];
    /* per chunk: angles whose coordinates over the whole tile lie inside the
     * detector edges, and angles where all of them lie beyond one edge */
    unsigned int inside[2], outside[2];
};

/* Angle of virtual index vi (angles of the subsets, in order). */
__device__ __forceinline__ int angle_of(const BpTileArgs &P, int vi)
{
    if (P.contiguous)
        return P.first_angle + vi;
    for (int k = 0; k < P.n_subsets; ++k) {
        if (vi < (int) P.sub_n[k])
            return (int) P.sub_offset[k] + vi;
        vi -= (int) P.sub_n[k];
    }
    return 0;
}

/* Detector coordinate of pixel (x, y) for one angle, exactly as the reference,
 * or with FM as the fast arithmetic sums it (sample_angles). */
template <bool FM>
__device__ __forceinline__ float det_coord(float fX, float fY, float cs, float sn, float shift)
{
    if (FM)
        return __fadd_rn(__fmul_rn(fX, cs), __fadd_rn(__fmul_rn(-fY, sn), shift));
    return __fadd_rn(__fsub_rn(__fmul_rn(fX, cs), __fmul_rn(fY, sn)), shift);
}

/*
 * Stages the windows of one chunk of angles. Each window starts at a detector
 * whose global address is 16-byte aligned, at most 3 before the leftmost
 * reachable tap, so the bulk of it moves in 16-byte cp.async copies; groups
 * that cross the ends of the detector row go element by element, with zeros
 * outside [0, n). A warp copies whole windows (lane = group of 4).
 *
 * The coordinate is monotone in each pixel index (every rounding step is, in
 * either order of the sum), so over the tile it lies between its values at the
 * corners, summed in the order of the samples: a tile decided inside by another
 * order can hold coordinates an ulp below the edge.
 */
template <class T, bool FM>
__device__ void load_chunk(const BpTileArgs &P, BpSmem<T> &S, int buf, int chunk, const float *sino, int x0, int y0,
                           const joseph::AxisConsts &k, float e0, float e1, float shift)
{
    const int lane = (int) threadIdx.x, warp = (int) threadIdx.y;
    const int first = chunk * kAC;
    const int count = min(kAC, P.total_angles - first);
    if (warp == 0) {
        bool in = false, out = false;
        if (lane < count) {
            const int a = angle_of(P, first + lane);
            const float cs = __ldg(P.cosv + a), sn = __ldg(P.sinv + a);
            const float fx0 = __fsub_rn(__fadd_rn((float) x0, 0.5f), k.os);
            const float fx1 = __fsub_rn(__fadd_rn((float) (x0 + T::TileX - 1), 0.5f), k.os);
            const float fy0 = __fsub_rn(__fadd_rn((float) y0, 0.5f), k.os);
            const float fy1 = __fsub_rn(__fadd_rn((float) (y0 + T::TileY - 1), 0.5f), k.os);
            const float c00 = det_coord<FM>(fx0, fy0, cs, sn, shift), c10 = det_coord<FM>(fx1, fy0, cs, sn, shift);
            const float c01 = det_coord<FM>(fx0, fy1, cs, sn, shift), c11 = det_coord<FM>(fx1, fy1, cs, sn, shift);
            const float lo = fminf(fminf(c00, c10), fminf(c01, c11));
            const float hi = fmaxf(fmaxf(c00, c10), fmaxf(c01, c11));
            in = lo >= e0 && hi <= e1;
            out = hi <= e0 || lo >= e1;
            const float clo = fminf(fmaxf(lo, e0), e1);
            const int w0 = align_window((int) floorf(__fsub_rn(clo, 0.5f)) - 2, sino + (size_t) a * P.n);
            BpAngle A;
            A.cs = joseph::splat(cs);
            A.sn = joseph::splat(sn);
            A.base = (uint32_t) __cvta_generic_to_shared(&S.win[buf][lane][0]) -
                     4u * (uint32_t) (w0 + joseph::kHalfFloorBits);
            A.w0 = w0;
            A.edge = hi <= e0 ? e0 : e1;
            A.pad_ = 0;
            S.ang[buf][lane] = A;
        }
        const unsigned int mi = __ballot_sync(0xffffffffu, in), mo = __ballot_sync(0xffffffffu, out);
        if (lane == 0) {
            S.inside[buf] = mi;
            S.outside[buf] = mo & ~mi;
        }
    }
    __syncthreads();
    for (int slot = warp; slot < count; slot += T::TY) {
        const int w0 = S.ang[buf][slot].w0;
        const float *src = sino + (size_t) angle_of(P, first + slot) * P.n + w0;
        copy_window<T>(S.win[buf][slot], src, w0, P.n);
    }
}

/* Whether the windows of a staged chunk hold a non-finite value, in the
 * groups this thread staged itself (load_chunk's loop; its own copies have
 * landed). x * 0 is NaN for infinities and NaNs and 0 for all else. */
template <class T>
__device__ __forceinline__ bool chunk_nonfinite(const BpSmem<T> &S, int buf, int count)
{
    float acc = 0.0f;
    for (int slot = (int) threadIdx.y; slot < count; slot += T::TY) {
#pragma unroll
        for (int g = 0; g < T::Win / 4; g += 32) {
            const int e = 4 * (g + (int) threadIdx.x);
            if (e >= T::Win)
                continue;
            const float4 w = *reinterpret_cast<const float4 *>(&S.win[buf][slot][e]);
            acc = fmaf(w.x, 0.0f, acc);
            acc = fmaf(w.y, 0.0f, acc);
            acc = fmaf(w.z, 0.0f, acc);
            acc = fmaf(w.w, 0.0f, acc);
        }
    }
    return !(acc == 0.0f);
}

/*
 * Angles [i0, i1) of one staged chunk for the thread's pixels, two pixels of a
 * row per packed instruction. CLAMP: coordinates are clamped to the detector
 * edges. FAST: every (clamped) coordinate is >= 0.5, so the three-step floor
 * applies. FIN: the windows hold finite values only, so the filter takes its
 * three-operation form (joseph::lerp2n).
 */
template <class T, bool CLAMP, bool FAST, bool FM, bool FIN>
__device__ __forceinline__ void sample_angles(const BpSmem<T> &S, int buf, int i0, int i1, const float2 (&fX)[T::H],
                                              const float2 (&nfY)[T::PR], float shift, float e0, float e1, float2 z2,
                                              float2 (&sum)[T::PR][T::H])
{
    constexpr uint32_t bits = FAST ? 0u : 4u * (uint32_t) (joseph::kFloorMagicBits - joseph::kHalfFloorBits);
    const float2 shift2 = joseph::splat(shift);
#pragma unroll T::Unroll
    for (int i = i0; i < i1; ++i) {
        const BpAngle A = S.ang[buf][i];
        float2 px[T::H], py[T::PR];
#pragma unroll
        for (int h = 0; h < T::H; ++h)
            px[h] = joseph::mul2z(fX[h], A.cs, z2);
#pragma unroll
        for (int p = 0; p < T::PR; ++p) {
            py[p] = joseph::mul2z(nfY[p], A.sn, z2);
            if (FM)
                py[p] = joseph::add2(py[p], shift2);
        }
        const uint32_t base = A.base - bits;
#pragma unroll
        for (int p = 0; p < T::PR; ++p)
#pragma unroll
            for (int h = 0; h < T::H; ++h) {
                /* fX * cos - fY * sin + shift, as fX*cos + (-fY)*sin + shift
                 * (fast arithmetic: fX*cos + ((-fY)*sin + shift)) */
                float2 sc = joseph::add2(px[h], py[p]);
                if (!FM)
                    sc = joseph::add2(sc, shift2);
                if (CLAMP) {
                    sc.x = fminf(fmaxf(sc.x, e0), e1);
                    sc.y = fminf(fmaxf(sc.y, e0), e1);
                }
                constexpr bool kFused = FIN && FAST && !FM;
                float2 t;
                const float2 y = kFused ? joseph::floor_half2n(sc, t)
                                        : FAST ? joseph::floor_half2(sc, t) : joseph::floor_any2(sc, t);
                const uint32_t a0 = base + 4u * (uint32_t) __float_as_int(y.x);
                const uint32_t a1 = base + 4u * (uint32_t) __float_as_int(y.y);
                const float2 t0 = make_float2(joseph::lds(a0), joseph::lds(a1));
                const float2 t1 = make_float2(joseph::lds(a0 + 4u), joseph::lds(a1 + 4u));
                if (FM)
                    sum[p][h] = joseph::lerp_acc_fast2(sum[p][h], t, t0, t1);
                else
                    sum[p][h] = joseph::add2(sum[p][h], kFused ? joseph::lerp2n(t, t0, t1, z2)
                                                               : joseph::lerp2(t, t0, t1, z2));
            }
    }
}

/* The same where the whole tile lies beyond one detector edge: every pixel's
 * coordinate is clamped to that edge, so all of them add one value. */
template <class T, bool FM>
__device__ __forceinline__ void edge_angles(const BpSmem<T> &S, int buf, int i0, int i1, float2 z2,
                                            float2 (&sum)[T::PR][T::H])
{
    for (int i = i0; i < i1; ++i) {
        const BpAngle A = S.ang[buf][i];
        float2 t;
        const float2 y = joseph::floor_any2(joseph::splat(A.edge), t);
        const uint32_t a = A.base + 4u * (uint32_t) (__float_as_int(y.x) -
                                                     (joseph::kFloorMagicBits - joseph::kHalfFloorBits));
        const float2 t0 = joseph::splat(joseph::lds(a)), t1 = joseph::splat(joseph::lds(a + 4u));
        const float2 val = joseph::lerp2(t, t0, t1, z2);
#pragma unroll
        for (int p = 0; p < T::PR; ++p)
#pragma unroll
            for (int h = 0; h < T::H; ++h)
                sum[p][h] = FM ? joseph::lerp_acc_fast2(sum[p][h], t, t0, t1) : joseph::add2(sum[p][h], val);
    }
}

/* One CTA's work: pixel tile `tile` of slice `slice`. */
template <class T, bool FM>
__device__ __forceinline__ void bp_tile(const BpTileArgs &P, BpSmem<T> &S, int tile, int slice)
{
    const int n = P.n;
    const int tiles_x = (n + T::TileX - 1) / T::TileX;
    const int x0 = (tile % tiles_x) * T::TileX;
    const int y0 = (tile / tiles_x) * T::TileY;
    const float *sino = P.sino + (size_t) slice * P.sino_stride;

    const joseph::AxisConsts k = joseph::axis_consts(n, P.axis);
    float e0, e1;
    joseph::bp_edges(k, n, P.axis, e0, e1);
    const float shift = __fsub_rn(k.os, k.ros);
    const float2 z2 = joseph::splat(P.neg_zero);

    /* pixel pairs: columns x + 64h and x + 64h + 32 of one row */
    const int x = x0 + (int) threadIdx.x;
    float2 fX[T::H], nfY[T::PR], sum[T::PR][T::H], v[T::PR][T::H];
#pragma unroll
    for (int h = 0; h < T::H; ++h)
        fX[h] = make_float2(__fsub_rn(__fadd_rn((float) (x + 2 * kTX * h), 0.5f), k.os),
                            __fsub_rn(__fadd_rn((float) (x + 2 * kTX * h + kTX), 0.5f), k.os));
#pragma unroll
    for (int p = 0; p < T::PR; ++p) {
        const int y = y0 + (int) threadIdx.y + T::TY * p;
        nfY[p] = joseph::splat(-__fsub_rn(__fadd_rn((float) y, 0.5f), k.os));
        const size_t row = (size_t) slice * P.vol_stride + (size_t) y * n;
#pragma unroll
        for (int h = 0; h < T::H; ++h) {
            const int xa = x + 2 * kTX * h, xb = xa + kTX;
            v[p][h] = make_float2((P.base && xa < n && y < n) ? P.base[row + xa] : 0.0f,
                                  (P.base && xb < n && y < n) ? P.base[row + xb] : 0.0f);
            sum[p][h] = make_float2(0.0f, 0.0f);
        }
    }
    /* clamped coordinates are >= min(e0, e1) */
    const bool fast = fminf(e0, e1) >= 0.5f;

    const int nchunks = (P.total_angles + kAC - 1) / kAC;
    int sub = 0;
    int sub_end = P.n_subsets > 0 ? (int) P.sub_n[0] : 0;
    if (nchunks > 0) {
        load_chunk<T, FM>(P, S, 0, 0, sino, x0, y0, k, e0, e1, shift);
        cp_async_commit();
    }
    for (int ch = 0; ch < nchunks; ++ch) {
        const int buf = ch & 1;
        if (ch + 1 < nchunks) {
            load_chunk<T, FM>(P, S, buf ^ 1, ch + 1, sino, x0, y0, k, e0, e1, shift);
            cp_async_commit();
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        const int first = ch * kAC, count = min(kAC, P.total_angles - first);
        bool fin = false;
        if (FM)
            __syncthreads();
        else
            fin = !__syncthreads_or(chunk_nonfinite<T>(S, buf, count));
        const unsigned int in = S.inside[buf], out = S.outside[buf];
        for (int i = 0; i < count;) {
            if (first + i == sub_end) {
                /* end of a subset: v = v + relax * sum (one BP launch of the reference) */
#pragma unroll
                for (int p = 0; p < T::PR; ++p)
#pragma unroll
                    for (int h = 0; h < T::H; ++h) {
                        v[p][h] = joseph::add2(v[p][h], joseph::mul2z(joseph::splat(P.relax), sum[p][h], z2));
                        sum[p][h] = make_float2(0.0f, 0.0f);
                    }
                ++sub;
                sub_end += (int) P.sub_n[sub];
                continue;
            }
            /* the run of angles of one form from here on */
            const bool is_in = (in >> i) & 1u, is_out = (out >> i) & 1u;
            const unsigned int same = (is_in ? in : is_out ? out : ~(in | out)) >> i;
            const int run = same == 0xffffffffu ? 32 : __ffs((int) ~same) - 1;
            const int end = min(min(count, sub_end - first), i + run);
            if (!fast)
                sample_angles<T, true, false, FM, false>(S, buf, i, end, fX, nfY, shift, e0, e1, z2, sum);
            else if (is_in && (FM || fin))
                sample_angles<T, false, true, FM, true>(S, buf, i, end, fX, nfY, shift, e0, e1, z2, sum);
            else if (is_out)
                edge_angles<T, FM>(S, buf, i, end, z2, sum);
            else
                sample_angles<T, true, true, FM, false>(S, buf, i, end, fX, nfY, shift, e0, e1, z2, sum);
            i = end;
        }
        __syncthreads();
    }
#pragma unroll
    for (int p = 0; p < T::PR; ++p) {
        const int y = y0 + (int) threadIdx.y + T::TY * p;
#pragma unroll
        for (int c = 0; c < T::COLS; ++c) {
            const int xc = x + kTX * c;
            float2 vv = v[p][c >> 1];
            if (P.n_subsets > 0)
                vv = joseph::add2(vv, joseph::mul2z(joseph::splat(P.relax), sum[p][c >> 1], z2));
            if (xc >= n || y >= n)
                continue;
            float r = (c & 1) ? vv.y : vv.x;
            if (P.cw)
                r = __fmul_rn(r, P.cw[(size_t) slice * P.cw_stride + (size_t) y * n + xc]);
            const size_t pix = (size_t) slice * P.vol_stride + (size_t) y * n + xc;
            if (P.add)
                r = __fadd_rn(r, P.add[pix]);
            P.dst[pix] = r;
        }
    }
}

template <class T, bool FM>
__global__ void __launch_bounds__(T::Threads, T::CTAS) bp_tiles_kernel(const __grid_constant__ BpTileArgs P)
{
    __shared__ BpSmem<T> S;
    bp_tile<T, FM>(P, S, (int) blockIdx.x, (int) blockIdx.y);
}

typedef ShapeM BatchShape;

/*
 * Mixed batch: the pixel tiles of many one-slice jobs (any size and angle
 * count) in one launch. CTA b belongs to the job j with item_start[j] <= b <
 * item_start[j + 1]; its record (the job's BpTileArgs) is staged in shared
 * memory. Jobs whose active flag is 0 are skipped.
 */
template <bool FM>
__global__ void __launch_bounds__(BatchShape::Threads, BatchShape::CTAS)
    bp_tiles_batch_kernel(const BpTileArgs *__restrict__ recs, const int *__restrict__ item_start, int n_jobs,
                          const int *__restrict__ job_index, const int *__restrict__ active)
{
    __shared__ BpSmem<BatchShape> S;
    __shared__ BpTileArgs rec;
    __shared__ int job_s;
    const int b = (int) blockIdx.x;
    const int tid = (int) (threadIdx.y * kTX + threadIdx.x);
    if (tid == 0) {
        int lo = 0, hi = n_jobs - 1;      /* last j with item_start[j] <= b */
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(item_start + mid) <= b)
                lo = mid;
            else
                hi = mid - 1;
        }
        job_s = lo;
    }
    __syncthreads();
    const int j = job_s;
    if (!__ldg(active + __ldg(job_index + j)))
        return;
    {
        const int *src = reinterpret_cast<const int *>(recs + j);
        int *dst = reinterpret_cast<int *>(&rec);
        for (int e = tid; e < (int) (sizeof(BpTileArgs) / sizeof(int)); e += BatchShape::Threads)
            dst[e] = __ldg(src + e);
    }
    __syncthreads();
    bp_tile<BatchShape, FM>(rec, S, b - __ldg(item_start + j), 0);
}

static_assert(sizeof(BpTileArgs) % sizeof(int) == 0, "records are copied as ints");

/* The arguments of one BP launch (udev_bp_tiles' contract) for one slice. */
static int fill_args(udev *d, const udev_geom *g, const ufoir_subset *subsets, int n_subsets, const float *sino,
                     const float *base, const float *cw, int cw_shared, const float *add, float *dst, float relax,
                     BpTileArgs &A)
{
    if (n_subsets > kMaxSub) {
        udev_set_error(d, "bp_tiles: %d subsets (at most %d)", n_subsets, kMaxSub);
        return UFOIR_ERR_UNSUPPORTED;
    }
    int total = 0;
    for (int i = 0; i < n_subsets; i++) {
        if (subsets[i].offset + (size_t) subsets[i].n > (size_t) g->n_angles) {
            udev_set_error(d, "bp: subset [%u, %u) outside [0, %d)", subsets[i].offset,
                           subsets[i].offset + subsets[i].n, g->n_angles);
            return UFOIR_ERR_INVALID;
        }
        total += (int) subsets[i].n;
    }
    memset(&A, 0, sizeof(A));
    A.sino = sino;
    A.base = base;
    A.cw = cw;
    A.add = add;
    A.dst = dst;
    A.sinv = g->d_sin;
    A.cosv = g->d_cos;
    A.n = g->n_dets;
    A.axis = g->axis;
    A.relax = relax;
    A.vol_stride = (long long) g->n_dets * g->n_dets;
    A.sino_stride = (long long) g->n_angles * g->n_dets;
    A.cw_stride = cw_shared ? 0 : A.vol_stride;
    A.n_subsets = n_subsets;
    A.total_angles = total;
    A.neg_zero = -0.0f;
    A.contiguous = 1;
    A.first_angle = n_subsets > 0 ? (int) subsets[0].offset : 0;
    for (int i = 1; i < n_subsets; i++)
        if (subsets[i].offset != subsets[i - 1].offset + subsets[i - 1].n)
            A.contiguous = 0;
    for (int i = 0; i < kMaxSub; i++) {
        A.sub_offset[i] = i < n_subsets ? subsets[i].offset : 0;
        A.sub_n[i] = i < n_subsets ? subsets[i].n : 0;
    }
    return UFOIR_OK;
}

template <class T>
static int launch_bp(udev *d, const BpTileArgs &B, int fast_arith, int n_slices)
{
    const unsigned int tiles = udev_div_up(B.n, T::TileX) * udev_div_up(B.n, T::TileY);
    const dim3 grid(tiles, (unsigned int) n_slices), block(kTX, T::TY);
    if (fast_arith)
        bp_tiles_kernel<T, true><<<grid, block, 0, d->stream>>>(B);
    else
        bp_tiles_kernel<T, false><<<grid, block, 0, d->stream>>>(B);
    return udev_after_launch(d, "bp_tiles_kernel");
}

}  // namespace

extern "C" size_t udev_bp_record_bytes(void)
{
    return sizeof(BpTileArgs);
}

extern "C" int udev_bp_record(udev *d, const udev_geom *g, const ufoir_subset *subsets, int n_subsets,
                              const float *sino, const float *base, const float *cw, const float *add, float *dst,
                              float relax, void *record, int *items)
{
    BpTileArgs A;
    const int rc = fill_args(d, g, subsets, n_subsets, sino, base, cw, 0, add, dst, relax, A);
    if (rc)
        return rc;
    memcpy(record, &A, sizeof(A));
    const int tiles_x = (g->n_dets + BatchShape::TileX - 1) / BatchShape::TileX;
    const int tiles_y = (g->n_dets + BatchShape::TileY - 1) / BatchShape::TileY;
    *items = tiles_x * tiles_y;
    return UFOIR_OK;
}

extern "C" int udev_bp_batch(udev *d, int fast_arith, const void *d_records, const int *d_item_start, int n_jobs,
                             const int *d_job_index, const int *d_active, int n_items)
{
    if (n_jobs <= 0 || n_items <= 0)
        return UFOIR_OK;
    UDEV_BIND(d);
    if (fast_arith)
        bp_tiles_batch_kernel<true><<<(unsigned int) n_items, dim3(kTX, BatchShape::TY), 0, d->stream>>>(
            static_cast<const BpTileArgs *>(d_records), d_item_start, n_jobs, d_job_index, d_active);
    else
        bp_tiles_batch_kernel<false><<<(unsigned int) n_items, dim3(kTX, BatchShape::TY), 0, d->stream>>>(
            static_cast<const BpTileArgs *>(d_records), d_item_start, n_jobs, d_job_index, d_active);
    return udev_after_launch(d, "bp_tiles_batch_kernel");
}

extern "C" int udev_bp_tiles(udev *d, const udev_geom *g, const ufoir_subset *subsets, int n_subsets,
                             const float *sino, const float *base, const float *cw, int cw_shared, const float *add,
                             float *dst, float relax, int n_slices)
{
    if (n_slices <= 0)
        return UFOIR_OK;
    BpTileArgs A;
    const int rc0 = fill_args(d, g, subsets, n_subsets, sino, base, cw, cw_shared, add, dst, relax, A);
    if (rc0)
        return rc0;
    UDEV_BIND(d);
    const int shape = bp_shape(d, g->n_dets, n_slices);
    for (int done = 0; done < n_slices;) {
        const int chunk = n_slices - done > 65535 ? 65535 : n_slices - done;
        BpTileArgs B = A;
        B.sino += (size_t) done * A.sino_stride;
        if (B.base)
            B.base += (size_t) done * A.vol_stride;
        if (B.cw)
            B.cw += (size_t) done * A.cw_stride;
        if (B.add)
            B.add += (size_t) done * A.vol_stride;
        B.dst += (size_t) done * A.vol_stride;
        const int rc = shape == 0   ? launch_bp<ShapeL>(d, B, g->fast_arith, chunk)
                       : shape == 1 ? launch_bp<ShapeM>(d, B, g->fast_arith, chunk)
                       : shape == 2 ? launch_bp<ShapeS>(d, B, g->fast_arith, chunk)
                                    : launch_bp<ShapeT>(d, B, g->fast_arith, chunk);
        if (rc)
            return rc;
        done += chunk;
    }
    return UFOIR_OK;
}
