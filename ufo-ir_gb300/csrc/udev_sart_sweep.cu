/*
 * udev_sart_sweep.cu - a run of SART angles in one kernel (sart-task.c:209-217
 * for the angles of one direction), for images that fit in the shared memory
 * of one thread-block cluster.
 *
 * Two kernels per angle spend most of a small image's time between kernels:
 * at 367^2 an angle took 5.3 us, of which launches, the hand-over through L2
 * and the first loads of each kernel were about 4. Here the cluster holds the
 * slice for the whole run: CTA (b, p) keeps the pixels of the 64-sample block
 * b (64 image rows, or 64 columns for horizontal rays) that part p of the
 * columns needs, projects the rays that cross the block there, and the CTAs
 * exchange the block sums over distributed shared memory. An angle at 367^2
 * takes 3.9 us (2.1 at 64^2, was 4.4), and a cluster being 16 SMs at most, as
 * long for 8 slices as for one (6.8 us for 8 before). Every value is computed
 * by the operations of the per-angle kernels in their order, so the results
 * are the same bits.
 */
#include <cuda_runtime.h>

#include "bp_shapes.cuh"
#include "joseph.cuh"
#include "tma.cuh"
#include "udev_internal.cuh"

namespace {

constexpr int kBlock = 64;         /* samples per block of a ray (the reference's BLOCK_SIZE) */
/* 16 warps of up to 128 registers: with 32 warps of 64 both halves of an angle
 * were slower (4.5 against 4.1 us at 367^2), the loads of a warp in flight
 * counting for more than the number of warps. */
constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kHalf = 32;          /* rows of a block per warp of a pair */
constexpr int kBatch = 4;          /* samples whose taps are in flight together, two batches at a time */
constexpr int kPerThread = 2;      /* rays that a thread finishes */
constexpr int kMaxCluster = 16;
constexpr int kMaxDets = kPerThread * kThreads;
constexpr int kHalo = 36;          /* columns kept beyond a part: 32 rows of slope <= UDEV_SART_SPLIT_SLOPE, two taps, rounding */
constexpr int kPad = 2;            /* zero columns at either end of a tile row */
constexpr int kResidPad = 4;

struct SweepArgs {
    float *x;                  /* [slices][n][n], updated in place */
    const float *table;        /* [n_angles][n_blocks][n] block-start coordinates */
    const float *src;
    const float *w;
    const float *sinv;
    const float *cosv;
    int n;
    int n_blocks;
    int parts;                 /* column parts per block */
    int part_cols;             /* columns of a part (the last may have fewer) */
    int pitch;                 /* of a tile row, odd */
    int first, end;            /* angles [first, end), all of direction dir */
    int dir;
    float axis;
    float scale;
    float os, shift, e0, e1;
    float relax;
    float neg_zero;
    const float *relax_dev;
    int skip_angle;            /* testing: angle whose exchange never completes (-1 = none) */
    int *err;
    long long vol_stride;
    long long sino_stride;
    long long w_stride;
};

__device__ __forceinline__ void cluster_sync_all()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

/* Stores v at the address `local` has here in CTA `rank`'s shared memory and
 * counts its 4 bytes on the barrier `bar` there (a release at cluster scope). */
__device__ __forceinline__ void st_async(float *local, uint64_t *bar, int rank, float v)
{
    uint32_t dst, rbar;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(tma::smem_addr(local)), "r"(rank));
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rbar) : "r"(tma::smem_addr(bar)), "r"(rank));
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst),
                 "r"(__float_as_uint(v)), "r"(rbar)
                 : "memory");
}

__device__ __forceinline__ bool try_wait_cluster(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(tma::smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

/* Waits for the sums and words of all CTAs; false, with the error word
 * set, after the limit of tma::mbar_wait. */
__device__ __forceinline__ bool wait_cluster(uint64_t *bar, uint32_t parity, int *err)
{
    if (try_wait_cluster(bar, parity))
        return true;
    const unsigned long long t0 = tma::global_ns();
    while (!try_wait_cluster(bar, parity)) {
        if (tma::global_ns() - t0 > tma::kWaitLimitNs) {
            tma::report(err, tma::kErrWaitTimeout);
            return false;
        }
    }
    return true;
}

/* Bytes that rank 0's barrier of angle `a` expects beyond the sums (testing). */
__device__ __forceinline__ uint32_t skip_bytes(const SweepArgs &P, int rank, int a)
{
    return rank == 0 && a == P.skip_angle ? 16u : 0u;
}

/* The rays that part `part` projects: those whose coordinate m0 + s * det_step
 * in the middle of the block lies in its columns. Every CTA of a block
 * evaluates the same expressions, so the parts' ranges meet exactly; a
 * rounding that moves a ray to the neighbour stays within the halo. */
__device__ __forceinline__ int part_bound(const SweepArgs &P, int part, float m0, float det_step)
{
    const bool up = det_step > 0.0f;
    if (part <= 0)
        return up ? 0 : P.n;
    if (part >= P.parts)
        return up ? P.n : 0;
    const float s = ceilf(__fdiv_rn(__fsub_rn((float) (part * P.part_cols), m0), det_step));
    return (int) fminf(fmaxf(s, 0.0f), (float) P.n);
}

/* What a CTA projects at an angle: rays [begin, end) of slope step. */
struct AngleRays {
    float sn, cs, step;
    int begin, end;
};

/* c0: ray 0's coordinate at the block start */
__device__ __forceinline__ AngleRays angle_rays(const SweepArgs &P, int part, float sn, float cs, float c0)
{
    AngleRays r;
    r.sn = sn;
    r.cs = cs;
    float det_step;
    joseph::ray_steps(P.dir, sn, cs, det_step, r.step);
    const float m0 = __fadd_rn(c0, __fmul_rn((float) (kBlock / 2), r.step));
    const int u = part_bound(P, part, m0, det_step), v = part_bound(P, part + 1, m0, det_step);
    r.begin = min(u, v);
    r.end = max(u, v);
    return r;
}

/* K samples of a ray from coordinate c on: fractions and taps. CLAMP:
 * coordinates may leave [lo, hi], beyond which both taps are zero columns. */
template <int K>
struct Batch {
    float t[K], t0[K], t1[K];
};

template <bool CLAMP, int K>
__device__ __forceinline__ void issue(Batch<K> &B, float &c, float step, uint32_t &row, uint32_t pitch, float lo,
                                      float hi)
{
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const float cm = __fsub_rn(CLAMP ? fminf(fmaxf(c, lo), hi) : c, 0.5f);
        const float y = __fadd_rd(cm, joseph::kFloorMagic);
        B.t[k] = __fsub_rn(cm, __fsub_rn(y, joseph::kFloorMagic));
        const uint32_t i = row + 4u * (uint32_t) __float_as_int(y);
        B.t0[k] = joseph::lds(i);
        B.t1[k] = joseph::lds(i + 4u);
        row += pitch;
        c = __fadd_rn(c, step);
    }
}

template <int K>
__device__ __forceinline__ void add(const Batch<K> &B, float &run)
{
#pragma unroll
    for (int k = 0; k < K; ++k)
        run = __fadd_rn(run, joseph::lerp(B.t[k], B.t0[k], B.t1[k]));
}

template <int K>
__device__ __forceinline__ void keep(const Batch<K> &B, float *&v)
{
#pragma unroll
    for (int k = 0; k < K; ++k)
        v[32 * k] = joseph::lerp(B.t[k], B.t0[k], B.t1[k]);
    v += 32 * K;
}

/* kHalf samples of a ray: their sum in order (SUM), or the samples in v. */
template <bool CLAMP, bool SUM>
__device__ __forceinline__ float half_block(float c, float step, uint32_t row, uint32_t pitch, float lo, float hi,
                                            float *v)
{
    constexpr int K = kBatch;
    float run = 0.0f;
    Batch<K> A, B;
    issue<CLAMP, K>(A, c, step, row, pitch, lo, hi);
#pragma unroll 1
    for (int r = 0; r < kHalf; r += 2 * K) {
        issue<CLAMP, K>(B, c, step, row, pitch, lo, hi);
        if (SUM)
            add<K>(A, run);
        else
            keep<K>(A, v);
        if (r + 2 * K < kHalf)
            issue<CLAMP, K>(A, c, step, row, pitch, lo, hi);
        if (SUM)
            add<K>(B, run);
        else
            keep<K>(B, v);
    }
    return run;
}

/* Barrier of the 64 threads of a warp pair: `pair` in 0 .. kWarps / 2 - 1. */
__device__ __forceinline__ void pair_sync(int pair)
{
    asm volatile("bar.sync %0, 64;" ::"r"(pair + 1) : "memory");
}

/* The pixels of a column in rows 0, kWarps, 2 kWarps, 3 kWarps from px on:
 * pixel + relax * (0 + sample). All loads come before the first store. fI:
 * the column's centre less the origin shift. */
template <bool T>
__device__ __forceinline__ void bp_column(const SweepArgs &P, float *px, float fI, int rows, const float2 (&qr)[2],
                                          float col_factor, uint32_t rs_base, float relax, float2 z2)
{
    float2 t[2], t0[2], t1[2], x[2];
    const float2 pc = joseph::splat(__fmul_rn(fI, col_factor));
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const float *pa = px + 2 * m * kWarps * P.pitch;
        float2 c = joseph::add2(T ? joseph::sub2(qr[m], pc) : joseph::sub2(pc, qr[m]), joseph::splat(P.shift));
        c = make_float2(fminf(fmaxf(c.x, P.e0), P.e1), fminf(fmaxf(c.y, P.e0), P.e1));
        const float2 y = joseph::floor_half2(c, t[m]);
        const uint32_t ia = rs_base + 4u * (uint32_t) __float_as_int(y.x);
        const uint32_t ib = rs_base + 4u * (uint32_t) __float_as_int(y.y);
        t0[m] = make_float2(joseph::lds(ia), joseph::lds(ib));
        t1[m] = make_float2(joseph::lds(ia + 4u), joseph::lds(ib + 4u));
        x[m] = make_float2(pa[0], pa[kWarps * P.pitch]);
    }
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        float *pa = px + 2 * m * kWarps * P.pitch;
        const float2 sum = joseph::add2(joseph::splat(0.0f), joseph::lerp2(t[m], t0[m], t1[m], z2));
        const float2 upd = joseph::add2(x[m], joseph::mul2z(joseph::splat(relax), sum, z2));
        /* the rows past the image stay zero */
        if (2 * m * kWarps < rows)
            pa[0] = upd.x;
        if ((2 * m + 1) * kWarps < rows)
            pa[kWarps * P.pitch] = upd.y;
    }
}

/*
 * A run of angles on one slice per cluster. Grid (n_blocks * parts, 1,
 * slices), cluster (n_blocks * parts, 1, 1).
 *
 * Per angle: warps 2g and 2g + 1 take the upper and lower 32 rows of the block
 * for 32 rays; the lower one keeps its samples and adds them, in order, to
 * the upper one's sum (…joseph.cl:84-92). The sums go to every CTA of the
 * cluster by st.async, counted in bytes on a barrier there, and beside them a
 * word from every CTA (two buffers, by the parity of the angle: a CTA sends its
 * word once it is done with the sums of the angle before, with or without rays
 * of its own, so past the wait of an angle nobody still reads the buffer that
 * the next angle's sums go to). The word costs 0.03 us an angle (3.86 -> 3.89
 * at 367^2; an mbarrier.arrive with release in its place 4.04, as it waits for
 * the loads in flight). Each CTA adds the blocks of all
 * rays in order and finishes the residual row itself, so the residual never
 * travels. The backprojection updates the CTA's tile, halo included, so parts
 * agree on the pixels that they both keep. The next angle's block starts
 * arrive by cp.async meanwhile, and one thread works out its ray range.
 *
 * An angle at 367^2 is about 8,000 cycles: 3,000 for the projection and 2,900
 * for the backprojection (12 CTAs; their shared-memory wavefronts are 1,200
 * and 2,000), 600 for the exchange and 500 for the sums over blocks. What is
 * left over is latency: 16 warps of dependent steps between barriers. More
 * CTAs cannot share a block's sum, which is a chain of 64 additions.
 */
template <bool T>
__global__ void __launch_bounds__(kThreads, 1) sart_sweep_kernel(SweepArgs P)
{
    extern __shared__ __align__(16) float sm[];
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ float word;              /* where the CTAs' words go; never read */
    __shared__ AngleRays rays_s[2];     /* by the parity of the angle */
    __shared__ float half_s[kWarps / 2][kHalf + 1][32];     /* a pair's first sum, second samples */
    const int n = P.n, nb = P.n_blocks, C = nb * P.parts;
    const int tid = (int) threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = (int) blockIdx.x, b = rank / P.parts, part = rank % P.parts;
    const int slice = (int) blockIdx.z;
    const int c_lo = part * P.part_cols, c_hi = min(n, c_lo + P.part_cols);
    const int h0 = max(0, c_lo - kHalo), h1 = min(n, c_hi + kHalo);
    const int row0 = b * kBlock, rows = min(kBlock, n - row0);
    float *tile = sm;                              /* [64][pitch] */
    float *rs = tile + kBlock * P.pitch;           /* residual row between zeros */
    float *tab = rs + n + 2 * kResidPad;           /* [2][n] */
    float *bs = tab + 2 * n;                       /* [2][nb][n] */
    float *vol = P.x + (size_t) slice * P.vol_stride;
    const float *tab_g = P.table + (size_t) b * n;
    const size_t tab_angle = (size_t) nb * n;

    for (int i = tid; i < kBlock * P.pitch; i += kThreads)
        tile[i] = 0.0f;
    for (int i = tid; i < n + 2 * kResidPad; i += kThreads)
        rs[i] = 0.0f;
    for (int i = tid; i < n; i += kThreads)
        bp::cp_async4(tab + i, tab_g + P.first * tab_angle + i);
    bp::cp_async_commit();
    __syncthreads();
    /* element (r, i) of the tile is pixel x = i, y = row0 + r, or with T x = row0 + r, y = i */
    if (T) {
        for (int i = h0 + (tid >> 6); i < h1; i += kThreads / 64)
            if ((tid & 63) < rows)
                tile[(tid & 63) * P.pitch + kPad + i - h0] = vol[(size_t) i * n + row0 + (tid & 63)];
    } else {
        for (int r = warp; r < rows; r += kThreads / 32)
            for (int i = h0 + lane; i < h1; i += 32)
                tile[r * P.pitch + kPad + i - h0] = vol[(size_t) (row0 + r) * n + i];
    }

    const joseph::AxisConsts kc = joseph::axis_consts(n, P.axis);
    const float relax = P.relax_dev ? *P.relax_dev : P.relax;
    const float2 z2 = joseph::splat(P.neg_zero);
    const float clamp_lo = (float) (h0 - 1), clamp_hi = (float) (h1 + 1);
    const uint32_t tile_u = (uint32_t) __cvta_generic_to_shared(tile);
    const uint32_t pitch_b = 4u * (uint32_t) P.pitch;
    const uint32_t fp_base = tile_u + 4u * (uint32_t) (kPad - h0 - joseph::kFloorMagicBits);
    const uint32_t rs_base = (uint32_t) __cvta_generic_to_shared(rs) +
                             4u * (uint32_t) (kResidPad - joseph::kHalfFloorBits);
    float2 fJ[2];
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const int ja = min(row0 + warp + 2 * m * kWarps, n - 1), jb = min(row0 + warp + (2 * m + 1) * kWarps, n - 1);
        fJ[m] = make_float2(__fsub_rn(__fadd_rn((float) ja, 0.5f), P.os), __fsub_rn(__fadd_rn((float) jb, 0.5f), P.os));
    }
    /* the last thread works out the next angle's rays while the first warps project */
    const bool planner = tid == kThreads - 1;
    float sn_next = 0.0f, cs_next = 0.0f, c0_next = 0.0f;
    const uint32_t sum_bytes = 4u * (uint32_t) (nb * n + C);
    if (planner)
        rays_s[0] = angle_rays(P, part, __ldg(P.sinv + P.first), __ldg(P.cosv + P.first),
                               __ldg(tab_g + P.first * tab_angle));
    if (tid == 0) {
        for (int k = 0; k < 2; ++k) {
            tma::mbar_init(&bars[k], 1);
            tma::mbar_arrive_expect_tx(&bars[k], sum_bytes + skip_bytes(P, rank, P.first + k));
        }
        tma::fence_mbar_init();
    }
    bool active[kPerThread];
    for (int k = 0; k < kPerThread; ++k)
        active[k] = !joseph::detector_inactive(kc, tid + k * kThreads);
    bool ok = true;
    /* every CTA of the cluster runs, its barriers armed, before the first remote store */
    cluster_sync_all();

#pragma unroll 1
    for (int a = P.first; a < P.end; ++a) {
        const int par = (a - P.first) & 1;
        /* this angle's src and w, the next one's sine, cosine and block starts */
        float src_v[kPerThread], w_v[kPerThread];
#pragma unroll
        for (int k = 0; k < kPerThread; ++k) {
            const int s = tid + k * kThreads;
            src_v[k] = w_v[k] = 0.0f;
            if (s < n) {
                src_v[k] = P.src[(size_t) slice * P.sino_stride + (size_t) a * n + s];
                if (P.w)
                    w_v[k] = P.w[(size_t) slice * P.w_stride + (size_t) a * n + s];
            }
        }
        const int a_next = min(a + 1, P.end - 1);
        if (planner) {
            sn_next = __ldg(P.sinv + a_next);
            cs_next = __ldg(P.cosv + a_next);
            c0_next = __ldg(tab_g + a_next * tab_angle);
        }
        bp::cp_async_wait<0>();
        __syncthreads();
        /* this CTA has read the other buffer, the angle before's: its word to
         * every CTA (the last warp is the first without rays) */
        if (warp == kWarps - 1 && lane < C)
            st_async(&word, &bars[par], lane, 0.0f);
        for (int i = tid; i < n; i += kThreads)
            bp::cp_async4(tab + (par ^ 1) * n + i, tab_g + a_next * tab_angle + i);
        bp::cp_async_commit();

        const float *tb = tab + par * n;
        float *bsum = bs + (size_t) par * nb * n;
        {
            const float step = rays_s[par].step;
            const int s_end = rays_s[par].end;
            const float reach = __fmul_rn((float) kBlock, step);
            float *out = bsum + b * n;
            if (planner)
                rays_s[par ^ 1] = angle_rays(P, part, sn_next, cs_next, c0_next);
            __syncwarp();
            const int half = warp & 1, pair = warp >> 1;
            float *mine = &half_s[pair][0][lane];
            const uint32_t row = fp_base + (half ? kHalf * pitch_b : 0u);
            for (int s0 = rays_s[par].begin + 32 * pair; s0 < s_end; s0 += 32 * (kWarps / 2)) {
                const int s = s0 + lane;
                float c = tb[min(s, s_end - 1)];
                const float c_end = __fadd_rn(c, reach);
                /* rays beside the image read zeros in the whole block */
                const bool out_left = c < -1.0f && c_end < -1.0f;
                const bool out_right = c > (float) (n + 1) && c_end > (float) (n + 1);
                const bool inside = c >= clamp_lo && c <= clamp_hi && c_end >= clamp_lo && c_end <= clamp_hi;
                const bool all_inside = __all_sync(0xffffffffu, inside);
                const bool any = __any_sync(0xffffffffu, !out_left && !out_right);
                float sum = 0.0f;
                if (any) {
                    if (half) {
#pragma unroll
                        for (int k = 0; k < kHalf; ++k)
                            c = __fadd_rn(c, step);
                        if (all_inside)
                            half_block<false, false>(c, step, row, pitch_b, clamp_lo, clamp_hi, mine + 32);
                        else
                            half_block<true, false>(c, step, row, pitch_b, clamp_lo, clamp_hi, mine + 32);
                        pair_sync(pair);
                        float v[kHalf + 1];
#pragma unroll
                        for (int k = 0; k <= kHalf; ++k)
                            v[k] = mine[32 * k];
                        sum = v[0];
#pragma unroll
                        for (int k = 1; k <= kHalf; ++k)
                            sum = __fadd_rn(sum, v[k]);
                    } else {
                        if (all_inside)
                            sum = half_block<false, true>(c, step, row, pitch_b, clamp_lo, clamp_hi, nullptr);
                        else
                            sum = half_block<true, true>(c, step, row, pitch_b, clamp_lo, clamp_hi, nullptr);
                        mine[0] = sum;
                        pair_sync(pair);
                    }
                }
                if (half && s < s_end)
#pragma unroll 1
                    for (int r = 0; r < C; ++r)
                        st_async(out + s, &bars[par], r, sum);
                /* before the next round's first sum replaces this one */
                if (any)
                    pair_sync(pair);
            }
        }
        ok = wait_cluster(&bars[par], (uint32_t) ((a - P.first) >> 1) & 1, P.err);
        /* before any CTA can send that angle's sums; never after a wait that ran
         * out, whose phase has no arrival left to take */
        if (ok && tid == 0 && a + 2 < P.end)
            tma::mbar_arrive_expect_tx(&bars[par], sum_bytes + skip_bytes(P, rank, a + 2));
#pragma unroll
        for (int k = 0; k < kPerThread; ++k) {
            const int s = tid + k * kThreads;
            if (s < n) {
                float result = src_v[k];
                if (active[k]) {
                    float detected = 0.0f;
                    const float *bj = bsum + s;
                    float v[kMaxCluster];
#pragma unroll
                    for (int j = 0; j < kMaxCluster; ++j, bj += n)
                        v[j] = j < nb ? *bj : 0.0f;
#pragma unroll
                    for (int j = 0; j < kMaxCluster; ++j)
                        if (j < nb)
                            detected = __fadd_rn(detected, v[j]);
                    result = __fadd_rn(result, __fmul_rn(detected, P.scale));
                }
                if (P.w)
                    result = __fmul_rn(result, w_v[k]);
                rs[kResidPad + s] = result;
            }
        }
        /* a wait ran out: this CTA leaves the angles, the others at their next wait */
        ok = __syncthreads_and(ok) != 0;
        if (!ok)
            break;
        /* tile += relax * (0 + sample): rows warp + 16 m, pairs (m, m + 1) */
        {
            const float sn = rays_s[par].sn, cs = rays_s[par].cs;
            float2 qr[2];
#pragma unroll
            for (int m = 0; m < 2; ++m)
                qr[m] = make_float2(__fmul_rn(fJ[m].x, T ? cs : sn), __fmul_rn(fJ[m].y, T ? cs : sn));
#pragma unroll 1
            for (int i = h0 + lane; i < h1; i += 32)
                bp_column<T>(P, tile + warp * P.pitch + kPad + i - h0, __fsub_rn(__fadd_rn((float) i, 0.5f), P.os),
                             rows - warp, qr, T ? sn : cs, rs_base, relax, z2);
        }
    }
    bp::cp_async_wait<0>();
    /* every CTA has read its halo (before the first cluster barrier). No CTA
     * leaves before all are here: the stores to a CTA whose wait ran out were
     * sent before their senders' last waits, so that limit has passed since,
     * or this one's has. */
    __syncwarp();
    cluster_sync_all();
    if (!ok)
        return;     /* this CTA's part of the image stays as it was */
    if (T) {
        for (int i = c_lo + (tid >> 6); i < c_hi; i += kThreads / 64)
            if ((tid & 63) < rows)
                vol[(size_t) i * n + row0 + (tid & 63)] = tile[(tid & 63) * P.pitch + kPad + i - h0];
    } else {
        for (int r = warp; r < rows; r += kThreads / 32)
            for (int i = c_lo + lane; i < c_hi; i += 32)
                vol[(size_t) (row0 + r) * n + i] = tile[r * P.pitch + kPad + i - h0];
    }
}

struct SweepPlan {
    int parts;
    int part_cols;
    int pitch;
    int cluster;
    size_t smem;
    double us;      /* estimated time of an angle */
};

constexpr int kMinPartCols = 64;   /* of a split block: the halos are computed twice */

/* an upper bound on the kernel's static shared memory */
constexpr size_t kStaticSmem = sizeof(float) * (kWarps / 2) * (kHalf + 1) * 32 + 256;

const void *sweep_func(int dir)
{
    return dir == 0 ? (const void *) sart_sweep_kernel<true> : (const void *) sart_sweep_kernel<false>;
}

}  // namespace

int udev_sart_sweep_init(udev *d)
{
    for (int dir = 0; dir < 2; ++dir) {
        const void *func = sweep_func(dir);
        cudaFuncAttributes fa;
        UDEV_CHECK(d, cudaFuncGetAttributes(&fa, func));
        UDEV_CHECK(d, cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           d->smem_optin - (int) fa.sharedSizeBytes));
        if (cudaFuncSetAttribute(func, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
            cudaGetLastError();     /* sizes above the portable one are then not offered */
    }
    return UFOIR_OK;
}

/* The cheapest split of the columns for n_slices slices: more parts make an
 * angle shorter (but their halos are computed twice), fewer let more clusters
 * run at once. False if none fits. An angle takes, per wave of clusters, 2.1 us
 * (64^2), 2.9 (256^2 in 4 parts), 3.9 (367^2 in 2), 4.9 (448^2 in 2), 5.7
 * (512^2 in 2), 8.7 (530^2 in 1) on 152 SMs, about 1.3 + 0.0142 us per column. */
static bool sweep_plan(udev *d, int n, bool split, int n_slices, SweepPlan *best)
{
    const int nb = (n + kBlock - 1) / kBlock;
    best->us = 0.0;
    for (int parts = split ? kMaxCluster / nb : 1; parts >= 1; --parts) {
        SweepPlan s;
        s.part_cols = (n + parts - 1) / parts;
        if (parts > 1 && (s.part_cols < kMinPartCols || (parts - 1) * s.part_cols >= n))
            continue;
        s.parts = parts;
        int width = s.part_cols + kHalo * (parts > 2 ? 2 : parts - 1);
        if (width > n)
            width = n;
        s.pitch = (width + 2 * kPad) | 1;
        s.smem = sizeof(float) *
                 ((size_t) kBlock * s.pitch + n + 2 * kResidPad + 2 * (size_t) n + 2 * (size_t) nb * n);
        s.cluster = nb * parts;
        if (s.smem + kStaticSmem > (size_t) d->smem_optin)
            continue;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        cfg.gridDim = dim3((unsigned int) s.cluster, 1, 1);
        cfg.blockDim = dim3(kThreads, 1, 1);
        cfg.dynamicSmemBytes = s.smem;
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned int) s.cluster;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, sweep_func(0), &cfg) != cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        if (clusters < 1)
            continue;
        s.us = ((n_slices + clusters - 1) / clusters) * (1.3 + 0.0142 * width);
        if (best->us == 0.0 || s.us < best->us)
            *best = s;
    }
    return best->us > 0.0;
}

extern "C" int udev_sart_sweep_serves(udev *d, const udev_geom *g, int split, int n_slices)
{
    const int n = g->n_dets;
    float os, shift, e0, e1;
    if (n < 1 || n > kMaxDets || (n + kBlock - 1) / kBlock > kMaxCluster || n_slices < 1 || n_slices > 65535)
        return 0;
    udev_sart_bp_consts(g, &os, &shift, &e0, &e1);
    if (!(e0 <= e1) || cudaSetDevice(d->device) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    SweepPlan s;
    if (!sweep_plan(d, n, split != 0, n_slices, &s))
        return 0;
    /* the per-angle kernels take at least this: 5.3 us (367^2), 5.5 (448^2,
     * 512^2), 5.9 (530^2), 6.8 (367^2 x 8), 11.2 (x 16), 14.2 (530^2 x 8), 28.5
     * (x 20) */
    double angles_us = 2.3 + 4.2e-6 * n_slices * n * n;
    if (angles_us < 5.3)
        angles_us = 5.3;
    return s.us < angles_us;
}

extern "C" int udev_sart_sweep(udev *d, const udev_geom *g, int first, int end, int dir, int split,
                               const float *table, const float *src, const float *w, int w_shared, float *x,
                               float scale, float relax, const float *relax_dev, int n_slices)
{
    const int n = g->n_dets;
    if (n_slices <= 0 || first >= end)
        return UFOIR_OK;
    if (first < 0 || end > g->n_angles || n < 1 || n > kMaxDets || n_slices > 65535) {
        udev_set_error(d, "sart_sweep: angles %d..%d of %d, n = %d, %d slices out of range", first, end, g->n_angles,
                       n, n_slices);
        return UFOIR_ERR_INVALID;
    }
    UDEV_BIND(d);
    SweepPlan s;
    if (!sweep_plan(d, n, split != 0, n_slices, &s)) {
        udev_set_error(d, "sart_sweep: n = %d does not fit a cluster", n);
        return UFOIR_ERR_UNSUPPORTED;
    }
    SweepArgs A;
    udev_sart_bp_consts(g, &A.os, &A.shift, &A.e0, &A.e1);
    A.x = x;
    A.table = table;
    A.src = src;
    A.w = w;
    A.sinv = g->d_sin;
    A.cosv = g->d_cos;
    A.n = n;
    A.n_blocks = (n + kBlock - 1) / kBlock;
    A.parts = s.parts;
    A.part_cols = s.part_cols;
    A.pitch = s.pitch;
    A.first = first;
    A.end = end;
    A.dir = dir;
    A.axis = g->axis;
    A.scale = scale;
    A.relax = relax;
    A.neg_zero = -0.0f;
    A.relax_dev = relax_dev;
    A.skip_angle = -1;
    if (d->inject_skip_angle >= first && d->inject_skip_angle < end) {     /* one-shot test injection */
        A.skip_angle = d->inject_skip_angle;
        d->inject_skip_angle = -1;
    }
    A.err = d->d_err;
    A.vol_stride = (long long) n * n;
    A.sino_stride = (long long) g->n_angles * n;
    A.w_stride = w_shared ? 0 : A.sino_stride;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned int) s.cluster, 1, (unsigned int) n_slices);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = s.smem;
    cfg.stream = d->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned int) s.cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = dir == 0 ? cudaLaunchKernelEx(&cfg, sart_sweep_kernel<true>, A)
                                   : cudaLaunchKernelEx(&cfg, sart_sweep_kernel<false>, A);
    if (e != cudaSuccess) {
        cudaGetLastError();
        udev_set_error(d, "sart_sweep_kernel launch: %s", cudaGetErrorString(e));
        return UFOIR_ERR_CUDA;
    }
    return udev_after_launch(d, "sart_sweep_kernel");
}
