/*
 * udev_sbtv.cu - the vector updates of split-Bregman TV's CGS
 * (sbtv-task.c:404-585) on a batch of slices in one launch each, every slice
 * with its own scalar, slices outside the mask left as they are. Every
 * operation rounds as the reference's (IEEE float, no contraction).
 *
 * One pass each, bound by HBM (or L2 at small sizes), instead of a launch and
 * a pass per operation and slice. Four slices of 724^2, one outer iteration:
 * 1700 launches of 8.1 ms in all became 370 of 1.9 ms, and the call (with the
 * inner products of udev_ops.cu) went from 78.5 to 49.1 ms.
 */
#include <cuda_runtime.h>

#include "udev_internal.cuh"

namespace {

constexpr int kThreads = 256;

struct SliceScalars {
    float m[UDEV_SBTV_SLICES];
    unsigned int mask;
};

/* u = r + m q;  p = u + m (q + m p);  first: u = p = r */
__global__ void __launch_bounds__(kThreads) cgs_dir_kernel(SliceScalars S, int first, const float *__restrict__ r,
                                                           const float *__restrict__ q, float *__restrict__ u,
                                                           float *__restrict__ p, size_t per_slice)
{
    if (!((S.mask >> blockIdx.y) & 1u))
        return;
    const float m = S.m[blockIdx.y];
    const size_t base = (size_t) blockIdx.y * per_slice;
    for (size_t i = (size_t) blockIdx.x * kThreads + threadIdx.x; i < per_slice; i += (size_t) gridDim.x * kThreads) {
        const size_t k = base + i;
        if (first) {
            u[k] = p[k] = r[k];
            continue;
        }
        const float qv = q[k];
        const float uv = __fadd_rn(r[k], __fmul_rn(m, qv));
        const float t = __fadd_rn(qv, __fmul_rn(m, p[k]));
        u[k] = uv;
        p[k] = __fadd_rn(uv, __fmul_rn(m, t));
    }
}

/* q = u + m v;  uh = u + q */
__global__ void __launch_bounds__(kThreads) cgs_step_kernel(SliceScalars S, const float *__restrict__ u,
                                                            const float *__restrict__ v, float *__restrict__ q,
                                                            float *__restrict__ uh, size_t per_slice)
{
    if (!((S.mask >> blockIdx.y) & 1u))
        return;
    const float m = S.m[blockIdx.y];
    const size_t base = (size_t) blockIdx.y * per_slice;
    for (size_t i = (size_t) blockIdx.x * kThreads + threadIdx.x; i < per_slice; i += (size_t) gridDim.x * kThreads) {
        const size_t k = base + i;
        const float uv = u[k];
        const float qv = __fadd_rn(uv, __fmul_rn(m, v[k]));
        q[k] = qv;
        uh[k] = __fadd_rn(uv, qv);
    }
}

/* out = a + m b (MODE 0), a - b (1) or a (2) */
template <int MODE>
__global__ void __launch_bounds__(kThreads) masked_kernel(SliceScalars S, const float *a, const float *b, float *out,
                                                          size_t per_slice)
{
    if (!((S.mask >> blockIdx.y) & 1u))
        return;
    const float m = S.m[blockIdx.y];
    const size_t base = (size_t) blockIdx.y * per_slice;
    for (size_t i = (size_t) blockIdx.x * kThreads + threadIdx.x; i < per_slice; i += (size_t) gridDim.x * kThreads) {
        const size_t k = base + i;
        out[k] = MODE == 0 ? __fadd_rn(a[k], __fmul_rn(m, b[k])) : MODE == 1 ? __fsub_rn(a[k], b[k]) : a[k];
    }
}

/* out = lambda (Dyt Dy in + Dxt Dx in) + mu at, the differences periodic
 * (ufo-ir-gradient-processor.cl:1-51; sbtv-task.c:587-635). */
__global__ void __launch_bounds__(kThreads) laplace_kernel(const float *__restrict__ in, const float *__restrict__ at,
                                                           float *__restrict__ out, int n, float lambda, float mu,
                                                           size_t per_slice)
{
    const int x = (int) (blockIdx.x * 32 + threadIdx.x), y = (int) (blockIdx.y * 8 + threadIdx.y);
    if (x >= n || y >= n)
        return;
    const float *p = in + (size_t) blockIdx.z * per_slice;
    const size_t k = (size_t) y * n + x;
    const float c = p[k];
    const float up = p[(size_t) (y == 0 ? n - 1 : y - 1) * n + x], down = p[(size_t) (y == n - 1 ? 0 : y + 1) * n + x];
    const float left = p[(size_t) y * n + (x == 0 ? n - 1 : x - 1)], right = p[(size_t) y * n + (x == n - 1 ? 0 : x + 1)];
    const float dy = __fsub_rn(__fsub_rn(c, up), __fsub_rn(down, c));
    const float dx = __fsub_rn(__fsub_rn(c, left), __fsub_rn(right, c));
    const float d = __fmul_rn(__fadd_rn(dy, dx), lambda);
    const size_t o = (size_t) blockIdx.z * per_slice + k;
    out[o] = __fadd_rn(d, __fmul_rn(at[o], mu));
}

SliceScalars scalars(const float *m, unsigned int mask)
{
    SliceScalars S;
    for (int i = 0; i < UDEV_SBTV_SLICES; ++i)
        S.m[i] = m && ((mask >> i) & 1u) ? m[i] : 0.0f;
    S.mask = mask;
    return S;
}

dim3 slice_grid(udev *d, size_t per_slice, int n_slices)
{
    const size_t want = (per_slice + kThreads - 1) / kThreads;
    const size_t cap = ((size_t) d->sm_count * 16 + (size_t) n_slices - 1) / (size_t) n_slices;
    return dim3((unsigned int) (want < cap ? want : cap), (unsigned int) n_slices);
}

int check(udev *d, int n_slices)
{
    if (n_slices > UDEV_SBTV_SLICES) {
        udev_set_error(d, "sbtv: %d slices (at most %d)", n_slices, UDEV_SBTV_SLICES);
        return UFOIR_ERR_INVALID;
    }
    return UFOIR_OK;
}

}  // namespace

extern "C" int udev_cgs_dir(udev *d, const float *beta, unsigned int mask, int first, const float *r, const float *q,
                            float *u, float *p, size_t per_slice, int n_slices)
{
    if (per_slice == 0 || n_slices <= 0 || mask == 0)
        return UFOIR_OK;
    int rc = check(d, n_slices);
    if (rc)
        return rc;
    UDEV_BIND(d);
    cgs_dir_kernel<<<slice_grid(d, per_slice, n_slices), kThreads, 0, d->stream>>>(scalars(beta, mask), first, r, q, u,
                                                                                  p, per_slice);
    return udev_after_launch(d, "cgs_dir_kernel");
}

extern "C" int udev_cgs_step(udev *d, const float *m, unsigned int mask, const float *u, const float *v, float *q,
                             float *uh, size_t per_slice, int n_slices)
{
    if (per_slice == 0 || n_slices <= 0 || mask == 0)
        return UFOIR_OK;
    int rc = check(d, n_slices);
    if (rc)
        return rc;
    UDEV_BIND(d);
    cgs_step_kernel<<<slice_grid(d, per_slice, n_slices), kThreads, 0, d->stream>>>(scalars(m, mask), u, v, q, uh,
                                                                                   per_slice);
    return udev_after_launch(d, "cgs_step_kernel");
}

extern "C" int udev_masked(udev *d, int op, const float *a, const float *b, const float *m, unsigned int mask,
                           float *out, size_t per_slice, int n_slices)
{
    if (per_slice == 0 || n_slices <= 0 || mask == 0)
        return UFOIR_OK;
    int rc = check(d, n_slices);
    if (rc)
        return rc;
    UDEV_BIND(d);
    const dim3 grid = slice_grid(d, per_slice, n_slices);
    const SliceScalars S = scalars(m, mask);
    switch (op) {
    case UDEV_ADD_SCALED: masked_kernel<0><<<grid, kThreads, 0, d->stream>>>(S, a, b, out, per_slice); break;
    case UDEV_SUB: masked_kernel<1><<<grid, kThreads, 0, d->stream>>>(S, a, b, out, per_slice); break;
    default: masked_kernel<2><<<grid, kThreads, 0, d->stream>>>(S, a, a, out, per_slice); break;
    }
    return udev_after_launch(d, "masked_kernel");
}

extern "C" int udev_laplace(udev *d, const float *in, const float *at, float *out, int n, float lambda, float mu,
                            int n_slices)
{
    if (n <= 0 || n_slices <= 0)
        return UFOIR_OK;
    int rc = check(d, n_slices);
    if (rc)
        return rc;
    UDEV_BIND(d);
    const dim3 grid(udev_div_up(n, 32), udev_div_up(n, 8), (unsigned int) n_slices);
    laplace_kernel<<<grid, dim3(32, 8), 0, d->stream>>>(in, at, out, n, lambda, mu, (size_t) n * n);
    return udev_after_launch(d, "laplace_kernel");
}
