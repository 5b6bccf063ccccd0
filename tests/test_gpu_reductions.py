"""The reference's float reductions, which are sums in a fixed order, computed
in parallel: equality is exact. The L1 norm's reference is numpy's running
float32 sum (one addition after another), the dot product's the oracle.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = ("normal", "ones", "ties", "growing", "stagnating", "subnormal", "sparse", "overflow", "inf", "nan")


def _values(kind, count):
    rng = np.random.default_rng(count)
    x = rng.standard_normal(count).astype(np.float32)
    if kind == "ones":
        x[:] = 1.0
    elif kind == "ties":        # half units of the running sum again and again
        x = (rng.integers(0, 8, count) * np.float32(0.5)).astype(np.float32)
        x[0] = 2.0 ** 23 - 1
    elif kind == "growing":     # a new binade every few elements
        x = np.exp2(np.linspace(-126, 100, count)).astype(np.float32) * np.sign(x)
    elif kind == "stagnating":
        x[: count // 7] *= np.float32(1e7)
        x[count // 7:] *= np.float32(1e-3)
    elif kind == "subnormal":
        x *= np.float32(1e-41)
    elif kind == "sparse":
        x[rng.random(count) < 0.98] = -0.0
    elif kind == "overflow":
        x *= np.float32(3e37)
    elif kind in ("inf", "nan"):
        x[count // 3] = np.inf
        if kind == "nan":
            x[count // 2] = np.nan
    return x


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("h,w", [(1, 1), (1, 5), (7, 73), (16, 32), (63, 65), (301, 433), (1200, 731)])
def test_compat_l1_norm_is_the_sequential_sum(ufoir_lib, gpu_ctx, h, w, kind):
    x = _values(kind, h * w).reshape(h, w)
    with np.errstate(over="ignore", invalid="ignore"):
        want = np.cumsum(np.abs(x).reshape(-1), dtype=np.float32)[-1]
    np.testing.assert_array_equal(np.float32(gpu_ctx.l1_norm(x, ufoir_lib.NORM_COMPAT)), want)


@pytest.mark.parametrize("h,w", [(1, 1), (3, 17), (33, 31), (65, 300), (367, 367)])
def test_dot_products(ufoir_lib, gpu_ctx, oracle, h, w):
    rng = np.random.default_rng(h)
    a, b = (rng.standard_normal((h, w)).astype(np.float32) for _ in range(2))
    assert np.float32(gpu_ctx.dot_product(a, b, ufoir_lib.NORM_COMPAT)) == np.float32(oracle.dot_product(a, b))
    want = oracle.dot_product(a, b, fp64=True)
    terms = float(np.abs(a.astype(np.float64)).max() * np.abs(b.astype(np.float64)).max()) * h * w
    # one rounding of the result to float, and FP64 rounding of every sum
    assert abs(gpu_ctx.dot_product(a, b) - want) <= 2.0 ** -24 * abs(want) + 2.0 ** -50 * terms


# The TV gradient computes its FP64 norm beside it: image edges on and beside
# the edges of its 32 x 32 tiles, fewer tiles than CTAs and more, several slices.
@pytest.mark.parametrize("n,slices", [(1, 1), (31, 2), (32, 1), (33, 3), (65, 1), (300, 2), (1500, 1)])
def test_tv_step_takes_the_norm_of_its_gradient(ufoir_lib, gpu_ctx, n, slices):
    rng = np.random.default_rng(n + slices)
    na = 4
    sinos = (rng.random((slices, na, n), dtype=np.float32) + 0.5) * n
    p = ufoir_lib.ParallelProjector(gpu_ctx, step=float(np.float32(np.pi / na)), is_forward=False)
    kw = dict(num_iterations=1, norm_mode=ufoir_lib.NORM_FP64,
              df_minimizer=dict(num_iterations=1, relaxation_factor=0.25))
    vol, x_tv, sc = ufoir_lib.asdpocs_state(p, sinos, **kw)
    p.close()
    for s in range(slices):
        # 20 sub-steps x -= (alpha dp / |g|_1) g from the volume before them, each
        # operation rounded to float; the norm's 64-bit sums differ in their order
        # only (a relative 2^-40 at most), so they round to the same float
        x = vol[s].astype(np.float32)
        dtgv = np.float32(0.2) * np.float32(sc[s]["dp"])
        for _ in range(20):
            g = ufoir_lib.tv_gradient(gpu_ctx, x[None])[0]
            factor = dtgv / np.float32(np.abs(g.astype(np.float64)).sum())
            x = x - factor * g
        assert np.array_equal(x_tv[s], x), np.abs(x_tv[s] - x).max()


@pytest.mark.parametrize("n,slices", [(65, 9), (367, 5), (530, 7), (1200, 2)])
def test_a_slice_of_a_stack_has_its_own_norms(ufoir_lib, gpu_ctx, n, slices):
    """ASD-POCS (FP64 norms): a slice's steps do not depend on the stack it is in."""
    na = 12
    sinos = np.random.default_rng(n).random((slices, na, n), dtype=np.float32) * n
    p = ufoir_lib.ParallelProjector(gpu_ctx, step=float(np.float32(np.pi / na)), is_forward=False)
    kw = dict(num_iterations=2, df_minimizer=dict(num_iterations=1, relaxation_factor=0.5))
    vol, x_tv, scalars = ufoir_lib.asdpocs_state(p, sinos, **kw)
    for s in (0, slices - 1):
        one = ufoir_lib.asdpocs_state(p, sinos[s], **kw)
        assert np.array_equal(one[0], vol[s]) and np.array_equal(one[1], x_tv[s])
        assert one[2][0] == scalars[s]
    p.close()


# Short slices are added by one thread, longer ones in chunks of 512 elements or
# more, 512 of them at most: counts on and beside those lines.
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("count", [15, 17, 1023, 1024, 1025, 2048, 8191, 8192, 8193, 8703, 8704, 8705, 262143, 262144, 262657])
def test_compat_l1_norm_of_short_and_chunked_slices(ufoir_lib, gpu_ctx, count, kind):
    x = _values(kind, count).reshape(1, count)
    with np.errstate(over="ignore", invalid="ignore"):
        want = np.cumsum(np.abs(x).reshape(-1), dtype=np.float32)[-1]
    np.testing.assert_array_equal(np.float32(gpu_ctx.l1_norm(x, ufoir_lib.NORM_COMPAT)), want)


@pytest.mark.parametrize("count,kernels", [(1, 1), (8192, 1), (8193, 3)])
def test_compat_l1_norm_of_a_short_slice_is_one_kernel(ufoir_lib, gpu_ctx, count, kernels):
    x = np.ones((1, count), np.float32)
    before = gpu_ctx.kernel_launches()
    assert gpu_ctx.l1_norm(x, ufoir_lib.NORM_COMPAT) == count
    assert gpu_ctx.kernel_launches() - before == kernels
