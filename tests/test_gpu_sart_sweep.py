"""SART's sweep kernel (a run of angles with the slice in a cluster's shared
memory) against the general per-angle kernels, which are compared with the
oracle elsewhere: the same operations in the same order, so the same bits.

Sizes: one block and part of a block, whole blocks and one ray more, one to
four column parts per block, the largest that fit, and two that the per-angle
kernels keep; axes beside the centre (inactive detectors, clamped pixels);
values that are not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sart(u, ctx, sinos, axis, iters):
    na = sinos.shape[1]
    p = u.ParallelProjector(ctx, step=float(np.float32(np.pi / na)), is_forward=False, axis_position=axis)
    before = ctx.kernel_launches()
    out = u.sart(p, sinos, num_iterations=iters, relaxation_factor=0.3)
    launches = ctx.kernel_launches() - before
    p.close()
    return out, launches


@pytest.mark.parametrize("n,na,axis,slices,swept", [
    (1, 4, -1.0, 1, True), (2, 5, -1.0, 2, True), (31, 20, 14.2, 1, True), (63, 30, -1.0, 1, True),
    (64, 30, 31.1, 3, True), (65, 30, -1.0, 2, True), (127, 24, -1.0, 1, True), (128, 24, 65.3, 1, True),
    (129, 24, -1.0, 2, True), (200, 31, 97.4, 3, True), (256, 40, -1.0, 1, True), (256, 40, -1.0, 10, True),
    (256, 40, -1.0, 30, True), (300, 45, 151.2, 1, True), (367, 60, -1.0, 2, True), (385, 20, 190.7, 2, True),
    (449, 16, -1.0, 1, True), (512, 12, 259.0, 9, True), (530, 10, -1.0, 1, False), (530, 10, -1.0, 8, True),
    (560, 8, 278.4, 8, True), (600, 6, -1.0, 9, False)])
def test_sweep_equals_the_per_angle_kernels(ufoir_lib, gpu_ctx, monkeypatch, n, na, axis, slices, swept):
    rng = np.random.default_rng(7 * n + na)
    sinos = rng.random((slices, na, n), dtype=np.float32) * n
    monkeypatch.delenv("UFOIR_SART_KERNELS", raising=False)
    got, few = _sart(ufoir_lib, gpu_ctx, sinos, axis, 2)
    monkeypatch.setenv("UFOIR_SART_KERNELS", "general")
    want, many = _sart(ufoir_lib, gpu_ctx, sinos, axis, 2)
    assert (few + 2 * na <= many) == swept, (few, many)
    assert np.array_equal(got, want), np.abs(got - want).max()


@pytest.mark.parametrize("n,na", [(65, 12), (300, 12)])
def test_sweep_passes_non_finite_values_on(ufoir_lib, gpu_ctx, monkeypatch, n, na):
    rng = np.random.default_rng(n)
    sinos = rng.random((1, na, n), dtype=np.float32)
    sinos[0, 3, n // 2] = np.inf
    sinos[0, na - 1, n // 3] = np.nan
    monkeypatch.delenv("UFOIR_SART_KERNELS", raising=False)
    got, _ = _sart(ufoir_lib, gpu_ctx, sinos, -1.0, 1)
    monkeypatch.setenv("UFOIR_SART_KERNELS", "general")
    want, _ = _sart(ufoir_lib, gpu_ctx, sinos, -1.0, 1)
    assert not np.isfinite(want).all()
    assert np.array_equal(got, want, equal_nan=True)


# Geometries where a column part has no rays at some angles (the last block's
# centre lies past the image, or the axis beside the image's centre): such a CTA
# sends no sums, and must keep up with the others all the same.
@pytest.mark.parametrize("n,na,axis,slices", [
    (129, 24, -1.0, 20), (200, 31, 97.4, 12), (257, 90, -1.0, 1), (262, 90, -1.0, 3), (277, 90, -1.0, 1),
    (256, 60, 168.0, 1), (256, 60, 208.0, 2), (367, 60, 263.5, 1)])
def test_sweep_with_parts_that_have_no_rays(ufoir_lib, gpu_ctx, monkeypatch, n, na, axis, slices):
    rng = np.random.default_rng(3 * n + na)
    sinos = rng.random((slices, na, n), dtype=np.float32) * n
    monkeypatch.delenv("UFOIR_SART_KERNELS", raising=False)
    got, few = _sart(ufoir_lib, gpu_ctx, sinos, axis, 25)
    monkeypatch.setenv("UFOIR_SART_KERNELS", "general")
    want, many = _sart(ufoir_lib, gpu_ctx, sinos, axis, 25)
    assert few < many / 4, (few, many)        # the sweep served
    assert np.array_equal(got, want), np.abs(got - want).max()
