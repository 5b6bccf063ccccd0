"""Forms of the tiled projectors that depend on the data or on the launch.

The projectors take a shorter filter form where their data are finite, and
other forms for angles whose whole tile lies inside or beyond the detector
edges; the launch shape follows the number of tiles. Every form must give
what the plain float32 sequence gives, infinities and NaNs included. The
reference is that sequence in numpy, one rounding per operation: each sample
reads its two taps in one row, (1 - t) * T0 + t * T1, zero outside. Equality
is exact (NaN where NaN).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

f32 = np.float32


def _lut(na, step):
    a = np.arange(na, dtype=f32) * f32(step)
    return np.sin(a.astype(np.float64)).astype(f32), np.cos(a.astype(np.float64)).astype(f32)


def _lerp(rows, c):
    """rows: [n] values with a zero border; c: float32 coordinates."""
    n = rows.shape[0]
    pad = np.zeros(n + 4, f32)
    pad[2:-2] = rows
    cm = c - f32(0.5)
    i0 = np.floor(cm)
    t = cm - i0
    k = i0.astype(np.int64)
    a, b = pad[np.clip(k, -2, n + 1) + 2], pad[np.clip(k + 1, -2, n + 1) + 2]
    return (f32(1) - t) * a + t * b


def _backward(sino, step, axis):
    """One slice, relaxation 1, volume starting at zero, one sum per direction run."""
    na, n = sino.shape
    sn, cs = _lut(na, step)
    w, ax = f32(n), f32(axis)
    diff = w - ax * f32(2)
    half = w - ax if diff < 0 else ax
    e0, e1 = ax - half + f32(0.5), ax + half - f32(0.5)
    os_, shift = w / f32(2), w / f32(2) - diff / f32(2)
    f = np.arange(n, dtype=f32) + f32(0.5) - os_
    v, total = np.zeros((n, n), f32), np.zeros((n, n), f32)
    vertical = np.abs(sn.astype(np.float64)) <= np.abs(cs.astype(np.float64))
    for a in range(na):
        if a and vertical[a] != vertical[a - 1]:
            v, total = v + total, np.zeros((n, n), f32)
        c = (f[None, :] * cs[a] - f[:, None] * sn[a]) + shift
        total = total + _lerp(sino[a], np.minimum(np.maximum(c, e0), e1))
    return v + total


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("slices,axis", [(1, 64.5), (12, 64.5), (137, 64.5), (304, 64.5), (12, 60.3), (1, 71.0)])
def test_backprojector_launch_shapes_and_non_finite_data(ufoir_lib, gpu_ctx, slices, axis, special):
    n, na = 129, 37      # one full chunk of 32 angles and a part; ragged tiles
    step = f32(np.pi / na)
    rng = np.random.default_rng(slices)
    sino = rng.standard_normal((slices, na, n)).astype(f32)
    if special:
        sino[0, 3, 40], sino[0, 20, 64], sino[-1, 33, 100] = np.inf, -np.inf, np.nan
        sino[0, 10, 0], sino[0, 11, n - 1] = np.inf, np.inf
    p = ufoir_lib.ParallelProjector(gpu_ctx, step=float(step), is_forward=0, axis_position=axis, angles_num=na)
    got = p.process(sino)
    p.close()
    with np.errstate(invalid="ignore"):
        for s in sorted({0, slices - 1}):
            np.testing.assert_array_equal(got[s], _backward(sino[s], step, axis))


def _forward(vol, na, step, axis):
    """One slice, scale 1, sinogram starting at zero: 64-sample blocks of a float coordinate recurrence."""
    n = vol.shape[0]
    sn, cs = _lut(na, step)
    diff = f32(n) - f32(axis) * f32(2)
    ros, os_, half_n = diff / f32(2), f32(n) / f32(2), f32(0.5) * f32(n)
    k = np.arange(n)
    off = (diff < 0) & (k < abs(diff)) | (diff > 0) & (k > f32(axis) * f32(2))
    out = np.zeros((na, n), f32)
    for a in range(na):
        vert = abs(float(sn[a])) <= abs(float(cs[a]))
        det = f32(1) / cs[a] if vert else f32(-1) / sn[a]
        st = sn[a] / cs[a] if vert else cs[a] / sn[a]
        c = ((0.5 + float(ros) + k - float(half_n)) * float(det) + float(-os_ * st) + float(half_n)).astype(f32)
        img = vol if vert else vol.T
        total, block = np.zeros(n, f32), np.zeros(n, f32)
        for r in range(n):
            block = block + _lerp(img[r], c)
            c = c + st
            if r % 64 == 63:
                total, block = total + block, np.zeros(n, f32)
        out[a] = np.where(off, f32(0), total + block)
    return out


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("n,slices,axis", [(129, 1, 64.5), (129, 40, 64.5), (800, 1, 400.0), (800, 40, 396.2), (61, 2, 34.0)])
def test_forward_projector_row_forms_and_non_finite_data(ufoir_lib, gpu_ctx, n, slices, axis, special):
    na = 37
    step = f32(np.pi / na)
    vol = np.random.default_rng(n).standard_normal((slices, n, n)).astype(f32)
    if special:
        vol[0, 5, 7], vol[0, n // 2, 3], vol[-1, n - 1, n - 1] = np.inf, -np.inf, np.nan
    p = ufoir_lib.ParallelProjector(gpu_ctx, step=float(step), is_forward=1, axis_position=axis, angles_num=na)
    got = p.process(vol)
    p.close()
    with np.errstate(invalid="ignore"):
        for s in sorted({0, slices - 1}):
            np.testing.assert_array_equal(got[s], _forward(vol[s], na, step, axis))


@pytest.mark.parametrize("n,na,axis", [(7, 6, 3.5), (64, 20, 32.0), (65, 12, 30.2), (200, 180, 104.0), (1100, 8, 550.0)])
def test_subset_projections(ufoir_lib, gpu_ctx, oracle, n, na, axis):
    """Subsets of one angle, several, and all of one direction, each as vertical
    and as horizontal rays (whichever the angles are), against the oracle's kernel."""
    import ctypes
    fp = ctypes.POINTER(ctypes.c_float)
    step = f32(np.pi / na)
    rng = np.random.default_rng(n)
    vol = rng.random((n, n), dtype=f32)
    p = ufoir_lib.ParallelProjector(gpu_ctx, step=float(step), angles_num=na, axis_position=axis, correction_scale=-1.0)
    p.get_requisition((n, n))
    s, c = oracle.lut(na, step)
    k, dims = oracle.kernels().contents, oracle.Dims(n, n, n, na)
    for off, cnt in [(1, 1), (na // 2, 1), (0, 3), (na // 4, na // 3)]:
        for direction in (0, 1):
            sino = rng.random((na, n), dtype=f32)
            want = sino.copy()
            k.fp(oracle.image(vol), oracle.image(want), s.ctypes.data_as(fp), c.ctypes.data_as(fp), dims, f32(axis),
                 oracle.Subset(off, cnt, direction), f32(-1.0))
            np.testing.assert_array_equal(p.subset_fp(vol, sino.copy(), off, cnt, direction), want)
    p.close()


@pytest.mark.parametrize("n,na,slices,axis", [(5, 3, 1, 2.5), (129, 37, 1, 64.5), (129, 33, 14, 60.1), (130, 17, 150, 71.3),
                                              (200, 40, 130, 100.0), (301, 70, 1, 150.5)])
def test_siddon_launch_shapes(ufoir_lib, gpu_ctx, oracle, n, na, slices, axis):
    """Each launch shape of the siddon model's tiles, ragged edges and off-centre
    axes among them, against the double oracle at the model's tolerance (bins
    that lie on pixel boundaries of an axis-aligned angle have no one answer:
    see the next test)."""
    step = f32(np.pi / na)
    rng = np.random.default_rng(n + slices)
    vols = rng.random((slices, n, n), dtype=f32)
    sinos = rng.random((slices, na, n), dtype=f32)
    fwd = ufoir_lib.ParallelProjector(gpu_ctx, step=float(step), is_forward=1, axis_position=axis, angles_num=na, model="siddon")
    bwd = ufoir_lib.ParallelProjector(gpu_ctx, step=float(step), is_forward=0, axis_position=axis, angles_num=na, model="siddon")
    got, back = fwd.process(vols), bwd.process(sinos)
    for i in sorted({0, slices - 1}):
        want, wantb = oracle.siddon_forward(n, na, step, vols[i], axis), oracle.siddon_backward(n, na, step, sinos[i], axis)
        assert np.linalg.norm(got[i] - want) <= 1e-5 * np.linalg.norm(want)
        assert np.linalg.norm(back[i] - wantb) <= 1e-5 * np.linalg.norm(wantb)
    fwd.close()
    bwd.close()


@pytest.mark.parametrize("n,na,axis", [(130, 16, 70.5), (129, 8, 60.0)])
def test_siddon_tiles_and_ray_walk_agree_on_pixel_boundaries(ufoir_lib, gpu_ctx, n, na, axis):
    """An axis half a bin off the centre puts every ray of the axis-aligned
    angles on a pixel boundary; whole sets (tiles) and subsets (the ray walk)
    must put them on the same side. Tolerance: two orders of n float roundings."""
    step = f32(np.pi / na)
    vol = np.random.default_rng(n).random((n, n), dtype=f32)
    p = ufoir_lib.ParallelProjector(gpu_ctx, step=float(step), is_forward=1, axis_position=axis, angles_num=na, model="siddon")
    whole = p.process(vol)
    part = np.zeros((na, n), f32)
    for off, cnt, direction in p.subsets():
        p.subset_fp(vol, part, off, cnt, direction)
    p.close()
    np.testing.assert_allclose(whole, part, rtol=0, atol=2 * n * 2.0 ** -24 * float(np.abs(part).max()))


# Launches of few tiles spread a tile's detectors over parts of whole rows or of
# column windows, by size and by how many tiles there are; launches of many tiles
# take other parts. The sums of a ray do not depend on it.
@pytest.mark.parametrize("n,na,axis,arithmetic", [
    (127, 16, -1.0, 0), (128, 16, 63.1, 0), (129, 24, -1.0, 0), (255, 60, 130.3, 0), (256, 200, -1.0, 0),
    (257, 24, -1.0, 1), (513, 24, 250.2, 0), (640, 280, -1.0, 0), (769, 90, -1.0, 0), (1024, 40, 517.7, 0),
    (1025, 200, -1.0, 1), (1449, 90, -1.0, 0), (1536, 30, 760.4, 0), (1537, 30, -1.0, 0)])
def test_few_tiles_give_what_many_give(ufoir_lib, gpu_ctx, n, na, axis, arithmetic):
    slices = 40 if n < 600 else 12
    rng = np.random.default_rng(n + na)
    vols = rng.standard_normal((slices, n, n), dtype=f32)
    p = ufoir_lib.ParallelProjector(gpu_ctx, step=float(f32(np.pi / na)), axis_position=axis, is_forward=True,
                                    angles_num=na, arithmetic=arithmetic)
    many = p.process(vols)
    for s in (0, slices - 1):
        one = p.process(vols[s])
        assert np.array_equal(one, many[s]), np.abs(one - many[s]).max()
    p.close()


# A warp's detectors may span the whole image: at a row one end ray lies left of
# it, the other right of it, and the rays between cross it. With the axis beside
# the centre that happens in whole chunks of rows. The siddon model's tiles are
# compared with its ray walk: two orders of n float roundings (an axis at half a
# bin puts rays on pixel boundaries, which the two put on the same side).
@pytest.mark.parametrize("n,na,axis", [(33, 720, 6.6), (34, 720, 25.5), (34, 720, 5.1), (35, 360, 26.25), (36, 720, 27.0)])
def test_rows_between_rays_on_either_side_of_the_image(ufoir_lib, gpu_ctx, n, na, axis):
    step = f32(np.pi / na)
    vol = np.random.default_rng(n).random((n, n), dtype=f32)
    kw = dict(step=float(step), is_forward=1, axis_position=axis, angles_num=na)
    p = ufoir_lib.ParallelProjector(gpu_ctx, **kw)
    np.testing.assert_array_equal(p.process(vol), _forward(vol, na, step, axis))
    p.close()
    p = ufoir_lib.ParallelProjector(gpu_ctx, model="siddon", **kw)
    whole, part = p.process(vol), np.zeros((na, n), f32)
    for off, cnt, direction in p.subsets():
        p.subset_fp(vol, part, off, cnt, direction)
    np.testing.assert_allclose(whole, part, rtol=0, atol=2 * n * 2.0 ** -24 * float(np.abs(part).max()))
    p.close()


# The tuner also tries shapes with more detectors per warp, which span larger images.
@pytest.mark.parametrize("n,na,axis", [(96, 60, 70.0), (256, 24, 184.3), (300, 40, 90.2)])
def test_tuned_shapes_off_centre(ufoir_lib, n, na, axis):
    step = f32(np.pi / na)
    vol = np.random.default_rng(n).random((n, n), dtype=f32)
    with ufoir_lib.Context(0) as ctx:
        p = ufoir_lib.ParallelProjector(ctx, step=float(step), is_forward=1, axis_position=axis, angles_num=na)
        p.get_requisition((n, n))
        p.autotune(1)
        np.testing.assert_array_equal(p.process(vol), _forward(vol, na, step, axis))
        p.close()


def _fma(a, b, c):
    """float32 a * b + c with one rounding: the product is exact in 64 bits, the
    sum is rounded to odd there, which the second rounding cannot tell from exact."""
    p, c = a.astype(np.float64) * b.astype(np.float64), c.astype(np.float64)
    s = p + c
    bb = s - p
    err = (p - (s - bb)) + (c - bb)
    bits = s.view(np.int64)
    odd = np.where((err != 0) & (bits & 1 == 0), np.where((err > 0) == (s > 0), 1, -1), 0)
    return (bits + odd).view(np.float64).astype(f32)


def _backward_fast(sino, step, axis):
    """_backward in the fast arithmetic: coordinates fX cos + ((-fY) sin + shift), samples (sum + T0) + t (T1 - T0)."""
    na, n = sino.shape
    sn, cs = _lut(na, step)
    w, ax = f32(n), f32(axis)
    diff = w - ax * f32(2)
    half = w - ax if diff < 0 else ax
    e0, e1 = ax - half + f32(0.5), ax + half - f32(0.5)
    shift = w / f32(2) - diff / f32(2)
    f = np.arange(n, dtype=f32) + f32(0.5) - w / f32(2)
    v, total = np.zeros((n, n), f32), np.zeros((n, n), f32)
    vertical = np.abs(sn.astype(np.float64)) <= np.abs(cs.astype(np.float64))
    for a in range(na):
        if a and vertical[a] != vertical[a - 1]:
            v, total = v + total, np.zeros((n, n), f32)
        c = np.minimum(np.maximum(f[None, :] * cs[a] + ((-f[:, None]) * sn[a] + shift), e0), e1) - f32(0.5)
        k = np.floor(c)
        row = np.append(sino[a], f32(0))
        t0, t1 = row[k.astype(np.int64)], row[k.astype(np.int64) + 1]
        total = _fma(c - k, t1 - t0, total + t0)
    return v + total


# At a quarter turn the last row of a centred image has its coordinates on the
# detector edge, or an ulp beside it, as the sum is ordered. Values in the first
# and last detector show which. All four launch shapes (slices).
@pytest.mark.parametrize("n,na,slices,axis", [(200, 20, 1, 100.0), (200, 20, 12, 100.0), (256, 60, 1, 128.0), (256, 60, 90, 128.0),
                                              (512, 16, 1, 256.0), (512, 16, 80, 256.0), (129, 37, 12, 60.3)])
def test_fast_backprojector_at_the_detector_edges(ufoir_lib, gpu_ctx, n, na, slices, axis):
    step = f32(np.pi / na)
    sino = np.random.default_rng(n).standard_normal((slices, na, n)).astype(f32)
    sino[:, :, [0, n - 1]] += f32(4)
    p = ufoir_lib.ParallelProjector(gpu_ctx, step=float(step), is_forward=0, axis_position=axis, angles_num=na,
                                    arithmetic=ufoir_lib.ARITH_FAST)
    got = p.process(sino)
    p.close()
    for s in sorted({0, slices - 1}):
        np.testing.assert_array_equal(got[s], _backward_fast(sino[s], step, axis))


@pytest.mark.parametrize("n,na", [(256, 60), (512, 400), (1024, 360)])
def test_fast_and_exact_backprojections_of_ones_agree(ufoir_lib, gpu_ctx, n, na):
    step = f32(np.pi / na)
    out = []
    for arithmetic in (ufoir_lib.ARITH_FAST, ufoir_lib.ARITH_EXACT):
        p = ufoir_lib.ParallelProjector(gpu_ctx, step=float(step), is_forward=0, angles_num=na, arithmetic=arithmetic)
        out.append(p.process(np.ones((na, n), f32)).astype(np.float64))
        p.close()
    assert np.linalg.norm(out[0] - out[1]) <= 1e-5 * np.linalg.norm(out[1])      # the path's bar


# Coordinates beyond 2^31, where the index of a tap saturates: an axis far
# outside, and a quarter turn walked as vertical rays (cos = -4e-8) by the kernel
# of one thread per ray, which serves subsets beyond 8192 detectors.
@pytest.mark.parametrize("na", [5, 20])
@pytest.mark.parametrize("axis", [3.0e9, 1.0e10, 1.0e30])
def test_an_axis_far_outside_gives_zeros(ufoir_lib, gpu_ctx, axis, na):
    n = 33
    rng = np.random.default_rng(na)
    p = ufoir_lib.ParallelProjector(gpu_ctx, step=float(f32(np.pi / na)), axis_position=axis, angles_num=na)
    assert not p.forward(rng.random((n, n), dtype=f32), np.zeros((na, n), f32)).any()
    assert not p.backward(np.zeros((n, n), f32), rng.random((na, n), dtype=f32)).any()
    p.close()
    p = ufoir_lib.ParallelProjector(gpu_ctx, step=float(f32(np.pi / na)), axis_position=axis, is_forward=0)
    assert not ufoir_lib.sart(p, rng.random((na, n), dtype=f32), num_iterations=1).any()
    p.close()


def test_a_quarter_turn_walked_as_vertical_rays(ufoir_lib, gpu_ctx):
    n, na = 8200, 2
    vol = np.random.default_rng(0).random((n, n), dtype=f32)
    p = ufoir_lib.ParallelProjector(gpu_ctx, step=float(f32(np.pi / na)), angles_num=na)
    p.get_requisition((n, n))
    got = p.subset_fp(vol, np.zeros((na, n), f32), 1, 1, 1)
    p.close()
    sn, cs = _lut(na, f32(np.pi / na))
    det, st, half = f32(1) / cs[1], sn[1] / cs[1], f32(0.5) * f32(n)
    c = ((0.5 + np.arange(n) - float(half)) * float(det) + float(-half * st) + float(half)).astype(f32)
    assert np.abs(c).max() > 2.0 ** 31
    total, block = np.zeros(n, f32), np.zeros(n, f32)
    for r in range(n):
        block = block + _lerp(vol[r], c)
        c = c + st
        if r % 64 == 63:
            total, block = total + block, np.zeros(n, f32)
    np.testing.assert_array_equal(got[1], total + block)
    assert not got[0].any()


@pytest.mark.parametrize("n,na,axis", [(130, 1600, 60.2), (200, 1250, 104.0)])
def test_subset_projections_of_many_angles(ufoir_lib, gpu_ctx, oracle, n, na, axis):
    """Subsets of more ray groups than the GPU has room for spread ones: one thread per ray."""
    test_subset_projections(ufoir_lib, gpu_ctx, oracle, n, na, axis)


# Whole sets of the siddon model go through tiles or the ray walk, whichever the
# launch's tiles make faster: few tiles of many columns, golden steps (tiles of
# one or two angles) and many full tiles, against the double oracle.
@pytest.mark.parametrize("n,na,slices,golden", [(776, 12, 1, False), (300, 60, 6, True), (200, 90, 1, True), (120, 400, 4, False)])
def test_siddon_tiles_and_walk_by_the_launch(ufoir_lib, gpu_ctx, oracle, n, na, slices, golden):
    step = f32(np.pi * (np.sqrt(5) - 1) / 2 if golden else np.pi / na)
    vols = np.random.default_rng(n).random((slices, n, n), dtype=f32)
    p = ufoir_lib.ParallelProjector(gpu_ctx, step=float(step), is_forward=1, axis_position=n / 2 + 0.3, angles_num=na, model="siddon")
    got = p.process(vols)
    p.close()
    for s in sorted({0, slices - 1}):
        want = oracle.siddon_forward(n, na, step, vols[s], n / 2 + 0.3)
        assert np.linalg.norm(got[s] - want) <= 1e-5 * np.linalg.norm(want)      # the model's tolerance


# The siddon model's limits hold whichever kernel would serve the call. Many
# slices or angles of a small image are what the tiles would take.
@pytest.mark.parametrize("n,na,slices", [(24, 1, 65536), (24, 65536, 1)])
def test_siddon_refuses_what_is_beyond_its_limits(ufoir_lib, gpu_ctx, n, na, slices):
    v, s = ufoir_lib.DeviceArray(gpu_ctx, (slices, n, n), zero=True), ufoir_lib.DeviceArray(gpu_ctx, (slices, na, n))
    p = ufoir_lib.ParallelProjector(gpu_ctx, step=1e-4, is_forward=1, angles_num=na, model="siddon")
    with pytest.raises(ufoir_lib.UfoirError) as e:
        p.process(v, s)
    assert e.value.status == ufoir_lib.ERR_INVALID
    p.close()
    v.close()
    s.close()


@pytest.mark.parametrize("n,na,axis,arithmetic", [(776, 300, -1.0, 0), (776, 400, 380.4, 1), (1100, 420, -1.0, 1), (1900, 200, -1.0, 1)])
def test_windows_serve_more_tiles_beyond_768_columns(ufoir_lib, gpu_ctx, n, na, axis, arithmetic):
    """39 to 57 tiles: column windows in one slice, whole rows in twelve."""
    test_few_tiles_give_what_many_give(ufoir_lib, gpu_ctx, n, na, axis, arithmetic)
