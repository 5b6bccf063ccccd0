"""Timing cases of the reconstruction path: what a program does with the
library through its Python binding (ufo-ir_gb300/ufoir), on data that live in
the GPU's memory.

  listed()             the standing cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  inputs and the handles a program keeps
  run(state)           one pass
  work(case)           the bytes and operations a pass cannot do without
  exact(case, seed)    the pass's results in 64 bits, in plain torch

Sinograms are those of random-ellipse phantoms (closed form, scaled to the
Joseph projector's samples-per-row unit), Poisson-noised at I0 = 1e5 and
log-transformed where a scan would be.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ufo-ir_gb300"))
import ufoir  # noqa: E402

RELAX = 0.25            # the methods' default relaxation factor
TV_STEPS = 20           # ASD-POCS sub-steps per outer iteration (fixed in the method)
CGS_ITERATIONS = 30     # SBTV's limit per outer iteration
EXACT_SAMPLES = 1.2e11  # interpolated samples that the 64-bit results are computed for at most


def _case(name, op, n, angles, slices=1, iters=1, axis=0.0, arith="exact", norm="fp64", subset=1, model="joseph"):
    """axis: offset of the rotation axis from the image centre, in bins; subset: angles per subset of a sweep."""
    c = {"op": op, "n": n, "angles": angles, "slices": slices, "iters": iters, "axis": axis, "arith": arith,
         "norm": norm, "subset": subset, "model": model}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a preview-sized forward and back projection: launches and host work count
        _case("project_64x60", "project", 64, 60),
        # the projector plugin on one full-size slice, as the reference's graph runs it
        _case("project_1448x1200", "project", 1448, 1200),
        # the exact line-integral model on the same slice
        _case("siddon_1448x1200", "project", 1448, 1200, model="siddon"),
        # a program's own Kaczmarz sweep through the operator interface, one angle per subset
        _case("subsets_724x90", "subsets", 724, 90),
        # plain SART at the smallest configured size
        _case("sart_367x180", "sart", 367, 180, iters=10),
        # SIRT on one slice per call, default iterations: the reference's own usage
        _case("sirt_1448x1200", "sirt", 1448, 1200, iters=10),
        # off-centre scan with ragged sizes, a few slices per call, the opt-in fast arithmetic
        _case("sirt_fast_1001x451x6", "sirt", 1001, 451, slices=6, iters=5, axis=-7.3, arith="fast"),
        # the headline batch: 64 resident slices
        _case("sirt_batch_1448x1200x64", "batch", 1448, 1200, slices=64, iters=2),
        # many small SIRT jobs of uneven size advanced together
        _case("mix_12_small", "mix", 724, 600, slices=12, iters=5),
        # sparse-view TV reconstruction at the largest configured size
        _case("asdpocs_2900x90", "asdpocs", 2900, 90),
        # the same method with norms summed as the reference sums them
        _case("asdpocs_530x24_compat", "asdpocs", 530, 24, iters=2, norm="compat"),
        # a slab of slices through split-Bregman TV
        _case("sbtv_724x360x4", "sbtv", 724, 360, slices=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["project", "project", "siddon", "subsets", "sart", "sart", "sirt", "sirt", "batch", "mix",
                     "asdpocs", "asdpocs", "sbtv"])
    axis = rng.choice([0.0, 0.0, round(rng.uniform(-9.0, 9.0), 1)])
    arith = rng.choice(["exact", "exact", "fast"])
    if op in ("project", "siddon"):
        n = _log_int(rng, 64, 2900)
        return _case(None, "project", n, _log_int(rng, 60, 1200), slices=rng.choice([1, 1, 2, 5]), axis=axis,
                     arith=arith if op == "project" else "exact", model="siddon" if op == "siddon" else "joseph")
    if op == "subsets":
        n, m = _log_int(rng, 128, 2900), rng.choice([1, 1, 4, 15])
        return _case(None, "subsets", n, m * rng.randint(4, 60 // m + 4), axis=axis, subset=m)
    if op == "sart":
        return _case(None, "sart", _log_int(rng, 128, 2900), _log_int(rng, 60, 360), slices=rng.choice([1, 1, 3]),
                     iters=rng.randint(1, 10), axis=axis)
    if op in ("sirt", "batch"):
        return _case(None, op, _log_int(rng, 128, 2048), _log_int(rng, 90, 1200), slices=rng.choice([1, 2, 4, 9]),
                     iters=rng.randint(2, 6), axis=axis, arith=arith)
    if op == "mix":
        return _case(None, "mix", _log_int(rng, 250, 1448), _log_int(rng, 120, 720), slices=rng.randint(4, 16),
                     iters=rng.randint(2, 6))
    if op == "asdpocs":
        norm = rng.choice(["fp64", "fp64", "compat"])
        n = _log_int(rng, 128, 900 if norm == "compat" else 2900)
        return _case(None, "asdpocs", n, _log_int(rng, 24, 180), iters=rng.randint(1, 2), axis=axis, norm=norm)
    return _case(None, "sbtv", _log_int(rng, 128, 900), _log_int(rng, 60, 400), slices=rng.choice([1, 2, 5]),
                 norm=rng.choice(["fp64", "fp64", "compat"]))


# ---------------------------------------------------------------- inputs


def _step(angles):
    return float(np.float32(np.pi / angles))


def _axis(case, n):
    return -1.0 if case["axis"] == 0.0 else float(np.float32(0.5 * n + case["axis"]))


def _members(case):
    """Sizes (n, angles) of a mixed batch: whole and half detectors, angle counts spread up to the case's."""
    k = case["slices"]
    return [(case["n"] if i % 2 else (case["n"] + 1) // 2, max(30, case["angles"] * (i + 1) // k)) for i in range(k)]


def _ellipses(gen, slices, n):
    """Parameters [slices, 10] of ellipses inside the disc of a phantom of side n / sqrt 2."""
    u = torch.rand(6, slices, 10, generator=gen, device="cuda", dtype=torch.float64)
    r = n / math.sqrt(2.0) / 2.0
    rad, ang = 0.6 * r * u[0].sqrt(), 2 * math.pi * u[1]
    return (rad * ang.cos(), rad * ang.sin(), r * (0.05 + 0.3 * u[2]), r * (0.05 + 0.3 * u[3]), math.pi * u[4], u[5])


def _volumes(gen, slices, n):
    x = torch.arange(n, device="cuda", dtype=torch.float64) + 0.5 - 0.5 * n
    vol = torch.zeros(slices, n, n, device="cuda")
    cx, cy, a, b, phi, rho = _ellipses(gen, slices, n)
    for s in range(slices):
        for e in range(10):
            c, q = phi[s, e].cos(), phi[s, e].sin()
            dx, dy = x[None, :] - cx[s, e], x[:, None] - cy[s, e]
            u, v = (dx * c + dy * q) / a[s, e], (dy * c - dx * q) / b[s, e]
            vol[s] += torch.where(u * u + v * v <= 1.0, rho[s, e], 0.0).float()
    return vol


def _sinograms(gen, slices, n, angles, axis, noisy):
    """Closed-form parallel projections of random-ellipse phantoms, [slices, angles, n] float32."""
    theta = torch.arange(angles, device="cuda", dtype=torch.float64)[:, None] * (math.pi / angles)
    t = torch.arange(n, device="cuda", dtype=torch.float64)[None, :] + 0.5 - (0.5 * n if axis < 0 else axis)
    per_row = torch.maximum(theta.cos().abs(), theta.sin().abs())
    out = torch.empty(slices, angles, n, device="cuda")
    cx, cy, a, b, phi, rho = _ellipses(gen, slices, n)
    for s in range(slices):
        p = torch.zeros(angles, n, device="cuda", dtype=torch.float64)
        for e in range(10):
            u, v = (theta + phi[s, e]).cos() * a[s, e], (theta + phi[s, e]).sin() * b[s, e]
            r2 = u * u + v * v
            d = t - (cx[s, e] * theta.cos() - cy[s, e] * theta.sin())
            p += 2 * a[s, e] * b[s, e] * rho[s, e] * (r2 - d * d).clamp(min=0.0).sqrt() / r2
        p *= per_row
        if noisy:
            kappa = 4.0 / p.max()
            counts = torch.poisson(1e5 * torch.exp(-kappa * p), generator=gen)
            p = -torch.log(counts.clamp(min=1.0) / 1e5) / kappa
        out[s] = p.float()
    return out


def _inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    n, na, s, op = case["n"], case["angles"], case["slices"], case["op"]
    if op == "project":
        return _volumes(gen, s, n), _sinograms(gen, s, n, na, _axis(case, n), False)
    if op == "mix":
        return [_sinograms(gen, 1, m, a, -1.0, True)[0] for m, a in _members(case)]
    return _sinograms(gen, s, n, na, _axis(case, n), not (op == "sart" and case["axis"] == 0.0))


# ---------------------------------------------------------------- the library's side

_CTX = None


def _context():
    """The program's one context."""
    global _CTX
    if _CTX is None:
        _CTX = ufoir.Context(0)
    return _CTX


class _Memory:
    """Library memory as torch sees it; freed when the last tensor over it goes."""

    def __init__(self, array):
        self.array = array
        self.__cuda_array_interface__ = {"shape": array.shape, "typestr": "<f4", "data": (array.ptr, False),
                                         "version": 3, "strides": None}

    def __del__(self):
        self.array.close()


class _State:
    def __init__(self, case):
        self.case = case
        self.ctx = _context()
        self.owned, self.views = [], []

    def keep(self, handle):
        self.owned.append(handle)
        return handle

    def array(self, tensor=None, shape=None):
        """Library memory holding `tensor` (or of `shape`), and its torch view."""
        a = ufoir.DeviceArray(self.ctx, tensor.shape if shape is None else shape)
        t = torch.as_tensor(_Memory(a), device="cuda")
        t.zero_() if tensor is None else t.copy_(tensor)
        self.views.append(t)
        return a, t

    def projector(self, n, forward, **kw):
        case = self.case
        return self.keep(ufoir.ParallelProjector(
            self.ctx, step=_step(case["angles"]), is_forward=int(forward), axis_position=_axis(case, n),
            angles_num=case["angles"], model=case["model"],
            arithmetic=ufoir.ARITH_FAST if case["arith"] == "fast" else ufoir.ARITH_EXACT, **kw))

    def __del__(self):
        for h in reversed(getattr(self, "owned", [])):
            h.close()


def prepare(case, seed):
    st = _State(case)
    n, na, s, op = case["n"], case["angles"], case["slices"], case["op"]
    data = _inputs(case, seed)
    if op == "project":
        st.vol, _ = st.array(data[0])
        st.sino, _ = st.array(data[1])
        st.sino_out, st.sino_t = st.array(shape=(s, na, n))
        st.vol_out, st.vol_t = st.array(shape=(s, n, n))
        st.fwd, st.bwd = st.projector(n, True), st.projector(n, False)
    elif op == "subsets":
        st.sino, _ = st.array(data[0])
        st.res, st.res_t = st.array(shape=(na, n))
        st.zero, _ = st.array(shape=(n, n))
        st.vol, st.vol_t = st.array(shape=(n, n))
        st.proj = st.projector(n, False, relaxation=float(np.float32(0.5 / (n * case["subset"]))),
                               correction_scale=-1.0)
        st.proj.get_requisition((n, na))
        st.subsets = _subsets(st.proj.subsets(), case["subset"])
    elif op == "mix":
        st.parts, jobs = [], []
        for (m, a), sino in zip(_members(case), data):
            b, _ = st.array(sino)
            x, x_t = st.array(shape=(m, m))
            jobs.append((b, x, dict(step=_step(a), relaxation_factor=RELAX)))
            st.parts.append(x_t)
        torch.cuda.synchronize()
        st.batch = st.keep(ufoir.Batch(st.ctx, jobs))
    else:
        st.sino, _ = st.array(data)
        st.vol, st.vol_t = st.array(shape=(s, n, n))
        st.proj = st.projector(n, False)
        if op == "batch":
            torch.cuda.synchronize()
            st.batch = st.keep(ufoir.SirtBatch(st.proj, st.sino, st.vol, relaxation_factor=RELAX))
            st.vol_parts = [st.vol_t[:2], st.vol_t[2:]] if s > 2 else [st.vol_t]
    torch.cuda.synchronize()
    return st


def _subsets(runs, m):
    """Ordered subsets of at most m angles that keep to one direction."""
    return [(off + k, min(m, count - k), d) for off, count, d in runs for k in range(0, count, m)]


def run(st):
    case, op = st.case, st.case["op"]
    norm = ufoir.NORM_COMPAT if case["norm"] == "compat" else ufoir.NORM_FP64
    if op == "project":
        st.fwd.process(st.vol, st.sino_out)
        st.bwd.process(st.sino, st.vol_out)
        return [st.sino_t, st.vol_t]
    if op == "subsets":
        lib, h = ufoir.lib(), st.ctx.handle
        st.ctx._check(lib.ufoir_memcpy(h, st.res.ptr, st.sino.ptr, st.sino.nbytes))
        st.ctx._check(lib.ufoir_memcpy(h, st.vol.ptr, st.zero.ptr, st.zero.nbytes))
        for off, count, direction in st.subsets:
            st.proj.subset_fp(st.vol, st.res, off, count, direction)
            st.proj.subset_bp(st.vol, st.res, off, count, direction)
        return [st.res_t, st.vol_t]
    if op == "mix":
        st.batch.run(case["iters"])
        return st.parts
    if op == "batch":
        st.batch.reset()
        st.batch.run(case["iters"])
        return st.vol_parts
    if op == "sart":
        ufoir.sart(st.proj, st.sino, st.vol, num_iterations=case["iters"], relaxation_factor=RELAX)
    elif op == "sirt":
        ufoir.sirt(st.proj, st.sino, st.vol, num_iterations=case["iters"], relaxation_factor=RELAX)
    elif op == "asdpocs":
        ufoir.asdpocs(st.proj, st.sino, st.vol, num_iterations=case["iters"], norm_mode=norm)
    else:
        ufoir.sbtv(st.proj, st.sino, st.vol, num_iterations=case["iters"], norm_mode=norm, **{"lambda": 0.05, "mu": 1.0})
    return [st.vol_t]


def _samples(case):
    """Interpolated samples of a pass: one per ray and row forward, one per pixel and angle backward."""
    n, na, s, it = case["n"], case["angles"], case["slices"], case["iters"]
    plane = float(n) * n * na
    op = case["op"]
    if op == "project":
        return 2 * plane * s
    if op == "subsets":
        return 2 * plane
    if op == "mix":
        return sum(2.0 * m * m * a for m, a in _members(case)) * it
    if op == "batch":
        return 2 * plane * s * it
    if op == "sart":
        return 2 * plane * s * it + plane                    # the ray weights: one forward projection
    if op == "sirt":
        return 2 * plane * s * it + 2 * plane                # ray and pixel weights
    if op == "asdpocs":
        return it * (2 * 10 + 1) * plane * s + plane         # ten SART sweeps and one residual per iteration
    return it * (2 * CGS_ITERATIONS + 2) * 2 * plane * s + plane * s


def work(case):
    # per sample: the coordinate, its fraction, two weights and two products, and the sum
    n, na, s = case["n"], case["angles"], case["slices"]
    if case["op"] == "mix":
        sizes = sum(a * m + 2 * m * m for m, a in _members(case))
    elif case["op"] == "project":
        sizes = 2 * s * (n * n + na * n)
    else:
        sizes = s * (na * n + n * n) + (na * n if case["op"] == "subsets" else 0)
    return {"bytes": 4.0 * sizes, "flops": 8.0 * _samples(case)}


# ---------------------------------------------------------------- 64-bit results

CHUNK = 4e7     # samples held at a time


class _Exact:
    """The projectors in double precision, on the library's float sine and cosine table."""

    def __init__(self, n, angles, axis, model="joseph"):
        angle = np.arange(angles, dtype=np.float32) * np.float32(_step(angles))
        to = dict(device="cuda", dtype=torch.float64)
        s32, c32 = np.sin(angle.astype(np.float64)).astype(np.float32), np.cos(angle.astype(np.float64)).astype(np.float32)
        self.n, self.na, self.model = n, angles, model
        self.sin, self.cos = torch.tensor(s32.astype(np.float64), **to), torch.tensor(c32.astype(np.float64), **to)
        self.vertical = self.sin.abs() <= self.cos.abs()
        self.axis = 0.5 * n if axis < 0 else axis
        self.k = torch.arange(n, **to)

    def _groups(self, angles):
        for d in (True, False):
            sel = angles[self.vertical[angles] == d]
            g = max(1, int(CHUNK // (self.n * self.n)))
            for i in range(0, len(sel), g):
                yield d, sel[i:i + g]

    def forward(self, vol, angles=None):
        """A vol for volumes [S, n, n]; only the rows of `angles` are computed."""
        n, S = self.n, vol.shape[0]
        out = torch.zeros(S, self.na, n, device="cuda", dtype=torch.float64)
        angles = torch.arange(self.na, device="cuda") if angles is None else angles
        pad = torch.zeros(S, 2, n, n + 2, device="cuda", dtype=torch.float64)
        pad[:, 1, :, 1:-1], pad[:, 0, :, 1:-1] = vol, vol.transpose(1, 2)
        rows = torch.arange(n, device="cuda")[None, None, :] * (n + 2)
        for vert, a in self._groups(angles):
            sn, cs = self.sin[a][:, None, None], self.cos[a][:, None, None]
            y, k = self.k[None, None, :], self.k[None, :, None]
            if self.model == "siddon":
                r = (sn * sn + cs * cs).sqrt()
                sn, cs, u0, e0 = sn / r, cs / r, (k + 0.5 - self.axis) / r, y - 0.5 * n
                slope = sn / cs if vert else cs / sn
                pa = (u0 + e0 * sn) / cs + 0.5 * n if vert else (e0 * cs - u0) / sn + 0.5 * n
                pb = (u0 + (e0 + 1) * sn) / cs + 0.5 * n if vert else ((e0 + 1) * cs - u0) / sn + 0.5 * n
                lo, hi = torch.minimum(pa, pb), torch.maximum(pa, pb)
                i0 = lo.floor()
                t = torch.where(hi > i0 + 1, 1 - (i0 + 1 - lo) / (hi - lo), torch.zeros_like(lo))
                unit = 1.0 / (cs if vert else sn).abs()[:, :, 0]
                del pa, pb, lo, hi, slope
            else:
                ros, det, step = (n - 2 * self.axis) / 2, (1 / cs if vert else -1 / sn), (sn / cs if vert else cs / sn)
                c = (0.5 + ros + k - 0.5 * n) * det - 0.5 * n * step + 0.5 * n + y * step - 0.5
                i0 = c.floor()
                t = c - i0
                diff = n - 2 * self.axis
                off = (self.k < -diff) if diff < 0 else ((self.k > 2 * self.axis) if diff > 0 else self.k < 0)
                unit = torch.where(off, 0.0, 1.0).double()[None, :]
            i0 = i0.clamp(-2, n + 1).long() + 1
            ia, ib = rows + i0.clamp(0, n + 1), rows + (i0 + 1).clamp(0, n + 1)
            for s in range(S):
                img = pad[s, 1 if vert else 0].reshape(-1)
                out[s, a] = ((1 - t) * img[ia] + t * img[ib]).sum(2) * unit
        return out

    def backward(self, sino, angles=None):
        """A^T sino for sinograms [S, angles, n]."""
        n, S = self.n, sino.shape[0]
        out = torch.zeros(S, n, n, device="cuda", dtype=torch.float64)
        angles = torch.arange(self.na, device="cuda") if angles is None else angles
        pad = torch.zeros(S, self.na, n + 2, device="cuda", dtype=torch.float64)
        pad[:, :, 1:-1] = sino
        f = self.k + 0.5 - 0.5 * n
        half = n - self.axis if n - 2 * self.axis < 0 else self.axis
        e0, e1 = self.axis - half + 0.5, self.axis + half - 0.5
        g = max(1, int(CHUNK // (n * n)))
        for i in range(0, len(angles), g):
            a = angles[i:i + g]
            sn, cs = self.sin[a][:, None, None], self.cos[a][:, None, None]
            uc = f[None, None, :] * cs - f[None, :, None] * sn + self.axis
            row = (a * (n + 2))[:, None, None]
            if self.model == "siddon":
                r = (sn * sn + cs * cs).sqrt()
                ca, sa = cs.abs() / r, sn.abs() / r
                i0 = (uc - 0.5).floor()
                ws = []
                for h in (0, 1):
                    d = (i0 + h + 0.5 - uc).abs() / r
                    slope = ((0.5 * (ca + sa) - d) / (ca * sa)).clamp(min=0.0)
                    ws.append(torch.where(d <= 0.5 * (ca - sa).abs(), 1 / torch.maximum(ca, sa), slope))
                wa, wb = ws
            else:
                c = uc.clamp(e0, e1) - 0.5
                i0 = c.floor()
                wb = c - i0
                wa = 1 - wb
            i0 = i0.clamp(-2, n + 1).long() + 1
            ia, ib = row + i0.clamp(0, n + 1), row + (i0 + 1).clamp(0, n + 1)
            for s in range(S):
                img = pad[s].reshape(-1)
                out[s] += (wa * img[ia] + wb * img[ib]).sum(0)
        return out

    def weights(self):
        ray = self.forward(torch.ones(1, self.n, self.n, device="cuda", dtype=torch.float64))
        return _inverse(ray), _inverse(self.backward(torch.ones(1, self.na, self.n, device="cuda", dtype=torch.float64)))

    def sirt(self, b, iters, relax):
        ray, pix = self.weights()
        x = torch.zeros(b.shape[0], self.n, self.n, device="cuda", dtype=torch.float64)
        for _ in range(iters):
            x = x + pix * (relax * self.backward((b - self.forward(x)) * ray))
        return x

    def sart(self, b, iters, relax, ray=None):
        ray = self.weights()[0] if ray is None else ray
        x = torch.zeros(b.shape[0], self.n, self.n, device="cuda", dtype=torch.float64)
        every = torch.arange(self.na, device="cuda")
        for _ in range(iters):
            for a in range(self.na):
                one = every[a:a + 1]
                res = torch.zeros_like(b)
                res[:, a] = (b[:, a] - self.forward(x, one)[:, a]) * ray[:, a]
                x = x + relax * self.backward(res, one)
        return x


def _inverse(v):
    return torch.where(v != 0, 1 / v, torch.zeros_like(v))


def _tv_gradient(x):
    """The TV stage's subgradient on one image [n, n], zero border."""
    p = torch.nn.functional.pad(x, (1, 1, 1, 1))
    f = {(i, j): p[1 + j:1 + j + x.shape[0], 1 + i:1 + i + x.shape[1]] for i in (-1, 0, 1) for j in (-1, 0, 1)}
    eps, c = float(np.float32(0.001)), f[0, 0]
    left, up, right, down = f[-1, 0], f[0, -1], f[1, 0], f[0, 1]

    def root(u, v):
        return (eps + u * u + v * v).sqrt()

    return ((2 * c - left - down) / root(c - left, c - down) - (right - c) / root(right - c, right - f[1, 1])
            - (up - c) / root(up - c, up - f[-1, -1]))


def _asdpocs(e, b, iters):
    """ASD-POCS with the default parameters on one sinogram."""
    ray = e.weights()[0]
    prev = torch.zeros(e.n, e.n, device="cuda", dtype=torch.float64)
    beta, dtgv, out = 1.0, 1.0, None
    for it in range(iters):
        x = e.sart(b, 10, float(np.float32(beta)), ray)[0].clamp(min=0.0)
        out = x.clone()
        dd = (b - e.forward(x[None])).abs().sum()
        dp = (x - prev).abs().sum()
        if it == 0:
            dtgv = float(np.float32(0.2)) * dp
        prev = x.clone()
        for _ in range(TV_STEPS):
            g = _tv_gradient(x)
            x = x - dtgv / g.abs().sum() * g
        dg = (x - prev).abs().sum()
        beta *= float(np.float32(0.995))
        if dg > float(np.float32(0.95)) * dp and dd > 0.001:
            dtgv = dtgv * float(np.float32(0.95))
    return out


class _Sbtv:
    """One outer iteration of split-Bregman TV on one sinogram (lambda 0.05, mu 1)."""

    def __init__(self, e):
        self.e, self.lam, self.mu = e, float(np.float32(0.05)), 1.0
        i = torch.arange(e.n, device="cuda")
        self.index = (i[:, None] * i[None, :]).reshape(-1)      # the method's inner product pairs elements part * i

    def dot(self, a, b):
        return (a.reshape(-1)[self.index] * b.reshape(-1)[self.index]).sum()

    def norm(self, a):
        return self.dot(a, a).sqrt()

    def apply(self, v):
        d = 4 * v - sum(torch.roll(v, k, ax) for k in (1, -1) for ax in (0, 1))
        return self.mu * self.e.backward(self.e.forward(v[None]))[0] + self.lam * d

    def first(self, b):
        for _ in range(2):
            lo, hi = b.min(), b.max()
            b = (b - lo) / (hi - lo)
        rhs = self.mu * self.e.backward(b[None])[0]
        x = torch.zeros_like(rhs)
        tol = float(np.float32(1e-6)) * self.norm(rhs)
        r = rhs - self.apply(x)
        best, rt, least, rho = x, r, self.norm(r), None
        u = p = q = None
        act, more, converged = least, 0, False
        for it in range(CGS_ITERATIONS):
            old, rho = rho, self.dot(rt, r)
            if it == 0:
                u, p = r, r
            else:
                beta = rho / old
                u = r + beta * q
                p = u + beta * (q + beta * p)
            v = self.apply(p)
            alpha = rho / self.dot(rt, v)
            q = u - alpha * v
            uh = u + q
            x = x + alpha * uh
            r = r - alpha * self.apply(uh)
            act = self.norm(r)
            if act <= tol or more:
                r = rhs - self.apply(r)
                act = self.norm(r)
                if act <= tol:
                    converged = True
                    break
                more += 1
                if more >= 5:
                    break
            if act < least:
                best, least = x, act
        if not converged and self.norm(rhs - self.apply(best)) <= act:
            x = best
        return x


def exact(case, seed):
    n, na, s, it, op = case["n"], case["angles"], case["slices"], case["iters"], case["op"]
    if op == "batch":
        some = min(s, 2)
    elif op in ("sirt", "project"):
        some = s
    else:
        some = 1 if op in ("asdpocs", "subsets") else s
    if op != "mix" and _samples(dict(case, slices=some)) > EXACT_SAMPLES:
        return None
    if op == "mix":
        if _samples(case) > EXACT_SAMPLES:
            return None
        return [_Exact(m, a, -1.0).sirt(b[None].double(), it, RELAX)[0]
                for (m, a), b in zip(_members(case), _inputs(case, seed))]
    e = _Exact(n, na, _axis(case, n), case["model"])
    data = _inputs(case, seed)
    if op == "project":
        return [e.forward(data[0].double()), e.backward(data[1].double())]
    b = data.double()
    if op == "batch":
        return [e.sirt(b[:some], it, RELAX)] + ([None] if s > 2 else [])
    if op == "sirt":
        return [e.sirt(b, it, RELAX)]
    if op == "sart":
        return [e.sart(b, it, RELAX)]
    if op == "asdpocs":
        return [_asdpocs(e, b[:1], it)[None].repeat(s, 1, 1)]
    if op == "sbtv":
        return [torch.stack([_Sbtv(e).first(b[k]) for k in range(s)])] if it == 1 else None
    every = torch.arange(na, device="cuda")
    relax = float(np.float32(0.5 / (n * case["subset"])))
    x, res, v = torch.zeros(1, n, n, device="cuda", dtype=torch.float64), b.clone(), e.vertical.tolist()
    runs, at = [], 0
    for a in range(1, na + 1):
        if a == na or v[a] != v[at]:
            runs.append((at, a - at, int(v[at])))
            at = a
    for off, count, _ in _subsets(runs, case["subset"]):
        a = every[off:off + count]
        res[:, a] -= e.forward(x, a)[:, a]
        x = x + relax * e.backward(res, a)
    return [res[0], x[0]]
