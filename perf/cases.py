"""The work a user of the framework has it do, as timed cases.

Each case is one call (or the few calls a program makes together) through the
package's public entry points: projector pairs, CGLS and split-Bregman
reconstructions, the framelet transform, batches of fan slices, and the
version-1 pair that an unmodified MATLAB program reaches. ``listed()`` names
twelve of them; ``draw(rng)`` gives more of the same ranges.

``exact(case, seed)`` is the same result in 64 bits from plain torch: an FP64
Siddon projector (every plane crossing of a ray, sorted), a framelet made of
circular shifts, and the solver loops over them. A plan that uses a scan's
turns and its reflection projects the scan whose angles are exact turns and
mirror images of the walked views; ``_angles`` gives those.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from framelab_gb300 import geometry as G
from framelab_gb300.batch import FanBatch
from framelab_gb300.projector import Plan
from framelab_gb300.solvers import NativeCGLS
from framelab_gb300.transforms import FrameletSystem, SplitBregmanSolver

_DT = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
_FAN = dict(SO=500.0, OD=500.0, L=256.0)          # the benchmark's fan scanner, mm
_CONE = dict(SO=600.0, SD=1200.0)                 # the benchmark's cone scanner, mm


def listed():
    return [
        # the smallest call: a quick look at a 64^2 slice, forward and back (latency, launches)
        dict(name="fan64_pair", kind="fan_pair", nx=64, ny=64, nd=96, nv=90),
        # the 2-D configuration: a slice from its sinogram (four CGLS iterations: on noisy data a few more
        # and the FP32 recurrence itself is what an output shows)
        dict(name="fan256_cgls", kind="fan_cgls", n=256, nd=512, nv=360, iters=4),
        # a rectangular slice with an odd, ragged size and view count (no symmetry to use)
        dict(name="fan_ragged_pair", kind="fan_pair", nx=501, ny=383, nd=701, nv=451),
        # a stack of uneven slices reconstructed together
        dict(name="fanbatch64_cgls", kind="fan_batch", slices=64, pick=7, iters=4),
        # the smallest volume, stored in 16 bits, forward and back (latency)
        dict(name="cone64_f16_pair", kind="cone_pair", n=64, nz=64, na=96, nb=80, nv=72, dtype="f16"),
        # the ordinary 3-D configuration, forward and back
        dict(name="cone256_pair", kind="cone_pair", n=256, nz=256, na=512, nb=384, nv=360, dtype="f32"),
        # the largest reconstruction: right-hand side from the sinogram, two CGLS iterations
        dict(name="cone512_cgls", kind="cone_cgls", n=512, na=1024, nb=768, nv=720, iters=2, mode="graph"),
        # a circular scan with odd sizes everywhere (no symmetry to use)
        dict(name="cone_ragged_pair", kind="cone_pair", n=151, nz=97, na=223, nb=161, nv=211, dtype="f32"),
        # a helical scan: the source moves along z
        dict(name="helix128_pair", kind="helix_pair", n=128, na=192, nb=64, nv=241),
        # the sparse-view reconstruction: two outer split-Bregman iterations of five CGLS each
        dict(name="sb256", kind="sb", n=256, na=512, nb=384, nv=90, outer=2),
        # the framelet transform and its adjoint on a volume of uneven sides
        dict(name="framelet3d_pair", kind="framelet", nx=200, ny=176, nz=144, levels=2, bank="linear"),
        # what an unmodified MATLAB program calls: the version-1 forward and backprojector
        dict(name="mex_v1_pair", kind="mex_pair", n=128, na=192, nb=160, nv=120),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fan_pair", "fan_pair", "fan_cgls", "fan_batch", "cone_pair", "cone_pair", "cone_cgls",
                       "helix_pair", "sb", "framelet", "mex_pair"])
    even = rng.random() < 0.6                      # most scans are set up with even, often round, sizes
    up = (lambda v, m: max(m, m * round(v / m))) if even else (lambda v, m: v)
    if kind == "fan_pair":
        nx = up(_log(rng, 48, 640), 4)
        ny = nx if rng.random() < 0.6 else up(_log(rng, 48, 640), 4)
        return dict(kind=kind, nx=nx, ny=ny, nd=up(int(max(nx, ny) * rng.uniform(1.2, 2.2)), 2), nv=up(_log(rng, 40, 720), 4))
    if kind == "fan_cgls":
        n = up(_log(rng, 64, 512), 4)
        return dict(kind=kind, n=n, nd=up(int(n * rng.uniform(1.3, 2.2)), 2), nv=up(_log(rng, 60, 720), 4), iters=rng.randint(1, 4))
    if kind == "fan_batch":
        return dict(kind=kind, slices=rng.randint(2, 48), pick=rng.randint(1, 10 ** 6), iters=rng.randint(1, 4))
    if kind == "cone_pair":
        n = up(_log(rng, 40, 224), 4)
        nz = n if rng.random() < 0.5 else up(max(8, int(n * rng.uniform(0.3, 1.1))), 2)
        return dict(kind=kind, n=n, nz=nz, na=up(int(n * rng.uniform(1.3, 2.1)), 2), nb=up(max(8, int(nz * rng.uniform(1.0, 1.7))), 2),
                    nv=up(_log(rng, 30, 400), 8 if rng.random() < 0.6 else 2), dtype=rng.choice(["f32", "f32", "f32", "f16", "bf16"]))
    if kind == "cone_cgls":
        n = up(_log(rng, 64, 256), 4)
        return dict(kind=kind, n=n, na=up(int(n * rng.uniform(1.4, 2.1)), 2), nb=up(int(n * rng.uniform(1.0, 1.6)), 2), nv=up(_log(rng, 60, 360), 8),
                    iters=rng.randint(1, 4), mode=rng.choice(["graph", "graph", "mixed"]))
    if kind == "helix_pair":
        n = up(_log(rng, 48, 192), 2)
        return dict(kind=kind, n=n, na=int(n * rng.uniform(1.2, 1.9)), nb=max(12, int(n * rng.uniform(0.2, 0.7))), nv=_log(rng, 60, 400))
    if kind == "sb":
        n = up(_log(rng, 40, 192), 4)
        return dict(kind=kind, n=n, na=up(int(n * rng.uniform(1.4, 2.1)), 2), nb=up(int(n * rng.uniform(1.0, 1.6)), 2), nv=up(_log(rng, 24, 120), 2),
                    outer=rng.randint(1, 3))
    if kind == "framelet":
        flat = rng.random() < 0.25
        side = (lambda: _log(rng, 64, 1500)) if flat else (lambda: _log(rng, 24, 256))
        return dict(kind=kind, nx=up(side(), 4), ny=up(side(), 4), nz=1 if flat else up(side(), 4), levels=rng.randint(1, 3),
                    bank=rng.choice(["linear", "linear", "haar"] + (["cubic"] if flat else [])))
    n = up(_log(rng, 32, 144), 2)
    return dict(kind="mex_pair", n=n, na=up(int(n * rng.uniform(1.2, 2.0)), 2), nb=up(int(n * rng.uniform(0.8, 1.5)), 2), nv=_log(rng, 24, 160))


# ----------------------------------------------------------------- geometry
def _fan_para(nx, ny, nd, nv):
    """The fan scanner over a field whose longer side is 256 mm; the detector spans the field's magnified diagonal."""
    pix = _FAN["L"] / max(nx, ny)
    Lx, Ly = nx * pix, ny * pix
    return G.fan_para(nx, ny, nd, nv, L=(Lx, Ly), SO=_FAN["SO"], OD=_FAN["OD"], Ly=2.0 * math.hypot(Lx, Ly))


def _cone_para(n, nz, na, nb, nv, dz=1.0):
    """The cone scanner over a field 256 mm wide; the panel keeps the benchmark's 512 mm width and its rows are square."""
    vox = 256.0 / n
    pitch = 512.0 / na
    return G.cone_para(n, n, nz, na, nb, nv, L=(256.0, 256.0, nz * vox * dz), SO=_CONE["SO"], OD=_CONE["SD"] - _CONE["SO"],
                       Ly=na * pitch, Lz=nb * pitch)


def _helix_para(c):
    """A helix over the length of the volume: three turns, a panel of fewer rows than columns."""
    n = c["n"]
    return G.cone_para(n, n, n, c["na"], c["nb"], L=(2.0, 2.0, 2.0), SO=6.0, OD=6.0, Ly=5.6, Lz=5.6 * c["nb"] / c["na"], scan="helix",
                       zmax=2.0, rps=3.0, vtab=2.0, fps=float(c["nv"] - 1))


def _batch_slices(c):
    """Uneven slices, the sizes and view counts of the batched benchmark."""
    r = np.random.default_rng(c["pick"])
    ns, nvs = r.choice(np.array((128, 192, 256, 384, 512)), c["slices"]), r.integers(180, 721, c["slices"])
    return [(int(n), int(v)) for n, v in zip(ns, nvs)]


def _paras(c):
    k = c["kind"]
    if k == "fan_pair":
        return [_fan_para(c["nx"], c["ny"], c["nd"], c["nv"])]
    if k == "fan_cgls":
        return [_fan_para(c["n"], c["n"], c["nd"], c["nv"])]
    if k == "fan_batch":
        return [_fan_para(n, n, 2 * n, v) for n, v in _batch_slices(c)]
    if k == "helix_pair":
        return [_helix_para(c)]
    if k == "framelet":
        return []
    return [_cone_para(c["n"], c.get("nz", c["n"]), c["na"], c["nb"], c["nv"])]


# ------------------------------------------------------------ synthetic data
def _gen(seed):
    return torch.Generator().manual_seed(seed)


def _ellipsoids(seed, count, dim):
    """Centres in [-0.6, 0.6]^dim, semi-axes 0.05 .. 0.45 and densities 0.1 .. 1, in units of half the field."""
    g = _gen(seed)
    return (torch.rand(count, dim, generator=g) * 1.2 - 0.6, torch.rand(count, dim, generator=g) * 0.4 + 0.05,
            torch.rand(count, generator=g) * 0.9 + 0.1)


def _image(seed, shape, count=8):
    """Piecewise constant phantom on the GPU: a sum of ellipsoids (shape z, y, x or y, x)."""
    cs, rs, ds = _ellipsoids(seed, count, len(shape))
    out = torch.zeros(shape, device="cuda")
    axes = [(torch.arange(n, device="cuda") + 0.5) * (2.0 / n) - 1.0 for n in shape]
    for c, r, d in zip(cs.tolist(), rs.tolist(), ds.tolist()):
        q = sum((((a - ci) / ri) ** 2).view([-1 if j == i else 1 for j in range(len(shape))])
                for i, (a, ci, ri) in enumerate(zip(axes, c, r)))
        out += d * (q <= 1.0)
    return out


def _detectors(p, phi, dtype, ivs):
    """Source and detector points of views `ivs` of a scan, in xy voxels from the isocentre: (v, 1, 1) and (v, nb, na)."""
    dev = "cuda"
    ph = torch.as_tensor(phi, dtype=torch.float64, device=dev)[ivs]
    c, s = ph.cos().to(dtype).view(-1, 1, 1), ph.sin().to(dtype).view(-1, 1, 1)
    u = torch.as_tensor(np.asarray(p["y_det"], np.float64), dtype=dtype, device=dev).view(1, 1, -1)
    SO, OD = float(p["SO"]), float(p["OD"])
    src, det = [-SO * c, -SO * s], [OD * c - u * s, OD * s + u * c]
    if "nz" in p:
        z0 = torch.as_tensor(np.asarray(p["sd_z"], np.float64), dtype=dtype, device=dev)[ivs].view(-1, 1, 1)
        v = torch.as_tensor(np.asarray(p["z_det"], np.float64), dtype=dtype, device=dev).view(1, -1, 1)
        src.append(z0)
        det.append(z0 + v)
    return src, det


def _sinogram(seed, p, noise=0.01, count=4):
    """Measured data of a scan: the line integrals of a few ellipsoids and 1 % of Gaussian noise."""
    phi = np.asarray(p["sd_phi"], np.float64)
    nv, na, nb = len(phi), len(p["y_det"]), len(p["z_det"]) if "nz" in p else 1
    half = [int(p["nx"]) / 2, int(p["ny"]) / 2] + ([int(p["nz"]) * float(p["dz"]) / 2] if "nz" in p else [])
    cs, rs, ds = _ellipsoids(seed + 1, count, len(half))
    y = torch.empty(nv, nb, na, device="cuda")
    step = max(1, 40_000_000 // (na * nb))
    for v0 in range(0, nv, step):
        ivs = torch.arange(v0, min(v0 + step, nv), device="cuda")
        src, det = _detectors(p, phi, torch.float32, ivs)
        out = y[v0:v0 + step].zero_()
        length = sum((d - s) ** 2 for s, d in zip(src, det)).sqrt() * float(p["scale"])
        for c, r, rho in zip(cs.tolist(), rs.tolist(), ds.tolist()):
            a = b = e = 0.0
            for s, d, h, ci, ri in zip(src, det, half, c, r):
                o, w = (s - ci * h) / (ri * h), (d - s) / (ri * h)
                a, b, e = a + w * w, b + o * w, e + o * o
            out += rho * 2.0 * (b * b - a * (e - 1.0)).clamp_(min=0.0).sqrt() / a * length
    g = torch.Generator(device="cuda").manual_seed(seed + 2)
    y += torch.randn(y.shape, device="cuda", generator=g) * (noise * float(y.max()))
    return y if "nz" in p else y.view(nv, na)


# ------------------------------------------------------------- prepare / run
def prepare(case, seed):
    k = case["kind"]
    if k == "framelet":
        shape = (case["ny"], case["nx"]) if case["nz"] == 1 else (case["nz"], case["ny"], case["nx"])
        return dict(kind=k, W=FrameletSystem(shape, case["bank"], case["levels"]), x=_image(seed, shape))
    paras = _paras(case)
    if k == "fan_batch":
        y = torch.cat([_sinogram(seed + 10 * i, p).reshape(-1) for i, p in enumerate(paras)])
        return dict(kind=k, B=FanBatch(paras), y=y, iters=case["iters"])
    p = paras[0]
    P = Plan(p)
    st = dict(kind=k, P=P, y=_sinogram(seed, p))
    if k in ("fan_pair", "cone_pair", "helix_pair", "mex_pair"):
        shape = (P.nz, P.ny, P.nx) if P.cone else (P.ny, P.nx)
        dt = _DT[case.get("dtype", "f32")]
        st["x"] = _image(seed, shape).view(P.vol_shape).to(dt)
        st["dt"], st["y"] = dt, st["y"].to(dt)
    elif k in ("fan_cgls", "cone_cgls"):
        st["cg"], st["iters"] = NativeCGLS(P, case.get("mode", "graph")), case["iters"]
    else:
        st["sb"], st["outer"] = SplitBregmanSolver(P, levels=2, kind="linear", mode="graph"), case["outer"]
        st["y"] = st["y"] * (4.0 / st["y"].max())
        st["u0"] = torch.zeros(P.vol_shape, device="cuda")
    return st


def run(st):
    k = st["kind"]
    if k == "framelet":
        coef = st["W"].forward(st["x"])
        return coef, st["W"].adjoint(coef)
    if k == "fan_batch":
        return st["B"].cgls(st["B"].adjoint(st["y"]), iters=st["iters"])
    P = st["P"]
    if k in ("fan_pair", "cone_pair", "helix_pair"):
        return P.forward(st["x"], out_dtype=st["dt"]), P.adjoint(st["y"], out_dtype=st["dt"])
    if k == "mex_pair":
        y, yn = P.forward_gao(st["x"])
        return y, yn, P.adjoint(st["y"], model="chord_ref")
    if k in ("fan_cgls", "cone_cgls"):
        return st["cg"].solve(P.adjoint(st["y"]), iters=st["iters"])
    return st["sb"].solve(st["y"], st["u0"], lam=0.01, mu=1.0, outer=st["outer"], cg_iters=5)


def _scan_sizes(c):
    """(rays, voxels, crossings) of a case's scans; a ray that meets the field crosses about 1.28 n voxels of an n-wide one."""
    rays = vox = isect = 0
    for p in _paras(c):
        n, cone = 0.5 * (int(p["nx"]) + int(p["ny"])), "nz" in p
        r = len(p["sd_phi"]) * len(p["y_det"]) * (len(p["z_det"]) if cone else 1)
        rays, vox, isect = rays + r, vox + int(p["nx"]) * int(p["ny"]) * (int(p["nz"]) if cone else 1), isect + int(1.28 * n * r * (0.5 if c["kind"] == "helix_pair" else 1.0))
    return rays, vox, isect


def _bands(c):
    nf = {"linear": 3, "haar": 2, "cubic": 5}[c.get("bank", "linear")]
    nb = nf ** (2 if c.get("nz", 2) == 1 else 3)
    lev = c.get("levels", 2)
    return lev * (nb - 1) + 1, nf


def work(case):
    k = case["kind"]
    if k == "framelet":
        n = case["nx"] * case["ny"] * case["nz"]
        nb, nf = _bands(case)
        taps = 5 if case["bank"] == "cubic" else 3
        return {"bytes": 4 * n * (1 + nb + nb + 1), "flops": 2 * 2 * taps * n * nb}
    rays, vox, isect = _scan_sizes(case)
    size = 4 if case.get("dtype", "f32") == "f32" else 2
    if k in ("fan_pair", "cone_pair", "helix_pair", "mex_pair"):
        more = rays * 4 if k == "mex_pair" else 0
        return {"bytes": 2 * size * (rays + vox) + more, "flops": 4 * isect}
    if k != "sb":
        return {"bytes": 4 * (rays + vox) + case["iters"] * 4 * 6 * vox, "flops": 2 * isect + case["iters"] * (4 * isect + 10 * vox)}
    nb, nf = _bands({})
    cg = 5 * (4 * isect + 10 * vox) + 4 * isect
    return {"bytes": 4 * (rays + vox) + case["outer"] * (4 * 36 * vox + 4 * 3 * nb * vox),
            "flops": 2 * isect + case["outer"] * (cg + 12 * nb * vox)}


# ------------------------------------------------------------- 64-bit results
def _angles(p, kind):
    """FP64 view angles of the scan a plan projects: the given ones, or where the scan has a half or quarter turn (and a
    reflection about the x axis), exact turns and mirror images of the walked views' given angles."""
    phi = np.asarray(p["sd_phi"], np.float64)
    nv, nx, ny, na = len(phi), int(p["nx"]), int(p["ny"]), len(p["y_det"])
    cone = "nz" in p
    if kind in ("helix_pair", "mex_pair"):
        return phi
    m = 4 if cone else 2
    half = nv % 2 == 0 and nx % m == 0 and ny % m == 0
    if cone:
        half = half and int(p["nz"]) % 2 == 0 and len(p["z_det"]) % 2 == 0
    quarter = half and nx == ny and nv % 4 == 0
    mirror = (cone or kind == "fan_batch") and na % 2 == 0
    turns = 4 if quarter else 2 if half else 1
    if quarter and nv % 8:
        mirror = False
    if turns == 1:
        mirror = mirror and not cone and nv % 2 == 1 and ny % 2 == 0
    out = phi.copy()
    q, turn = nv // turns, 2 * math.pi / turns
    for v in range(q if not mirror else q // 2 + 1):
        a = phi[v]
        if mirror and q % 2 == 0 and v == q // 2:
            a = math.pi / turns
        for j in range(turns):
            out[(v + j * q) % nv] = a + j * turn
            if mirror and v:
                out[(j * q - v) % nv] = j * turn - a
    return out


class _Siddon:
    """Exact intersection lengths of every ray of a scan with every voxel, in 64 bits, a few views at a time."""

    def __init__(self, p, kind):
        self.p, self.phi = p, _angles(p, kind)
        self.n = [int(p["nx"]), int(p["ny"])] + ([int(p["nz"])] if "nz" in p else [])
        self.pitch = [1.0, 1.0] + ([float(p["dz"])] if "nz" in p else [])
        self.nv, self.na, self.nb = len(self.phi), len(p["y_det"]), len(p["z_det"]) if "nz" in p else 1
        self.cross = sum(self.n) + len(self.n)
        self.kept = [] if self.nv * self.na * self.nb * self.cross <= 4e8 else None

    def _chunk(self, ivs):
        src, det = _detectors(self.p, self.phi, torch.float64, ivs)
        shape = (len(ivs), self.nb, self.na)
        S = [s.expand(shape).reshape(-1, 1) for s in src]
        D = [(d.expand(shape).reshape(-1, 1) - s) for d, s in zip(det, S)]
        xy = (D[0] ** 2 + D[1] ** 2).sqrt()
        for i, lim in enumerate([xy, xy] + [torch.full_like(xy, float(self.p["SO"]) + float(self.p["OD"]))] * (len(S) - 2)):
            tiny = D[i].abs() < 1e-9 * lim
            D[i] = torch.where(tiny, torch.where(D[i] < 0, -1e-9 * lim, 1e-9 * lim), D[i])
        t = torch.cat([((torch.arange(n + 1, device="cuda", dtype=torch.float64) - n // 2) * h - s) / d
                       for n, h, s, d in zip(self.n, self.pitch, S, D)], 1)
        t = t.sort(1).values
        seg = t[:, 1:] - t[:, :-1]
        mid = 0.5 * (t[:, 1:] + t[:, :-1])
        idx, ok, stride = 0, True, 1
        for n, h, s, d in zip(self.n, self.pitch, S, D):
            j = torch.floor((s + mid * d) / h).long() + n // 2
            ok = ok & (j >= 0) & (j < n)
            idx = idx + j.clamp_(0, n - 1) * stride
            stride *= n
        length = sum(d * d for d in D).sqrt() * float(self.p["scale"])
        return seg.mul_(length).mul_(ok), idx

    def chunks(self):
        if self.kept:
            yield from self.kept
            return
        step = max(1, int(2.5e7 // (self.na * self.nb * self.cross)))
        for v0 in range(0, self.nv, step):
            c = (v0, *self._chunk(torch.arange(v0, min(v0 + step, self.nv), device="cuda")))
            if self.kept is not None:
                self.kept.append(c)
            yield c

    def _rays(self, v0, w):
        return slice(v0 * self.nb * self.na, v0 * self.nb * self.na + w.shape[0])

    def forward(self, x):
        x, y = x.double().reshape(-1), torch.zeros(self.nv * self.nb * self.na, device="cuda", dtype=torch.float64)
        for v0, w, idx in self.chunks():
            y[self._rays(v0, w)] = (w * x[idx]).sum(1)
        return y

    def adjoint(self, y):
        y, x = y.double().reshape(-1), torch.zeros(math.prod(self.n), device="cuda", dtype=torch.float64)
        for v0, w, idx in self.chunks():
            x.index_add_(0, idx.reshape(-1), (w * y[self._rays(v0, w)].view(-1, 1)).reshape(-1))
        return x

    def both(self, x, y):
        x, y = x.double().reshape(-1), y.double().reshape(-1)
        Ax, Aty = torch.zeros_like(y), torch.zeros_like(x)
        for v0, w, idx in self.chunks():
            r = self._rays(v0, w)
            Ax[r] = (w * x[idx]).sum(1)
            Aty.index_add_(0, idx.reshape(-1), (w * y[r].view(-1, 1)).reshape(-1))
        return Ax, Aty


def _cgls(A, b, u, lam, iters, tol):
    normal = lambda v: A.adjoint(A.forward(v)) + lam * v
    r = normal(u) - b
    p, gamma = -r, float(r @ r)
    for _ in range(iters):
        if gamma == 0.0:
            break
        q = normal(p)
        alpha = gamma / float(p @ q)
        u, r = u + alpha * p, r + alpha * q
        new = float(r @ r)
        p, gamma = -r + (new / gamma) * p, new
        if gamma < tol:
            break
    return u


_BANK = {  # analysis and synthesis taps
    "linear": ([[0.25, 0.5, 0.25], [-math.sqrt(2) / 4, 0, math.sqrt(2) / 4], [-0.25, 0.5, -0.25]],
               [[0.25, 0.5, 0.25], [math.sqrt(2) / 4, 0, -math.sqrt(2) / 4], [-0.25, 0.5, -0.25]]),
    "haar": ([[0, 0.5, 0.5], [0, -0.5, 0.5]], [[0.5, 0.5, 0], [0.5, -0.5, 0]]),
    "cubic": ([[1 / 16, 4 / 16, 6 / 16, 4 / 16, 1 / 16], [-1 / 8, -2 / 8, 0, 2 / 8, 1 / 8],
               [-math.sqrt(6) / 16, 0, 2 * math.sqrt(6) / 16, 0, -math.sqrt(6) / 16], [-1 / 8, 2 / 8, 0, -2 / 8, 1 / 8],
               [-1 / 16, 4 / 16, -6 / 16, 4 / 16, -1 / 16]],
              [[1 / 16, 4 / 16, 6 / 16, 4 / 16, 1 / 16], [1 / 8, 2 / 8, 0, -2 / 8, -1 / 8],
               [-math.sqrt(6) / 16, 0, 2 * math.sqrt(6) / 16, 0, -math.sqrt(6) / 16], [1 / 8, -2 / 8, 0, 2 / 8, -1 / 8],
               [-1 / 16, 4 / 16, -6 / 16, 4 / 16, -1 / 16]]),
}


class _Framelet:
    """The undecimated framelet by circular shifts: bands i, j, k along y, x, z (2-D: i, j along x, y)."""

    def __init__(self, shape, bank, levels):
        self.shape, self.levels, (self.D, self.R) = tuple(shape), levels, _BANK[bank]
        self.dims = (1, 2, 0) if len(shape) == 3 else (1, 0)

    @staticmethod
    def _corr(x, taps, dim, step):
        c = (len(taps) - 1) // 2
        return sum(w * torch.roll(x, -(t - c) * step, dim) for t, w in enumerate(taps) if w)

    def forward(self, x):
        x, out = x.double().reshape(self.shape), []
        for lev in range(self.levels):
            bands = [x]
            for dim in self.dims:
                bands = [self._corr(b, f, dim, 1 << lev) for b in bands for f in self.D]
            x = bands[0]
            out += bands if lev == self.levels - 1 else bands[1:]
        return torch.cat([b.reshape(-1) for b in out])

    def adjoint(self, coef):
        c = list(coef.double().view(-1, *self.shape))
        nb, low = len(self.D) ** len(self.dims), None
        for lev in range(self.levels - 1, -1, -1):
            at = lev * (nb - 1)
            bands = c[at:at + nb] if low is None else [low] + c[at:at + nb - 1]
            for dim in reversed(self.dims):
                bands = [sum(self._corr(bands[i + f], self.R[f], dim, 1 << lev) for f in range(len(self.D)))
                         for i in range(0, len(bands), len(self.D))]
            low = bands[0]
        return low


def _elements(c):
    """Plane crossings all projections of a case sort or read again, in 64 bits."""
    per = sum(len(p["sd_phi"]) * len(p["y_det"]) * (len(p["z_det"]) if "nz" in p else 1) *
              (int(p["nx"]) + int(p["ny"]) + (int(p["nz"]) if "nz" in p else 0) + 3) for p in _paras(c))
    k = c["kind"]
    if k.endswith("_pair"):
        return per, 1
    if k == "sb":
        return per, 1 + c["outer"] * 12
    return per, 3 + 2 * c["iters"]


def exact(case, seed):
    k = case["kind"]
    if k == "framelet":
        n = case["nx"] * case["ny"] * case["nz"] * _bands(case)[0]
        if n > 6e8:
            return None
        shape = (case["ny"], case["nx"]) if case["nz"] == 1 else (case["nz"], case["ny"], case["nx"])
        W = _Framelet(shape, case["bank"], case["levels"])
        coef = W.forward(_image(seed, shape))
        return coef, W.adjoint(coef)
    per, times = _elements(case)
    if (times == 1 and per > 1.6e9) or (times > 1 and (per > 4e8 or per * times > 6e9)):
        return None
    paras = _paras(case)
    if k == "fan_batch":
        out = []
        for i, p in enumerate(paras):
            A = _Siddon(p, k)
            b = A.adjoint(_sinogram(seed + 10 * i, p))
            out.append(_cgls(A, b, torch.zeros_like(b), 0.0, case["iters"], 0.0))
        return torch.cat(out)
    p = paras[0]
    A, y = _Siddon(p, k), _sinogram(seed, p)
    if k.endswith("_pair"):
        dt = _DT[case.get("dtype", "f32")]
        shape = tuple(reversed(A.n))
        x, y = _image(seed, shape).to(dt), y.to(dt)
        if k != "mex_pair":
            Ax, Aty = A.both(x, y)
            sino = (A.nv, A.nb, A.na) if len(A.n) == 3 else (A.nv, A.na)
            return Ax.view(sino), Aty.view(1, *shape)
        # the version-1 pair: lengths in physical units forward (and divided by the ray's length), in voxels times the pitch back
        Ax, _ = A.both(x, y)
        src, det = _detectors(p, A.phi, torch.float64, torch.arange(A.nv, device="cuda"))
        length = sum((d - s) ** 2 for s, d in zip(src, det)).sqrt() * float(p["scale"])
        Ax = Ax.view(A.nv, A.nb, A.na)
        return Ax, Ax / length, None
    b = A.adjoint(y)
    if k in ("fan_cgls", "cone_cgls"):
        shape = (1, *reversed(A.n))
        return _cgls(A, b, torch.zeros_like(b), 0.0, case["iters"], 1e-14).view(shape)
    y = y * (4.0 / y.max())
    b0 = A.adjoint(y)
    shape = (int(p["nz"]), int(p["ny"]), int(p["nx"]))
    W, mu, tau = _Framelet(shape, "linear", 2), 1.0, 0.01
    u = torch.zeros_like(b0)
    v, b = W.forward(u), b0
    keep = slice(26 * u.numel(), 27 * u.numel())       # the low band of the last level is not shrunk
    for _ in range(case["outer"]):
        u = _cgls(A, b, u, mu, 5, 1e-10)
        s = v + W.forward(u)
        a = s.sign() * (s.abs() - tau).clamp(min=0.0)
        a[keep] = s[keep]
        v = s - a
        b = b0 + mu * W.adjoint(a - v).reshape(-1)
    return u.view(1, *shape)
