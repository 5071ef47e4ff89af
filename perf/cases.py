"""The work that users of this library have it do, as timed cases.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare``/``run`` build a case's state on the GPU and make one pass through
the public entry points (``hycadv.Context``, ``hycadv.Ensemble``), ``work``
counts what a pass cannot do without and ``exact`` restates the pass in plain
64-bit torch.

Inputs are seeded synthetic ocean states in the reference's layout and units:
a coast and islands (closed) or a re-entrant channel with ~30 % land
(periodic), layers of 10-500 m, an eddying flow at a given Courant number
with a small divergent part, temperature and salinity with eddies, passive
tracers with log-uniform values and sharp fronts, and a grid spacing that
varies with latitude.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hycom-src_gb300"))

import hycadv  # noqa: E402

NB = 6  # nbdy of every case: the reference's halo width
ONEM = 9806.0  # Pa per metre
ONEMU = 9806.0e-12
THBASE, ONETA0, RA2FAC, TEMDF2 = 34.0, 0.1, 0.125, 0.015
F64 = torch.float64
DEV = "cuda"
MOST_UPDATES = 4500 * 3298 * 41 * 2  # the largest listed case, in cells x layers x tracers


def listed():
    ts = dict(kind="tsadvc", scheme=2, ntr=0, btrmas=False, courant=0.5, dt=1800.0)
    ens = dict(kind="ens", precision="mixed", scheme=2, basins=1, steps=3, diffusion=False, courant=0.8, dt=240.0)
    return [
        # one slice of one field: a host program that calls advem itself (latency, launches)
        dict(name="advem_257x193", kind="advem", scheme=2, nx=257, ny=193, periodic=False, courant=0.5, dt=1800.0),
        # the small closed basin of the tests and of model development: T and S
        dict(ts, name="tsadvc_fct2_257x193x10", nx=257, ny=193, kdm=10, periodic=False),
        # the global basin, the drop-in's FP64 step: T and S, FCT2
        dict(ts, name="tsadvc_fct2_4500x3298x41", nx=4500, ny=3298, kdm=41, periodic=True, courant=0.8, dt=240.0),
        # FCT4 with two passive tracers, an odd row length
        dict(ts, name="tsadvc_fct4_1201x901x22_t4", scheme=4, nx=1201, ny=901, kdm=22, ntr=2, periodic=True),
        # MPDATA on a regional basin
        dict(ts, name="tsadvc_mpdata_1500x1100x32", scheme=1, nx=1500, ny=1100, kdm=32, periodic=False),
        # FCT2 with the barotropic mass flux (advem_fct2c)
        dict(ts, name="tsadvc_btrmas_900x700x32", nx=900, ny=700, kdm=32, periodic=False, btrmas=True),
        # the whole tracer step of a model: filter save, advection, diffusion and density, filter
        dict(name="step_1500x1100x41", kind="step", scheme=2, nx=1500, ny=1100, kdm=41, ntr=0, periodic=True,
             courant=0.5, dt=600.0),
        # the continuity equation with biharmonic interface diffusion
        dict(name="cnuity_1500x1100x41", kind="cnuity", nx=1500, ny=1100, kdm=41, periodic=False, thkdf=4,
             courant=0.5, dt=600.0),
        # an ensemble of uneven basins (nx 120-1500), 2-6 tracers, in the plain precision
        dict(ens, name="ens_fp64_6basins", precision="fp64", basins=6, nx=1500, ny=1100, kdm=41, ntr=4,
             periodic=False, courant=0.5, dt=1800.0),
        # the FP32-mixed form on the global basin, T and S
        dict(ens, name="ens_mixed_4500x3298x41", nx=4500, ny=3298, kdm=41, ntr=2, periodic=True),
        # the FP32-mixed form on many uneven basins
        dict(ens, name="ens_mixed_24basins", basins=24, nx=1500, ny=1100, kdm=41, ntr=6, steps=6, periodic=False,
             courant=0.5, dt=1800.0),
        # the FP32-mixed form with ten tracers, MPDATA, two regional basins
        dict(ens, name="ens_mixed_mpdata_t10", scheme=1, basins=2, nx=800, ny=600, kdm=41, ntr=10, periodic=False,
             courant=0.9, dt=600.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["advem", "tsadvc", "tsadvc", "tsadvc", "step", "cnuity", "ens", "ens", "ens"])
    c = dict(kind=kind, periodic=rng.random() < 0.5, courant=round(rng.uniform(0.3, 0.9), 2),
             dt=rng.choice([240.0, 600.0, 1800.0]))
    c["nx"] = _log(rng, 60, 4500)
    c["ny"] = max(40, int(c["nx"] * rng.uniform(0.5, 0.9)))
    if kind == "advem":
        c["scheme"] = rng.choice([0, 1, 2, 4])
        return c
    c["kdm"] = rng.choice([3, 10, 22, 32, 41])
    if kind == "tsadvc":
        c.update(scheme=rng.choice([0, 1, 2, 2, 4]), ntr=rng.choice([0, 0, 1, 3]), btrmas=False)
        if c["scheme"] == 2 and rng.random() < 0.2:
            c["btrmas"] = True
    elif kind == "step":
        c.update(scheme=rng.choice([1, 2, 4]), ntr=rng.choice([0, 0, 1]))
    elif kind == "cnuity":
        c["thkdf"] = rng.choice([0, 2, 4])
    else:
        c.update(precision=rng.choice(["mixed", "mixed", "fp64"]), basins=rng.choice([1, 1, 4, 12]), diffusion=False,
                 ntr=rng.choice([2, 3, 5, 10]), steps=rng.choice([1, 3]))
        c["scheme"] = rng.choice([1, 2, 2, 4] if c["precision"] == "mixed" else [0, 1, 2, 4])
        c["diffusion"] = c["precision"] == "mixed" and rng.random() < 0.3
        if c["basins"] > 1:
            c["nx"], c["ny"] = max(c["nx"] // 2, 150), max(c["ny"] // 2, 100)
    # no costlier than the largest listed case: fewer layers, then a smaller basin
    slow = {"advem": 1, "tsadvc": 8 if c.get("btrmas") else 2, "step": 8, "cnuity": 4}.get(kind, 1)
    if kind == "ens":
        slow = c["steps"] * c["basins"] * (4 if c["precision"] == "fp64" else 2)
    while c["nx"] * c["ny"] * c["kdm"] * _fields(c) * slow > MOST_UPDATES:
        if c["kdm"] > 10:
            c["kdm"] -= 9
        else:
            c["nx"], c["ny"] = int(c["nx"] * 0.8), int(c["ny"] * 0.8)
    return c


def _fields(c):
    """Advected fields of a case."""
    return {"advem": 1, "cnuity": 1, "ens": c.get("ntr", 0)}.get(c["kind"], 2 + c.get("ntr", 0))


# ----------------------------------------------------------------------
# geometry: it belongs to the case, not to the seed
# ----------------------------------------------------------------------


def _no_one_point_seas(land, periodic):
    while True:
        p = np.pad(land, 1, constant_values=True)
        if periodic:
            p[1:-1, 0], p[1:-1, -1] = land[:, -1], land[:, 0]
        bad = ~land & p[1:-1, :-2] & p[1:-1, 2:] & p[:-2, 1:-1] & p[2:, 1:-1]
        if not bad.any():
            return land
        land = land | bad


@functools.lru_cache(maxsize=64)
def _geometry(nx, ny, periodic, salt=0):
    """(depth, masks, nreg, scp2, scp2i, dx) of a basin; dx(j) the grid spacing of each row."""
    rng = np.random.default_rng([nx, ny, int(periodic), salt])
    if periodic:
        x, y = (np.arange(nx, dtype=np.float32) + 0.5) / nx, (np.arange(ny, dtype=np.float32) + 0.5) / ny
        kx, ky = rng.integers(1, 9, 10), rng.uniform(0.5, 8.0, 10)
        px, py = rng.uniform(0, 2 * np.pi, (2, 10))
        noise = ((np.sin(2 * np.pi * y[:, None] * ky + py) / (kx + ky)).astype(np.float32)
                 @ np.sin(2 * np.pi * x[:, None] * kx + px).astype(np.float32).T)
        land = noise > np.quantile(noise[:: max(1, ny // 500), :: max(1, nx // 500)], 0.7)
        land[:2], land[-2:] = True, True
        land[ny // 2 - 1: ny // 2 + 2, -2:] = False  # sea in the last column: the basin is re-entrant
    else:
        land = np.zeros((ny, nx), bool)
        land[:2], land[-2:], land[:, :2], land[:, -2:] = True, True, True, True
        for _ in range(6):
            w, h = int(rng.integers(3, max(4, nx // 8))), int(rng.integers(3, max(4, ny // 8)))
            i, j = int(rng.integers(4, max(5, nx - w - 4))), int(rng.integers(4, max(5, ny - h - 4)))
            land[j:j + h, i:i + w] = True
    land = _no_one_point_seas(land, periodic)
    depth = np.zeros((ny + 2 * NB, nx + 2 * NB))
    depth[NB:-NB, NB:-NB] = np.where(land, 0.0, 4000.0)
    depth, masks, nreg = hycadv.bigrid(depth, NB)
    lat = (np.arange(1 - NB, ny + NB + 1) - 0.5) / ny
    dx = 1.0e4 * (0.6 + 0.4 * np.cos(1.2 * (lat - 0.4)))
    scp2 = np.ascontiguousarray(np.broadcast_to((dx * dx)[:, None], depth.shape))
    return depth, masks, nreg, scp2, 1.0 / scp2, dx


class _Grid:
    """Masks and metrics of a basin as CUDA tensors, for the generator and exact()."""

    def __init__(self, nx, ny, periodic, salt=0):
        depth, self.masks, self.nreg, self.scp2_np, self.scp2i_np, self.dx_np = _geometry(nx, ny, periodic, salt)
        self.nx, self.ny, self.ld1, self.ld2 = nx, ny, nx + 2 * NB, ny + 2 * NB
        self.periodic = self.nreg == 1
        self.ip = torch.from_numpy(depth > 0).to(DEV)
        self.iu = self.ip & _w(self.ip)
        self.iv = self.ip & _s(self.ip)
        self.scp2 = torch.from_numpy(self.scp2_np).to(DEV)
        self.scp2i = torch.from_numpy(self.scp2i_np).to(DEV)
        self.dx = torch.from_numpy(self.dx_np).to(DEV)[:, None]
        self.sea = torch.zeros_like(self.ip)
        self.sea[NB:-NB, NB:-NB] = self.ip[NB:-NB, NB:-NB]

    def spec(self, kdm, ntr):
        return dict(idm=self.nx, jdm=self.ny, kdm=kdm, nbdy=NB, nreg=self.nreg, ntr=ntr, ip=self.masks["ip"],
                    iu=self.masks["iu"], iv=self.masks["iv"], scp2=self.scp2_np, scp2i=self.scp2i_np)

    def context(self, kdm):
        return hycadv.Context.from_masks(self.masks, self.scp2_np, self.scp2i_np, kdm=kdm, nreg=self.nreg, nbdy=NB)

    def halo(self, a, w):
        """The halo fill, w wide, in place: zero across a closed edge, a copy across a periodic one."""
        o, nx, ny = NB, self.nx, self.ny
        a[..., o - w:o, o:o + nx] = 0.0
        a[..., o + ny:o + ny + w, o:o + nx] = 0.0
        rows = slice(o - w, o + ny + w)
        for k in range(1, w + 1):
            a[..., rows, o - k] = a[..., rows, o + nx - k] if self.periodic else 0.0
            a[..., rows, o + nx - 1 + k] = a[..., rows, o - 1 + k] if self.periodic else 0.0
        return a


# the neighbour to the west, east, south, north (the outermost ring is never used)
def _w(a):
    return a.roll(1, -1)


def _e(a):
    return a.roll(-1, -1)


def _s(a):
    return a.roll(1, -2)


def _n(a):
    return a.roll(-1, -2)


# ----------------------------------------------------------------------
# inputs: sums of separable terms, evaluated as batched products on the GPU
# ----------------------------------------------------------------------


def _coords(g):
    i, j = torch.arange(1 - NB, g.nx + NB + 1, dtype=F64), torch.arange(1 - NB, g.ny + NB + 1, dtype=F64)
    if g.periodic:
        i = torch.remainder(i - 1, g.nx) + 1
    return i.to(DEV), j.to(DEV)


def _waves(g, rng, n, terms, kmax, out=None, amp=1.0, eddies=0):
    """(n, ld2, ld1): smooth fields within +-amp; `eddies` of their terms are Gaussian eddies of 3-20 cells."""
    i, j = _coords(g)
    t = terms + eddies
    kx = rng.integers(1, kmax + 1, (n, t)) if g.periodic else rng.uniform(0.5, kmax, (n, t))
    par = [rng.uniform(0.5, kmax, (n, t)), rng.uniform(0, 2 * np.pi, (n, t)), rng.uniform(0, 2 * np.pi, (n, t)),
           rng.uniform(1, g.nx, (n, t)), rng.uniform(1, g.ny, (n, t)), rng.uniform(3, 20, (n, t)),
           rng.uniform(0.5, 1.0, (n, t)) * rng.choice([-1.0, 1.0], (n, t))]
    kx, ky, px, py, ci, cj, rad, s = (torch.from_numpy(np.asarray(v, dtype=np.float64)).to(DEV)[..., None]
                                      for v in [kx] + par)
    X = torch.sin(2 * math.pi * kx * (i - 0.5) / g.nx + px)
    Y = torch.sin(2 * math.pi * ky * (j - 0.5) / g.ny + py)
    if eddies:
        d = i - ci[:, terms:]
        if g.periodic:
            d = torch.remainder(d + g.nx / 2, g.nx) - g.nx / 2
        X[:, terms:] = torch.exp(-(d / rad[:, terms:]) ** 2)
        Y[:, terms:] = torch.exp(-((j - cj[:, terms:]) / rad[:, terms:]) ** 2)
    Y = Y * s
    Y[:, :terms] *= amp / max(terms, 1)
    Y[:, terms:] *= amp
    return torch.matmul(Y.transpose(1, 2), X, out=out)


def _flow(g, kdm, rng, courant, dt):
    """dp (2, kdm, ld2, ld1), uflx, vflx (kdm, ld2, ld1): level 2 (index 1) is the new thickness."""
    dp = torch.empty((2, kdm, g.ld2, g.ld1), dtype=F64, device=DEV)
    _waves(g, rng, kdm, 3, 3, out=dp[1], amp=1.0)
    dp[1].mul_(245.0 * ONEM).add_(255.0 * ONEM).clamp_(10.0 * ONEM, 500.0 * ONEM)
    dp[1].mul_((4000.0 * ONEM / dp[1].sum(0)).clamp_(max=1.0))
    _waves(g, rng, kdm, 2, 4, out=dp[0], amp=0.02)
    dp[0].add_(1.0).mul_(dp[1])
    g.halo(dp, NB)
    dp.clamp_(min=ONEM)
    uflx, vflx = torch.empty_like(dp[0]), torch.empty_like(dp[0])
    per = max(1, (1 << 26) // (g.ld1 * g.ld2))
    vel = courant * g.dx / dt
    for k0 in range(0, kdm, per):
        k = slice(k0, min(kdm, k0 + per))
        n = k.stop - k0
        psi, chi = _waves(g, rng, n, 8, 8), _waves(g, rng, n, 4, 6)
        u, v = psi - _n(psi), _e(psi) - psi
        m = torch.maximum(u[:, 2:-2, 2:-2].abs().amax((1, 2)), v[:, 2:-2, 2:-2].abs().amax((1, 2)))[:, None, None]
        u /= m
        v /= m
        ud, vd = chi - _w(chi), chi - _s(chi)
        m = torch.maximum(ud[:, 2:-2, 2:-2].abs().amax((1, 2)), vd[:, 2:-2, 2:-2].abs().amax((1, 2)))[:, None, None]
        u += 0.05 * ud / m
        v += 0.05 * vd / m
        m = (u[:, 2:-2, 2:-2].abs().amax((1, 2)) + v[:, 2:-2, 2:-2].abs().amax((1, 2)))[:, None, None]
        d = dp[1, k]
        uflx[k] = torch.where(g.iu, u / m * vel * (0.5 * g.dx) * (d + _w(d)), 0.0)
        vflx[k] = torch.where(g.iv, v / m * vel * (0.5 * g.dx) * (d + _s(d)), 0.0)
    return dp, uflx, vflx


def _tracer(g, kdm, rng, kind, out):
    """out (2, kdm, ld2, ld1): index 0 at time t, index 1 at t-1."""
    base = torch.linspace(0.0, 1.0, kdm, dtype=F64, device=DEV)[:, None, None]
    if kind == 0:  # temperature
        _waves(g, rng, kdm, 3, 4, out=out[0], amp=1.5, eddies=8)
        out[0].add_(27.0 - 25.0 * base).clamp_(-2.0, 30.0)
    elif kind == 1:  # salinity
        _waves(g, rng, kdm, 3, 4, out=out[0], amp=0.5, eddies=8)
        out[0].add_(34.0 + base).clamp_(30.0, 38.0)
    else:  # passive: log-uniform patches with sharp fronts
        i, j = _coords(g)
        bx, by = rng.integers(5, 60, 2)  # quarter patches along each direction
        ex, ey = (torch.from_numpy(10.0 ** rng.uniform(-3, 1, (kdm, 64))).to(DEV) for _ in range(2))
        X = ex[:, (i * float(bx) / (4 * g.nx)).long().remainder(64)]
        Y = ey[:, (j * float(by) / (4 * g.ny)).long().remainder(64)]
        torch.mul(Y[:, :, None], X[:, None, :], out=out[0])
    _waves(g, rng, kdm, 2, 5, out=out[1], amp=(0.01, 0.002, 0.01)[min(kind, 2)])
    out[0].mul_(g.ip)  # land carries zeros
    out[1].add_(1.0).mul_(out[0])
    return out


def _pair(g, kdm):
    return torch.empty((2, kdm, g.ld2, g.ld1), dtype=F64, device=DEV)


def _inputs(case, seed):
    """The model arrays of a case (one basin), as a dict of CUDA tensors, and its grid."""
    g = _Grid(case["nx"], case["ny"], case["periodic"])
    kdm = case.get("kdm", 1)
    rng = np.random.default_rng([seed, 77])
    f = {}
    f["dp"], f["uflx"], f["vflx"] = _flow(g, kdm, rng, case["courant"], case["dt"])
    if case["kind"] == "cnuity":
        return g, _cnuity_inputs(g, kdm, f)
    f["temp"] = _tracer(g, kdm, rng, 0, _pair(g, kdm))
    if case["kind"] != "advem":
        f["saln"] = _tracer(g, kdm, rng, 1, _pair(g, kdm))
    if case.get("ntr"):
        f["tracer"] = torch.empty((case["ntr"], 2, kdm, g.ld2, g.ld1), dtype=F64, device=DEV)
        for q in range(case["ntr"]):
            _tracer(g, kdm, rng, 2, f["tracer"][q])
    if case.get("btrmas"):
        f["oneta"] = g.halo(_waves(g, rng, 2, 3, 4, amp=0.02), NB).add_(1.0)
    if case["kind"] == "step":
        f["pbot"] = f["dp"][1].sum(0)
        f["pbavg"] = _waves(g, rng, 3, 3, 4, amp=0.02) * f["pbot"]
        f["oneta"] = torch.ones((2, g.ld2, g.ld1), dtype=F64, device=DEV)
        f["onetao"] = torch.ones_like(f["oneta"])
        f["th3d"] = _sig(f["temp"], f["saln"]) - THBASE
        f["dpo"] = f["dp"].clone()
        f["dpo"][1].mul_(1.01)
        for k in ("temp", "saln", "th3d"):
            f["o" + k] = torch.zeros_like(f["dp"][0])
        if case.get("ntr"):
            f["otracer"] = torch.zeros_like(f["tracer"][:, 0])
    return g, f


def _cnuity_inputs(g, kdm, f):
    dp = f["dp"]
    dp *= g.ip
    f["dpu"], f["dpv"] = 0.5 * (dp + _w(dp)) * g.iu, 0.5 * (dp + _s(dp)) * g.iv
    f["u"], f["v"] = torch.empty_like(dp), torch.empty_like(dp)
    f["u"][:] = torch.where(g.iu, f["uflx"] / (f["dpu"][1].clamp(min=1.0) * g.dx), 0.0)
    f["v"][:] = torch.where(g.iv, f["vflx"] / (f["dpv"][1].clamp(min=1.0) * g.dx), 0.0)
    f["ubavg"] = torch.zeros((3, g.ld2, g.ld1), dtype=F64, device=DEV)
    f["vbavg"] = torch.zeros_like(f["ubavg"])
    f["ubavg"][:] = 0.1 * f["u"][0, 0]
    f["vbavg"][:] = 0.1 * f["v"][0, 0]
    f["pbot"] = dp[0].sum(0)
    f["p"] = torch.zeros((kdm + 1, g.ld2, g.ld1), dtype=F64, device=DEV)
    f["p"][1:] = torch.cumsum(dp[0], 0)
    f["dpo"] = torch.zeros_like(dp)
    f["uflx"].zero_()
    f["vflx"].zero_()
    f["depthu"], f["depthv"] = torch.minimum(f["pbot"], _w(f["pbot"])), torch.minimum(f["pbot"], _s(f["pbot"]))
    f["thkd"] = (0.01 * g.dx ** 3 * torch.ones_like(g.scp2)).contiguous()
    return f


def _ens_sizes(case):
    """(nx, ny, kdm, ntr) of each basin: the first at the case's size, the rest uneven below it."""
    rng = np.random.default_rng([case["nx"], case["ny"], case["basins"], case["ntr"]])
    out = [(case["nx"], case["ny"], case["kdm"], case["ntr"])]
    for _ in range(1, case["basins"]):
        out.append((int(rng.integers(min(120, case["nx"]), case["nx"] + 1)),
                    int(rng.integers(min(90, case["ny"]), case["ny"] + 1)),
                    int(rng.integers((case["kdm"] + 1) // 2, case["kdm"] + 1)),
                    int(rng.integers(2, max(2, case["ntr"]) + 1)) if case["ntr"] < 10 else case["ntr"]))
    return out


def _ens_basin(case, seed, i):
    """(grid, dp, uflx, vflx, tracer generator) of basin i of an ensemble case."""
    nx, ny, kdm, ntr = _ens_sizes(case)[i]
    g = _Grid(nx, ny, case["periodic"], salt=i)
    dp, uflx, vflx = _flow(g, kdm, np.random.default_rng([seed, 88, i]), case["courant"], case["dt"])
    buf = _pair(g, kdm)

    def tracer(q):
        return _tracer(g, kdm, np.random.default_rng([seed, 99, i, q]), q, buf)

    return g, kdm, ntr, dp, uflx, vflx, tracer


def _diff_grid(g):
    one = torch.ones_like(g.scp2)
    d = (g.dx * one).contiguous()
    return dict(aspux=one, aspvy=one, scuy=d, scvx=d)


# ----------------------------------------------------------------------
# prepare and run
# ----------------------------------------------------------------------


def prepare(case, seed):
    if case["kind"] == "ens":
        return _prepare_ens(case, seed)
    g, f = _inputs(case, seed)
    kdm = case.get("kdm", 1)
    state = {"case": case, "f": f, "step": 0, "ctx": g.context(kdm), "g": g}
    ctx = state["ctx"]
    if case["kind"] == "advem":
        fco, fcn = _thickness(g, f["dp"][1, 0], f["uflx"][0], f["vflx"][0], case["dt"])
        fld, fldc = g.halo(f["temp"][1, 0].clone(), 5), g.halo(f["temp"][0, 0].clone(), 5)
        state["args"] = (fld, fldc, g.halo(f["uflx"][0].clone(), 5), g.halo(f["vflx"][0].clone(), 5), fco, fcn,
                         256.0 if case["scheme"] == 1 else 0.0, g.scp2, g.scp2i, case["dt"])
        return state
    for k, a in f.items():
        if k in hycadv.FIELDS:
            ctx.bind(k, a)
    if case["kind"] == "step":
        ctx.set_diffusion_grid(**{k: a.cpu().numpy() for k, a in _diff_grid(g).items()})
    if case["kind"] == "cnuity":
        d = np.ascontiguousarray(np.broadcast_to(g.dx_np[:, None], g.scp2_np.shape))
        th = f["thkd"].cpu().numpy() if case["thkdf"] else None
        ctx.set_cnuity_grid(d, d, f["depthu"].cpu().numpy(), f["depthv"].cpu().numpy(), th, th)
    return state


def _prepare_ens(case, seed):
    sizes = _ens_sizes(case)
    grids = [_Grid(nx, ny, case["periodic"], salt=i) for i, (nx, ny, _, _) in enumerate(sizes)]
    ens = hycadv.Ensemble([g.spec(s[2], s[3]) for g, s in zip(grids, sizes)], precision=case["precision"])
    outs = []
    for i in range(len(sizes)):
        g, kdm, ntr, dp, uflx, vflx, tracer = _ens_basin(case, seed, i)
        ens.put(i, "dp", dp[1])
        ens.put(i, "uflx", uflx)
        ens.put(i, "vflx", vflx)
        for q in range(ntr):
            t = tracer(q)
            ens.put(i, "cur", t[0], q * kdm, kdm)
            ens.put(i, "old", t[1], q * kdm, kdm)
            if case["scheme"] == 1 and q == 0:
                ens.set_posdef(i, 0, 256.0)
        if case["diffusion"]:
            ens.set_diffusion(i, TEMDF2, **_diff_grid(g))
        del dp, uflx, vflx, tracer
        outs.append(torch.empty((ntr, kdm, g.ld2, g.ld1), dtype=F64, device=DEV))
    ens.tune(case["scheme"], case["dt"])
    return {"case": case, "ens": ens, "outs": outs}


def run(state):
    case = state["case"]
    kind, dt = case["kind"], case["dt"]
    if kind == "ens":
        ens = state["ens"]
        ens.step(case["scheme"], dt, nsteps=case["steps"], graph=True)
        for i, o in enumerate(state["outs"]):
            ens.get(i, "cur", o)
        return state["outs"]
    ctx, f = state["ctx"], state["f"]
    if kind == "advem":
        ctx.advem(case["scheme"], *state["args"])
        return state["args"][0]
    state["step"] += 1
    s = state["step"]
    m, n = (s + 1) % 2 + 1, s % 2 + 1  # the leapfrog levels of the s-th step
    if kind == "cnuity":
        ctx.cnuity(m, n, delt1=dt, nstep=s, thkdf=case["thkdf"], ra2fac=RA2FAC)
        return [f[k] for k in ("dp", "dpo", "uflx", "vflx", "p")]
    ntr = case["ntr"]
    flags = np.zeros(max(ntr, 1), np.int32)
    if kind == "tsadvc":
        ctx.tsadvc(m, n, delt1=dt, advtyp=case["scheme"], btrmas=case["btrmas"], ntracr=ntr, trcflg=flags, nstep=s)
        return [f["temp"][n - 1], f["saln"][n - 1]] + ([f["tracer"]] if ntr else [])
    ctx.asselin_save(m, n, oneta0=ONETA0, ntracr=ntr)
    ctx.tsadvc(m, n, delt1=dt, advtyp=case["scheme"], ntracr=ntr, trcflg=flags, nstep=s)
    ctx.tsdff(m, n, delt1=dt, temdf2=TEMDF2, thbase=THBASE, ntracr=ntr)
    ctx.asselin_filter(m, n, ra2fac=RA2FAC, oneta0=ONETA0, thbase=THBASE, ntracr=ntr)
    return [f[k] for k in ("temp", "saln", "th3d", "dp")] + ([f["tracer"]] if ntr else [])


def work(case):
    """Bytes: each input read once, each output written once.  Flops: the schemes' additions, products and
    divisions per cell, layer and field, and the thickness prep per cell and layer."""
    per = {0: 20.0, 1: 75.0, 2: 65.0, 4: 75.0}
    if case["kind"] == "ens":
        b = fl = 0.0
        st, sf = (4, 4) if case["precision"] == "mixed" else (8, 8)
        lev = 3 if case["scheme"] in (2, 4) else 2
        for nx, ny, kdm, ntr in _ens_sizes(case):
            n = float(nx * ny)
            b += case["steps"] * (n * kdm * (lev * st * ntr + 2 * sf + 8) + 19 * n) + n * kdm * ntr * (st + 8)
            fl += case["steps"] * n * kdm * (ntr * (per[case["scheme"]] + (15 if case["diffusion"] else 0)) + 12)
        return {"bytes": b, "flops": fl}
    n = float(case["nx"] * case["ny"])
    if case["kind"] == "advem":
        lev = 3 if case["scheme"] in (2, 4) else 2
        return {"bytes": n * (8 * (lev + 4 + 2) + 3), "flops": n * (per[case["scheme"]] + 4)}
    nk, nf = n * case["kdm"], _fields(case)
    if case["kind"] == "cnuity":  # dp(n), dp(m), u, v, dpu, dpv in; dp(n), dp(m), dpo(n), dpo(m), uflx, vflx, p out
        return {"bytes": nk * 13 * 8 + 19 * n, "flops": nk * (100 if case["thkdf"] else 75)}
    lev = 3 if case["scheme"] in (2, 4) else 2
    adv = nk * 8 * (lev * nf + 3) + 19 * n
    fl = nk * (nf * per[case["scheme"]] * (1.3 if case.get("btrmas") else 1) + 12)
    if case["kind"] == "tsadvc":
        return {"bytes": adv, "flops": fl}
    # the step: save (fields and th3d copied), diffusion (fields in and out, dp in, th3d out), filter (three
    # levels of every field in, one out, dp and dpo in, dp and th3d out)
    return {"bytes": adv + nk * 8 * (2 * (nf + 1) + (2 * nf + 2) + (4 * nf + 6)), "flops": fl + nk * (28 * nf + 130)}


# ----------------------------------------------------------------------
# exact: the same passes restated in 64-bit torch
# ----------------------------------------------------------------------


def _thickness(g, dp, u, v, dt, om=1.0):
    o = om * dp
    div = ((_e(u) - u) + (_n(v) - v)) * dt * g.scp2i
    return (o + div).clamp_(min=0.0), o.clamp(min=0.0)


def _five(g, a, op):
    """op over a cell and its sea neighbours."""
    r = a
    for nb in (_w, _e, _s, _n):
        r = op(r, torch.where(nb(g.ip), nb(a), a))
    return r


def _div(g, x, y, dt):
    return ((_e(x) - x) + (_n(y) - y)) * dt * g.scp2i


def _advect(g, scheme, f, c, u, v, fco, fcn, dt, posdef):
    """The new level of one field, a slice or a stack of slices (land and halo as in f)."""
    zero = torch.zeros((), dtype=F64, device=DEV)
    up = lambda a, nb, vel: torch.where(vel >= 0, nb(a), a)  # noqa: E731
    hn = fcn + ONEMU
    pd = posdef if scheme == 1 else 0.0
    fx = torch.where(g.iu, u * (up(f, _w, u) + pd), zero)
    fy = torch.where(g.iv, v * (up(f, _s, v) + pd), zero)
    fmx, fmn = _five(g, f, torch.maximum) + pd, _five(g, f, torch.minimum) + pd
    fd = _div(g, fx, fy, dt)
    lo = torch.maximum(fmn, torch.minimum(fmx, ((f + pd) * (fco + ONEMU) - fd) / hn))
    if scheme == 0:
        return torch.where(g.sea, lo, f)
    pos, neg = (lambda a: a.clamp(min=0.0)), (lambda a: a.clamp(max=0.0))
    if scheme == 1:
        h = fco + fcn
        ax = torch.where(g.iu, 0.5 * u.abs() * (f - _w(f)) - u * (fd + _w(fd)) / ((h + _w(h)) + ONEMU), zero)
        ay = torch.where(g.iv, 0.5 * v.abs() * (f - _s(f)) - v * (fd + _s(fd)) / ((h + _s(h)) + ONEMU), zero)
        fe, fn = _e(ax), _n(ay)
        rp = (fmx - lo) * (fcn * g.scp2) / ((ONEMU - ((neg(fe) - pos(ax)) + (neg(fn) - pos(ay)))) * dt)
        rm = (lo - fmn) * (fcn * g.scp2) / ((ONEMU + ((pos(fe) - neg(ax)) + (pos(fn) - neg(ay)))) * dt)
        rp, rm = rp.clamp(max=1.0), rm.clamp(max=1.0)
        lx = pos(ax) * torch.minimum(rp, _w(rm)) + neg(ax) * torch.minimum(_w(rp), rm)
        ly = pos(ay) * torch.minimum(rp, _s(rm)) + neg(ay) * torch.minimum(_s(rp), rm)
        lx, ly = torch.where(g.iu, lx, zero), torch.where(g.iv, ly, zero)
        r = torch.maximum(fmn, torch.minimum(fmx, lo - _div(g, lx, ly, dt) / hn)) - pd
        return torch.where(g.sea, r, f)
    hx, hy = u * 0.5 * (c + _w(c)), v * 0.5 * (c + _s(c))
    if scheme == 4:
        a, b = 7.0 / 12.0, -1.0 / 12.0
        hx = torch.where(_w(g.iu) & _e(g.iu), u * (a * (c + _w(c)) + b * (_e(c) + _w(_w(c)))), hx)
        hy = torch.where(_s(g.iv) & _n(g.iv), v * (a * (c + _s(c)) + b * (_n(c) + _s(_s(c)))), hy)
    ax, ay = torch.where(g.iu, hx - fx, zero), torch.where(g.iv, hy - fy, zero)
    mx, mn = torch.maximum(torch.maximum(f, c), lo), torch.minimum(torch.minimum(f, c), lo)
    qx, qn = _five(g, mx, torch.maximum), _five(g, mn, torch.minimum)
    rp, rm = _ratios(g, ax, ay, torch.where(_e(g.ip), _e(ax), ax), torch.where(_n(g.ip), _n(ay), ay),
                     (qx - lo) * fcn * g.scp2 * (1.0 / dt), (lo - qn) * fcn * g.scp2 * (1.0 / dt), 0.0)
    lx, ly = _limit(ax, ay, rp, rm)
    r = torch.maximum(qn, torch.minimum(qx, lo - _div(g, lx, ly, dt) / hn))
    return torch.where(g.sea, r, f)


def _ratios(g, ax, ay, axe, ayn, qp, qm, eps):
    pos, neg = (lambda a: a.clamp(min=0.0)), (lambda a: a.clamp(max=0.0))
    amax = pos(ax) - neg(axe) + pos(ay) - neg(ayn)
    amin = pos(axe) - neg(ax) + pos(ayn) - neg(ay)
    rp = torch.where(amax > eps, torch.where(qp < amax, qp / amax, 1.0), 0.0)
    rm = torch.where(amin > eps, torch.where(qm < amin, qm / amin, 1.0), 0.0)
    return torch.where(g.ip, rp, 0.0), torch.where(g.ip, rm, 0.0)


def _limit(ax, ay, rp, rm):
    return (ax * torch.where(ax < 0, torch.minimum(_w(rp), rm), torch.minimum(rp, _w(rm))),
            ay * torch.where(ay < 0, torch.minimum(_s(rp), rm), torch.minimum(rp, _s(rm))))


def _fct2c(g, f, c, u, v, fco, dt):
    """advem_fct2c: five donor-cell passes with a local time step, then the Zalesak limiter."""
    eps = 1.0e-10
    z = lambda: torch.zeros_like(f)  # noqa: E731
    h, lo, ucum, vcum, fxc, fyc, live = fco.clone(), f.clone(), z(), z(), z(), z(), torch.ones_like(f, dtype=torch.bool)
    q = _e(u).clamp(min=0) - u.clamp(max=0) + _n(v).clamp(min=0) - v.clamp(max=0)
    for _ in range(5):
        dl = torch.where(q > 0, (h / (q * g.scp2i)).clamp(max=dt), dt)
        left = dt - ucum
        du = torch.where(g.iu & (ucum != dt), torch.minimum(left, torch.where(u >= 0, _w(dl), dl)), 0.0)
        left = dt - vcum
        dv = torch.where(g.iv & (vcum != dt), torch.minimum(left, torch.where(v >= 0, _s(dl), dl)), 0.0)
        ul, vl = du * u, dv * v
        fx, fy = torch.where(u >= 0, _w(lo), lo) * ul, torch.where(v >= 0, _s(lo), lo) * vl
        ucum, vcum, fxc, fyc = ucum + du, vcum + dv, fxc + fx, fyc + fy
        qp = h - (_e(ul) - ul + _n(vl) - vl) * g.scp2i
        on = live & g.ip
        lo2 = ((eps + h) * lo - (_e(fx) - fx + _n(fy) - fy) * g.scp2i) / (eps + qp)
        lo = torch.where(on & (qp > 0), lo2, lo)
        h = torch.where(on, qp, h)
        live = torch.where(on, (_e(ucum) != dt) | (ucum != dt) | (_n(vcum) != dt) | (vcum != dt), live)
        g.halo(h, 5)
        g.halo(lo, 5)
    ax = torch.where(g.iu, u * 0.5 * (c + _w(c)) - fxc / dt, 0.0)
    ay = torch.where(g.iv, v * 0.5 * (c + _s(c)) - fyc / dt, 0.0)
    qx, qn = _five(g, lo, torch.maximum), _five(g, lo, torch.minimum)
    rp, rm = _ratios(g, ax, ay, _e(ax), _n(ay), (qx - lo) * h * g.scp2 * (1.0 / dt), (lo - qn) * h * g.scp2 * (1.0 / dt), eps)
    lx, ly = _limit(ax, ay, rp, rm)
    r = torch.where(h > 0, ((eps + h) * lo - _div(g, lx, ly, dt)) / (eps + h), lo)
    return torch.where(g.sea, r, f)


def _chunks(g, kdm):
    per = max(1, (1 << 24) // (g.ld1 * g.ld2))
    return [slice(k, min(kdm, k + per)) for k in range(0, kdm, per)]


def _sig(t, s):
    """The 17-term equation of state, sigma at 2000 dbar."""
    p = 2000.0
    c = [9.9984085444849347e+02, 7.3471625860981584e+00, -5.3211231792841769e-02, 3.6492439109814549e-04,
         2.5880571023991390e+00, 6.7168282786692355e-03, 1.9203202055760151e-03, 1.0, 7.2815210113327091e-03,
         -4.4787265461983921e-05, 3.3851002965802430e-07, 1.3651202389758572e-10, 1.7632126669040377e-03,
         8.8066583251206474e-06, 1.8832689434804897e-10, 5.7463776745432097e-06, 1.4716275472242334e-09,
         1.1798263740430364e-02, 9.8920219266399117e-08, 4.6996642771754730e-06, 2.5862187075154352e-08,
         3.2921414007960662e-12, 6.7103246285651894e-06, 2.4461698007024582e-17, 9.1534417604289062e-18]
    num = (c[0] + (c[17] - c[20] * p) * p) + t * (c[1] + t * ((c[2] + (c[18] - c[21] * p) * p) + t * c[3])) + s * (
        (c[4] + c[19] * p) - t * c[5] + s * c[6])
    den = (c[7] + c[22] * p) + t * ((c[8] - c[24] * p ** 3) + t * (c[9] + t * ((c[10] - c[23] * p ** 2) + t * c[11])))
    den = den + s * (c[12] - t * (c[13] + t * t * c[14]) + torch.sqrt(s.clamp(min=0)) * (c[15] + t * t * c[16]))
    return num / den - 1000.0


def _diffuse(g, flds, h, dt):
    """tsdff of a stack of slices of each field, in place (sea points of the interior)."""
    d = _diff_grid(g)
    h0 = h.clamp(min=0.0)
    har = lambda a, b: 2.0 * a * b / (a + b).clamp(min=2.0e-20)  # noqa: E731
    fu = torch.where(g.iu, TEMDF2 * d["aspux"] * d["scuy"] * har(_w(h0), h0), 0.0)
    fv = torch.where(g.iv, TEMDF2 * d["aspvy"] * d["scvx"] * har(_s(h0), h0), 0.0)
    fac = -dt / (g.scp2 * h.clamp(min=1.0e-20))
    for f in flds:
        x, y = fu * (_w(f) - f), fv * (_s(f) - f)
        f.copy_(torch.where(g.sea, f + ((_e(x) - x) + (_n(y) - y)) * fac, f))


def exact(case, seed):
    kind = case["kind"]
    if kind == "ens":
        return [_exact_basin(case, seed, i) for i in range(case["basins"])]
    g, f = _inputs(case, seed)
    if kind == "cnuity":
        return _exact_cnuity(g, f, case)
    scheme, dt = case["scheme"], case["dt"]
    w = 2 if scheme == 0 else 5
    if kind == "advem":
        fco, fcn = _thickness(g, f["dp"][1, 0], f["uflx"][0], f["vflx"][0], dt)
        fld, fldc, u, v = (g.halo(a, 5) for a in (f["temp"][1, 0], f["temp"][0, 0], f["uflx"][0], f["vflx"][0]))
        return _advect(g, scheme, fld, fldc, u, v, fco, fcn, dt, 256.0)
    if kind == "step":
        _exact_save(g, f)
    for k in ("temp", "saln", "uflx", "vflx", "tracer"):
        if k in f:
            g.halo(f[k], w)
    flds = [(f["temp"], 256.0), (f["saln"], 0.0)] + [(f["tracer"][q], 0.0) for q in range(case["ntr"])]
    om = f["oneta"][1] if case.get("btrmas") else 1.0
    for k in _chunks(g, case["kdm"]):
        u, v = f["uflx"][k], f["vflx"][k]
        fco, fcn = _thickness(g, f["dp"][1, k], u, v, dt, om)
        for a, posdef in flds:
            a[1, k] = (_fct2c(g, a[1, k], a[0, k], u, v, fco, dt) if case.get("btrmas") else
                       _advect(g, scheme, a[1, k], a[0, k], u, v, fco, fcn, dt, posdef))
    if kind == "tsadvc":
        return [f["temp"][1], f["saln"][1]] + ([f["tracer"]] if case["ntr"] else [])
    g.halo(f["th3d"], w)
    for k in ("temp", "saln", "th3d", "tracer"):
        if k in f:
            g.halo(f[k][..., 1, :, :, :], 2)
    for k in _chunks(g, case["kdm"]):
        _diffuse(g, [a[1, k] for a, _ in flds], f["dp"][1, k] * f["oneta"][1], dt)
        f["th3d"][1, k] = torch.where(g.sea, _sig(f["temp"][1, k], f["saln"][1, k]) - THBASE, f["th3d"][1, k])
    _exact_filter(g, f, case)
    return [f[k] for k in ("temp", "saln", "th3d", "dp")] + ([f["tracer"]] if case["ntr"] else [])


def _exact_save(g, f):
    new = (1.0 + f["pbavg"][:2] / f["pbot"]).clamp(min=ONETA0)
    for k in ("oneta", "onetao"):
        f[k] = g.halo(torch.where(g.sea, new, f[k]), 6)
    for k in ("temp", "saln", "th3d"):
        f["o" + k][:, NB:-NB, NB:-NB] = f[k][1][:, NB:-NB, NB:-NB]
    if "tracer" in f:
        f["otracer"][..., NB:-NB, NB:-NB] = f["tracer"][:, 1, :, NB:-NB, NB:-NB]


def _exact_filter(g, f, case):
    on, om = f["oneta"][1], f["oneta"][0]
    for k in _chunks(g, case["kdm"]):
        old, mid, new = f["dpo"][1, k] * f["onetao"][1], f["dpo"][0, k] * f["onetao"][0], f["dp"][1, k] * on
        h = mid + 0.5 * RA2FAC * (old + new - 2.0 * mid)
        f["dp"][0, k] = torch.where(g.sea, h / om, f["dp"][0, k])
        live = g.sea & (h > 9806.0e-20)

        def filt(a, o):
            lo = torch.minimum(torch.minimum(o, a[0, k]), a[1, k])
            so, sm, sn = old * (o - lo), mid * (a[0, k] - lo), new * (a[1, k] - lo)
            a[0, k] = torch.where(live, lo + (sm + 0.5 * RA2FAC * (so + sn - 2.0 * sm)) / h, a[0, k])

        for n in ("saln", "temp"):
            filt(f[n], f["o" + n][k])
        f["th3d"][0, k] = torch.where(live, _sig(f["temp"][0, k], f["saln"][0, k]) - THBASE, f["th3d"][0, k])
        for q in range(case["ntr"]):
            filt(f["tracer"][q], f["otracer"][q, k])


def _exact_basin(case, seed, i):
    g, kdm, ntr, dp, u, v, tracer = _ens_basin(case, seed, i)
    g.halo(u, 5)
    g.halo(v, 5)
    out = torch.empty((ntr, kdm, g.ld2, g.ld1), dtype=F64, device=DEV)
    for q in range(ntr):
        t = tracer(q)
        cur, old = g.halo(t[0], 5), g.halo(t[1], 5)
        new = cur.clone()
        for _ in range(case["steps"]):
            for k in _chunks(g, kdm):
                fco, fcn = _thickness(g, dp[1, k], u[k], v[k], case["dt"])
                r = _advect(g, case["scheme"], old[k], cur[k], u[k], v[k], fco, fcn, case["dt"], 256.0 if q == 0 else 0.0)
                if case["diffusion"]:
                    g.halo(r, 5)
                    _diffuse(g, [r], dp[1, k], case["dt"])
                new[k] = torch.where(g.sea, r, new[k])
                if g.periodic:  # the wrap of the sea cells, five wide
                    for d in range(5):
                        for to, at in ((NB - 1 - d, NB + g.nx - 1 - d), (NB + g.nx + d, NB + d)):
                            new[k, :, to] = torch.where(g.sea[:, at], new[k, :, at], new[k, :, to])
            old, cur, new = cur, new, old
        out[q] = cur
    return out


def _exact_cnuity(g, f, case):
    dt, kdm, mm, nn = case["dt"], case["kdm"], 0, 1
    dp, dpo, p, uflx, vflx = (f[k] for k in ("dp", "dpo", "p", "uflx", "vflx"))
    eps = 1.0e-11
    box = []
    for m in range(7):
        b = torch.zeros_like(g.ip)
        b[NB - m:NB + g.ny + m, NB - m:NB + g.nx + m] = True
        box.append(b)

    def put(dst, m, mask, val):
        dst.copy_(torch.where(box[m] & mask, val, dst))

    pos, neg = (lambda a: a.clamp(min=0.0)), (lambda a: a.clamp(max=0.0))
    g.halo(dp, 6)
    for k in ("dpu", "dpv", "u", "v", "ubavg", "vbavg"):
        g.halo(f[k][mm], 6)
    dpo[nn] = dp[nn]
    z = lambda: torch.zeros_like(g.scp2)  # noqa: E731
    uf, vf, u2, v2, utn, vtn, t1, t2, depth = (z() for _ in range(9))
    for k in range(kdm):
        d = dp[nn, k]
        for fl, f2, out, vel, bar, th, lim, mask, nb in (
                (uf, u2, uflx[k], f["u"][mm, k], f["ubavg"][mm], f["dpu"][mm, k], f["depthu"], g.iu, _w),
                (vf, v2, vflx[k], f["v"][mm, k], f["vbavg"][mm], f["dpv"][mm, k], f["depthv"], g.iv, _s)):
            tot = (vel + bar) * g.dx
            q = torch.where(tot >= 0, torch.minimum(nb(d), pos(lim - nb(depth))), torch.minimum(d, pos(lim - depth)))
            put(fl, 5, mask, tot * q)
            put(f2, 5, mask, tot * th - fl)
            put(out, 5, mask, fl)
        put(depth, 4, g.ip, depth + d)
        put(d, 4, g.ip, d - _div(g, uf, vf, dt))
        put(dpo[mm, k], 4, g.ip, d)
        put(t1, 4, g.ip, (_five(g, d, torch.maximum) - d) / (
            ((pos(u2) - neg(_e(u2))) + (pos(v2) - neg(_n(v2))) + eps) * dt * g.scp2i))
        put(t2, 4, g.ip, (pos(_five(g, d, torch.minimum)) - d) / (
            ((neg(u2) - pos(_e(u2))) + (neg(v2) - pos(_n(v2))) - eps) * dt * g.scp2i))
        for fl, f2, tn, out, mask, nb in ((uf, u2, utn, uflx[k], g.iu, _w), (vf, v2, vtn, vflx[k], g.iv, _s)):
            clip = torch.where(f2 >= 0, torch.minimum(t1.clamp(max=1.0), nb(t2)), torch.minimum(t2.clamp(max=1.0), nb(t1)))
            put(tn, 3, mask, tn + f2 * (1.0 - clip))
            put(fl, 3, mask, f2 * clip)
            put(out, 3, mask, out + fl)
        put(d, 2, g.ip, d - _div(g, uf, vf, dt))
        put(p[k + 1], 2, g.ip, p[k] + d)
    bottom = p[kdm].clone()
    for k in range(kdm):
        d = dp[nn, k]
        q = d / bottom
        for fl, tn, out, mask, nb in ((uf, utn, uflx[k], g.iu, _w), (vf, vtn, vflx[k], g.iv, _s)):
            put(fl, 1, mask, tn * torch.where(tn >= 0, nb(q), q))
            put(out, 1, mask, out + fl)
        put(d, 0, g.ip, d - _div(g, uf, vf, dt))
        put(p[k + 1], 0, g.ip, p[k] + d)
    q = f["pbot"] / p[kdm]
    for k in range(kdm):
        put(dp[nn, k], 0, g.ip, dp[nn, k] * q)
        put(p[k + 1], 0, g.ip, p[k] + dp[nn, k])
    if case["thkdf"]:
        _exact_thkdf(g, f, case, box, put, uf, vf, t1, t2)
    g.halo(dp[nn], 6)
    mid = dp[mm].clone()
    new = mid + 0.5 * RA2FAC * (dpo[nn] + dp[nn] - 2.0 * mid)
    put(dpo[mm], 6, g.ip, mid)
    put(dp[mm], 6, g.ip, new)
    return [dp, dpo, uflx, vflx, p]


def _exact_thkdf(g, f, case, box, put, uf, vf, t1, t2):
    """Interface diffusion of the first step: biharmonic (upwards, nstep odd) or Laplacian (downwards)."""
    dt, kdm, nn = case["dt"], case["kdm"], 1
    dp, p, uflx, vflx, th = f["dp"], f["p"], f["uflx"], f["vflx"], dt * f["thkd"]
    bih, flip, onecm = case["thkdf"] == 4, True, 9.806 / (1.0 / 1000.0) * 0.01
    g.halo(dp[nn], 6)
    g.halo(p[1:], 6)
    uf.copy_(torch.where(g.iu, 0.0, uf))
    vf.copy_(torch.where(g.iv if bih else g.ip | g.iv, 0.0, vf))
    pold = torch.where(g.ip, p[kdm], 0.0)

    def side(a, nb, other):  # the neighbour if sea, else the opposite one if sea, else the point itself
        return torch.where(nb(g.ip), nb(a), torch.where(other(g.ip), other(a), a))

    for k in (range(kdm - 1, 0, -1) if bih else range(1, kdm)):
        pk, dk, dm = p[k], dp[nn, k], dp[nn, k - 1]
        if bih:
            thick = torch.minimum(dk, dm) >= onecm
            for t, a, b in ((t1, _w, _e), (t2, _s, _n)):
                c = pk - 0.5 * (side(pk, a, b) + side(pk, b, a))
                thin = torch.where(c > 0, torch.minimum(side(dk, a, b), side(dk, b, a)),
                                   torch.minimum(side(dm, a, b), side(dm, b, a))) < onecm
                put(t, 5, g.ip, torch.where(thick & ~thin, c, 0.0))
        G, H = 0.25 * (p[kdm] - pk) * g.scp2, 0.25 * (pold - pk) * g.scp2
        for fl, t, out, mask, nb in ((uf, t1, uflx, g.iu, _w), (vf, t2, vflx, g.iv, _s)):
            hi, lo = G, -nb(G)
            if bih and flip:
                hi, lo = torch.minimum(hi, fl + H), torch.maximum(lo, fl - nb(H))
            drive = (nb(t) - t) if bih else (nb(pk) - pk)
            put(fl, 4, mask, torch.minimum(hi, torch.maximum(lo, th * drive)))
            put(out[k - 1], 4, mask, out[k - 1] + fl * (1.0 / dt))
            put(out[k], 4, mask, out[k] - fl * (1.0 / dt))
        put(pold, 4, g.ip, pk)
        put(pk, 4, g.ip, pk - ((_e(uf) - uf) + (_n(vf) - vf)) * g.scp2i)
    for k in range(kdm):
        put(p[k + 1], 4, g.ip, torch.maximum(p[k + 1], p[k]))
        put(dp[nn, k], 4, g.ip, p[k + 1] - p[k])
