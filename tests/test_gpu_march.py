"""The strip kernels (csrc/hyc_march.cuh) against the oracle, bit for bit,
where its geometry ends: strips of 58 columns, short and ragged segments, odd
counts of fields, and tracers that leave the range of the integer
multiplication and division or the FP32 limiter test.  The layer counts put
every case above the size from which the launch goes to this kernel."""
import numpy as np
import pytest

from helpers import basin, np_case, oneta_field, oracle_grid, same
from test_gpu_parity import bind_all, compare, gpu_steps, make_ctx, oracle_steps, torchify

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,kdm,periodic", [(57, 41, 52, False), (58, 33, 56, True), (59, 20, 80, False),
                                                (117, 18, 40, True), (175, 45, 20, False)])
@pytest.mark.parametrize("advtyp,ntr", [(0, 0), (0, 1), (1, 0), (1, 3), (2, 0), (2, 1), (4, 3)])
def test_strip_edges(cuda, nx, ny, kdm, periodic, advtyp, ntr):
    b = basin(nx, ny, periodic, seed=nx)
    g = oracle_grid(b)
    c = np_case(b, g, kdm=kdm, ntracr=ntr, seed=nx, courant=0.8, delt1=240.0)
    c["delt1"] = 240.0
    t = torchify(c, cuda)
    ctx = make_ctx(b, g, kdm)
    bind_all(ctx, t)
    flg = np.zeros(ntr, np.int32) if ntr else None
    oracle_steps(g, c, (1, 2), advtyp, trcflg=flg)
    gpu_steps(ctx, t, (1, 2), advtyp, ntracr=ntr, trcflg=flg)
    compare(c, t)


@pytest.mark.parametrize("advtyp", [0, 1, 4])
def test_with_oneta(cuda, advtyp):
    b = basin(90, 70, True, seed=5)
    g = oracle_grid(b)
    c = np_case(b, g, kdm=24, ntracr=0, seed=5, courant=0.7, delt1=600.0)
    c["delt1"] = 600.0
    oneta = oneta_field(b, 5)
    t = torchify(dict(c, oneta=oneta), cuda)
    ctx = make_ctx(b, g, 24)
    bind_all(ctx, t, extra=("oneta",))
    oracle_steps(g, c, (1, 2), advtyp, btrmas=True, oneta=oneta)
    gpu_steps(ctx, t, (1, 2), advtyp, btrmas=True)
    compare(c, t)


@pytest.mark.parametrize("advtyp", [0, 1, 2])
@pytest.mark.parametrize("scale", [0.0, 1e-306, 1e-40, 1e30, 1e150])
def test_tracer_ranges(cuda, scale, advtyp):
    """Constant, tiny and huge tracers: what the limiter's FP32 test cannot
    decide and what the integer arithmetic hands to the FP64 pipe."""
    b = basin(100, 60, False, seed=9)
    g = oracle_grid(b)
    c = np_case(b, g, kdm=26, ntracr=2, seed=9, courant=0.8, delt1=240.0)
    c["delt1"] = 240.0
    c["tracer"] *= scale
    c["tracer"][1, :, :, 30:, :] = 0.0  # half of one tracer is exactly zero
    t = torchify(c, cuda)
    ctx = make_ctx(b, g, 26)
    bind_all(ctx, t)
    flg = np.zeros(2, np.int32)
    oracle_steps(g, c, (1, 2), advtyp, trcflg=flg)
    gpu_steps(ctx, t, (1, 2), advtyp, ntracr=2, trcflg=flg)
    compare(c, t)


@pytest.mark.parametrize("advtyp", [0, 1, 2, 4])
def test_one_field_slice(cuda, advtyp):
    """advem on one long slice: the one-field form."""
    b = basin(59, 9800, False, seed=11)
    g = oracle_grid(b)
    c = np_case(b, g, kdm=1, ntracr=0, seed=11, courant=0.7, delt1=600.0)
    fld, fldc, u, v = (c[k][l].copy() for k, l in (("temp", (1, 0)), ("temp", (0, 0)), ("uflx", 0), ("vflx", 0)))
    for a in (fld, fldc, u, v):
        g.xctilr(a, 5, 5)
    dpn = c["dp"][1, 0]
    fd = np.zeros_like(dpn)
    fd[:-1, :-1] = ((u[:-1, 1:] - u[:-1, :-1]) + (v[1:, :-1] - v[:-1, :-1])) * 600.0 * c["scp2i"][:-1, :-1]
    fco, fcn = np.maximum(dpn + fd, 0.0), np.maximum(dpn, 0.0)
    ref, got = fld.copy(), fld.copy()
    g.advem(advtyp, ref, fldc, u, v, fco, fcn, 0.0, c["scp2"], c["scp2i"], 600.0)
    make_ctx(b, g, 1).advem(advtyp, got, fldc, u, v, fco, fcn, 0.0, c["scp2"], c["scp2i"], 600.0)
    assert same(got, ref) and not np.array_equal(got, fld)


@pytest.mark.parametrize("advtyp", [0, 1, 2, 4])
@pytest.mark.parametrize("mode", ["hybrid", "isopycnic", "conserve"])
def test_field_lists(cuda, advtyp, mode):
    """Fields with layer ranges of their own: th3d above nhybrd, q2/q2l with a
    layer offset, the isopycnic layer 1; and the conserving rescale."""
    b = basin(83, 61, True, seed=131)
    g = oracle_grid(b)
    kdm = 28
    c = np_case(b, g, kdm=kdm, ntracr=2, seed=131, courant=0.7, delt1=600.0)
    c["delt1"] = 600.0
    kw = {"hybrid": dict(advflg=1, nhybrd=11, mxlmy=True), "isopycnic": dict(isopyc=True, nhybrd=0, mxlmy=True),
          "conserve": {}}[mode]
    q2 = {}
    if kw:
        rng = np.random.default_rng(131)
        q2 = dict(q2=0.01 + rng.random((2, kdm + 2, b.ld2, b.ld1)) * 0.1, q2l=0.1 + rng.random((2, kdm + 2, b.ld2, b.ld1)))
    c.update(q2)
    t = torchify(c, cuda)
    ctx = make_ctx(b, g, kdm)
    bind_all(ctx, t, extra=tuple(q2))
    flg = np.array([0, 2], np.int32)
    if mode == "conserve":
        ctx.set_conserve(True)
        g.set_conserve(True)
    oracle_steps(g, c, (1, 2), advtyp, trcflg=flg, **q2, **kw)
    gpu_steps(ctx, t, (1, 2), advtyp, ntracr=2, trcflg=flg, **kw)
    compare(c, t, keys=("temp", "saln", "th3d", "tracer") + tuple(q2))
