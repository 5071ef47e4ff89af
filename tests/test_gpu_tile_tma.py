"""The tile kernels staged by TMA against the oracle, bit for bit: launches
between one and two 32x16 tiles an SM (one field: up to four or eight), where
they are chosen by size, and the shapes that a caller fixes.  TMA wants an
even ld1; an odd one takes plain loads.  Every case asserts its kernel."""
import numpy as np
import pytest

import dispatch
from helpers import basin, np_case, oracle_grid, same
from test_gpu_parity import bind_all, compare, gpu_steps, make_ctx, oracle_steps, torchify

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def exe(built_lib, tmp_path_factory):
    return dispatch.build(tmp_path_factory.mktemp("dispatch"))


def layers_for(cuda, nx, ny, per_sm):
    """Layers of an nx x ny basin that make per_sm 32x16 tiles an SM."""
    import torch

    nsm = torch.cuda.get_device_properties(cuda).multi_processor_count
    return round(per_sm * nsm / (((nx + 31) // 32) * ((ny + 15) // 16)))


def check(cuda, nx, ny, kdm, periodic, advtyp, ntr, tile=None, **kw):
    b = basin(nx, ny, periodic, seed=nx)
    g = oracle_grid(b)
    c = np_case(b, g, kdm=kdm, ntracr=ntr, seed=nx, courant=0.8, delt1=240.0)
    c["delt1"] = 240.0
    t = torchify(c, cuda)
    ctx = make_ctx(b, g, kdm, tile=tile)
    bind_all(ctx, t)
    flg = np.zeros(ntr, np.int32) if ntr else None
    oracle_steps(g, c, (1, 2), advtyp, trcflg=flg, **kw)
    gpu_steps(ctx, t, (1, 2), advtyp, ntracr=ntr, trcflg=flg, **kw)
    compare(c, t)


@pytest.mark.parametrize("nx,ny,periodic", [(58, 37, False), (70, 45, True), (61, 40, False)])
@pytest.mark.parametrize("advtyp", [1, 2, 4])
def test_chosen_by_size(cuda, exe, nx, ny, periodic, advtyp):
    kdm = layers_for(cuda, nx, ny, 1.5)
    shape = "16x16" if advtyp == 1 else "32x16"
    assert dispatch.routes(exe, [(advtyp, nx, ny, kdm, 3)]) == [f"tile {shape} tma"]
    check(cuda, nx, ny, kdm, periodic, advtyp, 1)


@pytest.mark.parametrize("advtyp", [1, 2, 4])
def test_one_field(cuda, exe, advtyp):
    nx = 58
    ny = 8 * layers_for(cuda, nx, 16, 3.0) * 2 + 3  # three tiles an SM in one slice
    shape = "16x16" if advtyp == 1 else "32x16"
    assert dispatch.routes(exe, [(advtyp, nx, ny, 1, 1)]) == [f"tile {shape} tma"]
    b = basin(nx, ny, False, seed=12)
    g = oracle_grid(b)
    c = np_case(b, g, kdm=1, ntracr=0, seed=12, courant=0.7, delt1=600.0)
    fld, fldc, u, v = (c[k][l].copy() for k, l in (("temp", (1, 0)), ("temp", (0, 0)), ("uflx", 0), ("vflx", 0)))
    for a in (fld, fldc, u, v):
        g.xctilr(a, 5, 5)
    fcn = np.maximum(c["dp"][1, 0], 0.0)
    ref, got = fld.copy(), fld.copy()
    posdef = 256.0 if advtyp == 1 else 0.0
    g.advem(advtyp, ref, fldc, u, v, fcn, fcn, posdef, c["scp2"], c["scp2i"], 600.0)
    make_ctx(b, g, 1).advem(advtyp, got, fldc, u, v, fcn, fcn, posdef, c["scp2"], c["scp2i"], 600.0)
    assert same(got, ref) and not np.array_equal(got, fld)


@pytest.mark.parametrize("tile", ["16x16", "32x16", "32x32"])
@pytest.mark.parametrize("advtyp", [0, 1, 2, 4])
def test_fixed_by_the_caller(cuda, exe, tile, advtyp):
    nx, ny = 94, 53
    kdm = layers_for(cuda, nx, ny, 3.0)  # the strip kernels' size
    tma = "plain" if tile == "32x32" and advtyp < 2 else "tma"
    assert dispatch.routes(exe, [(advtyp, nx, ny, kdm, 2)]) == ["strip"]
    assert dispatch.routes(exe, [(advtyp, nx, ny, kdm, 2)], tile) == [f"tile {tile} {tma}"]
    check(cuda, nx, ny, kdm, True, advtyp, 0, tile=tile)


def test_strip_kernel_tests_reach_it(cuda, exe):
    """The sizes of test_gpu_march.py and test_gpu_ens_queue.py go to the strip kernels."""
    import test_gpu_march as tm

    marks = {m.args[0]: m.args[1] for m in tm.test_strip_edges.pytestmark}
    launches = [(s, nx, ny, kdm, 2 + ntr) for nx, ny, kdm, _ in marks["nx,ny,kdm,periodic"]
                for s, ntr in marks["advtyp,ntr"]]
    launches += [(s, 90, 70, 24, 2) for s in (0, 1, 4)]
    launches += [(s, 100, 60, 26, 4) for s in (0, 1, 2)]
    launches += [(s, 59, 9800, 1, 1) for s in (0, 1, 2, 4)]
    launches += [(s, 83, 61, 28, 4) for s in (0, 1, 2, 4)]
    launches += [(s, 175, 45, 20, 3) for s in (0, 1)]
    assert dispatch.routes(exe, launches) == ["strip"] * len(launches)
