"""The ensemble's data path on the GPU: a get into device memory and the
FP32/FP64 conversions of put and get, the mixed form's work items over the
rows with sea, and the FP64 strip kernels of PCM and MPDATA under graph
capture."""
import numpy as np
import pytest

import hycadv
from helpers import basin, np_case, oracle_grid, same
from test_gpu_ensemble import DELT1, load, make_members, spec_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_get_into_device_memory(cuda, precision):
    """Every kind of value, whole and by slices at an odd offset, equals the
    host's own conversion and the get into host memory."""
    import torch

    m = make_members([(61, 45, False, 3, 2, 401, 0.5, 1800.0)])[0]
    ens = hycadv.Ensemble([spec_of(m)], precision=precision)
    b = m["b"]
    rng = np.random.default_rng(3)
    x = rng.standard_normal((2, 3, b.ld2, b.ld1)) * 10.0 ** rng.uniform(-60, 60, (2, 3, b.ld2, b.ld1))
    x.view(np.uint64)[0, 0] = rng.integers(0, 2 ** 64, (b.ld2, b.ld1), dtype=np.uint64)  # any bits
    f = np.float32(1.0) + np.arange(b.ld1, dtype=np.float64) * 2.0 ** -25  # halfway cases
    x[1, 0] = f
    special = [0.0, -0.0, np.inf, -np.inf, np.nan, 1e-45, 1.2e-38, 2.0 ** -126, 2.0 ** -149, 2.0 ** -150, 3.4028235e38,
               2.0 ** 128 - 2.0 ** 103, 2.0 ** 127, 5e-324, 1e300]
    rows = x[1, 1, b.nbdy]
    rows[b.nbdy:b.nbdy + len(special)] = special
    ens.put(0, "cur", x)
    with np.errstate(over="ignore", invalid="ignore"):
        want = x.astype(np.float32).astype(np.float64) if precision == "mixed" else x
    host, dev = np.zeros_like(x), torch.zeros(x.shape, dtype=torch.float64, device=cuda)
    ens.get(0, "cur", host)
    ens.get(0, "cur", dev)
    part = torch.zeros(1 + 2 * b.ld1 * b.ld2, dtype=torch.float64, device=cuda)
    view = part[1:].view(2, b.ld2, b.ld1)
    ens.get(0, "cur", view, 2, 2)
    inner = (Ellipsis, slice(b.nbdy, -b.nbdy), slice(b.nbdy, -b.nbdy))
    assert same(host[inner], want[inner])
    assert same(dev.cpu().numpy(), host)
    assert same(view.cpu().numpy(), host.reshape(6, b.ld2, b.ld1)[2:4])
    ens.get_async(0, "cur", dev.zero_())
    ens.wait()
    assert same(dev.cpu().numpy(), host)


@pytest.mark.parametrize("advtyp,diffusion", [(2, False), (4, False), (1, False), (2, True)])
def test_rows_without_sea(cuda, advtyp, diffusion):
    """A basin with wide belts of land: the same bits whatever the segments,
    and the FP64 form's values within the mixed form's error."""
    b = basin(130, 300, True, seed=17)
    b.depth[b.nbdy + 60:b.nbdy + 150] = 0.0
    b.depth[b.nbdy + 200:b.nbdy + 220, : b.nbdy + 70] = 0.0
    g = oracle_grid(b)
    c = np_case(b, g, kdm=2, ntracr=1, seed=17, courant=0.6, delt1=DELT1)
    trc = np.concatenate([c["saln"][None], c["tracer"]], axis=0)
    m = dict(b=b, g=g, c=c, ntr=2, kdm=2, trc=trc)
    sc, _ = b.metrics()
    d = dict(aspux=np.ones_like(sc), aspvy=np.ones_like(sc), scuy=np.full_like(sc, 1e4), scvx=np.full_like(sc, 1e4))
    got = {}
    for tile in (32, 128, 2048):
        ens = hycadv.Ensemble([spec_of(m)], precision="mixed")
        ens.set_tile(56, tile)
        load(ens, [m])
        if diffusion:
            ens.set_diffusion(0, 0.015, **d)
        ens.step(advtyp, DELT1, 2)
        got[tile] = np.zeros((2, 2, b.ld2, b.ld1))
        ens.get(0, "cur", got[tile])
        ens.close()
    assert same(got[32], got[128]) and same(got[32], got[2048])
    if diffusion:
        return
    ens = hycadv.Ensemble([spec_of(m)], precision="fp64")
    load(ens, [m])
    ens.step(advtyp, DELT1, 2)
    ref = np.zeros_like(got[32])
    ens.get(0, "cur", ref)
    ens.close()
    sea = np.zeros((b.ld2, b.ld1), bool)
    sea[b.J, b.I] = g.masks["ip"][b.J, b.I] != 0
    for q in range(2):
        assert np.abs(got[32][q][:, sea] - ref[q][:, sea]).max() < 2e-6 * np.abs(ref[q][:, sea]).max()


@pytest.mark.parametrize("advtyp", [0, 1])
def test_strip_kernels_under_capture(cuda, advtyp):
    out = []
    for graph in (False, True):
        members = make_members([(175, 45, True, 20, 3, 411, 0.7, 1800.0)])
        ens = hycadv.Ensemble([spec_of(members[0])], precision="fp64")
        load(ens, members)
        ens.step(advtyp, DELT1, 3, graph=graph)
        ens.step(advtyp, DELT1, 3, graph=graph)
        a = np.zeros((3, 20, members[0]["b"].ld2, members[0]["b"].ld1))
        ens.get(0, "cur", a)
        out.append(a)
        ens.close()
    assert same(out[0], out[1])
