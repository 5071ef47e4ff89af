"""cnuity's launches over batches of layers (csrc/hyc_cnuity.cu) against the
oracle, bit for bit: more layers than a batch holds (1 GiB of work slices), in
both directions of the interface diffusion, and one layer alone."""
import pytest

from helpers import same
from test_gpu_cnuity import compare, setup

pytestmark = pytest.mark.gpu


def test_more_layers_than_a_batch(cuda):
    kdm = 45  # slices of 712 x 612 cells: 44 layers a batch
    b, g, c, t, ctx = setup(cuda, 700, 600, True, 95, kdm=kdm, thkdf=4)
    assert (1 << 30) // (7 * 8 * b.ld1 * b.ld2) < kdm
    for step in (1, 2):
        m, n = ((step + 1) % 2) + 1, (step % 2) + 1
        want = g.cnuity(m, n, c, delt1=1800.0, nstep=step, thkdf4=True)
        got = ctx.cnuity(m, n, delt1=1800.0, nstep=step, thkdf=4, want_dpkmin=True)
        assert same(got, want)
        compare(c, t)


def test_one_layer(cuda):
    b, g, c, t, ctx = setup(cuda, 41, 33, False, 96, kdm=1)
    for step in (1, 2):
        m, n = ((step + 1) % 2) + 1, (step % 2) + 1
        want = g.cnuity(m, n, c, delt1=1800.0, nstep=step)
        got = ctx.cnuity(m, n, delt1=1800.0, nstep=step, want_dpkmin=True)
        assert same(got, want)
        compare(c, t)
