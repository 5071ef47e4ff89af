"""cnuity with one layer a launch, as on slices so large (or a device so full)
that the work slices hold no more, against the oracle, bit for bit."""
import pytest

from helpers import same
from test_gpu_cnuity import compare, setup

pytestmark = pytest.mark.gpu


def test_one_layer_a_launch(cuda):
    b, g, c, t, ctx = setup(cuda, 3100, 3140, False, 97, kdm=3, thkdf=4)
    assert (1 << 30) // (7 * 8 * b.ld1 * b.ld2) == 1  # layers in 1 GiB of work slices
    for step in (1, 2):
        m, n = ((step + 1) % 2) + 1, (step % 2) + 1
        want = g.cnuity(m, n, c, delt1=1800.0, nstep=step, thkdf4=True)
        got = ctx.cnuity(m, n, delt1=1800.0, nstep=step, thkdf=4, want_dpkmin=True)
        assert same(got, want)
        compare(c, t)
