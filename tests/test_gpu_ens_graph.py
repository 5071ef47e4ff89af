"""Step graphs between longer eager runs on the GPU: the same bits as eager
steps alone (the graph is recorded again once its queue counters move)."""
import numpy as np
import pytest

import hycadv
from helpers import same
from test_gpu_ensemble import DELT1, SPECS, get_cur, load, make_members, spec_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,advtyp", [("fp64", 2), ("fp64", 1), ("mixed", 2)])
def test_graph_after_a_longer_run(cuda, precision, advtyp):
    runs = [(3, True), (5, False), (1, False), (3, True)]  # the second graph run starts at the first one's rotation
    out = []
    for graphs in (True, False):
        members = make_members(SPECS[:2])
        ens = hycadv.Ensemble([spec_of(m) for m in members], precision=precision)
        load(ens, members)
        for n, graph in runs:
            ens.step(advtyp, DELT1, n, graph=graph and graphs)
        out.append([get_cur(ens, i, m) for i, m in enumerate(members)])
        ens.close()
    assert all(np.isfinite(a).all() for a in out[1])
    assert all(same(a, b) for a, b in zip(*out))
