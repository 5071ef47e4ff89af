"""The FP64 ensemble's queue with several work items a CTA (csrc/hyc_march.cuh,
march_queue_kernel) against the oracle, bit for bit: uneven basins, closed and
periodic, odd counts of fields, ragged last segments and strips."""
import numpy as np
import pytest

import hycadv
from helpers import levels, same
from test_gpu_ensemble import DELT1, get_cur, load, make_members, oracle_step, sea_interior, spec_of

pytestmark = pytest.mark.gpu

SPECS = [  # nx, ny, periodic, kdm, ntr, seed, courant, delt1
    (131, 103, False, 60, 5, 501, 0.7, 1800.0),
    (70, 41, True, 24, 3, 502, 0.8, 1800.0),
    (59, 50, False, 17, 1, 503, 0.6, 1800.0),
    (116, 27, True, 9, 2, 504, 0.5, 1800.0),
]


@pytest.mark.parametrize("advtyp", [2, 4])
def test_many_items(cuda, advtyp):
    import torch

    nsm = torch.cuda.get_device_properties(cuda).multi_processor_count
    # strips of 58 columns, segments of at least 24 rows, pairs of fields; four CTAs an SM
    items = sum(-(-nx // 58) * -(-ny // 32) * k * -(-ntr // 2) for nx, ny, _, k, ntr, *_ in SPECS)
    assert items > 3 * 4 * nsm
    members = make_members(SPECS)
    ens = hycadv.Ensemble([spec_of(m) for m in members], precision="fp64")
    load(ens, members)
    for step in (1, 2):
        ens.step(advtyp, DELT1, 1)
        for i, m in enumerate(members):
            want, got, ip = oracle_step(m, step, advtyp), get_cur(ens, i, m), sea_interior(m)
            assert same(got[..., ip], want[..., ip]), f"basin {i} step {step}"
            mm, nn = levels(step + 1)
            ens.put(i, "dp", np.ascontiguousarray(m["c"]["dp"][nn - 1]))
    ens.close()
