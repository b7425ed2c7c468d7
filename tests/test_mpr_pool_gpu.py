"""The FP64 MPR kernel at the batch sizes where its distribution over blocks
changes, with and without penetration, and at its bounds: bit for bit the
oracle's results."""
import numpy as np
import pytest

from distance3d_gb300 import workloads
from distance3d_gb300.mpr import mpr_batch
from distance3d_gb300.store import ColliderStore
from oracle import oracle

pytestmark = pytest.mark.gpu

SLOTS = 2 * 152 * 256  # pairs the GPU holds at once


def check(cs, i1, i2, **opt):
    r = {k: v.cpu().numpy() for k, v in mpr_batch(ColliderStore(cs), i1, i2, **opt).items()}
    ref = oracle.mpr(cs, i1, i2, **{"tolerance" if k == "mpr_tolerance" else k: v for k, v in opt.items()})
    for k in r:
        assert np.array_equal(r[k], ref[k], equal_nan=ref[k].dtype.kind == "f"), k


@pytest.mark.parametrize("penetration", [True, False])
@pytest.mark.parametrize("n", [1, 31, 303, 305, 4095, 4097, 20011, SLOTS - 1, SLOTS + 300])
def test_batch_sizes(n, penetration):
    check(*workloads.pairs_all_types(n, seed=n, margin_fraction=0.2), penetration=penetration)


@pytest.mark.parametrize("opt", [dict(mpr_tolerance=1e-9), dict(max_iterations=1), dict(refine_limit=1),
                                 dict(mpr_tolerance=0.1, max_iterations=2)])
def test_bounds(opt):
    check(*workloads.pairs_all_types(2003, seed=4, types=workloads.ALL_TYPES_MESH), **opt)
