"""The mixed form gives a pair the same bits in every batch: small batches run
spread over the grid with shared hull scans, large ones on full warps."""
import numpy as np
import pytest

from distance3d_gb300 import workloads
from distance3d_gb300.epa import epa_batch
from distance3d_gb300.gjk import gjk_distance_batch
from distance3d_gb300.store import ColliderStore

pytestmark = pytest.mark.gpu

FULL = 90001  # more pairs than the GPU holds lanes of the first phase (152 SMs x 512)


def run(st, i, j):
    return {k: v.cpu().numpy() for k, v in gjk_distance_batch(st, i, j, precision="mixed").items()}


@pytest.mark.parametrize("types", [workloads.ALL_TYPES, workloads.ALL_TYPES_MESH])
def test_any_batch_size(types):
    cs, _, _ = workloads.pairs_all_types(700, seed=3, center_half_width=0.5, types=types)
    rng = np.random.default_rng(1)
    i = rng.integers(0, len(cs), FULL).astype(np.int32)
    j = rng.integers(0, len(cs), FULL).astype(np.int32)
    st = ColliderStore(cs)
    whole = run(st, i, j)
    for n in (1, 2, 15, 16, 17, 305, 2433, 4095, 4097, 30011, 77823, 77824):
        lo = int(rng.integers(0, FULL - n + 1))
        part = run(st, i[lo:lo + n], j[lo:lo + n])
        for k in whole:
            assert np.array_equal(part[k], whole[k][lo:lo + n], equal_nan=whole[k].dtype.kind == "f"), (n, k)
    hit = np.flatnonzero((whole["dist"] == 0) & (whole["n_simplex"] == 4))
    e = epa_batch(st, i[hit], j[hit], whole["simplex"][hit], precision="mixed")
    for n in (1, 33, 700):
        p = epa_batch(st, i[hit[:n]], j[hit[:n]], whole["simplex"][hit[:n]], precision="mixed")
        for k in p:
            assert np.array_equal(p[k].cpu().numpy(), e[k][:n].cpu().numpy(), equal_nan=k == "mtv"), (n, k)
