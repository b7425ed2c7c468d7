"""The batch sizes at which a dispatch changes form, from the SM count of the
GPU at hand: one size below each and one at it."""
import numpy as np
import pytest
import torch

from distance3d_gb300 import workloads
from distance3d_gb300.epa import epa_batch
from distance3d_gb300.gjk import gjk_distance_batch, gjk_intersection_batch
from distance3d_gb300.mpr import mpr_batch
from distance3d_gb300.store import ColliderStore
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    cs, _, _ = workloads.pairs_all_types(900, seed=21, center_half_width=0.4, types=workloads.ALL_TYPES_MESH,
                                         margin_fraction=0.2)
    rng = np.random.default_rng(3)
    n = 3 * 512 * sms // 2
    i, j = (rng.integers(0, len(cs), n).astype(np.int32) for _ in range(2))
    return cs, ColliderStore(cs), i, j, sms


# slots the FP64 pools hold at once (2 blocks of 256 per SM), and blocks of them
@pytest.mark.parametrize("n", [lambda sms: 2 * sms - 1, lambda sms: 2 * sms, lambda sms: 2 * sms + 1,
                               lambda sms: 2 * 255 * sms, lambda sms: 2 * 255 * sms + 1,
                               lambda sms: 512 * sms, lambda sms: 512 * sms + 1])
def test_fp64_pools(scene, n):
    cs, st, i, j, sms = scene
    n = n(sms)
    i, j = i[:n], j[:n]
    r = {k: v.cpu().numpy() for k, v in gjk_distance_batch(st, i, j).items()}
    ref = oracle.gjk_distance(cs, i, j)
    for k in ("dist", "cp1", "cp2", "simplex", "n_simplex", "status", "iterations"):
        assert np.array_equal(r[k], ref[k], equal_nan=ref[k].dtype.kind == "f"), k
    assert np.array_equal(gjk_intersection_batch(st, i, j)["hit"].cpu().numpy(), oracle.gjk_intersection(cs, i, j)["hit"])
    m = {k: v.cpu().numpy() for k, v in mpr_batch(st, i, j).items()}
    ref = oracle.mpr(cs, i, j)
    for k in m:
        assert np.array_equal(m[k], ref[k], equal_nan=ref[k].dtype.kind == "f"), k


def test_mixed_forms(scene):
    """The FP32 phase's full grid (512 lanes per SM: the sort, and a pair on every lane), the
    refinement pass's blocks (from 16 to 128 pairs) and the spread's lanes per warp: a pair has the
    same bits in all of them."""
    cs, st, i, j, sms = scene
    whole = {k: v.cpu().numpy() for k, v in gjk_distance_batch(st, i, j, precision="mixed").items()}
    for n in (16 * sms - 1, 16 * sms, 16 * sms + 1, 32 * sms, 32 * sms + 1, 256 * sms - 1, 256 * sms, 256 * sms + 1,
              512 * sms - 1, 512 * sms, 512 * sms + 1):
        part = gjk_distance_batch(st, i[-n:], j[-n:], precision="mixed")
        for k in whole:
            assert np.array_equal(part[k].cpu().numpy(), whole[k][-n:], equal_nan=whole[k].dtype.kind == "f"), (n, k)


def test_search_forms(scene):
    """The FP32 polytope search: a whole warp per pair up to two pairs per resident warp (24 per SM),
    8 or 16 lanes above."""
    cs, st, i, j, sms = scene
    r = gjk_distance_batch(st, i, j, precision="mixed")
    k = np.flatnonzero(((r["dist"] == 0) & (r["n_simplex"] == 4)).cpu().numpy())
    i, j, s = i[k], j[k], r["simplex"].cpu().numpy()[k]
    assert len(k) > 48 * sms + 2
    for kw in (dict(), dict(max_faces=256, max_loose_edges=128)):
        runs = {n: epa_batch(st, i[:n], j[:n], s[:n], precision="mixed", **kw)
                for n in (24 * sms, 48 * sms, 48 * sms + 1, 48 * sms + 2)}
        for n, e in runs.items():
            for key, v in runs[48 * sms + 2].items():
                assert np.array_equal(e[key].cpu().numpy(), v[:n].cpu().numpy(), equal_nan=key == "mtv"), (n, key)
