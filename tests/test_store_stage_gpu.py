"""A collider set on either side of the size up to which its arrays reach the
device in one copy gives the same store."""
import numpy as np
import pytest
import torch

from distance3d_gb300 import store as store_module
from distance3d_gb300 import workloads
from distance3d_gb300.store import STAGE_BYTES, ColliderStore
from oracle import oracle

pytestmark = pytest.mark.gpu


def staged_bytes(cs):
    boxes = int(((np.asarray(cs.types) & 0xff) == 2).sum())
    n = len(cs.types)
    # types, poses, params, vertex offsets and counts; vertices (hulls, meshes, boxes); links
    return n * (4 + 96 + 32 + 8 + 4) + 32 * max(len(cs.vertices) + 8 * boxes, 1) + 4 * len(cs.links)


def around(types):
    """Sets just below and just above STAGE_BYTES."""
    sets = [workloads.pairs_all_types(n, seed=5, types=types, margin_fraction=0.3)[0] for n in range(2, 130, 2)]
    sizes = [staged_bytes(cs) for cs in sets]
    below = max((s, k) for k, s in enumerate(sizes) if s <= STAGE_BYTES)[1]
    above = min((s, k) for k, s in enumerate(sizes) if s > STAGE_BYTES)[1]
    return sets[below], sets[above], sets[0]


@pytest.mark.parametrize("types", [workloads.ALL_TYPES, workloads.ALL_TYPES_MESH])
def test_both_sides(types, monkeypatch):
    copies = []
    real = store_module._staged
    monkeypatch.setattr(store_module, "_staged", lambda *a: copies.append(1) or real(*a))
    below, above, small = around(types)
    for cs, staged in ((small, 1), (below, 1), (above, 0)):
        copies.clear()
        monkeypatch.setattr(store_module, "STAGE_BYTES", STAGE_BYTES)
        a = ColliderStore(cs)
        assert len(copies) == staged
        monkeypatch.setattr(store_module, "STAGE_BYTES", -1)
        b = ColliderStore(cs)
        assert len(copies) == staged
        n = len(cs.types)
        for k in ("rec64", "rec32", "meta"):
            assert torch.equal(getattr(a, k)[:n].view(torch.int32), getattr(b, k)[:n].view(torch.int32)), k
        rows = len(cs.vertices) + 8 * int(((np.asarray(cs.types) & 0xff) == 2).sum())  # (a store without has one unused)
        for k in ("verts64", "verts32"):
            assert torch.equal(getattr(a, k)[:rows].view(torch.int32), getattr(b, k)[:rows].view(torch.int32)), k
        assert (a.links is None) == (b.links is None) and (a.links is None or torch.equal(a.links, b.links))
        d = np.random.default_rng(1).standard_normal((n, 3))
        s = a.support(np.arange(n), torch.from_numpy(d)).cpu().numpy()
        assert np.array_equal(s, oracle.support_batch(cs, np.arange(n), d))
