"""EPA with horizons of 30 to 60 edges on polytopes of about 64 faces: the
FP64 block kernel's loose-edge list that outgrows a warp's lanes, and the FP32
search's horizons wider than its segments.

The pairs are pyramids over a many-sided rim, their base a very flat cone, and
a point.  From a tetrahedron of three rim vertices and the top, EPA fills in
the rim, whose side faces are nearer to the origin than the base, until the
base is nearest; its apex then sees the whole fan of base faces at once."""
import numpy as np
import pytest

from distance3d_gb300.collider_set import HULL, ColliderSet
from oracle import oracle

TOP = 10.0


def fans(n, seed, rim=256, reach=(0.98, 0.994)):
    """Colliders, pairs and starting simplices; side faces of chords below
    `reach` of the radius are nearer than the base."""
    rng = np.random.default_rng(seed)
    points, offset, count, simplex, rows = [], [], [], [], 0
    for _ in range(n):
        c, z = rng.uniform(*reach), 0.0
        for _ in range(50):  # the base as far from the origin as the side face of a chord at distance c
            z = c * TOP / np.hypot(c, TOP + z)
        angle = (np.arange(rim) + rng.uniform(-0.2, 0.2, rim)) * 2 * np.pi / rim
        p = np.concatenate([np.stack([np.cos(angle), np.sin(angle), np.full(rim, -z)], 1),
                            [[0.0, 0.0, TOP], [0.0, 0.0, -z - 0.01]]])
        q = np.linalg.qr(rng.standard_normal((3, 3)))[0]
        q[:, 0] *= np.sign(np.linalg.det(q))
        p = p @ q.T
        start = (np.array([0.0, 120.0, 240.0]) + rng.uniform(0, 30, 3)) * rim / 360
        a, b, d = start.astype(int) % rim
        simplex.append(p[[a, d, b, rim]])  # faces wound outwards
        points += [p, np.zeros((1, 3))]
        offset += [rows, rows + rim + 2]
        count += [rim + 2, 1]
        rows += rim + 3
    poses = np.tile(np.concatenate([np.eye(3).reshape(9), np.zeros(3)]), (2 * n, 1))
    cs = ColliderSet(np.full(2 * n, HULL), poses, np.zeros((2 * n, 4)), np.array(offset), np.array(count),
                     np.concatenate(points))
    k = np.arange(n, dtype=np.int32)
    return cs, 2 * k, 2 * k + 1, np.array(simplex)


def test_the_pairs_have_long_edge_lists():
    """With at most 64 faces before it, an expansion of these pairs takes more
    than 29, 32 and 33 loose edges."""
    cs, i, j, s = fans(400, 1)
    def faces(t, e):
        return oracle.epa(cs, i, j, s, max_iter=t, max_faces=256, max_loose_edges=e)["n_faces"]
    whole = {t: faces(t, 128) for t in range(16, 33)}
    for e, least in ((29, 40), (32, 20), (33, 10)):
        hit = np.zeros(len(i), bool)
        same = np.ones(len(i), bool)
        for t in range(17, 33):
            d = faces(t, e) != whole[t]
            hit |= same & d & (whole[t - 1] <= 64)
            same &= ~d
        assert hit.sum() >= least, (e, hit.sum())


@pytest.mark.gpu
@pytest.mark.parametrize("opt", [dict(max_loose_edges=e) for e in (28, 29, 30, 31, 32, 33, 34, 36, 48, 128, 255)] +
                         [dict(max_loose_edges=128, max_faces=f) for f in (64, 65, 66, 67, 130)] +
                         [dict(max_loose_edges=128, max_iter=t) for t in (24, 27, 30, 32)])
def test_fp64(opt):
    from distance3d_gb300.epa import epa_batch
    from distance3d_gb300.store import ColliderStore
    cs, i, j, s = fans(400, 1)
    opt = {"max_faces": 256, **opt}
    r = {k: v.cpu().numpy() for k, v in epa_batch(ColliderStore(cs), i, j, s, return_faces=True, **opt).items()}
    ref = oracle.epa(cs, i, j, s, want_faces=True, **opt)
    assert np.array_equal(r["status"], ref["status"])
    assert np.array_equal(r["n_faces"], ref["n_faces"])
    assert np.array_equal(r["mtv"], ref["mtv"], equal_nan=True)
    for k, n in enumerate(ref["n_faces"]):
        assert np.array_equal(r["faces"][k, :n], ref["faces"][k, :n], equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("opt", [dict(max_faces=255, max_loose_edges=255), dict(max_faces=128, max_loose_edges=64)])
def test_fp32_search(opt):
    import torch
    from distance3d_gb300.epa import epa_batch
    from distance3d_gb300.store import ColliderStore
    n = 600
    cs, i, j, s = fans(n, 2, rim=48)  # few enough sides for the search to end
    st = ColliderStore(cs)

    def run(copies, **kw):
        r = epa_batch(st, np.tile(i, copies), np.tile(j, copies), np.tile(s, (copies, 1, 1)), return_faces=True,
                      precision="mixed", **{**opt, **kw})
        r["faces"] = torch.where(torch.arange(r["faces"].shape[1], device=r["faces"].device)[None, :, None, None]
                                 < r["n_faces"][:, None, None, None], r["faces"], 0.0)
        return {k: v.cpu().numpy() for k, v in r.items()}

    few = run(1)  # a whole warp per pair
    # the same bits with 8 or 16 lanes per pair (more pairs than two per resident warp)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    many = run((2 * 24 * sms) // n + 2)
    for k in few:
        assert np.array_equal(many[k][:n], few[k], equal_nan=True) and np.array_equal(many[k][-n:], few[k],
                                                                                      equal_nan=True), k
    # a shorter list sends the pairs with longer horizons to the FP64 search, whose faces differ
    for edges, least in ((24, n // 8), (32, n // 20)):
        short = run(1, max_loose_edges=edges)
        assert (short["faces"] != few["faces"]).any(axis=(1, 2, 3)).sum() > least, edges
    # The search stops where the support is within 32 ulp of the polytope's size of the face, and
    # the depth along the face's normal is above the true one by no more than that; the normal's and
    # the offset's own roundings are a few ulp more.
    ref = oracle.epa(cs, i, j, s, **{**opt, "max_iter": 64})
    ok = (few["status"] == 0) & (ref["status"] == 0)
    depth, true = np.linalg.norm(few["mtv"], axis=1)[ok], np.linalg.norm(ref["mtv"], axis=1)[ok]
    assert ok.sum() > n // 4
    assert np.abs(depth - true).max() <= 48 * 2.0 ** -23 * (TOP + 0.1)
