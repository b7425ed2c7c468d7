"""The work that users of distance3d_gb300 have it do, as measurable cases.

``listed()`` gives a fixed set of cases, ``draw(rng)`` one more of the same
ranges.  ``prepare(case, seed)`` makes what a program holds before the call
(colliders on the device, index lists, a captured batch), ``run(state)`` is one
pass through the public entry points, ``work(case)`` the bytes and operations
that pass cannot do without, and ``exact(case, seed)`` the distances it should
return, from a plain 64-bit GJK written here in torch.

Kinds of case:

* ``pair``    the drop-in ``gjk.gjk(collider1, collider2)`` on two objects
* ``gjk``     ``gjk_distance_batch`` on a resident store
* ``hit``     ``gjk_intersection_batch``
* ``epa``     ``epa_batch`` on intersecting pairs and their GJK simplices
* ``mpr``     ``mpr_batch``, with or without penetration
* ``collide`` ``CollisionBatch`` (GJK, then EPA where it intersects) from host
              index lists to results in host memory
* ``scene``   ``collide_scene``: AABBs, tree, overlapping pairs, GJK and EPA
* ``tree``    ``LBVH`` built over boxes, then queried with other boxes
* ``robot``   ``SelfCollisionBatch.run``: joint values to contacts

Collider sets: ``scb`` (sphere, capsule, box), ``six`` (with cylinder,
ellipsoid and convex hulls of 8 to 256 vertices), ``ten`` (with disk, ellipse,
cone, MeshGraph, a quarter of them wrapped in Margin).  Sizes follow the
package's workloads: radii 0.05-0.3, heights 0.1-0.5.  ``half`` is the half
width of the cube the centers lie in: 0.38 gives ~30% intersecting six-type
pairs, 1.0 about 3%.
"""
import math

import numpy as np
import torch

SPHERE, CAPSULE, BOX, CYLINDER, ELLIPSOID, HULL, DISK, ELLIPSE, CONE, MESH = range(10)
MARGIN = 0x100
TYPES = {"scb": (SPHERE, CAPSULE, BOX),
         "six": (SPHERE, CAPSULE, BOX, CYLINDER, ELLIPSOID, HULL),
         "ten": tuple(range(10))}
ONE = {"sphere": SPHERE, "capsule": CAPSULE, "box": BOX, "cylinder": CYLINDER, "ellipsoid": ELLIPSOID, "hull": HULL,
       "disk": DISK, "ellipse": ELLIPSE, "cone": CONE}


def listed():
    return [
        # one query of a planner or an interactive program: two collider objects
        {"name": "pair_capsule_hull", "kind": "pair", "first": "capsule", "second": "hull", "half": 0.38},
        # a small batch, the reference's own benchmark setting: primitives only, mostly apart
        {"name": "gjk_f64_scb_1000", "kind": "gjk", "set": "scb", "n": 1000, "half": 1.0, "precision": "fp64"},
        # exact distances of a large batch of mixed shapes
        {"name": "gjk_f64_six_100003", "kind": "gjk", "set": "six", "n": 100003, "half": 0.38, "precision": "fp64"},
        # every collider type with margins and meshes, tolerance-bound distances
        {"name": "gjk_mixed_ten_20011", "kind": "gjk", "set": "ten", "n": 20011, "half": 0.38, "precision": "mixed"},
        # boolean collision checks, as motion planning asks for them
        {"name": "hit_f64_six_65536", "kind": "hit", "set": "six", "n": 65536, "half": 0.6},
        # exact penetration depths with the reference's default limits
        {"name": "epa_f64_six_6007", "kind": "epa", "set": "six", "n": 6007, "faces": 64, "edges": 32,
         "precision": "fp64"},
        # contact estimation with MPR, exact form
        {"name": "mpr_f64_ten_50021", "kind": "mpr", "set": "ten", "n": 50021, "half": 0.38, "precision": "fp64",
         "penetration": True},
        # one request of a collision service over a resident store
        {"name": "collide_mixed_six_3000", "kind": "collide", "set": "six", "n": 3000, "half": 0.38, "faces": 64,
         "edges": 32, "precision": "mixed"},
        # the throughput workload: a million mixed pairs, large polytopes
        {"name": "collide_mixed_six_1048576", "kind": "collide", "set": "six", "n": 1048576, "half": 0.38,
         "faces": 256, "edges": 128, "precision": "mixed"},
        # a whole scene, broad and narrow phase
        {"name": "scene_mixed_six_131072", "kind": "scene", "set": "six", "n": 131072, "precision": "mixed"},
        # broad phase alone: static geometry against a set of query boxes
        {"name": "tree_200003_by_30011", "kind": "tree", "n": 200003, "m": 30011},
        # self-collision of sampled arm configurations
        {"name": "robot_mixed_1024", "kind": "robot", "configs": 1024, "bodies": 30, "dof": 7, "precision": "mixed"},
    ]


def _log(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, max(lo, n + rng.randint(-3, 3)))


def draw(rng):
    kind = rng.choice(["pair", "gjk", "gjk", "hit", "epa", "mpr", "collide", "collide", "scene", "tree", "robot"])
    precision = rng.choice(["fp64", "mixed"])
    some = rng.choice(["scb", "six", "ten"])
    half = round(rng.uniform(0.3, 1.0), 3)
    if kind == "pair":
        first, second = rng.choice(sorted(ONE)), rng.choice(sorted(ONE))
        return {"kind": kind, "first": first, "second": second, "half": half}
    if kind == "gjk":
        n = _log(rng, 32, 100003 if precision == "fp64" else 400000)
        return {"kind": kind, "set": some, "n": n, "half": half, "precision": precision}
    if kind == "hit":
        return {"kind": kind, "set": some, "n": _log(rng, 32, 100003), "half": half}
    if kind == "epa":
        faces, edges = rng.choice([(64, 32), (128, 64), (256, 128)])
        n = _log(rng, 32, 30000 if precision == "fp64" else 60000)
        return {"kind": kind, "set": some, "n": n, "faces": faces, "edges": edges, "precision": precision}
    if kind == "mpr":
        n = _log(rng, 32, 200003 if precision == "fp64" else 600000)
        return {"kind": kind, "set": some, "n": n, "half": half, "precision": precision,
                "penetration": rng.random() < 0.7}
    if kind == "collide":
        faces, edges = rng.choice([(64, 32), (256, 128)])
        n = _log(rng, 100, 60000 if precision == "fp64" else 500000)
        return {"kind": kind, "set": some, "n": n, "half": half, "faces": faces, "edges": edges,
                "precision": precision}
    if kind == "scene":
        n = _log(rng, 300, 30000 if precision == "fp64" else 131072)
        return {"kind": kind, "set": some, "n": n, "precision": precision}
    if kind == "tree":
        return {"kind": kind, "n": _log(rng, 100, 400000), "m": _log(rng, 50, 100000)}
    return {"kind": kind, "configs": _log(rng, 16, 2048 if precision == "fp64" else 8192),
            "bodies": rng.randint(8, 30), "dof": rng.randint(4, 8), "precision": precision}


# ---------------------------------------------------------------- inputs
class _Colliders:
    """Plain arrays of one batch of colliders, on the GPU (float64 / int64)."""


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * (int(seed) % 2000000) + 17)
    return g


def _uniform(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _rotations(g, n):
    q = torch.randn(n, 4, generator=g, device="cuda", dtype=torch.float64)
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                        2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                        2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1).reshape(n, 3, 3)


def _octasphere(level, scale):
    """Vertices and triangles of a subdivided octahedron, stretched per axis:
    6, 18 or 66 vertices, convex."""
    v = [(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)]
    v = [np.array(p, dtype=float) for p in v]
    tri = [(0, 2, 4), (2, 1, 4), (1, 3, 4), (3, 0, 4), (2, 0, 5), (1, 2, 5), (3, 1, 5), (0, 3, 5)]
    for _ in range(level):
        mid, new = {}, []

        def between(i, j):
            k = (min(i, j), max(i, j))
            if k not in mid:
                p = v[i] + v[j]
                v.append(p / np.linalg.norm(p))
                mid[k] = len(v) - 1
            return mid[k]
        for a, b, c in tri:
            ab, bc, ca = between(a, b), between(b, c), between(c, a)
            new += [(a, ab, ca), (ab, b, bc), (ca, bc, c), (ab, bc, ca)]
        tri = new
    return np.array(v) * np.asarray(scale), np.array(tri)


def _meshes():
    """The mesh shapes that MeshGraph colliders share, as links of a robot do."""
    scales = [(0.2, 0.2, 0.2), (0.1, 0.25, 0.15), (0.08, 0.08, 0.3), (0.3, 0.12, 0.2), (0.06, 0.1, 0.07),
              (0.25, 0.25, 0.1)]
    return [_octasphere(k % 3, s) for k, s in enumerate(scales)]


def _colliders(g, n, types, half):
    c = _Colliders()
    choice = torch.tensor(types, device="cuda")
    c.types = choice[torch.randint(len(types), (n,), generator=g, device="cuda")]
    c.R = _rotations(g, n)
    c.t = _uniform(g, -half, half, n, 3)
    u = _uniform(g, 0.05, 0.3, n, 3)
    h = _uniform(g, 0.1, 0.5, n)
    p = torch.zeros(n, 4, device="cuda", dtype=torch.float64)
    is_ = lambda *ts: torch.isin(c.types, torch.tensor(ts, device="cuda"))  # noqa: E731
    round_ = is_(SPHERE, CAPSULE, CYLINDER, DISK, CONE)
    p[:, 0] = torch.where(round_, u[:, 0], p[:, 0])
    p[:, 1] = torch.where(is_(CAPSULE, CYLINDER, CONE), h, p[:, 1])
    p[:, :3] = torch.where(is_(BOX)[:, None], 2 * u, p[:, :3])
    p[:, :3] = torch.where(is_(ELLIPSOID)[:, None], u, p[:, :3])
    p[:, :2] = torch.where(is_(ELLIPSE)[:, None], u[:, :2], p[:, :2])
    # hulls: points on a sphere, in world space
    hull = is_(HULL).nonzero().flatten()
    count = torch.exp(_uniform(g, math.log(8), math.log(256.99), len(hull))).floor().long().clamp(8, 256)
    owner = torch.repeat_interleave(hull, count)
    pts = torch.randn(len(owner), 3, generator=g, device="cuda", dtype=torch.float64)
    pts = pts / pts.norm(dim=1, keepdim=True) * u[owner, :1] + c.t[owner]
    c.count = torch.zeros(n, device="cuda", dtype=torch.int64)
    c.offset = torch.full((n,), -1, device="cuda", dtype=torch.int64)
    c.count[hull] = count
    c.offset[hull] = torch.cumsum(count, 0) - count
    c.R[hull] = torch.eye(3, device="cuda", dtype=torch.float64)
    c.t[hull] = 0.0
    c.R[is_(SPHERE)] = torch.eye(3, device="cuda", dtype=torch.float64)
    # meshes: a few shared shapes, in their own frame
    c.mesh_of = torch.full((n,), -1, device="cuda", dtype=torch.int64)
    mesh = is_(MESH).nonzero().flatten()
    if len(mesh):
        shapes = _meshes()
        k = torch.randint(len(shapes), (len(mesh),), generator=g, device="cuda")
        sizes = torch.tensor([len(v) for v, _ in shapes], device="cuda")
        first = len(pts) + torch.cumsum(sizes, 0) - sizes
        c.mesh_of[mesh] = k
        c.count[mesh] = sizes[k]
        c.offset[mesh] = first[k]
        pts = torch.cat([pts] + [torch.tensor(v, device="cuda", dtype=torch.float64) for v, _ in shapes])
    c.verts = pts
    c.wrapped = torch.zeros(n, device="cuda", dtype=torch.bool)
    if MESH in types:
        c.wrapped = torch.rand(n, generator=g, device="cuda") < 0.25
        p[:, 3] = torch.where(c.wrapped, _uniform(g, 0.01, 0.05, n), p[:, 3])
    c.params = p
    return c


def _packed(c):
    """The package's ColliderSet of the same colliders."""
    from distance3d_gb300.collider_set import ColliderSet, mesh_links
    host = lambda t: t.cpu().numpy()  # noqa: E731
    params = host(c.params)
    links = []
    mesh_of = host(c.mesh_of)
    if (mesh_of >= 0).any():
        at, first, low = 0, [], []
        for v, tri in _meshes():
            block = mesh_links(v, tri)
            first.append(at)
            low.append(float(tri.min()))
            links.append(block)
            at += len(block)
        m = mesh_of >= 0
        params[m, 0] = np.array(first)[mesh_of[m]]
        params[m, 1] = np.array(low)[mesh_of[m]]
    types = c.types.to(torch.int32) | torch.where(c.wrapped, MARGIN, 0).to(torch.int32)
    poses = torch.cat([c.R.reshape(-1, 9), c.t], 1)
    verts = torch.cat([c.verts, torch.zeros(len(c.verts), 1, device="cuda", dtype=torch.float64)], 1)
    return ColliderSet(host(types), host(poses), params, host(c.offset), host(c.count.to(torch.int32)), host(verts),
                       np.concatenate(links) if links else None)


def _pairs(case, seed, n=None):
    """2 n colliders; pair k is (2 k, 2 k + 1)."""
    n = case["n"] if n is None else n
    return _colliders(_gen(seed), 2 * n, TYPES[case["set"]], case.get("half", 0.38))


def _half(n):
    # the package's scene density: 131,072 colliders in [-20, 20]^3
    return 20.0 * (n / 131072) ** (1 / 3)


def _turn(g):
    """A rotation that permutes the axes (all three negated where the
    permutation is odd) and a shift.  A scene of another seed is the same world
    turned, shifted and listed in another order, so that the number of its
    overlapping pairs does not depend on the seed."""
    k = int(torch.randint(6, (1,), generator=g, device="cuda"))
    perm = [(0, 1, 2), (1, 2, 0), (2, 0, 1), (1, 0, 2), (0, 2, 1), (2, 1, 0)][k]
    Q = torch.zeros(3, 3, device="cuda", dtype=torch.float64)
    for i in range(3):
        Q[i, perm[i]] = 1.0 if k < 3 else -1.0
    return Q, _uniform(g, -1.0, 1.0, 3)


def _scene(case, seed):
    c = _colliders(_gen(case["n"]), case["n"], TYPES[case["set"]], _half(case["n"]))
    g = _gen(seed)
    Q, shift = _turn(g)
    order = torch.randperm(case["n"], generator=g, device="cuda")
    hull, sphere = c.types == HULL, c.types == SPHERE
    turned = torch.matmul(Q, c.R)
    c.R = torch.where((hull | sphere)[:, None, None], c.R, turned)
    c.t = torch.where(hull[:, None], c.t, c.t @ Q.T + shift)
    world = int(c.count[hull].sum())  # mesh vertices, kept after these, are in their own frame
    c.verts = torch.cat([c.verts[:world] @ Q.T + shift, c.verts[world:]])
    for k in ("types", "R", "t", "params", "count", "offset", "mesh_of", "wrapped"):
        setattr(c, k, getattr(c, k)[order].contiguous())
    return c


def _indices(n):
    k = torch.arange(n, device="cuda", dtype=torch.int32)
    return 2 * k, 2 * k + 1


def _boxes(case, seed):
    g, h = _gen(case["n"] + case["m"]), _gen(seed)
    Q, shift = _turn(h)
    got = []
    for n in (case["n"], case["m"]):
        center = _uniform(g, -_half(case["n"]), _half(case["n"]), n, 3) @ Q.T + shift
        ext = _uniform(g, 0.05, 0.4, n, 3) @ Q.abs().T
        order = torch.randperm(n, generator=h, device="cuda")
        got.append(torch.stack([center - ext, center + ext], 2)[order].contiguous())
    return got


def _arm(case, seed):
    """A serial arm: joints alternating z and y, bodies spread over its links
    (capsules, boxes, cylinders along them), and joint values."""
    rng = np.random.default_rng(int(seed))
    dof, nb = case["dof"], case["bodies"]
    length = rng.uniform(0.1, 0.4, dof)
    axis = np.array([[0.0, 0.0, 1.0] if j % 2 == 0 else [0.0, 1.0, 0.0] for j in range(dof)])
    origin = np.zeros((dof, 12))
    origin[:, [0, 4, 8]] = 1.0
    origin[1:, 11] = length[:-1]
    link = np.arange(nb) * (dof + 1) // nb
    along = np.where(link > 0, length[np.maximum(link - 1, 0)], 0.15)
    kind = rng.choice([CAPSULE, BOX, CYLINDER], nb)
    params = np.zeros((nb, 4))
    params[:, 0] = rng.uniform(0.04, 0.08, nb)
    params[:, 1] = rng.uniform(0.3, 0.8, nb) * along
    box = kind == BOX
    params[box, :2] = rng.uniform(0.04, 0.12, (int(box.sum()), 2))
    params[box, 2] = rng.uniform(0.3, 0.8, int(box.sum())) * along[box]
    ang = rng.uniform(-0.3, 0.3, nb)
    body = np.zeros((nb, 12))
    body[:, 0], body[:, 4], body[:, 5], body[:, 7], body[:, 8] = (1.0, np.cos(ang), -np.sin(ang), np.sin(ang),
                                                                  np.cos(ang))
    body[:, 9:11] = rng.uniform(-0.03, 0.03, (nb, 2))
    body[:, 11] = rng.uniform(0.1, 0.9, nb) * along
    q = rng.uniform(-math.pi, math.pi, (case["configs"], dof))
    return axis, origin, link, body, kind, params, q


def _object(c, i):
    """Collider i as the object a user constructs."""
    from distance3d_gb300 import colliders as col
    t = int(c.types[i])
    pose = np.eye(4)
    pose[:3, :3] = c.R[i].cpu().numpy()
    pose[:3, 3] = c.t[i].cpu().numpy()
    p = [float(x) for x in c.params[i].cpu()]
    if t == SPHERE:
        return col.Sphere(pose[:3, 3], p[0])
    if t == CAPSULE:
        return col.Capsule(pose, p[0], p[1])
    if t == BOX:
        return col.Box(pose, np.array(p[:3]))
    if t == CYLINDER:
        return col.Cylinder(pose, p[0], p[1])
    if t == ELLIPSOID:
        return col.Ellipsoid(pose, np.array(p[:3]))
    if t == HULL:
        o, k = int(c.offset[i]), int(c.count[i])
        return col.ConvexHullVertices(c.verts[o:o + k].cpu().numpy())
    if t == DISK:
        return col.Disk(pose[:3, 3], p[0], pose[:3, 2].copy())
    if t == ELLIPSE:
        return col.Ellipse(pose[:3, 3], pose[:3, :2].T.copy(), np.array(p[:2]))
    return col.Cone(pose, p[0], p[1])


def _two(case, seed):
    g = _gen(seed)
    parts = [_colliders(g, 1, (ONE[case[k]],), case["half"]) for k in ("first", "second")]
    return parts


# ---------------------------------------------------------------- prepare and run
def prepare(case, seed):
    from distance3d_gb300.store import ColliderStore
    kind = case["kind"]
    if kind == "pair":
        a, b = _two(case, seed)
        return {"kind": kind, "a": _object(a, 0), "b": _object(b, 0)}
    if kind in ("gjk", "hit", "mpr"):
        i1, i2 = _indices(case["n"])
        return {"kind": kind, "case": case, "store": ColliderStore(_packed(_pairs(case, seed))), "i1": i1, "i2": i2}
    if kind == "epa":
        from distance3d_gb300.gjk import gjk_distance_batch
        some = 5 * case["n"] + 300
        store = ColliderStore(_packed(_pairs(case, seed, some)))
        i1, i2 = _indices(some)
        r = gjk_distance_batch(store, i1, i2, precision=case["precision"])
        k = ((r["dist"] == 0.0) & (r["n_simplex"] == 4)).nonzero().flatten()[:case["n"]]
        return {"kind": kind, "case": case, "store": store, "i1": i1[k].contiguous(), "i2": i2[k].contiguous(),
                "simplex": r["simplex"][k].contiguous()}
    if kind == "collide":
        from distance3d_gb300.serve import CollisionBatch
        store = ColliderStore(_packed(_pairs(case, seed)))
        kw = dict(max_faces=case["faces"], max_loose_edges=case["edges"])
        i1, i2 = (x.cpu().numpy() for x in _indices(case["n"]))
        return {"kind": kind, "batch": CollisionBatch(store, case["n"], precision=case["precision"], epa_kw=kw),
                "i1": i1, "i2": i2}
    if kind == "scene":
        return {"kind": kind, "case": case, "store": ColliderStore(_packed(_scene(case, seed)))}
    if kind == "tree":
        leaves, boxes = _boxes(case, seed)
        return {"kind": kind, "leaves": leaves, "boxes": boxes}
    from distance3d_gb300.robot import SelfCollisionBatch, SerialArm
    axis, origin, link, body, types, params, q = _arm(case, seed)
    arm = SerialArm(axis, origin, link, body, types, params)
    return {"kind": kind, "batch": SelfCollisionBatch(arm, case["configs"], precision=case["precision"]), "q": q}


def run(state):
    kind = state["kind"]
    if kind == "pair":
        from distance3d_gb300.gjk import gjk
        return gjk(state["a"], state["b"])
    if kind == "gjk":
        from distance3d_gb300.gjk import gjk_distance_batch
        return gjk_distance_batch(state["store"], state["i1"], state["i2"], precision=state["case"]["precision"])
    if kind == "hit":
        from distance3d_gb300.gjk import gjk_intersection_batch
        return gjk_intersection_batch(state["store"], state["i1"], state["i2"])
    if kind == "epa":
        from distance3d_gb300.epa import epa_batch
        c = state["case"]
        return epa_batch(state["store"], state["i1"], state["i2"], state["simplex"], max_faces=c["faces"],
                         max_loose_edges=c["edges"], precision=c["precision"])
    if kind == "mpr":
        from distance3d_gb300.mpr import mpr_batch
        c = state["case"]
        return mpr_batch(state["store"], state["i1"], state["i2"], precision=c["precision"],
                         penetration=c["penetration"])
    if kind == "collide":
        state["batch"].submit(state["i1"], state["i2"])
        return state["batch"].results()
    if kind == "scene":
        from distance3d_gb300.pipeline import collide_scene
        return collide_scene(state["store"], precision=state["case"]["precision"])
    if kind == "tree":
        from distance3d_gb300.bvh import LBVH
        tree = LBVH(state["leaves"])
        return {"self": tree.self_pairs(), "query": tree.query(state["boxes"])}
    return state["batch"].run(state["q"])


# ---------------------------------------------------------------- work
# operations per unit of the path: one pair of supports and one simplex solve
# (GJK, MPR), one expansion (EPA), one box test
_STEP, _EXPAND = 250.0, 900.0
_OUT = 154.0       # bytes a pair's GJK results take
_EPA_OUT = 29.0


def _bytes_of(case, colliders):
    hull = {"scb": 0.0, "six": 1 / 6, "ten": 1 / 10}[case["set"]] * 73 * 24.0
    return colliders * (124.0 + hull)


def work(case):
    kind, n = case["kind"], case.get("n", 1)
    if kind == "pair":
        return {"bytes": 2 * 124.0 + 73 * 24.0 + _OUT, "flops": 15 * _STEP}
    if kind == "gjk":
        return {"bytes": n * (8 + _OUT) + _bytes_of(case, 2 * n), "flops": n * 12 * _STEP}
    if kind == "hit":
        return {"bytes": n * 10.0 + _bytes_of(case, 2 * n), "flops": n * 5 * _STEP}
    if kind == "mpr":
        return {"bytes": n * (10.0 + (56 if case["penetration"] else 0)) + _bytes_of(case, 2 * n),
                "flops": n * 6 * _STEP}
    if kind == "epa":
        return {"bytes": n * (8 + 96 + _EPA_OUT) + _bytes_of(case, 2 * n), "flops": n * 20 * _EXPAND}
    if kind == "collide":
        return {"bytes": n * (8 + _OUT + _EPA_OUT) + _bytes_of(case, 2 * n),
                "flops": n * 12 * _STEP + 0.3 * n * 20 * _EXPAND}
    if kind == "scene":
        pairs = 0.67 * n
        return {"bytes": _bytes_of(case, n) + pairs * (8 + _OUT + _EPA_OUT),
                "flops": pairs * (12 * _STEP + 0.4 * 20 * _EXPAND) + n * 17 * 12.0}
    if kind == "tree":
        m = case["m"]
        return {"bytes": (n + m) * 48.0 + (1.5 * n + 3.0 * m) * 8, "flops": (n + m) * 17 * 12.0}
    pairs = case["configs"] * case["bodies"] * (case["bodies"] - 1) / 2 * 0.7
    return {"bytes": case["configs"] * case["dof"] * 8.0 + pairs * 33, "flops": pairs * 10 * _STEP}


# ---------------------------------------------------------------- exact distances
def exact(case, seed):
    """Distances in 64 bits (closest points, simplices, contact normals and
    depths depend on where the algorithms stop and have no such value)."""
    kind = case["kind"]
    if kind == "pair":
        a, b = _two(case, seed)
        return [float(_distances(a, b, torch.zeros(1, device="cuda", dtype=torch.long),
                                 torch.zeros(1, device="cuda", dtype=torch.long))[0]), None, None, None]
    if kind in ("gjk", "collide"):
        c = _pairs(case, seed)
        i1, i2 = (x.long() for x in _indices(case["n"]))
        d = _distances(c, c, i1, i2)
        return {"dist": d.cpu().numpy() if kind == "collide" else d}
    if kind == "scene":
        c = _scene(case, seed)
        i, j = _overlaps(*_aabbs(c))
        return [None, {"dist": _distances(c, c, i, j)}]
    if kind == "robot":
        axis, origin, link, body, types, params, q = _arm(case, seed)
        c = _posed(axis, origin, link, body, types, params, q)
        a, b = np.triu_indices(len(link), k=1)
        keep = np.abs(link[a] - link[b]) > 1
        base = torch.arange(len(q), device="cuda")[:, None] * len(link)
        i1 = (base + torch.tensor(a[keep], device="cuda")).flatten()
        i2 = (base + torch.tensor(b[keep], device="cuda")).flatten()
        return {"dist": _distances(c, c, i1, i2).reshape(len(q), -1), "mtv": None}
    return None


def _unit(v):
    n = v.norm(dim=1, keepdim=True)
    return torch.where(n > 0, v / n.clamp_min(1e-300), torch.zeros_like(v))


def _support(c, idx, d):
    """Farthest points of colliders idx along d."""
    R, t, p, ty = c.R[idx], c.t[idx], c.params[idx], c.types[idx]
    local = (R * d[:, :, None]).sum(1)
    flat = torch.cat([_unit(local[:, :2]), torch.zeros_like(local[:, :1])], 1)
    end = torch.where(local[:, 2:] >= 0, 1.0, -1.0).to(torch.float64)
    z = torch.zeros_like(local)
    z[:, 2] = 1.0
    rad, height = p[:, :1], p[:, 1:2]
    out = _unit(local) * rad  # sphere
    is_ = lambda k: (ty == k)[:, None]  # noqa: E731
    out = torch.where(is_(CAPSULE), out + z * end * height / 2, out)
    out = torch.where(is_(BOX), torch.where(local >= 0, 0.5, -0.5) * p[:, :3], out)
    out = torch.where(is_(CYLINDER), flat * rad + z * end * height / 2, out)
    out = torch.where(is_(ELLIPSOID), _unit(local * p[:, :3]) * p[:, :3], out)
    out = torch.where(is_(DISK), flat * rad, out)
    pq = torch.cat([p[:, :2], torch.zeros_like(p[:, :1])], 1)
    out = torch.where(is_(ELLIPSE), _unit(local * pq) * pq, out)
    rim = (flat * local).sum(1, keepdim=True) * rad >= local[:, 2:] * height
    out = torch.where(is_(CONE), torch.where(rim, flat * rad, z * height), out)
    poly = ((ty == HULL) | (ty == MESH)).nonzero().flatten()
    if len(poly):
        cnt, off = c.count[idx[poly]], c.offset[idx[poly]]
        owner = torch.repeat_interleave(torch.arange(len(poly), device="cuda"), cnt)
        start = torch.cumsum(cnt, 0) - cnt
        row = off[owner] + torch.arange(len(owner), device="cuda") - start[owner]
        s = (c.verts[row] * local[poly][owner]).sum(1)
        top = torch.full((len(poly),), -math.inf, device="cuda", dtype=torch.float64)
        top.scatter_reduce_(0, owner, s, "amax")
        best = torch.full((len(poly),), 1 << 60, device="cuda", dtype=torch.long)
        best.scatter_reduce_(0, owner, torch.where(s == top[owner], row, torch.full_like(row, 1 << 60)), "amin")
        out[poly] = c.verts[best]
    out = (R * out[:, None, :]).sum(2) + t
    return out + torch.where(c.wrapped[idx][:, None], _unit(d) * p[:, 3:], torch.zeros_like(d))


_SUBSETS = [[0], [1], [2], [3], [0, 1], [0, 2], [0, 3], [1, 2], [1, 3], [2, 3], [0, 1, 2], [0, 1, 3], [0, 2, 3],
            [1, 2, 3]]


def _closest(Y, have):
    """Closest point to the origin of each simplex (rows Y where `have`), its
    squared length, the rows that carry it, and whether it encloses the origin."""
    best = torch.full((len(Y),), math.inf, device="cuda", dtype=torch.float64)
    v, used = torch.zeros(len(Y), 3, device="cuda", dtype=torch.float64), torch.zeros_like(have)
    for sub in _SUBSETS:
        ok = have[:, sub].all(1)
        a = Y[:, sub[0]]
        if len(sub) == 1:
            x = a
        elif len(sub) == 2:
            e = Y[:, sub[1]] - a
            s = -(a * e).sum(1) / (e * e).sum(1).clamp_min(1e-300)
            x = a + e * s[:, None]
            ok = ok & (s > 0) & (s < 1)
        else:
            e, f = Y[:, sub[1]] - a, Y[:, sub[2]] - a
            nrm = torch.linalg.cross(e, f)
            nn = (nrm * nrm).sum(1)
            s = (torch.linalg.cross(-a, f) * nrm).sum(1) / nn.clamp_min(1e-300)
            r = (torch.linalg.cross(e, -a) * nrm).sum(1) / nn.clamp_min(1e-300)
            x = nrm * ((a * nrm).sum(1) / nn.clamp_min(1e-300))[:, None]
            ok = ok & (nn > 1e-28 * (e * e).sum(1) * (f * f).sum(1)) & (s > 0) & (r > 0) & (s + r < 1)
        l = (x * x).sum(1)
        take = ok & (l < best)
        best = torch.where(take, l, best)
        v = torch.where(take[:, None], x, v)
        mask = torch.zeros(4, dtype=torch.bool, device="cuda")
        mask[sub] = True
        used = torch.where(take[:, None], mask[None], used)
    full = have.all(1)
    inside = full
    for i, j, k, o in ((0, 1, 2, 3), (0, 1, 3, 2), (0, 2, 3, 1), (1, 2, 3, 0)):
        nrm = torch.linalg.cross(Y[:, j] - Y[:, i], Y[:, k] - Y[:, i])
        up = Y[:, o] - Y[:, i]
        so, sv = -(nrm * Y[:, i]).sum(1), (nrm * up).sum(1)
        flat = sv.abs() <= 1e-9 * nrm.norm(dim=1) * up.norm(dim=1)
        inside = inside & (so * sv >= 0) & ~flat
    return v, best, used, inside


def _distances(ca, cb, i1, i2, rounds=250):
    """Distance of each pair by GJK with an exhaustive sub-simplex search."""
    n = len(i1)
    dist = torch.zeros(n, device="cuda", dtype=torch.float64)
    for lo in range(0, n, 1 << 18):
        pid = torch.arange(lo, min(n, lo + (1 << 18)), device="cuda")
        a, b = i1[pid], i2[pid]
        d = torch.zeros(len(pid), 3, device="cuda", dtype=torch.float64)
        d[:, 0] = 1.0
        Y = torch.zeros(len(pid), 4, 3, device="cuda", dtype=torch.float64)
        have = torch.zeros(len(pid), 4, device="cuda", dtype=torch.bool)
        Y[:, 0] = _support(ca, a, d) - _support(cb, b, -d)
        have[:, 0] = True
        v = Y[:, 0].clone()
        vv = (v * v).sum(1)
        for _ in range(rounds):
            if not len(pid):
                break
            w = _support(ca, a, -v) - _support(cb, b, v)
            done = (vv - (v * w).sum(1) <= 1e-13 * vv) | (vv <= 1e-24)
            slot = (~have).to(torch.int8).argmax(1)
            rows = torch.arange(len(pid), device="cuda")
            Y2, have2 = Y.clone(), have.clone()
            Y2[rows, slot] = w
            have2[rows, slot] = True
            nv, nvv, used, inside = _closest(Y2, have2)
            stuck = ~inside & (nvv >= vv * (1 - 1e-15))
            end = done | stuck | inside
            dist[pid[end]] = torch.where(inside & ~done, 0.0, torch.sqrt(vv))[end]
            go = ~end
            pid, a, b = pid[go], a[go], b[go]
            Y, have, v, vv = Y2[go], used[go], nv[go], nvv[go]
        dist[pid] = torch.sqrt(vv) if len(pid) else dist[pid]
    # touching pairs come back at the rounding of the search
    return torch.where(dist < 1e-10, torch.zeros_like(dist), dist)


def _aabbs(c):
    n = len(c.types)
    idx = torch.arange(n, device="cuda")
    e = torch.eye(3, device="cuda", dtype=torch.float64)
    hi = torch.stack([_support(c, idx, e[k].expand(n, 3))[:, k] for k in range(3)], 1)
    lo = torch.stack([_support(c, idx, -e[k].expand(n, 3))[:, k] for k in range(3)], 1)
    # the reference's box of an ellipsoid is not its extent: the largest entry per axis of R diag(radii) R^T
    ell = (c.types == ELLIPSOID)[:, None]
    m = torch.where(c.wrapped, c.params[:, 3], torch.zeros_like(c.params[:, 3]))[:, None]
    ext = (c.R @ (c.R * c.params[:, None, :3]).transpose(1, 2)).amax(1)
    lo, hi = torch.where(ell, c.t - ext - m, lo), torch.where(ell, c.t + ext + m, hi)
    # a cone's: its base disk's box and its tip
    cone = (c.types == CONE)[:, None]
    ax, r, h = c.R[:, :, 2], c.params[:, :1], c.params[:, 1:2]
    ext = torch.sqrt((1 - ax * ax).clamp_min(0)) * r
    lo = torch.where(cone, torch.minimum(c.t - ext, c.t + h * ax) - m, lo)
    hi = torch.where(cone, torch.maximum(c.t + ext, c.t + h * ax) + m, hi)
    return lo, hi


def _overlaps(lo, hi):
    """Every pair i < j whose closed boxes overlap, ascending."""
    n, got = len(lo), []
    for a in range(0, n, 2048):
        b = min(n, a + 2048)
        hit = torch.ones(b - a, n - a, device="cuda", dtype=torch.bool)
        for k in range(3):
            hit &= (lo[a:b, k, None] <= hi[None, a:, k]) & (hi[a:b, k, None] >= lo[None, a:, k])
        i, j = hit.nonzero(as_tuple=True)
        keep = j > i
        got.append(torch.stack([i[keep] + a, j[keep] + a], 1))
    pairs = torch.cat(got)
    return pairs[:, 0], pairs[:, 1]


def _posed(axis, origin, link, body, types, params, q):
    """The arm's bodies at joint values q, as colliders."""
    dev = dict(device="cuda", dtype=torch.float64)
    q = torch.tensor(q, **dev)
    n, nb = len(q), len(link)

    def frame(x):
        T = torch.eye(4, **dev)
        T[:3, :3] = torch.tensor(x[:9].reshape(3, 3), **dev)
        T[:3, 3] = torch.tensor(x[9:], **dev)
        return T
    T = torch.eye(4, **dev).expand(n, 4, 4)
    frames = [T]
    for j in range(len(axis)):
        x, y, z = axis[j]
        K = torch.tensor([[0, -z, y], [z, 0, -x], [-y, x, 0]], **dev)
        J = torch.eye(4, **dev).repeat(n, 1, 1)
        J[:, :3, :3] += torch.sin(q[:, j])[:, None, None] * K + (1 - torch.cos(q[:, j]))[:, None, None] * (K @ K)
        T = T @ frame(origin[j]) @ J
        frames.append(T)
    all_ = torch.stack([frames[link[b]] @ frame(body[b]) for b in range(nb)], 1).reshape(n * nb, 4, 4)
    c = _Colliders()
    c.types = torch.tensor(types, device="cuda").long().repeat(n)
    c.R, c.t = all_[:, :3, :3].contiguous(), all_[:, :3, 3].contiguous()
    c.params = torch.tensor(params, **dev).repeat(n, 1)
    c.count = torch.zeros(n * nb, device="cuda", dtype=torch.long)
    c.offset = c.count - 1
    c.verts = torch.zeros(0, 3, **dev)
    c.wrapped = torch.zeros(n * nb, device="cuda", dtype=torch.bool)
    return c
