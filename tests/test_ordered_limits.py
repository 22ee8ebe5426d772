"""Where the ordered traversal's hit may differ from preorder traversal's: only where the preorder hit is one whose reported t
lies in front of its own leaf's box, by more than the slack subtrees are skipped with (kCullSlack, wide_bvh.cuh). Rays that
graze the triangles of a smooth mesh and rays through slivers, where the triangle test's determinant is at the level of its
rounding. Any-hit queries have no such exception."""
import numpy as np
import pytest

CULL_SLACK = 1.0 + 1.0 / 1024.0


def _scene(wfb, verts):
    base = wfb.Scene.generate("cornell36", 24, 16, 1234, 16).export()
    verts = np.ascontiguousarray(verts, np.float32).reshape(-1, 3)
    tris = np.zeros(len(verts) // 3, wfb.TRIANGLE)
    tris["i0"], tris["i1"], tris["i2"] = (np.arange(len(tris)) * 3 + k for k in range(3))
    arrays = dict(base, vertices=verts, triangles=tris, spheres=np.zeros(0, wfb.SPHERE), nodes=None, prim_order=None,
                  lights=None)
    scene = wfb.Scene.from_arrays(arrays, finalize_bins=8)
    return scene, dict(arrays, **{k: scene.export()[k] for k in ("nodes", "prim_order", "lights")})


def _smooth_mesh():
    x, y = np.meshgrid(np.linspace(-1, 1, 61), np.linspace(-1, 1, 61), indexing="ij")
    p = np.stack([x, y, 0.05 * np.sin(5 * x) * np.cos(4 * y)], -1)
    a, b, c, d = p[:-1, :-1], p[1:, :-1], p[1:, 1:], p[:-1, 1:]
    return np.concatenate([np.stack(t, -2).reshape(-1, 3, 3) for t in ((a, b, c), (a, c, d))])


def _unit(rng, n):
    d = rng.normal(size=(n, 3))
    return d / np.linalg.norm(d, axis=1, keepdims=True)


def _slivers(rng, n=3000, width=1e-5):
    c, e = rng.uniform(-1, 1, (n, 1, 3)), _unit(rng, n)[:, None, :]
    v = np.concatenate([c, c + e * rng.uniform(0.5, 1, (n, 1, 1)), c + 0.5 * e + width * _unit(rng, n)[:, None, :]], 1)
    return np.take_along_axis(v, rng.permuted(np.tile(np.arange(3), (n, 1)), axis=1)[:, :, None], 1)


def _rays_at(wfb, rng, verts, d, distance):
    n = len(d)
    target = (verts * rng.dirichlet([1, 1, 1], n)[:, :, None]).sum(1)
    d = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.zeros(n, wfb.RAY)
    rays["o"], rays["d"] = target - d * distance, d
    rays["tmin"], rays["tmax"] = np.float32(1e-4), np.float32(3.402823466e38)
    return rays


def _leaf_entry(arrays, rays, prims):
    """Entry distance, in 64 bits, of the box of each given primitive's leaf."""
    nodes, order = arrays["nodes"], arrays["prim_order"]
    leaf_of = np.zeros(len(order), np.int64)
    for i in np.flatnonzero(nodes["prim_count"] > 0):
        leaf_of[order[nodes["prim_start"][i] : nodes["prim_start"][i] + nodes["prim_count"][i]]] = i
    box = nodes[leaf_of[prims]]
    o, d = rays["o"].astype(np.float64), rays["d"].astype(np.float64)
    t = np.stack([(box["lo"] - o) / d, (box["hi"] - o) / d])
    return t.min(0).max(1)


@pytest.mark.parametrize("case,n", [("grazing", 150000), ("slivers", 100000)])
def test_differences_are_hits_in_front_of_their_own_leaf(wfb, orc, case, n):
    rng = np.random.default_rng(8)
    verts = _smooth_mesh() if case == "grazing" else _slivers(rng)
    scene, arrays = _scene(wfb, verts)
    at = verts[rng.integers(0, len(verts), n)]
    d = _unit(rng, n)
    if case == "grazing":
        normal = np.cross(at[:, 1] - at[:, 0], at[:, 2] - at[:, 0])
        normal /= np.linalg.norm(normal, axis=1, keepdims=True)
        d -= normal * (d * normal).sum(1, keepdims=True)
        d = d / np.linalg.norm(d, axis=1, keepdims=True) + normal * 1e-5 * rng.normal(size=(n, 1))
        distance = 10 ** rng.uniform(-3, 1.5, (n, 1))
    else:
        distance = 30.0
    rays = _rays_at(wfb, rng, at, d, distance)
    want = orc.intersect(arrays, rays)
    got, counts = scene.test_traverse_ordered(rays)
    assert counts["tree"] > 0
    differ = (got["prim"] != want["prim"]) | (got["t"].view(np.uint32) != want["t"].view(np.uint32))
    assert differ.mean() < 1e-3
    if case == "grazing":
        assert differ.any()  # the exception does occur
    assert (want["prim"][differ] >= 0).all()
    entry = _leaf_entry(arrays, rays[differ], want["prim"][differ])
    assert (want["t"][differ] * CULL_SLACK < entry).all()
    any_got, _ = scene.test_traverse_ordered(rays, anyhit=True)
    assert np.array_equal(any_got["prim"] >= 0, orc.intersect(arrays, rays, anyhit=True)["prim"] >= 0)
