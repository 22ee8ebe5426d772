"""The ordered traversal of the wide tree against preorder traversal, bit for bit: its steps on the host
(wfb_test_traverse_ordered) against the oracle's traversal (WVM/include/wf/bvh.hpp:91-116), and on a
B200 the films it makes against those of the plain preorder steps (speculation off). No tolerance: both
sides run the same primitive tests, so a hit is the same bits or a different hit."""
import zlib

import numpy as np
import pytest

from test_traversal_steps import _coplanar_quads, _rays, _same


def _ball_scene(wfb, n_balls, seed, width=48, height=27):
    """Cornell box with balls of every material among its triangles (leaves of spheres, triangles and both)."""
    rng = np.random.default_rng(seed)
    a = wfb.Scene.generate("cornell36", width, height, 1234, 16).export()
    mats = np.zeros(len(a["materials"]) + 2, wfb.MATERIAL)
    mats[:-2] = a["materials"]
    mats[-2]["type"], mats[-2]["ior"], mats[-2]["albedo"] = 1, 1.0, (0.9, 0.8, 0.7)
    mats[-1]["type"], mats[-1]["ior"], mats[-1]["albedo"] = 2, 1.5, (1.0, 1.0, 1.0)
    balls = np.zeros(n_balls, wfb.SPHERE)
    balls["center"] = rng.uniform(0.1, 0.9, (n_balls, 3))
    balls["radius"] = rng.uniform(0.01, 0.12, n_balls)
    balls["material"] = rng.choice([0, len(mats) - 2, len(mats) - 1], n_balls)
    arrays = dict(a, spheres=balls, materials=mats, nodes=None, prim_order=None, lights=None)
    scene = wfb.Scene.from_arrays(arrays, finalize_bins=8)
    return scene, dict(arrays, **{k: scene.export()[k] for k in ("nodes", "prim_order", "lights")})


def _broken(arrays, how):
    """Trees that do not qualify: a leaf box that leaves its parent's, one that misses part of its primitive
    (shrunk, so the boxes still nest), one primitive entry in two leaves."""
    nodes = arrays["nodes"].copy()
    leaves = np.flatnonzero(nodes["prim_count"] > 0)
    if how == "grown":
        nodes["hi"][leaves[0]] += np.float32(1.0)
    elif how == "shrunk":
        leaf = leaves[len(leaves) // 2]
        ax = int(np.argmax(nodes["hi"][leaf] - nodes["lo"][leaf]))
        nodes["hi"][leaf, ax] = 0.5 * (nodes["hi"][leaf, ax] + nodes["lo"][leaf, ax])
    else:
        nodes["lo"][leaves[1]] = np.minimum(nodes["lo"][leaves[0]], nodes["lo"][leaves[1]])
        nodes["hi"][leaves[1]] = np.maximum(nodes["hi"][leaves[0]], nodes["hi"][leaves[1]])
        nodes["prim_start"][leaves[1]] = nodes["prim_start"][leaves[0]]
    return dict(arrays, nodes=nodes)


def _arrays(wfb, name):
    if name == "balls":
        return _ball_scene(wfb, 300, 3)[1]
    if name == "one_leaf":
        return _ball_scene(wfb, 0, 3)[1] | _single_triangle(wfb)
    return wfb.Scene.generate(name, 16, 9, 1234, 16).export()


def _single_triangle(wfb):
    """A scene of one triangle: the root is a leaf, the wide tree a single node with one child."""
    a = wfb.Scene.generate("cornell36", 16, 9, 1234, 16).export()
    one = dict(a, triangles=a["triangles"][:1].copy(), nodes=None, prim_order=None, lights=None)
    scene = wfb.Scene.from_arrays(one, finalize_bins=8)
    return dict(one, **{k: scene.export()[k] for k in ("nodes", "prim_order", "lights")})


@pytest.mark.parametrize("name", ["cornell36", "icospheres", "balls", "one_leaf"])
@pytest.mark.parametrize("anyhit", [False, True])
def test_ordered_traversal_equals_preorder(wfb, orc, name, anyhit):
    arrays = _arrays(wfb, name)
    scene = wfb.Scene.from_arrays(arrays)
    rays = _rays(wfb, arrays, 6000, seed=zlib.crc32(f"ordered/{name}/{anyhit}".encode()))
    if anyhit:
        rays["tmax"] = np.where(np.arange(len(rays)) % 2, np.float32(0.7), rays["tmax"])
    want = orc.intersect(arrays, rays, anyhit=anyhit)
    got, counts = scene.test_traverse_ordered(rays, anyhit=anyhit)
    assert counts["tree"] > 0
    # half of the rays have a zero direction component and take the preorder steps; most others do not
    assert counts["redone"] < 0.6 * len(rays)
    if anyhit:
        assert np.array_equal(got["prim"] >= 0, want["prim"] >= 0)
    else:
        assert _same(got, want)


def test_ordered_traversal_on_coplanar_quads(wfb, orc):
    """Hits of many leaves within a few ulp of each other: ties, and leaf boxes entered after their own hits."""
    scene, arrays = _coplanar_quads(wfb, seed=1)
    rng = np.random.default_rng(3)
    n = 100000
    o = np.stack([rng.uniform(-3, 0.5, n), rng.uniform(-2, 2, n), rng.uniform(-2, 2, n)], 1)
    tgt = np.stack([np.ones(n), rng.uniform(-1, 2, n), rng.uniform(-1, 2, n)], 1)
    d = (tgt - o) / np.linalg.norm(tgt - o, axis=1, keepdims=True)
    rays = np.zeros(n, wfb.RAY)
    rays["o"], rays["d"] = o.astype(np.float32), d.astype(np.float32)
    rays["tmin"], rays["tmax"] = np.float32(1e-4), np.float32(3.402823466e38)
    got, counts = scene.test_traverse_ordered(rays)
    assert counts["redone"] > 0  # the ties do occur
    assert _same(got, orc.intersect(arrays, rays))


@pytest.mark.parametrize("how", ["grown", "shrunk", "shared"])
def test_trees_that_do_not_qualify(wfb, orc, how):
    arrays = _broken(_arrays(wfb, "icospheres"), how)
    scene = wfb.Scene.from_arrays(arrays)
    rays = _rays(wfb, arrays, 1500, seed=11)
    got, counts = scene.test_traverse_ordered(rays)
    assert counts["tree"] == 0 and counts["redone"] == len(rays)
    assert _same(got, orc.intersect(arrays, rays))


def _chain(wfb, n, overlap):
    """A BVH that is a chain: every internal node has one leaf and the rest. Triangles in a row along x; with `overlap`
    stacked along z instead, so that a ray along z meets every box."""
    rng = np.random.default_rng(n)
    base = wfb.Scene.generate("cornell36", 24, 16, 1234, 16).export()
    verts = np.zeros((3 * n, 3), np.float32)
    for k in range(n):
        at = np.array([0.5, 0.5, -0.01 * k] if overlap else [k / n, 0.5, 0.0])
        verts[3 * k : 3 * k + 3] = at + rng.uniform(-0.4, 0.4, (3, 3)) * ([1, 1, 0.001] if overlap else [1 / n, 1, 0.2])
    tris = np.zeros(n, wfb.TRIANGLE)
    tris["i0"], tris["i1"], tris["i2"] = np.arange(n) * 3, np.arange(n) * 3 + 1, np.arange(n) * 3 + 2
    lo, hi = verts.reshape(n, 3, 3).min(1), verts.reshape(n, 3, 3).max(1)
    nodes = np.zeros(2 * n - 1, wfb.BVH_NODE)
    nodes["prim_start"] = -1
    for k in range(n):
        leaf = 2 * k + 1 if k < n - 1 else 2 * k
        nodes["lo"][leaf], nodes["hi"][leaf] = lo[k], hi[k]
        nodes["prim_start"][leaf], nodes["prim_count"][leaf] = k, 1
        nodes["skip"][leaf] = leaf + 1 if k < n - 1 else -1
        if k < n - 1:
            nodes["lo"][2 * k], nodes["hi"][2 * k], nodes["skip"][2 * k] = lo[k:].min(0), hi[k:].max(0), -1
    return dict(base, vertices=verts, triangles=tris, spheres=np.zeros(0, wfb.SPHERE), nodes=nodes,
                prim_order=np.arange(n, dtype=np.int32), lights=np.zeros(0, wfb.LIGHT), env=[1.0, 0.9, 0.8])


# 2 triangles; one node and its levels in one block; several launches of levels and a lane stack that overflows
# (every box met, 3 leaves left behind per level); more levels than the wide tree may have
CHAINS = [(2, False), (100, True), (250, False), (250, True), (400, True)]


@pytest.mark.parametrize("n,overlap", CHAINS)
@pytest.mark.parametrize("anyhit", [False, True])
def test_ordered_traversal_on_chains(wfb, orc, n, overlap, anyhit):
    arrays = _chain(wfb, n, overlap)
    scene = wfb.Scene.from_arrays(arrays)
    rng = np.random.default_rng(5)
    rays = _rays(wfb, arrays, 1200, seed=n)
    rays["o"][600:] = rng.uniform([0.2, 0.2, 1.0], [0.8, 0.8, 2.0], (600, 3))  # along the stack, all boxes in a row
    rays["d"][600:] = np.array([0.01, 0.02, -0.9997], np.float32)
    rays["o"][900:, 2] -= np.float32(0.01 * n + 4.0)
    rays["d"][900:, 2] = np.float32(0.9997)
    want = orc.intersect(arrays, rays, anyhit=anyhit)
    got, _ = scene.test_traverse_ordered(rays, anyhit=anyhit)
    assert np.array_equal(got["prim"] >= 0, want["prim"] >= 0)
    if not anyhit:
        assert _same(got, want)


def _film(wfb, scene, mode, on, spp, depth, **knobs):
    r = wfb.GpuRenderer(scene, mode)
    if knobs:
        r.configure(**knobs)
    r.set_speculation(on)
    r.reset()
    r.run_passes(0, spp, wfb.RenderParams(spp=spp, seed=5, max_depth=depth))
    sums = r.download_sums()
    r.close()
    return np.concatenate([s.ravel() for s in sums]).view(np.uint32)


@pytest.mark.gpu
@pytest.mark.parametrize("n,overlap", CHAINS)
def test_films_of_chains(wfb, n, overlap):
    arrays = _chain(wfb, n, overlap)
    scene = wfb.Scene.from_arrays(arrays)
    for mode in (wfb.MEGAKERNEL, wfb.WAVEFRONT):
        assert np.array_equal(_film(wfb, scene, mode, True, 3, 8), _film(wfb, scene, mode, False, 3, 8))


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(256, 255), (256, 256), (256, 257)])
def test_downloads_either_side_of_the_staged_size(wfb, w, h):
    """Films below, at and above 1 MB of resolved bytes, whole and in parts, against the raw sums."""
    scene = wfb.Scene.generate("cornell36", w, h, 1234, 16)
    r = wfb.GpuRenderer(scene, wfb.MEGAKERNEL)
    out = r.render(wfb.RenderParams(spp=4, seed=2, max_depth=4))
    rgb, lum, lum2 = r.download_sums()
    inv = np.float32(1.0) / np.float32(4)
    assert np.array_equal(out.rgb.view(np.uint32), (rgb * inv).view(np.uint32))
    m, m2 = lum.astype(np.float64) / 4, lum2.astype(np.float64) / 4
    assert np.array_equal(out.lum_var, np.maximum(0.0, m2 - m * m).astype(np.float32))
    assert np.array_equal(r.download_mean(4).view(np.uint32), out.rgb.view(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("arm", ["megakernel", "wavefront"])
@pytest.mark.parametrize("case", ["cornell36", "icospheres", "balls", "one_leaf", "coplanar", "grown", "shrunk", "shared"])
def test_films_equal_the_preorder_steps(wfb, case, arm):
    """Odd sizes, one and several samples per pixel (the two commit paths), every launch variant of the
    megakernel on the first scene."""
    if case == "coplanar":
        _, arrays = _coplanar_quads(wfb, seed=1)
    elif case in ("grown", "shrunk", "shared"):
        arrays = _broken(_arrays(wfb, "icospheres"), case)
    else:
        arrays = _arrays(wfb, case)
    mode = wfb.MEGAKERNEL if arm == "megakernel" else wfb.WAVEFRONT
    for w, h, spp, depth in ((61, 37, 1, 8), (133, 75, 5, 8), (1, 1, 3, 2)):
        scene = wfb.Scene.from_arrays(dict(arrays, width=w, height=h))
        want = _film(wfb, scene, mode, False, spp, depth)
        assert np.array_equal(_film(wfb, scene, mode, True, spp, depth), want), (w, h, spp)
        if case == "cornell36" and arm == "megakernel":
            for block, occupancy, min_active in ((64, 0, 1), (256, 0, 32), (128, 6, 4), (128, 8, 16), (128, 10, 8)):
                got = _film(wfb, scene, mode, True, spp, depth, block=block, occupancy=occupancy, min_active=min_active)
                assert np.array_equal(got, want), (w, h, spp, block, occupancy, min_active)
