"""The ordered traversal on rays that come from far away compared with the boxes they pass, where the rounding of a slab
distance is longer than a whole wide node: hits against the oracle's preorder traversal (WVM/include/wf/bvh.hpp:91-116) on
the host, films against those of the plain preorder steps on the device. No tolerance."""
import numpy as np
import pytest

from test_traversal_steps import _same


def _cluster(wfb, half, distance, n=2000, width=40, height=24):
    """A cluster of small triangles of half-width `half` around the origin, a wall of two triangles behind it, and the camera
    at `distance`, its view as narrow as the cluster."""
    rng = np.random.default_rng(17)
    base = wfb.Scene.generate("cornell36", width, height, 1234, 16).export()
    at = rng.uniform(-half, half, (n, 1, 3))
    cluster = (at + rng.normal(0.0, 0.05 * half, (n, 3, 3))).reshape(-1, 3)
    side, z = 4.0 * half, -3.0 * half
    wall = np.array([[-side, -side, z], [side, -side, z], [side, side, z], [-side, side, z]])
    verts = np.concatenate([cluster, wall]).astype(np.float32)
    tris = np.zeros(n + 2, wfb.TRIANGLE)
    tris["i0"][:n], tris["i1"][:n], tris["i2"][:n] = (np.arange(n) * 3 + k for k in range(3))
    tris["i0"][n:], tris["i1"][n:], tris["i2"][n:] = 3 * n, (3 * n + 1, 3 * n + 2), (3 * n + 2, 3 * n + 3)
    arrays = dict(base, vertices=verts, triangles=tris, spheres=np.zeros(0, wfb.SPHERE), nodes=None, prim_order=None,
                  lights=None, env=[1.0, 0.9, 0.8], cam_position=[0.2 * distance, 0.3 * distance, distance],
                  cam_look_at=[0.0, 0.0, 0.0], cam_vfov_deg=float(np.degrees(3.0 * half / distance)))
    scene = wfb.Scene.from_arrays(arrays, finalize_bins=8)
    return scene, dict(arrays, **{k: scene.export()[k] for k in ("nodes", "prim_order", "lights")})


def _far_rays(wfb, half, distance, n, seed):
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n, 3))
    d[:, 2] = -np.abs(d[:, 2]) - 0.5
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    target = rng.uniform(-1.2 * half, 1.2 * half, (n, 3))
    rays = np.zeros(n, wfb.RAY)
    rays["o"] = (target - distance * d).astype(np.float32)
    rays["d"] = d.astype(np.float32)
    rays["tmin"], rays["tmax"] = np.float32(1e-4), np.float32(3.402823466e38)
    return rays


# extent over distance from 1e-3 (every box wider than a rounding) to 1e-7 (all of the cluster within a few)
FAR = [(1.0, 1e3), (0.01, 1e3), (0.01, 1e4), (0.1, 1e5), (1.0, 1e6), (0.001, 1e4)]


@pytest.mark.parametrize("half,distance", FAR)
@pytest.mark.parametrize("anyhit", [False, True])
def test_far_rays_equal_preorder(wfb, orc, half, distance, anyhit):
    scene, arrays = _cluster(wfb, half, distance)
    rays = _far_rays(wfb, half, distance, 20000, seed=3)
    want = orc.intersect(arrays, rays, anyhit=anyhit)
    got, counts = scene.test_traverse_ordered(rays, anyhit=anyhit)
    assert counts["tree"] > 0 and (want["prim"] >= 0).mean() > 0.1
    assert np.array_equal(got["prim"] >= 0, want["prim"] >= 0)
    if not anyhit:
        assert _same(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("half,distance", FAR)
def test_films_seen_from_far_away(wfb, half, distance):
    scene, _ = _cluster(wfb, half, distance)
    assert scene.wide_nodes() > 0
    for mode in (wfb.MEGAKERNEL, wfb.WAVEFRONT):
        films = []
        for on in (True, False):
            r = wfb.GpuRenderer(scene, mode)
            r.set_speculation(on)
            r.reset()
            r.run_passes(0, 4, wfb.RenderParams(spp=4, seed=5, max_depth=6))
            films.append(np.concatenate([s.ravel() for s in r.download_sums()]).view(np.uint32))
            r.close()
        assert np.array_equal(*films)
