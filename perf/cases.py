"""Performance cases: what a user of the path-tracing engine has it do, through its public entry points.

A case is a plain dict with a "kind":

  render       one whole film: GpuRenderer.render on a renderer the program keeps (either arm)
  progressive  an interactive preview: reset, then passes of a few samples each, then the film
  frame        a new scene per frame: Scene.from_arrays, GpuRenderer, render, close
  batch        many jobs in one persistent launch: Batch.clear/add/run and every job's film
  serve        a burst of jobs into the continuous-batching Server, collected as they finish
  queue        the stream-ordered queue primitives: exclusive scan and stable compaction of uint32

listed() holds one case per kind and size that stands for a use; draw() takes more of the same
ranges; prepare() makes the scene, renderer, batch, server or device arrays from a seed; run() is one
pass and returns its films or arrays; work() is what a pass cannot do without; exact() gives the
64-bit values where there are any (the films are Monte Carlo estimates whose paths branch on every
rounding, so they have none).
"""
import importlib
import math

import numpy as np
import torch

wfb = importlib.import_module("graphics-book-tutorials_b200")

SCENES = wfb.MIX_SCENES
# (primitives, rays per sample at depth 8) of the generated scenes: camera, bounce and shadow rays
SCENE_FACTS = {"cornell36": (36, 6.0), "icospheres": (163844, 2.7), "heightfield": (2093060, 2.2)}


def listed():
    return [
        # the smallest call: a thumbnail of a 36-triangle scene, one sample per pixel
        {"name": "thumbnail", "kind": "render", "scene": "cornell36", "arm": "megakernel",
         "width": 64, "height": 36, "spp": 1, "depth": 8},
        # the Cornell box preview of the benchmark's first configuration
        {"name": "cornell_preview", "kind": "render", "scene": "cornell36", "arm": "megakernel",
         "width": 320, "height": 180, "spp": 16, "depth": 8},
        # the benchmark's headline frame: mixed materials, 164K triangles
        {"name": "icospheres_720p", "kind": "render", "scene": "icospheres", "arm": "megakernel",
         "width": 1280, "height": 720, "spp": 64, "depth": 8},
        # the benchmark's large scene: 2.1M triangles, sky and sun
        {"name": "heightfield_720p", "kind": "render", "scene": "heightfield", "arm": "megakernel",
         "width": 1280, "height": 720, "spp": 64, "depth": 8},
        # the largest job of the benchmark's job mix, at its shorter depth
        {"name": "icospheres_1080p", "kind": "render", "scene": "icospheres", "arm": "megakernel",
         "width": 1920, "height": 1080, "spp": 64, "depth": 4},
        # the wavefront arm on the headline scene, an ordinary frame
        {"name": "wavefront_720p", "kind": "render", "scene": "icospheres", "arm": "wavefront",
         "width": 1280, "height": 720, "spp": 16, "depth": 8},
        # the wavefront arm on the small preview, where barriers and tails count
        {"name": "wavefront_preview", "kind": "render", "scene": "cornell36", "arm": "wavefront",
         "width": 320, "height": 180, "spp": 16, "depth": 8},
        # an interactive viewer in an odd-sized window: one sample per pixel and pass
        {"name": "viewer", "kind": "progressive", "scene": "heightfield", "arm": "megakernel",
         "width": 333, "height": 187, "passes": 6, "spp": 1, "depth": 8},
        # a changing scene: arrays in, film out, nothing kept between frames
        {"name": "new_scene_frame", "kind": "frame", "scene": "icospheres", "arm": "megakernel",
         "width": 640, "height": 360, "spp": 4, "depth": 8},
        # a render farm's batch: jobs of uneven size over all three scenes
        {"name": "batch_mix", "kind": "batch", "scene": "mix", "arm": "megakernel", "jobs": 16,
         "largest": 1280, "spp": 16},
        # a burst of requests at the render server
        {"name": "serve_burst", "kind": "serve", "scene": "mix", "arm": "megakernel", "jobs": 12,
         "largest": 640, "spp": 16},
        # queue primitives on a ragged array of flags and ids
        {"name": "queue_16m", "kind": "queue", "n": 16000003, "keep": 0.4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges: sizes spread over their logarithm, odd ones among them."""
    kind = rng.choice(["render", "render", "render", "render", "progressive", "frame", "batch", "serve", "queue"])
    if kind == "queue":
        return {"kind": kind, "n": _log_int(rng, 100, 16000003), "keep": round(rng.uniform(0.02, 0.98), 3)}
    if kind in ("batch", "serve"):
        return {"kind": kind, "scene": "mix", "arm": "megakernel", "jobs": rng.randint(3, 16 if kind == "batch" else 12),
                "largest": _log_int(rng, 256, 1280 if kind == "batch" else 640), "spp": _log_int(rng, 1, 16)}
    case = {"kind": kind, "scene": rng.choice(SCENES), "arm": "megakernel",
            "width": _log_int(rng, 40, 1920), "height": _log_int(rng, 24, 1080), "spp": _log_int(rng, 1, 64),
            "depth": rng.choice([1, 2, 4, 8, 8, 8])}
    if kind == "render" and rng.random() < 0.3:
        case["arm"] = "wavefront"
        case["spp"] = min(case["spp"], 16)
    if kind == "progressive":
        case.update(width=_log_int(rng, 40, 1280), height=_log_int(rng, 24, 720), spp=rng.randint(1, 4),
                    passes=rng.randint(2, 8))
    if kind == "frame":
        case.update(width=_log_int(rng, 40, 1280), height=_log_int(rng, 24, 720), spp=_log_int(rng, 1, 16),
                    scene=rng.choice(["cornell36", "icospheres"]))
    return case


def _mode(case):
    return wfb.WAVEFRONT if case["arm"] == "wavefront" else wfb.MEGAKERNEL


def _mix_jobs(case, seed):
    """Jobs like the benchmark's mix, up to `largest` pixels wide: scene, size, samples and depth are the
    case's own, cameras and sample seeds come from the seed."""
    shape, rng = np.random.default_rng(case["jobs"]), np.random.default_rng(seed)
    big = case["largest"]
    sizes = [(max(8, int(big * f)), max(8, int(big * f * 9 / 16))) for f in (0.2, 0.35, 0.6, 1.0)]
    spps = [max(1, int(case["spp"] * f)) for f in (0.1, 0.25, 0.5, 1.0)]
    # the server's scenes change often, so they are the two that build quickly
    scenes = SCENES if case["kind"] == "batch" else SCENES[:2]
    jobs = []
    for i in range(case["jobs"]):
        k = int(shape.integers(len(sizes)))
        jobs.append({"scene": scenes[i % len(scenes)], "width": sizes[k][0], "height": sizes[k][1],
                     "spp": spps[int(shape.integers(len(spps)))], "max_depth": (4, 8)[int(shape.integers(2))],
                     "seed": i + 1 + (seed & 0xFFFF), "azimuth": float(rng.uniform(0, 360)),
                     "elevation": float(rng.uniform(10, 40))})
    return scenes, jobs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "queue":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        n = case["n"]
        flags = (torch.rand(n, device="cuda", generator=gen) < case["keep"]).to(torch.int32)
        values = torch.randint(0, 2**31 - 1, (n,), device="cuda", generator=gen, dtype=torch.int32)
        return {"kind": kind, "n": n, "flags": flags, "values": values, "ws": wfb.ScanWorkspace(n),
                "scan": torch.zeros(n, dtype=torch.int32, device="cuda"),
                "kept": torch.zeros(n, dtype=torch.int32, device="cuda"),
                "counts": torch.zeros(2, dtype=torch.int32, device="cuda")}
    if kind in ("batch", "serve"):
        names, jobs = _mix_jobs(case, seed)
        scenes = {name: wfb.Scene.generate(name, 64, 36, seed) for name in names}
        work = [(scenes[j["scene"]], wfb.mix_job_desc(j, scenes[j["scene"]])) for j in jobs]
        if kind == "batch":
            return {"kind": kind, "work": work, "batch": wfb.Batch(max_jobs=max(16, len(jobs)), mode=_mode(case))}
        return {"kind": kind, "work": work, "server": wfb.Server(budget_bytes=2 << 30, max_jobs=64)}
    scene = wfb.Scene.generate(case["scene"], case["width"], case["height"], seed)
    params = wfb.RenderParams(spp=case["spp"] * case.get("passes", 1), seed=seed & 0xFFFFFF, max_depth=case["depth"])
    state = {"kind": kind, "params": params, "mode": _mode(case)}
    if kind == "frame":
        state["arrays"] = scene.export()
        return state
    state.update(renderer=wfb.GpuRenderer(scene, _mode(case)), passes=case.get("passes", 1), per_pass=case["spp"])
    return state


def _film(result):
    return [result.rgb, result.lum_var]


def run(state):
    kind = state["kind"]
    if kind == "render":
        return _film(state["renderer"].render(state["params"]))
    if kind == "progressive":
        r, k = state["renderer"], state["per_pass"]
        r.reset()
        for i in range(state["passes"]):
            r.run_passes(i * k, k, state["params"])
        return _film(r.download(state["passes"] * k))
    if kind == "frame":
        scene = wfb.Scene.from_arrays(state["arrays"])
        r = wfb.GpuRenderer(scene, state["mode"])
        film = _film(r.render(state["params"]))
        r.close()
        scene.close()
        return film
    if kind == "batch":
        b = state["batch"]
        b.clear()
        ids = [b.add(scene, job) for scene, job in state["work"]]
        b.run()
        return [_film(b.download(i)) for i in ids]
    if kind == "serve":
        s = state["server"]
        tickets = [s.submit(scene, job) for scene, job in state["work"]]
        films = []
        for t in tickets:
            s.wait(t)
            films.append(_film(s.result(t)[0]))
        return films
    n, ws = state["n"], state["ws"]
    flags, counts = state["flags"].data_ptr(), state["counts"].data_ptr()
    ws.scan_exclusive_u32(flags, state["scan"].data_ptr(), n, counts)
    ws.compact_u32(state["values"].data_ptr(), flags, state["kept"].data_ptr(), counts + 4, n)
    return [state["scan"], state["kept"], state["counts"]]


def _render_work(scene, width, height, spp, depth):
    """A film: every ray descends one root-to-leaf path (a slab test per level, 25 operations) and tests
    one primitive (50); a path event costs about 100 more. Memory: the scene is read once (or what its rays
    touch, if that is less) and the film, 16 bytes a pixel, written once."""
    prims, rays = SCENE_FACTS[scene]
    rays *= min(1.0, (depth + 1) / 4)
    n_rays = width * height * spp * rays
    levels = math.log2(prims)
    scene_bytes = min(prims * (2 * 32 + 48 + 16), n_rays * (32 * levels + 48))
    return {"bytes": scene_bytes + 16 * width * height, "flops": n_rays * (25 * levels + 150)}


def work(case):
    kind = case["kind"]
    if kind == "queue":
        # the scan reads the flags and writes the offsets; the compaction reads flags and values and
        # writes the kept ones
        n = case["n"]
        return {"bytes": 4 * n * (4 + case["keep"]), "flops": 2 * n}
    if kind in ("batch", "serve"):
        _, jobs = _mix_jobs(case, 1)
        parts = [_render_work(j["scene"], j["width"], j["height"], j["spp"], j["max_depth"]) for j in jobs]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    w = _render_work(case["scene"], case["width"], case["height"], case["spp"] * case.get("passes", 1), case["depth"])
    return {"bytes": float(w["bytes"]), "flops": float(w["flops"])}


def exact(case, seed):
    if case["kind"] != "queue":
        return None
    s = prepare(case, seed)
    flags = s["flags"].cpu().numpy().astype(np.int64)
    values = s["values"].cpu().numpy()
    scan = (np.cumsum(flags) - flags).astype(np.int32)
    kept = np.zeros(case["n"], np.int32)
    chosen = values[flags != 0]
    kept[: chosen.size] = chosen
    return [scan, kept, np.array([flags.sum(), chosen.size], np.int32)]
