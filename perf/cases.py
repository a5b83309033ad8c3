"""The work that users of this library have it do, as cases that can be timed.

A case is one call (or the few calls that belong together) through the public
Python layer: device traces of ray batches in each walk, with and without the
access traces; the host-buffer calls a simulator makes; a batch of scenes in
one launch; the RT-unit replay and prefetch decision that consume the traces;
and the treelet predictor's loss and gradients.  Scenes, ray batches and sizes
are those of the benchmark and the tests, or smaller ones of the same kind.

Scenes are kept from one preparation to the next, as a program that traces many
batches keeps its scene; rays, traces, parameters and samples are made anew
from the seed.
"""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "treelet-prefetching-for-rt_gb300"))

import treelet_rt as rt  # noqa: E402
from treelet_rt import learned  # noqa: E402

BUDGET = 8192  # bytes per treelet, the reference's default
SCENES = {"terrain": rt.SCENE_TERRAIN_INSTANCES, "cube_plane": rt.SCENE_CUBE_PLANE, "blobs": rt.SCENE_BLOBS,
          "cube": rt.SCENE_CUBE, "shared": rt.SCENE_SHARED_BLAS}
MODES = {"plain": rt.MODE_PLAIN, "treelet": rt.MODE_TREELET, "staged": rt.MODE_STAGED}
# transactions a ray makes, rounded (from the walks' own counts on these scenes)
VISITS = {"primary": 51, "bounce": 60, "ao": 40}


def listed():
    return [
        # one simulated warp handed over from the cycle loop, its transaction lists wanted back at once
        {"name": "warp_host_traced", "path": "packed", "scene": "cube_plane", "tris": 16384, "width": 8, "height": 4,
         "spp": 1, "rays": "primary", "mode": "treelet", "capacity": 256},
        # the frame sizes that cycle-level simulation can afford, traces for the timing model
        {"name": "frame_64x64_traced", "path": "trace", "scene": "terrain", "tris": 131072, "width": 64, "height": 64,
         "spp": 1, "rays": "primary", "mode": "treelet", "capacity": 256},
        # an odd-sized preview frame's bounce rays, hits only
        {"name": "bounce_251x187_plain", "path": "trace", "scene": "terrain", "tris": 131072, "width": 251,
         "height": 187, "spp": 1, "rays": "bounce", "mode": "plain", "capacity": 0},
        # the benchmark's frame: 2M-triangle terrain with 64 instances, 1024 x 1024 x 2 primary rays
        {"name": "primary_2m_staged", "path": "trace", "scene": "terrain", "tris": 2097152, "width": 1024,
         "height": 1024, "spp": 2, "rays": "primary", "mode": "staged", "capacity": 0},
        # its bounce rays, the incoherent half of the frame, in the reference's default order
        {"name": "bounce_2m_plain", "path": "trace", "scene": "terrain", "tris": 2097152, "width": 1024,
         "height": 1024, "spp": 2, "rays": "bounce", "mode": "plain", "capacity": 0},
        # bounce rays with both traces written, what the reference hands its timing model for every ray
        {"name": "bounce_1m_treelet_traced", "path": "trace", "scene": "terrain", "tris": 2097152, "width": 1024,
         "height": 1024, "spp": 1, "rays": "bounce", "mode": "treelet", "capacity": 256},
        # ambient occlusion: short any-hit rays, four per primary hit
        {"name": "ao_treelet", "path": "trace", "scene": "blobs", "tris": 1000000, "width": 960, "height": 540,
         "spp": 1, "rays": "ao", "mode": "treelet", "capacity": 0},
        # host buffers in, hits and packed per-ray transaction lists out
        {"name": "packed_host_640x480", "path": "packed", "scene": "terrain", "tris": 131072, "width": 640,
         "height": 480, "spp": 1, "rays": "primary", "mode": "treelet", "capacity": 256},
        # many scenes of very different sizes in one launch
        {"name": "batch_48_scenes", "path": "batch", "scenes": 48, "tris": 300000, "rays": "mixed", "mode": "treelet"},
        # the traces' consumer: RT units replayed with treelet prefetching
        {"name": "replay_4096", "path": "replay", "scene": "terrain", "tris": 131072, "width": 64, "height": 32,
         "units": 16, "prefetcher": rt.UNIT_PF_TREELET},
        # the RT units' prefetch decision for one simulated GPU, 16 resident warps each
        {"name": "decide_152x512", "path": "decide", "scene": "terrain", "tris": 131072, "units": 152, "lanes": 512},
        # the predictor's forward and backward on a full mini-batch of treelet transitions
        {"name": "predictor_grad_4096", "path": "grad", "scene": "cube", "tris": 60000, "n": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["trace"] * 7 + ["host", "packed", "batch", "replay", "decide", "grad"])
    if path == "grad":
        return {"path": path, "scene": "cube", "tris": _log(rng, 2000, 60000), "n": _log(rng, 33, 4096)}
    if path == "decide":
        return {"path": path, "scene": rng.choice(["cube_plane", "terrain"]), "tris": _log(rng, 4000, 131072),
                "units": _log(rng, 1, 152), "lanes": rng.randint(32, 512)}
    if path == "replay":
        return {"path": path, "scene": rng.choice(["cube_plane", "terrain"]), "tris": _log(rng, 4000, 131072),
                "width": rng.randint(16, 60), "height": rng.randint(8, 32), "units": rng.choice([4, 8, 16, 30]),
                "prefetcher": rng.choice([rt.UNIT_PF_NONE, rt.UNIT_PF_TREELET, rt.UNIT_PF_TREELET, rt.UNIT_PF_STRIDE])}
    if path == "batch":
        return {"path": path, "scenes": rng.randint(3, 48), "tris": _log(rng, 5000, 300000), "rays": "mixed",
                "mode": rng.choice(["plain", "treelet"])}
    c = {"path": path, "scene": rng.choice(["terrain", "terrain", "cube_plane", "blobs", "shared"]),
         "tris": _log(rng, 1000, 2000000), "width": 1, "height": 1, "spp": 1,
         "rays": rng.choice(["primary", "bounce", "bounce", "ao"]), "mode": rng.choice(list(MODES)), "capacity": 0}
    if c["scene"] == "shared":
        c["tris"] = min(c["tris"], 200000)
    pixels = {"host": (32, 20000), "packed": (32, 300000), "trace": (32, 900000)}[path]
    n = _log(rng, *pixels)
    if c["rays"] == "ao":  # four rays a hit
        n = max(32, n // 4)
    c["width"] = max(1, int(math.sqrt(n * rng.uniform(0.6, 1.8))))
    c["height"] = max(1, n // c["width"])
    if path == "packed" or (path == "trace" and rng.random() < 0.4):
        c["capacity"] = rng.choice([64, 250, 256])
    return c


@functools.lru_cache(maxsize=1)
def _context():
    return rt.Context(0)


@functools.lru_cache(maxsize=12)
def _scene(kind, tris):
    scene = rt.Scene(_context(), rt.Blob.gen(SCENES[kind], tris, 1))
    scene.form_treelets(BUDGET)
    return scene


@functools.lru_cache(maxsize=2)
def _batch_scenes(count, tris):
    sizes = np.exp(np.random.default_rng(1).uniform(np.log(1000), np.log(tris), count)).astype(int)
    made = []
    for k, t in enumerate(sizes):
        scene = rt.Scene(_context(), rt.Blob.gen(rt.SCENE_CUBE, int(t), k + 1))
        scene.form_treelets(BUDGET)
        made.append(scene)
    return made


def _bytes(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()).cuda()


def _rays(scene, kind, width, height, spp, what, seed):
    """Device rays (a uint8 tensor of 32-byte rays): jittered camera rays, or rays from their hits."""
    cam = rt.default_camera(SCENES[kind])
    prim = rt.camera_rays(cam, width, height, spp, seed + 1, 1e-4, 1e30)
    d = _bytes(prim)
    if what == "primary":
        return d
    n = len(prim)
    hits = torch.empty(n * 64, dtype=torch.uint8, device="cuda")
    scene.trace(d, hits, rt.MODE_PLAIN, n=n)
    if what == "ao":
        # four rays a hit, as many hits as pixels (the frame's hits taken round and round)
        hit = torch.nonzero(hits.view(torch.int32).view(n, 16)[:, 0] != 0).view(-1)
        if hit.numel() == 0:
            hit = torch.arange(n, device="cuda")
        pick = hit[torch.arange(n, device="cuda") % hit.numel()].repeat_interleave(4)
        d = d.view(n, 32)[pick].view(-1)
        hits = hits.view(n, 64)[pick].view(-1)
        n *= 4
    out = torch.empty(n * 32, dtype=torch.uint8, device="cuda")
    scene.bounce(d, hits, out, seed=seed + 7, tmin=1e-4, tmax=0.1 if what == "ao" else 1e30, n=n)
    torch.cuda.synchronize()
    return out


def _treelet_traces(scene, kind, width, height, seed, capacity=256):
    """Primary and bounce rays of a frame, their hit records and treelet-order traces."""
    prim = _rays(scene, kind, width, height, 1, "primary", seed)
    rays = torch.cat([prim, _rays(scene, kind, width, height, 1, "bounce", seed)])
    n = rays.numel() // 32
    hits = torch.zeros(n * 64, dtype=torch.uint8, device="cuda")
    visits = torch.zeros((n, capacity), dtype=torch.int32, device="cuda")
    treelets = torch.zeros((n, capacity), dtype=torch.int32, device="cuda")
    scene.trace(rays, hits, rt.MODE_TREELET, visits=visits, treelets=treelets, capacity=capacity, n=n)
    torch.cuda.synchronize()
    return rays, hits, visits, treelets, n


def _grad_inputs(case, seed):
    """Parameters and transitions: what a partly trained predictor and its next mini-batch hold."""
    scene = _scene(case["scene"], case["tris"])
    c = scene.treelet_info["n_treelets"]
    rays, hits, _, treelets, n = _treelet_traces(scene, case["scene"], 96, 96, seed)
    trans = learned.transitions(rays.cpu().numpy().view(rt.RAY_DTYPE), hits.cpu().numpy().view(rt.HIT_DTYPE),
                                treelets.cpu().numpy().view(np.uint32), scene.treelets()["roots"])
    rng = np.random.default_rng(seed)
    samples = trans[rng.integers(0, len(trans), case["n"])]
    scale = np.concatenate([np.full(16 * c, 0.1), np.full(22 * 64, 0.2), np.full(64, 0.05), np.full(64 * 64, 0.125),
                            np.full(64, 0.05), np.full(64 * c, 0.125), np.full(c, 0.05)])
    params = (rng.uniform(-1, 1, len(scale)) * scale).astype(np.float32)
    return c, params, samples


def prepare(case, seed):
    path = case["path"]
    if path == "batch":
        scenes = _batch_scenes(case["scenes"], case["tris"])
        rng = np.random.default_rng(1)  # the batches' sizes are the case's, their rays the seed's
        parts, begin = [], [0]
        for k, s in enumerate(scenes):
            half = int(np.exp(rng.uniform(np.log(2048), np.log(24576))))
            w = max(8, int(math.sqrt(half)))
            for what in ("primary", "bounce"):
                parts.append(_rays(s, "cube", w, max(4, half // w), 1, what, seed + 64 * k))
            begin.append(begin[-1] + (parts[-1].numel() + parts[-2].numel()) // 32)
        batch = rt.Batch(_context(), scenes)
        batch.set_items(begin, list(range(len(scenes))))
        rays = torch.cat(parts)
        return {"path": path, "batch": batch, "rays": rays, "mode": MODES[case["mode"]],
                "hits": torch.zeros(rays.numel() * 2, dtype=torch.uint8, device="cuda")}
    scene = _scene(case["scene"], case["tris"])
    if path == "grad":
        c, params, samples = _grad_inputs(case, seed)
        mlp = learned.Mlp(_context(), c, 1)
        mlp.set_params(params)
        return {"path": path, "mlp": mlp, "samples": _bytes(samples), "n": case["n"]}
    if path == "replay":
        _, hits, visits, _, n = _treelet_traces(scene, case["scene"], case["width"], case["height"], seed)
        # the stride prefetcher queues only while its queue holds at least max_queue requests
        limit = 0 if case["prefetcher"] == rt.UNIT_PF_STRIDE else 4096
        cfg = rt.unit_config(n_rt_units=case["units"], prefetcher=case["prefetcher"], max_queue=limit)
        stats = torch.zeros(case["units"] * rt.UNIT_STATS_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
        return {"path": path, "scene": scene, "hits": hits, "visits": visits, "n": n, "cfg": cfg, "stats": stats}
    if path == "decide":
        units, lanes = case["units"], case["lanes"]
        _, hits, visits, _, n = _treelet_traces(scene, case["scene"], 128, 64, seed)
        g = torch.Generator(device="cuda").manual_seed(seed)
        # resident warps are 32 neighbouring rays, each at some transaction of its list; one lane in eight is idle
        warp = torch.randint(0, n // 32, (units, (lanes + 31) // 32), device="cuda", generator=g)
        ray = (warp[:, :, None] * 32 + torch.arange(32, device="cuda")).reshape(units, -1)[:, :lanes].reshape(-1)
        count = hits.view(torch.int32).view(n, 16)[:, 11].long()[ray].clamp(1, 256)
        at = (torch.rand(ray.numel(), device="cuda", generator=g) * count).long()
        nxt = torch.bitwise_right_shift(visits[ray, at], 3)
        nxt[torch.rand(ray.numel(), device="cuda", generator=g) < 0.125] = -1
        state = torch.full((units, 4), -1, dtype=torch.int32, device="cuda")
        state[:, 3] = 0
        params = rt.PrefetchParams(0, 4096, 0.75, 1, rt.PREFETCH_MAIN_BLOCK)
        return {"path": path, "scene": scene, "next": nxt, "units": units, "lanes": lanes, "params": params,
                "unit_state": state, "out": torch.zeros((units, 8), dtype=torch.int32, device="cuda")}
    rays = _rays(scene, case["scene"], case["width"], case["height"], case["spp"], case["rays"], seed)
    n, cap = rays.numel() // 32, case["capacity"]
    state = {"path": path, "scene": scene, "n": n, "mode": MODES[case["mode"]], "cap": cap,
             "flags": rt.RAY_FLAG_OPAQUE | (rt.RAY_FLAG_TERMINATE_ON_FIRST_HIT if case["rays"] == "ao" else 0)}
    if path == "trace":
        state.update(rays=rays, hits=torch.zeros(n * 64, dtype=torch.uint8, device="cuda"))
        if cap:
            state["visits"] = torch.zeros((n, cap), dtype=torch.int32, device="cuda")
            state["treelets"] = torch.zeros((n, cap), dtype=torch.int32, device="cuda")
    elif path == "host":
        state["rays"] = rays.cpu().numpy().view(rt.RAY_DTYPE)
    else:  # the caller's own page-locked arrays, as the C interface takes them
        def pinned(count, dtype):
            return torch.zeros(count, dtype=dtype).pin_memory()
        state["room"] = 160 * n
        state.update(rays=rays.cpu().pin_memory(), hits=pinned(16 * n, torch.int32), offsets=pinned(n + 1, torch.int64),
                     visits=pinned(state["room"], torch.int32), treelets=pinned(state["room"], torch.int32))
    return state


def run(state):
    path = state["path"]
    if path == "trace":
        state["scene"].trace(state["rays"], state["hits"], state["mode"], default_flags=state["flags"],
                             visits=state.get("visits"), treelets=state.get("treelets"), capacity=state["cap"],
                             stream=torch.cuda.current_stream().cuda_stream, n=state["n"])
        out = {"hits": state["hits"].view(torch.int32)}
        if state["cap"]:
            out.update(visits=state["visits"], treelets=state["treelets"])
        return out
    if path == "host":
        hits, _, _ = state["scene"].trace_host(state["rays"], state["mode"], default_flags=state["flags"])
        return {"hits": hits.view(np.int32)}
    if path == "packed":
        total = ctypes.c_uint64(0)
        status = rt.lib().rt_trace_host_packed(
            state["scene"].handle, state["rays"].data_ptr(), None, state["flags"], state["n"], state["mode"],
            state["cap"], state["hits"].data_ptr(), state["offsets"].data_ptr(), state["visits"].data_ptr(),
            state["treelets"].data_ptr(), state["room"], ctypes.byref(total))
        if status:
            raise rt.RTError(status, rt.lib().rt_last_error().decode())
        return {k: state[k] for k in ("hits", "offsets", "visits", "treelets")}
    if path == "batch":
        state["batch"].trace(state["rays"], state["hits"], state["mode"],
                             stream=torch.cuda.current_stream().cuda_stream)
        return {"hits": state["hits"].view(torch.int32)}
    if path == "replay":
        state["scene"].unit_replay(state["hits"], state["visits"], state["n"], 256, state["cfg"], state["stats"],
                                   stream=torch.cuda.current_stream().cuda_stream)
        return {"stats": state["stats"].view(torch.int64)}
    if path == "decide":
        state["scene"].prefetch_decide(state["next"], state["units"], state["lanes"], state["params"],
                                       state["unit_state"], state["out"],
                                       stream=torch.cuda.current_stream().cuda_stream)
        return {"decisions": state["out"], "state": state["unit_state"]}
    loss, grads = state["mlp"].loss_grad(state["samples"], state["n"])
    return {"loss": loss, "grads": grads}


def work(case):
    """Rays, the scene's nodes and the outputs once each; six slab tests of 24 operations an internal node."""
    path = case["path"]
    if path == "grad":
        c, n = 0.44 * case["tris"], case["n"]
        return {"bytes": 4 * 81 * c * 2 + 32 * n, "flops": 2 * n * (3 * 64 * c + 3 * (22 * 64 + 64 * 64))}
    if path == "decide":
        return {"bytes": case["units"] * (case["lanes"] * 12 + 64), "flops": 0}
    if path == "replay":
        n = 2 * case["width"] * case["height"]
        return {"bytes": n * (64 + 4 * 55) + 184 * case["units"], "flops": 0}
    if path == "batch":
        n, visits, scene = 2 * 9000 * case["scenes"], 45, 20e3 * case["scenes"] * 88
    else:
        n = case["width"] * case["height"] * case["spp"] * (4 if case["rays"] == "ao" else 1)
        visits, scene = VISITS[case["rays"]], 88 * case["tris"]
    traced = 8 * visits * n if case.get("capacity") else 0
    return {"bytes": 96 * n + traced + min(scene, 64 * visits * n), "flops": n * visits * 0.7 * 6 * 24}


def exact(case, seed):
    """The predictor's loss and gradients in 64 bits; the other paths' outputs are bit patterns with no tolerance."""
    if case["path"] != "grad":
        return None
    c, params, samples = _grad_inputs(case, seed)
    p = torch.from_numpy(params).cuda().double().requires_grad_(True)
    e, w1, b1, w2, b2, w3, b3 = torch.split(p, [16 * c, 22 * 64, 64, 64 * 64, 64, 64 * c, c])
    s = {k: torch.from_numpy(np.ascontiguousarray(samples[k]).astype(np.float64 if k in ("origin", "dir")
                                                                     else np.int64)).cuda() for k in samples.dtype.names}
    x = torch.cat([s["origin"], s["dir"], e.view(c, 16)[s["current"]]], dim=1)
    h = torch.nn.functional.gelu(x @ w1.view(22, 64) + b1)
    h = torch.nn.functional.gelu(h @ w2.view(64, 64) + b2)
    loss = torch.nn.functional.cross_entropy(h @ w3.view(64, c) + b3, s["target"])
    loss.backward()
    return {"loss": float(loss), "grads": p.grad}
