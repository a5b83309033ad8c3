"""GPU RT-unit replay (rt_unit_replay, one CUDA thread per RT unit) against
the oracle's restatement of the same model: every counter of every unit
must be equal, on traces the GPU traversal produced."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CAP = 256


def _gpu_traces(ctx, kind, budget):
    import torch

    import treelet_rt as rt

    if kind == "cube_plane":
        blob = rt.Blob.gen(rt.SCENE_CUBE_PLANE, 8000, 2)
        cam = rt.default_camera(rt.SCENE_CUBE_PLANE)
        side = 48
    elif kind == "terrain":
        blob = rt.Blob.gen(rt.SCENE_TERRAIN_INSTANCES, 2 * 48 * 48, 5)
        cam = rt.default_camera(rt.SCENE_TERRAIN_INSTANCES)
        side = 40
    else:
        blob = rt.Blob.gen(rt.SCENE_SHARED_BLAS, 400, 4)
        cam = rt.default_camera(rt.SCENE_SHARED_BLAS)
        side = 40
    scene = rt.Scene(ctx, blob)
    scene.form_treelets(budget)
    prim = rt.camera_rays(cam, side, side, 1, 3, 1e-4, 1e30)
    n = len(prim)
    dp = torch.from_numpy(prim.view(np.uint8)).cuda()
    hp = torch.empty(n * 64, dtype=torch.uint8, device="cuda")
    scene.trace(dp, hp, rt.MODE_PLAIN, n=n)
    db = torch.empty(n * 32, dtype=torch.uint8, device="cuda")
    scene.bounce(dp, hp, db, seed=9, n=n)
    rays = torch.cat([dp, db])
    n2 = 2 * n
    hits = torch.empty(n2 * 64, dtype=torch.uint8, device="cuda")
    vis = torch.zeros(n2 * CAP, dtype=torch.int32, device="cuda")
    scene.trace(rays, hits, rt.MODE_TREELET, visits=vis, capacity=CAP, n=n2)
    torch.cuda.synchronize()
    return blob, scene, hits, vis, n2


CONFIGS = [
    dict(prefetcher=0),
    dict(prefetcher=1, heuristic=0),
    dict(prefetcher=1, heuristic=1, threshold=0.3),
    dict(prefetcher=1, heuristic=2, second_prefetch=1),
    dict(prefetcher=1, heuristic=3, scheduler=1, prefetch_delay=3),
    dict(prefetcher=1, heuristic=0, scheduler=2),
    dict(prefetcher=1, heuristic=0, load_metadata=1, max_queue=2048),
    dict(prefetcher=1, heuristic=0, load_metadata=1, wait_metadata=1, max_queue=2048),
    dict(prefetcher=2, max_queue=0),
    dict(prefetcher=1, heuristic=0, max_queue=64),
]


@pytest.mark.parametrize("kind,budget", [("cube_plane", 2048), ("terrain", 8192), ("shared_blas", 512)])
@pytest.mark.parametrize("extra", CONFIGS)
def test_replay_matches_oracle(ctx, kind, budget, extra):
    import torch

    import treelet_rt as rt
    from oracle import oracle as orc

    blob, scene, hits, vis, n = _gpu_traces(ctx, kind, budget)
    cfg = rt.unit_config(n_rt_units=5, max_warps=6, l1_sets=8, l1_ways=4, hit_latency=3, miss_latency=60, **extra)
    d_stats = torch.zeros(cfg.n_rt_units * rt.UNIT_STATS_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    scene.unit_replay(hits, vis, n, CAP, cfg, d_stats)
    got = np.frombuffer(d_stats.cpu().numpy().tobytes(), rt.UNIT_STATS_DTYPE)
    h = np.frombuffer(hits.cpu().numpy().tobytes(), rt.HIT_DTYPE)
    v = vis.cpu().numpy().view(np.uint32).reshape(n, CAP)
    exp = orc.unit_replay(orc.Treelets(blob.bytes(), budget), h, v, cfg)
    for f in rt.UNIT_STATS_DTYPE.names:
        assert np.array_equal(got[f], exp[f]), (f, got[f], exp[f])
    assert (got["status"] == 0).all()
    if extra["prefetcher"]:
        assert got["prefetch_issued"].sum() > 0
    scene.close()


def test_replay_bad_config_is_an_error(ctx):
    import torch

    import treelet_rt as rt

    blob, scene, hits, vis, n = _gpu_traces(ctx, "cube_plane", 2048)
    d_stats = torch.zeros(4 * rt.UNIT_STATS_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    for bad in (dict(max_warps=17), dict(l1_sets=6), dict(miss_latency=5000), dict(prefetch_delay=0),
                dict(prefetcher=3)):
        cfg = rt.unit_config(n_rt_units=4, **bad)
        with pytest.raises(rt.RTError):
            scene.unit_replay(hits, vis, n, CAP, cfg, d_stats)
    scene.close()


def _replay(scene, blob, budget, hits, vis, n, cfg):
    """Counters of the replay and of the oracle's, for device traces."""
    import torch

    import treelet_rt as rt
    from oracle import oracle as orc

    d_stats = torch.zeros(cfg.n_rt_units * rt.UNIT_STATS_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    scene.unit_replay(hits, vis, n, CAP, cfg, d_stats)
    got = np.frombuffer(d_stats.cpu().numpy().tobytes(), rt.UNIT_STATS_DTYPE)
    h = np.frombuffer(hits.cpu().numpy().tobytes(), rt.HIT_DTYPE)
    v = vis.cpu().numpy().view(np.uint32).reshape(n, CAP)
    return got, orc.unit_replay(orc.Treelets(blob.bytes(), budget), h, v, cfg)


EDGES = [
    dict(max_warps=16, l1_sets=64, l1_ways=32, prefetcher=1, heuristic=0),  # 2,048 lines: more than shared memory takes
    dict(max_warps=16, l1_sets=128, l1_ways=16, prefetcher=2, max_queue=0),
    dict(max_warps=16, l1_sets=16, l1_ways=32, prefetcher=1, heuristic=2, second_prefetch=1),
    dict(max_warps=16, l1_sets=16, l1_ways=16, prefetcher=1, scheduler=1, load_metadata=1, wait_metadata=1, max_queue=2048),
    dict(max_warps=16, l1_sets=1, l1_ways=1, prefetcher=1, scheduler=2, prefetch_delay=7),
    dict(max_warps=1, l1_sets=8, l1_ways=4, prefetcher=1, heuristic=3, second_prefetch=1, prefetch_delay=2),
    dict(max_warps=16, l1_sets=8, l1_ways=4, prefetcher=1, prefetch_delay=1000),
    dict(max_warps=6, l1_sets=8, l1_ways=4, prefetcher=1, hit_latency=1, miss_latency=1),
    dict(max_warps=6, l1_sets=8, l1_ways=4, prefetcher=1, miss_latency=4000, load_metadata=1, max_queue=2048, n_rt_units=40),
    dict(max_warps=16, l1_sets=8, l1_ways=4, prefetcher=1, n_rt_units=150),  # units without warps
]


@pytest.mark.parametrize("kind,budget", [("cube_plane", 1024), ("terrain", 8192)])
@pytest.mark.parametrize("extra", EDGES)
def test_replay_at_its_limits(ctx, kind, budget, extra):
    """As many resident warps as there may be and one, lines in shared memory
    and outside it, rare decisions, equal and long latencies, idle units."""
    import treelet_rt as rt

    blob, scene, hits, vis, n = _gpu_traces(ctx, kind, budget)
    cfg = rt.unit_config(**{**dict(n_rt_units=7, hit_latency=3, miss_latency=60), **extra})
    got, exp = _replay(scene, blob, budget, hits, vis, n, cfg)
    for f in rt.UNIT_STATS_DTYPE.names:
        assert np.array_equal(got[f], exp[f]), (f, got[f], exp[f])
    scene.close()


@pytest.mark.parametrize("max_cycles", [1, 2, 61, 64, 777, 4096, 20011])
def test_replay_stops_at_max_cycles(ctx, max_cycles):
    """The limit falls where it may, into skipped idle cycles too."""
    import treelet_rt as rt

    blob, scene, hits, vis, n = _gpu_traces(ctx, "terrain", 8192)
    for extra in (dict(prefetcher=0), dict(prefetcher=1, prefetch_delay=3), dict(prefetcher=1, prefetch_delay=100)):
        cfg = rt.unit_config(n_rt_units=5, max_warps=2, l1_sets=8, l1_ways=4, hit_latency=3, miss_latency=60,
                             max_cycles=max_cycles, **extra)
        got, exp = _replay(scene, blob, 8192, hits, vis, n, cfg)
        assert (exp["status"] == 2).all()
        for f in rt.UNIT_STATS_DTYPE.names:
            assert np.array_equal(got[f], exp[f]), (extra, f, got[f], exp[f])
    scene.close()


def test_replay_with_a_full_prefetch_ring(ctx):
    """Prefetches that never issue (each waits for metadata that nobody loads)
    pile up until the ring of 2^18 entries is full: that is reported, and the
    counters that a full ring cannot change are the oracle's."""
    import treelet_rt as rt

    blob, scene, hits, vis, n = _gpu_traces(ctx, "terrain", 65536)
    cfg = rt.unit_config(n_rt_units=5, max_warps=1, l1_sets=16, l1_ways=4, hit_latency=3, miss_latency=60,
                         prefetcher=1, heuristic=0, wait_metadata=1, max_queue=1 << 31)
    got, exp = _replay(scene, blob, 65536, hits, vis, n, cfg)
    full = exp["prefetch_queued"] - exp["prefetch_removed"] > 1 << 18
    assert full.any() and not exp["prefetch_issued"].any()
    assert (got["status"][full] == 1).all()
    for f in rt.UNIT_STATS_DTYPE.names:
        if f not in ("status", "prefetch_removed"):
            assert np.array_equal(got[f], exp[f]), (f, got[f], exp[f])
    scene.close()


@pytest.mark.parametrize("budget", [192, 256, 8192])
@pytest.mark.parametrize("extra", [dict(heuristic=0), dict(heuristic=0, wait_metadata=1),
                                   dict(heuristic=2, second_prefetch=1), dict(heuristic=0, max_queue=8)])
def test_replay_of_members_that_share_addresses(ctx, budget, extra):
    """A quad leaf in the second half of an instance leaf: both members of a
    treelet queue requests of the same addresses."""
    import kat_blob as K
    import torch

    import treelet_rt as rt

    full = ((0, 0, 0), (64, 64, 64))
    units = [
        K._header(256, (-1, -1, 0), (3, 3, 4)),                     # 0: TLAS root is unit 4
        K._header(64, (-1, -1, 0), (3, 3, 4)),                      # 1: BLAS root is unit 2
        K._internal((-1, -1, 0), 4, (4, 4, 4), [(1, 4) + full] * 3),  # 2: leaves 6, 7, 8
        bytes(64),
        K._internal((-1, -1, 0), 1, (4, 4, 4), [(2, 1) + full]),    # 4
        K._instance((1 << 64) - 256, 7),                            # 5-6: BLAS header is unit 1
        K._quad(1.0, 100), K._quad(2.0, 101),                       # 7, 8
    ]
    data = np.frombuffer(b"".join(units), np.uint8).copy()
    blob = rt.Blob.wrap(data)
    scene = rt.Scene(ctx, blob)
    scene.form_treelets(budget)
    assert {5, 6} <= set(scene.treelets()["members"].tolist())
    rays = np.resize(K.grid_rays(16), 1024)
    h, v, _ = scene.trace_host(rays, rt.MODE_TREELET, capacity=CAP, want_visits=True)
    hits = torch.from_numpy(h.view(np.uint8).copy()).cuda()
    vis = torch.from_numpy(v.view(np.uint8).copy()).cuda().view(torch.int32)
    cfg = rt.unit_config(n_rt_units=3, max_warps=4, l1_sets=1, l1_ways=2, hit_latency=3, miss_latency=40, prefetcher=1,
                         **extra)
    got, exp = _replay(scene, blob, budget, hits, vis, len(rays), cfg)
    for f in rt.UNIT_STATS_DTYPE.names:
        assert np.array_equal(got[f], exp[f]), (f, got[f], exp[f])
    assert got["prefetch_queued"].sum() > 0
    scene.close()
