"""The walks that give a ray one lane, in launches too large for eight lanes a
ray (more than 32,768 rays, 24,576 staged): tunings that are theirs alone,
boxes and rays that the fast box test must not see, a unit used in two roles,
stacks that run over."""
import numpy as np
import pytest

import kat_blob
from helpers import assert_hits_equal, assert_traces_equal, edge_rays
from test_gpu_failure import _check_overflow
from test_gpu_parity import _check_all_modes
from test_gpu_walks import _odd_rays, _swap_bounds

pytestmark = pytest.mark.gpu

OFF = 0xFFFFFFFF
N = 40001
CAP = 160


@pytest.mark.parametrize("tuning", [dict(block_threads=32, staged_threads=32), dict(block_threads=64, staged_threads=64),
                                    dict(block_threads=256, refill_lanes=32), dict(refill_lanes=1),
                                    dict(pinned_bytes=OFF), dict(pinned_bytes=1024), dict(pinned_bytes=16384),
                                    dict(pinned_bytes=16384, staged_threads=256, refill_lanes=1),
                                    dict(staged_slots=1, staged_epoch=1, staged_min_votes=1),
                                    dict(stack_depth=48, short_stack=1), dict(stack_depth=160)])
def test_tunings(ctx, tuning):
    import treelet_rt as rt
    from oracle import oracle as orc

    blob = rt.Blob.gen(rt.SCENE_CUBE_PLANE, 16384, 10)
    prim = rt.camera_rays(rt.default_camera(rt.SCENE_CUBE_PLANE), 64, 64, 1, 1, 1e-4, 1e30)
    ph, _, _ = orc.trace(blob.bytes(), prim, 0, threads=8)
    rays = np.concatenate([prim, rt.bounce_rays_host(blob, prim, ph, seed=11), edge_rays()])
    _check_all_modes(ctx, blob, np.resize(rays, N), cap=CAP, tuning=tuning)


@pytest.mark.parametrize("every", [0, 1, 5])
@pytest.mark.parametrize("tuning", [{}, dict(staged_slots=2, staged_epoch=1, staged_min_votes=1, pinned_bytes=OFF)])
def test_unordered_boxes_and_nonfinite_rays(ctx, every, tuning):
    import treelet_rt as rt
    from oracle import oracle as orc

    data = rt.Blob.gen(rt.SCENE_CUBE_PLANE, 3000, 6).bytes()
    if every:
        data = _swap_bounds(data, every)
    scene = rt.Scene(ctx, rt.Blob.wrap(data))
    scene.form_treelets(1024)
    scene.set_tuning(**tuning)
    tl = orc.Treelets(data, 1024)
    rays = np.resize(_odd_rays(45), N)
    finite = np.isfinite(rays["origin"]).all(axis=1) & np.isfinite(rays["dir"]).all(axis=1)
    for mode, omode in ((rt.MODE_PLAIN, 0), (rt.MODE_TREELET, 1), (rt.MODE_STAGED, 1)):
        hits, vis, tids = scene.trace_host(rays, mode, capacity=CAP, want_visits=True, want_treelets=True)
        oh, ov, ot = orc.trace(data, rays, omode, tl, capacity=CAP, want_visits=True, want_treelets=True, threads=8)
        assert np.array_equal(hits["n_visits"], oh["n_visits"])
        assert_traces_equal(vis, ov, oh["n_visits"], f"visits, mode {mode}")
        assert_traces_equal(tids, ot, oh["n_visits"], f"treelet ids, mode {mode}")
        assert_hits_equal(hits[finite], oh[finite], f"hits, mode {mode}")
    scene.close()


def test_unit_that_is_node_and_leaf(ctx):
    """A unit one parent lists as an internal node and another as a quad leaf."""
    import treelet_rt as rt
    from oracle import oracle as orc

    def unit(b, u):
        return b[u * 64:u * 64 + 64]

    b = rt.Blob.gen(rt.SCENE_CUBE, 2000, 3).bytes()
    top = int(b[:8].view(np.uint64)[0]) // 64
    leaf = top + int(unit(b, top)[12:16].view(np.int32)[0])
    hdr = leaf + int(unit(b, leaf + 1)[:8].view(np.uint64)[0]) // 64
    root = hdr + int(unit(b, hdr)[:8].view(np.uint64)[0]) // 64
    node = unit(b, root + int(unit(b, root)[12:16].view(np.int32)[0]))  # the root's first child
    assert (unit(b, root)[22] >> 2) & 15 == 0 and node[22] & 3
    node[12:16] = np.array([1], np.int32).view(np.uint8)  # its siblings, read as quad leaves
    for i in range(22, 28):
        if node[i] & 3:
            node[i] = 4 << 2 | 1
    rays = np.resize(rt.camera_rays(rt.default_camera(rt.SCENE_CUBE), 40, 31, 1, 2, 1e-4, 1e30), N)
    scene = rt.Scene(ctx, rt.Blob.wrap(b))
    hits, vis, _ = scene.trace_host(rays, rt.MODE_PLAIN, capacity=CAP, want_visits=True)
    oh, ov, _ = orc.trace(b, rays, 0, None, capacity=CAP, want_visits=True, threads=8)
    assert np.array_equal(hits["n_visits"], oh["n_visits"])
    assert_traces_equal(vis, ov, oh["n_visits"], "visits")
    scene.close()


def test_stack_overflow(ctx):
    import treelet_rt as rt

    chain = rt.Blob.wrap(kat_blob.deep_chain_blob(11))
    assert _check_overflow(ctx, chain, np.resize(kat_blob.grid_rays(16), N), 8192, (48, 96)) > 0
    tris = np.random.default_rng(5).uniform(0, 1, (4000, 9)).astype(np.float32)
    ident = np.array([[1, 0, 0], [0, 1, 0], [0, 0, 1], [0, 0, 0]], np.float32)
    rays = rt.camera_rays(rt.default_camera(rt.SCENE_CUBE), 48, 48, 1, 3, 1e-4, 1e30)
    overlapping = rt.Blob.build([tris], [(0, ident, 0)])
    assert _check_overflow(ctx, overlapping, np.resize(rays, N), 8192, (48, 96, 160)) > 0


@pytest.mark.parametrize("n,depth", [(786431, 96), (786432, 96), (786433, 48), (786432, 160)])
def test_large_any_hit_launches(ctx, n, depth):
    """Staged any-hit launches on both sides of the size from which they run four CTAs per SM."""
    import torch

    import treelet_rt as rt
    from oracle import oracle as orc

    blob = rt.Blob.gen(rt.SCENE_CUBE_PLANE, 2000, 4)
    prim = rt.camera_rays(rt.default_camera(rt.SCENE_CUBE_PLANE), 64, 64, 1, 2, 1e-4, 1e30)
    ph, _, _ = orc.trace(blob.bytes(), prim, 0)
    few = np.concatenate([prim, rt.bounce_rays_host(blob, prim, ph, seed=5)])
    flags = rt.RAY_FLAG_OPAQUE | rt.RAY_FLAG_TERMINATE_ON_FIRST_HIT
    tl = orc.Treelets(blob.bytes(), 1024)
    oh, _, _ = orc.trace(blob.bytes(), few, 1, tl, default_flags=flags, threads=8)
    pick = np.resize(np.arange(len(few)), n)
    scene = rt.Scene(ctx, blob)
    scene.form_treelets(1024)
    scene.set_tuning(stack_depth=depth)
    d_rays = torch.from_numpy(few[pick].view(np.uint8)).cuda()
    d_hits = torch.zeros(n * 64, dtype=torch.uint8, device="cuda")
    scene.trace(d_rays, d_hits, rt.MODE_STAGED, default_flags=flags, n=n)
    hits = d_hits.cpu().numpy().view(rt.HIT_DTYPE)
    scene.close()
    assert_hits_equal(hits, oh[pick], f"{n} any-hit rays, depth {depth}")
