"""The walks' box test against the oracle where its planes cannot be told
apart by the direction's sign (a scene with quantized lower bounds above the
upper ones) and for rays that are not finite."""
import numpy as np
import pytest

from helpers import assert_hits_equal, assert_traces_equal, edge_rays

pytestmark = pytest.mark.gpu

CAP = 512


def _swap_bounds(blob_bytes, every):
    """Swaps lower and upper bounds on one axis of every k-th node's children, breadth first from the root."""
    b = blob_bytes.copy()
    work, done = [int(b[:8].view(np.uint64)[0]) // 64], 0
    while work and done < 400:
        u = work.pop(0)
        p = b[u * 64:u * 64 + 64]
        c = u + int(p[12:16].view(np.int32)[0])
        for i in range(6):
            info = int(p[22 + i])
            if info & 3 and (info >> 2) & 15 == 0:
                work.append(c)
            c += info & 3
        if done % every == 0:
            row = 28 + 12 * (done % 3)
            lo = p[row:row + 6].copy()
            p[row:row + 6] = p[row + 6:row + 12]
            p[row + 6:row + 12] = lo
        done += 1
    return b


def _odd_rays(n):
    """Camera rays with every eighth one made non-finite in some component."""
    import treelet_rt as rt

    rays = rt.camera_rays(rt.default_camera(rt.SCENE_CUBE_PLANE), n, 37, 1, 4, 1e-4, 1e30)
    bad = np.array([np.inf, -np.inf, np.nan], np.float32)
    for j, k in enumerate(range(0, len(rays), 8)):
        f = ("origin", "dir")[j % 2]
        rays[f][k, (j // 2) % 3] = bad[(j // 6) % 3]
    rays["tmax"][4::8] = np.inf
    return np.concatenate([rays, edge_rays()])


@pytest.mark.parametrize("every", [0, 1, 5])
def test_unordered_boxes_and_nonfinite_rays(ctx, every):
    import treelet_rt as rt
    from oracle import oracle as orc

    data = rt.Blob.gen(rt.SCENE_CUBE_PLANE, 3000, 6).bytes()
    if every:
        data = _swap_bounds(data, every)
    scene = rt.Scene(ctx, rt.Blob.wrap(data))
    scene.form_treelets(1024)
    tl = orc.Treelets(data, 1024)
    rays = _odd_rays(45)
    for mode, omode in ((rt.MODE_PLAIN, 0), (rt.MODE_TREELET, 1), (rt.MODE_STAGED, 1)):
        hits, vis, tids = scene.trace_host(rays, mode, capacity=CAP, want_visits=True, want_treelets=True)
        oh, ov, ot = orc.trace(data, rays, omode, tl, capacity=CAP, want_visits=True, want_treelets=True)
        assert np.array_equal(hits["n_visits"], oh["n_visits"])
        assert_traces_equal(vis, ov, oh["n_visits"], f"visits, mode {mode}")
        assert_traces_equal(tids, ot, oh["n_visits"], f"treelet ids, mode {mode}")
        finite = np.isfinite(rays["origin"]).all(axis=1) & np.isfinite(rays["dir"]).all(axis=1)
        assert_hits_equal(hits[finite], oh[finite], f"hits, mode {mode}")
    scene.close()


def test_unit_that_is_node_and_leaf(ctx):
    """A unit one parent lists as an internal node and another as a quad leaf."""
    import treelet_rt as rt
    from oracle import oracle as orc

    b = rt.Blob.gen(rt.SCENE_CUBE, 2000, 3).bytes()
    top = int(b[:8].view(np.uint64)[0]) // 64
    leaf = top + int(b[top * 64 + 12:top * 64 + 16].view(np.int32)[0])  # the TLAS root's instance leaf
    hdr = leaf + int(b[leaf * 64 + 64:leaf * 64 + 72].view(np.uint64)[0]) // 64
    root = hdr + int(b[hdr * 64:hdr * 64 + 8].view(np.uint64)[0]) // 64
    child = root + int(b[root * 64 + 12:root * 64 + 16].view(np.int32)[0])
    info = b[child * 64 + 22:child * 64 + 28]
    assert (b[root * 64 + 22] >> 2) & 15 == 0 and info[0] & 3  # the root's first child is internal
    # the first child's children become its siblings, read as quad leaves
    b[child * 64 + 12:child * 64 + 16] = np.array([1], np.int32).view(np.uint8)
    for i in range(6):
        if info[i] & 3:
            info[i] = 4 << 2 | 1
    rays = rt.camera_rays(rt.default_camera(rt.SCENE_CUBE), 40, 31, 1, 2, 1e-4, 1e30)
    scene = rt.Scene(ctx, rt.Blob.wrap(b))
    hits, vis, _ = scene.trace_host(rays, rt.MODE_PLAIN, capacity=CAP, want_visits=True)
    oh, ov, _ = orc.trace(b, rays, 0, None, capacity=CAP, want_visits=True)
    assert np.array_equal(hits["n_visits"], oh["n_visits"])
    assert_traces_equal(vis, ov, oh["n_visits"], "visits")
    scene.close()
