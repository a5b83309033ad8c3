"""The walks against the oracle where their kernels branch: the box test of a
scene whose planes cannot be told apart by the direction's sign (quantized
lower bounds above the upper ones) and of rays that are not finite, nodes used
in two roles, and launches on both sides of the sizes at which a ray gets eight
lanes, and a warp fewer rays."""
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


@pytest.mark.parametrize("n", [256, 40001])
def test_node_of_both_levels(ctx, n):
    """A node the TLAS root lists as its child and an instance has as its BLAS
    root: as a top-level node its quad leaf is an instance leaf, whose BLAS is
    reached no other way."""
    import kat_blob as K

    import treelet_rt as rt
    from oracle import oracle as orc

    def box(size, typ):
        return size, typ, (0, 0, 0), (64, 64, 64)

    wide = (-262144.0,) * 3
    second = bytearray(64)  # the second half of the quad leaf's instance: its BLAS header is unit 8
    second[0:8] = np.uint64(128).tobytes()
    units = [
        K._header(128, (-1, -1, 0), (3, 3, 4)),                             # 0: TLAS root is unit 2
        K._header(128, (-1, -1, 0), (3, 3, 4)),                             # 1: BLAS root is unit 3
        K._internal((-1, -1, 0), 1, (4, 4, 4), [box(1, 0), box(2, 1)]),     # 2
        K._internal((-1, -1, 0), 3, (4, 4, 4), [box(1, 4)]),                # 3: a node of both levels
        K._instance((1 << 64) - 192, 7),                                    # 4-5: BLAS header is unit 1
        K._quad(1.0, 100),                                                  # 6
        bytes(second),                                                      # 7
        K._header(64, (-1, -1, 0), (3, 3, 4)),                              # 8: BLAS root is unit 9
        K._internal(wide, 1, (20, 20, 20), [(1, 4, (0, 0, 0), (128, 128, 128)), (1, 0, (0, 0, 0), (128, 128, 128))]),
        K._quad(2.0, 200),                                                  # 10
        K._internal(wide, 1, (20, 20, 20), [(1, 4, (0, 0, 0), (128, 128, 128))]),  # 11
        K._quad(3.0, 300),                                                  # 12
    ]
    b = np.frombuffer(b"".join(units), np.uint8).copy()
    rays = np.resize(K.grid_rays(16), n)
    oh, ov, _ = orc.trace(b, rays, 0, None, capacity=32, want_visits=True, threads=8)
    reached = ov[np.arange(32)[None, :] < np.minimum(oh["n_visits"], 32)[:, None]] >> 3
    assert {3, 6, 9, 11} <= set(reached.tolist())
    scene = rt.Scene(ctx, rt.Blob.wrap(b))
    hits, vis, _ = scene.trace_host(rays, rt.MODE_PLAIN, capacity=32, want_visits=True)
    assert_hits_equal(hits, oh, "hits")
    assert_traces_equal(vis, ov, oh["n_visits"], "visits")
    scene.close()


@pytest.mark.parametrize("n", [1, 7, 33, 4864, 4865, 9729, 24576, 24577, 32768, 32769, 40001])
def test_launch_sizes(ctx, n):
    """Eight lanes a ray (one, two or four rays a warp) up to 32,768 rays (24,576 staged), one
    lane a ray above: hits and traces, any-hit rays among them, with a row
    capacity that some rays exceed and rows that start off a 32-byte boundary."""
    import torch

    import treelet_rt as rt
    from oracle import oracle as orc

    blob = rt.Blob.gen(rt.SCENE_TERRAIN_INSTANCES, 2 * 40 * 40, 5)
    scene = rt.Scene(ctx, blob)
    scene.form_treelets(2048)
    tl = orc.Treelets(blob.bytes(), 2048)
    rays = rt.camera_rays(rt.default_camera(rt.SCENE_TERRAIN_INSTANCES), 250, 161, 1, 3, 1e-4, 1e30)
    rays = np.ascontiguousarray(rays[np.random.default_rng(n).permutation(len(rays))[:n]])
    flags = np.random.default_rng(n + 1).choice(np.array([0, 1, 5], np.uint32), size=n)
    d_rays = torch.from_numpy(rays.view(np.uint8).copy()).cuda()
    d_flags = torch.from_numpy(flags.view(np.uint8).copy()).cuda()
    for mode, omode in ((rt.MODE_PLAIN, 0), (rt.MODE_TREELET, 1), (rt.MODE_STAGED, 1)):
        for cap, skew in ((48, 0), (48, 1), (45, 0)):
            d_hits = torch.zeros(n * 64, dtype=torch.uint8, device="cuda")
            d_vis = torch.zeros(n * cap + skew, dtype=torch.int32, device="cuda")[skew:]
            d_tl = torch.zeros(n * cap, dtype=torch.int32, device="cuda")
            scene.trace(d_rays, d_hits, mode, flags=d_flags, visits=d_vis, treelets=d_tl, capacity=cap, n=n)
            torch.cuda.synchronize()
            hits = np.frombuffer(d_hits.cpu().numpy().tobytes(), rt.HIT_DTYPE)
            oh, ov, ot = orc.trace(blob.bytes(), rays, omode, tl, flags=flags, capacity=cap, want_visits=True,
                                   want_treelets=True, threads=8)
            assert_hits_equal(hits, oh, f"hits, mode {mode}, {n} rays")
            assert_traces_equal(d_vis.cpu().numpy().view(np.uint32).reshape(n, cap), ov, oh["n_visits"], "visits")
            assert_traces_equal(d_tl.cpu().numpy().view(np.uint32).reshape(n, cap), ot, oh["n_visits"], "treelet ids")
            node_bytes = scene.stats()["node_bytes"]
            assert mode != rt.MODE_STAGED or scene.stats()["smem_reads"] > 0
        untraced = torch.zeros(n * 64, dtype=torch.uint8, device="cuda")
        scene.trace(d_rays, untraced, mode, flags=d_flags, n=n)
        torch.cuda.synchronize()
        got = np.frombuffer(untraced.cpu().numpy().tobytes(), rt.HIT_DTYPE).copy()
        got["status"] |= np.where(got["n_visits"] > cap, rt.RAY_TRACE_OVERFLOW, 0).astype(np.uint32)
        assert_hits_equal(got, hits, f"untraced hits, mode {mode}, {n} rays")
        assert scene.stats()["node_bytes"] == node_bytes
    scene.close()


@pytest.mark.parametrize("n", [1, 8192, 8193, 16384, 16385, 131073])
@pytest.mark.parametrize("pinned", [True, False])
def test_packed_call_sizes(ctx, n, pinned):
    """Packed traces where the call changes its way: one block or four kernels
    for the offsets, straight into page-locked arrays or through copies, one or
    two chunks; arrays one entry too small; treelet ids alone."""
    import ctypes as C

    import torch

    import treelet_rt as rt

    scene = rt.Scene(ctx, rt.Blob.gen(rt.SCENE_CUBE_PLANE, 3000, 6))
    scene.form_treelets(1024)
    cam = rt.default_camera(rt.SCENE_CUBE_PLANE)
    rays = np.resize(rt.camera_rays(cam, 190, 97, 1, 2, 1e-4, 1e30), n)
    cap = 24  # some rays have more
    hits, vis, tids = scene.trace_host(rays, rt.MODE_TREELET, capacity=cap, want_visits=True, want_treelets=True)
    keep = np.arange(cap)[None, :] < hits["n_visits"][:, None]
    total = int(keep.sum())
    want_off = np.concatenate([[0], np.cumsum(keep.sum(axis=1))])

    def array(a):
        t = torch.from_numpy(a)
        return t.pin_memory() if pinned else t.clone()

    d_rays = array(rays.view(np.uint8).copy())
    for visits, room in ((True, total), (True, total - 1), (False, total)):
        h, off = array(np.zeros(n * 64, np.uint8)), array(np.zeros(n + 1, np.int64))
        v, t = array(np.zeros(max(room, 1), np.int32)), array(np.zeros(max(room, 1), np.int32))
        got = C.c_uint64(0)
        st = rt.lib().rt_trace_host_packed(scene.handle, d_rays.data_ptr(), None, 1, n, rt.MODE_TREELET, cap,
                                           h.data_ptr(), off.data_ptr(), v.data_ptr() if visits else None,
                                           t.data_ptr(), room, C.byref(got))
        assert st == (0 if room >= total else 6), rt.lib().rt_last_error().decode()
        assert got.value == total
        assert np.array_equal(off.numpy(), want_off)
        assert_hits_equal(h.numpy().view(rt.HIT_DTYPE), hits, "packed hits")
        if room >= total:
            assert np.array_equal(t.numpy().view(np.uint32)[:total], tids[keep])
            if visits:
                assert np.array_equal(v.numpy().view(np.uint32)[:total], vis[keep])
    scene.close()


@pytest.mark.parametrize("n", [(1 << 19) - 1, 1 << 19, (1 << 19) + 33])
def test_staged_rays_taken_together(ctx, n):
    """Staged launches on both sides of the size from which a warp of
    neighbouring camera rays waits for its last one: camera rays, then the same
    from other points and in other directions, mixed within the warps."""
    import torch

    import treelet_rt as rt
    from oracle import oracle as orc

    blob = rt.Blob.gen(rt.SCENE_TERRAIN_INSTANCES, 2 * 40 * 40, 5)
    scene = rt.Scene(ctx, blob)
    scene.form_treelets(1024)
    rays = np.resize(rt.camera_rays(rt.default_camera(rt.SCENE_TERRAIN_INSTANCES), 1024, 512, 1, 3, 1e-4, 1e30), n)
    rng = np.random.default_rng(n)
    spread = np.arange(n) % 4096 > 3000
    spread &= rng.random(n) < 0.5
    rays["origin"][spread] += rng.uniform(-0.1, 0.1, (int(spread.sum()), 3)).astype(np.float32)
    rays["dir"][spread] = rng.normal(size=(int(spread.sum()), 3)).astype(np.float32)
    rays["dir"][7::5001] = np.nan
    d_rays = torch.from_numpy(rays.view(np.uint8).copy()).cuda()
    hits = torch.zeros(n * 64, dtype=torch.uint8, device="cuda")
    scene.trace(d_rays, hits, rt.MODE_STAGED, n=n)
    torch.cuda.synchronize()
    oh, _, _ = orc.trace(blob.bytes(), rays, 1, orc.Treelets(blob.bytes(), 1024), threads=8)
    assert_hits_equal(hits.cpu().numpy().view(rt.HIT_DTYPE), oh, "staged")
    scene.close()


def test_forming_treelets_waits_for_traces_in_flight(ctx):
    """Plain traces queued on a stream of the caller's own are over when
    rt_treelets_form, or a change of the device offset, returns: both rewrite
    nodes that the traces read."""
    import torch

    import treelet_rt as rt

    n = 1 << 21
    scene = rt.Scene(ctx, rt.Blob.gen(rt.SCENE_CUBE_PLANE, 3000, 6))
    rays = np.resize(rt.camera_rays(rt.default_camera(rt.SCENE_CUBE_PLANE), 190, 97, 1, 2, 1e-4, 1e30), n)
    d_rays = torch.from_numpy(rays.view(np.uint8).copy()).cuda()
    want = torch.zeros(n * 64, dtype=torch.uint8, device="cuda")
    scene.trace(d_rays, want, rt.MODE_PLAIN, n=n)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    for change in (lambda: scene.form_treelets(1024), lambda: scene.form_treelets(2048),
                   lambda: scene.set_device_offset(64), lambda: scene.set_device_offset(0)):
        hits = [torch.zeros(n * 64, dtype=torch.uint8, device="cuda") for _ in range(4)]
        torch.cuda.synchronize()
        for k in range(200):  # at least a tenth of a second of work: longer than the calls take by themselves
            scene.trace(d_rays, hits[k % 4], rt.MODE_PLAIN, n=n, stream=stream.cuda_stream)
        change()
        assert stream.query()
        assert all(torch.equal(h, want) for h in hits)
    scene.close()


def test_packed_arrays_lie_in_one_registration(ctx):
    """A small packed call packs into an array anywhere inside one page-locked
    registration; an array across two of them (back to back here, so that all
    of it is page-locked) is refused as the copies of larger calls refuse it, and
    the next call is none the worse."""
    import ctypes as C
    import mmap

    import torch

    import treelet_rt as rt

    n, cap, page = 300, 24, mmap.PAGESIZE
    scene = rt.Scene(ctx, rt.Blob.gen(rt.SCENE_CUBE_PLANE, 3000, 6))
    scene.form_treelets(1024)
    rays = np.ascontiguousarray(rt.camera_rays(rt.default_camera(rt.SCENE_CUBE_PLANE), 30, 10, 1, 2, 1e-4, 1e30)[:n])
    hits, vis, _ = scene.trace_host(rays, rt.MODE_TREELET, capacity=cap, want_visits=True)
    keep = np.arange(cap)[None, :] < hits["n_visits"][:, None]
    total = int(keep.sum())
    half = -(-n * 64 // page) * page  # bytes of a registration: the hit records fit one
    room = mmap.mmap(-1, 2 * half)
    base = np.frombuffer(room, np.uint8)
    cudart = torch.cuda.cudart()
    for k in range(2):
        assert int(cudart.cudaHostRegister(base.ctypes.data + k * half, half, 0)) == 0
    off = torch.zeros(n + 1, dtype=torch.int64).pin_memory()
    v = torch.zeros(total, dtype=torch.int32).pin_memory()
    try:
        for at, ok in ((0, True), (half, True), (half - 64 * 7, False), (2 * half - 64 * n, True)):
            base[:] = 0
            got = C.c_uint64(0)
            st = rt.lib().rt_trace_host_packed(scene.handle, rays.ctypes.data, None, 1, n, rt.MODE_TREELET, cap,
                                               base.ctypes.data + at, off.data_ptr(), v.data_ptr(), None, total,
                                               C.byref(got))
            assert st == (0 if ok else 2), rt.lib().rt_last_error().decode()
            if ok:
                assert got.value == total
                assert_hits_equal(base[at:at + 64 * n].copy().view(rt.HIT_DTYPE), hits, "packed hits")
                assert np.array_equal(v.numpy().view(np.uint32), vis[keep])
    finally:
        for k in range(2):
            cudart.cudaHostUnregister(base.ctypes.data + k * half)
    scene.close()


@pytest.mark.parametrize("epoch", [16, 64])
def test_staged_epoch_counts_node_visits(ctx, epoch):
    """Warp slots: a warp votes every staged_epoch visits.  A visit is of 32
    nodes at most, on average of far fewer, so the warps vote more than (nodes
    read) / (32 epoch) times; with one slot, one vote enough, and rays all over a
    scene of many treelets, nearly every vote stages one.  And they vote no more
    often than the visits allow, at once and then every epoch."""
    import torch

    import treelet_rt as rt

    n = 2_000_000
    scene = rt.Scene(ctx, rt.Blob.gen(rt.SCENE_BLOBS, 60000, 5))
    info = scene.form_treelets(1024)
    assert info["n_treelets"] > 1000
    rng = np.random.default_rng(3)
    rays = np.zeros(n, rt.RAY_DTYPE)
    rays["origin"] = rng.uniform(0, 1, (n, 3))
    rays["dir"] = rng.normal(size=(n, 3))
    rays["tmax"] = 1e30
    d_rays = torch.from_numpy(rays.view(np.uint8).copy()).cuda()
    want = torch.zeros(n * 64, dtype=torch.uint8, device="cuda")
    scene.trace(d_rays, want, rt.MODE_TREELET, n=n)
    scene.set_tuning(staged_slots=1, staged_min_votes=1, staged_epoch=epoch, staged_threads=128,
                     pinned_bytes=rt.TUNING_OFF)
    hits = torch.zeros_like(want)
    scene.trace(d_rays, hits, rt.MODE_STAGED, n=n)
    torch.cuda.synchronize()
    assert torch.equal(hits, want)
    st = scene.stats()
    nodes = st["smem_reads"] + st["gmem_reads"]
    assert st["stagings"] > nodes / (32 * epoch)
    assert st["stagings"] <= nodes / epoch + 152 * 64
    scene.close()


@pytest.mark.parametrize("cap,skew", [(8, 0), (16, 0), (40, 0), (40, 1), (45, 0)])
def test_ids_of_short_rows(ctx, cap, skew):
    """Rows on both sides of eight entries (rays that miss, or leave the scene at once): the walk
    writes the ids of shorter ones, the pass after it the others', and none past a row's entries."""
    import torch

    import treelet_rt as rt
    from oracle import oracle as orc

    blob = rt.Blob.gen(rt.SCENE_BLOBS, 2000, 5)
    few = rt.camera_rays(rt.default_camera(rt.SCENE_BLOBS), 96, 80, 1, 3, 1e-4, 1e30)
    tl = orc.Treelets(blob.bytes(), 1024)
    n = 40003
    pick = np.random.default_rng(1).integers(0, len(few), n)
    d_rays = torch.from_numpy(few[pick].view(np.uint8)).cuda()
    scene = rt.Scene(ctx, blob)
    scene.form_treelets(1024)
    for mode, omode in ((rt.MODE_PLAIN, 0), (rt.MODE_TREELET, 1), (rt.MODE_STAGED, 1)):
        oh, ov, ot = orc.trace(blob.bytes(), few, omode, tl, capacity=cap, want_visits=True, want_treelets=True, threads=8)
        assert (oh["n_visits"] < 8).any() and (oh["n_visits"] >= 8).any()
        d_hits = torch.zeros(n * 64, dtype=torch.uint8, device="cuda")
        d_vis = torch.full((n * cap + skew,), -1, dtype=torch.int32, device="cuda")[skew:]
        d_tl = torch.full((n * cap,), -1, dtype=torch.int32, device="cuda")
        scene.trace(d_rays, d_hits, mode, visits=d_vis, treelets=d_tl, capacity=cap, n=n)
        keep = np.arange(cap)[None, :] < np.minimum(oh["n_visits"], cap)[pick][:, None]
        for got, expect, what in ((d_vis, ov, "visits"), (d_tl, ot, "treelet ids")):
            g = got.cpu().numpy().view(np.uint32).reshape(n, cap)
            assert np.array_equal(g[keep], expect[pick][keep]), f"{what}, mode {mode}"
            assert (g[~keep] == 0xFFFFFFFF).all(), f"{what} past a row's entries, mode {mode}"
    scene.close()
