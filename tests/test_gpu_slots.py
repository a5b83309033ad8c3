"""Warp slots (rt_tuning.staged_slots): nodes read from a slot that holds the
first bytes of a treelet's image."""
import numpy as np
import pytest

from helpers import assert_hits_equal, assert_traces_equal

pytestmark = pytest.mark.gpu

CAP = 256
OFF = 0xFFFFFFFF


def _cut_leaves(blob, budget):
    """Slot sizes that end in the middle of an instance leaf of some treelet's image."""
    import treelet_rt as rt

    g = rt.Partition(blob, budget).get()
    first, size = g["member_first"].astype(np.int64), g["member_bytes"].astype(np.int64)
    at = np.cumsum(size) - size
    at -= np.repeat(at[first[:-1]], np.diff(first))  # within the treelet's image
    return sorted({int(o) + 64 for o in at[(size == 128) & (at % 128 == 64)]})


@pytest.mark.parametrize("kind,budget,pick", [("TERRAIN_INSTANCES", 8192, 0), ("TERRAIN_INSTANCES", 8192, -1),
                                              ("TERRAIN_INSTANCES", 2048, 1), ("SHARED_BLAS", 512, 0)])
def test_slot_ends_in_an_instance_leaf(ctx, kind, budget, pick):
    """The second half of the leaf is not in the slot: the leaf is read from global memory."""
    import treelet_rt as rt
    from oracle import oracle as orc

    kind = getattr(rt, "SCENE_" + kind)
    blob = rt.Blob.gen(kind, 2000, 1)
    slot_bytes = _cut_leaves(blob, budget)[pick]
    prim = rt.camera_rays(rt.default_camera(kind), 48, 40, 1, 5, 1e-4, 1e30)
    ph, _, _ = orc.trace(blob.bytes(), prim, 0)
    rays = np.concatenate([prim, rt.bounce_rays_host(blob, prim, ph, seed=11)])
    tl = orc.Treelets(blob.bytes(), budget)
    oh, ov, ot = orc.trace(blob.bytes(), rays, 1, tl, capacity=CAP, want_visits=True, want_treelets=True, threads=8)
    scene = rt.Scene(ctx, blob)
    scene.form_treelets(budget)
    scene.set_tuning(pinned_bytes=OFF, staged_slots=2, staged_slot_bytes=slot_bytes, staged_epoch=1,
                     staged_min_votes=1)
    hits, vis, tids = scene.trace_host(rays, rt.MODE_STAGED, capacity=CAP, want_visits=True, want_treelets=True)
    assert_hits_equal(hits, oh, f"slots of {slot_bytes} bytes: hits")
    assert_traces_equal(vis, ov, oh["n_visits"], "visits")
    assert_traces_equal(tids, ot, oh["n_visits"], "treelet ids")
    assert scene.stats()["smem_reads"] > 0
    scene.close()
