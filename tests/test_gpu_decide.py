"""The prefetch decision's counting table and searches at the edges of their
ranges (one lane, odd counts, 1,024 lanes that all differ, ties) against the
oracle's decision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NONE = 0xFFFFFFFF


@pytest.mark.parametrize("lanes", [1, 31, 33, 511, 513, 1024])
@pytest.mark.parametrize("spread", ["distinct", "pairs", "one"])
def test_decide_lane_counts(ctx, lanes, spread):
    import torch

    import treelet_rt as rt
    from oracle import oracle as orc

    blob = rt.Blob.gen(rt.SCENE_CUBE_PLANE, 6000, 2)
    scene = rt.Scene(ctx, blob)
    scene.form_treelets(512)
    tl = orc.Treelets(blob.bytes(), 512)
    roots = scene.treelets()["roots"].astype(np.uint32)
    assert len(roots) > 1024
    rng = np.random.default_rng(lanes)
    units = 5
    nxt = np.empty((units, lanes), np.uint32)
    for u in range(units):
        some = rng.permutation(roots)
        # every lane its own treelet; two lanes a treelet (ties go to the lowest root); the first or last root only
        nxt[u] = {"distinct": some[:lanes], "pairs": np.resize(some[:(lanes + 1) // 2], lanes),
                  "one": np.full(lanes, roots[0] if u % 2 else roots[-1])}[spread]
    nxt[4, 1:] = NONE
    state = np.zeros(units, rt.PREFETCH_STATE_DTYPE)
    for f in ("last_prefetched", "last_prefetched_second", "last_rejected"):
        state[f] = NONE
    params = rt.PrefetchParams(0, 4096, 0.5, 1, 0)
    d_state = torch.from_numpy(state.view(np.uint8).copy()).cuda()
    d_next = torch.from_numpy(nxt.view(np.uint8).copy().reshape(-1)).cuda()
    for _ in range(2):
        d_out = torch.zeros(units * 32, dtype=torch.uint8, device="cuda")
        scene.prefetch_decide(d_next, units, lanes, params, d_state, d_out)
        torch.cuda.synchronize()
        got = np.frombuffer(d_out.cpu().numpy().tobytes(), rt.PREFETCH_DECISION_DTYPE)
        got_state = np.frombuffer(d_state.cpu().numpy().tobytes(), rt.PREFETCH_STATE_DTYPE)
        for u in range(units):
            exp, state[u] = orc.prefetch_decide(tl, nxt[u], heuristic=0, max_queue=4096, threshold=0.5,
                                                second_prefetch=True, state=state[u])
            assert got[u].tobytes() == exp.tobytes(), (u, got[u], exp)
            assert got_state[u].tobytes() == state[u].tobytes()
        state["queue_len"] = 0  # drained: the second treelet may follow
        d_state = torch.from_numpy(state.view(np.uint8).copy()).cuda()
    scene.close()
