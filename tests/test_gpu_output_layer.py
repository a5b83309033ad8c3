"""The predictor's loss and gradients where its output layer's split changes:
single and ragged row tiles and column chunks, several tiles and
chunks a CTA, and CTAs whose share starts or ends inside a split."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# BF16 activations and FP32 accumulation against a float64 oracle with
# BF16-rounded weights and inputs: relative Frobenius error per group, as for
# the sizes of test_gpu_mlp.py.
GRAD_RTOL = 1e-2
LOSS_RTOL = 1e-4


@pytest.mark.parametrize("n_treelets,n", [(1, 1), (128, 128), (129, 129), (384, 127), (385, 300), (3000, 4096),
                                          (1700, 3201), (20000, 257), (40001, 128)])
def test_gradients_across_splits(ctx, n_treelets, n):
    import torch

    from oracle import mlp_oracle as mo
    from treelet_rt import learned as L

    C = n_treelets
    mlp = L.Mlp(ctx, C, seed=5)
    rng = np.random.default_rng(n)
    s = np.zeros(n, L.SAMPLE_DTYPE)
    s["origin"] = rng.uniform(0, 1, (n, 3))
    s["dir"] = rng.uniform(-1, 1, (n, 3))
    s["current"] = rng.integers(0, C, n)
    s["target"] = rng.integers(0, C, n)
    s["target"][-1] = C - 1
    loss, g = mlp.loss_grad(torch.from_numpy(s.view(np.uint8).copy()).cuda(), n)
    p = mlp.get_params()
    rl, rg = mo.loss_and_grad(p, s, C)
    assert abs(loss - rl) <= LOSS_RTOL * max(abs(rl), 1e-3)
    offs = np.cumsum([0, C * 16, 22 * 64, 64, 64 * 64, 64, 64 * C, C])
    for k, (a, b) in enumerate(zip(offs[:-1], offs[1:])):
        if C == 1:  # one class: every gradient is zero up to the rounding of exp(z - lse)
            assert np.abs(g[a:b]).max() <= 1e-5
            continue
        err = np.linalg.norm(g[a:b] - rg[a:b]) / max(1e-30, np.linalg.norm(rg[a:b]))
        assert err <= GRAD_RTOL, (k, err)
    mlp.close()
