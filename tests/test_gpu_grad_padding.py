"""The rows past n of a gradient batch are padding, whatever they hold: the
head's gradients (w3, b3) and the loss do not depend on them."""
import numpy as np
import pytest

from farm_gb300.engine import Store

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,rows", [(1, 128), (100, 128), (128, 256), (300, 640)])
@pytest.mark.parametrize("fill", [0.0, 1e4, float("inf"), float("nan")])
def test_gpu_head_gradients_ignore_padding(gpu_lib, n, rows, fill):
    import torch

    rng = np.random.default_rng(n)
    X = np.zeros((rows, 576), np.float32)
    X[:n, :520] = rng.random((n, 520))
    y = torch.from_numpy((rng.random(rows) < 0.5).astype(np.uint8)).cuda()
    with Store() as st:
        st.mlp_init(seed=7)
        clean = st.mlp_grad(torch.from_numpy(X).to(torch.bfloat16).cuda(), y, n)
        X[n:] = fill
        loss, g = st.mlp_grad(torch.from_numpy(X).to(torch.bfloat16).cuda(), y, n)
    # sums of n terms by atomics: their order may differ, so do some roundings
    assert abs(loss - clean[0]) <= 1e-5 * clean[0]
    assert np.all(np.isfinite(g[-257:])), "NaN reached the head's gradients"
    assert np.max(np.abs(g[-257:] - clean[1][-257:])) <= n * 2.0 ** -23 * np.max(np.abs(clean[1][-257:]))
