"""The fused training step (one kernel for forward and backward, csrc/mlp.cu) against the same step as
separate mma.sync GEMMs, transposes and elementwise passes (CUBE_MLP_MMA_SYNC).

Both multiply the same BF16 operands and add in FP32, so gradients differ only by the order of the sums over
the batch: a random walk of B roundings of 2^-24, about sqrt(B) 2^-24 of the sum of magnitudes, which
may cancel to a fraction of that.  Batches: one row tile not full, exactly full, one and a
remainder, and several.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [16, 128, 144, 1024])
def test_fused_step_matches_separate_passes(gpu, monkeypatch, batch):
    import torch
    from cube2_b200 import learned as Ln
    rng = np.random.default_rng(batch)
    p = Ln.unflatten(Ln.init_params(3))
    for k in ("b1", "b2", "b3", "b4"):
        p[k] = (0.1 * rng.standard_normal(p[k].shape)).astype(np.float32)
    X = torch.from_numpy(rng.standard_normal((3000, Ln.K_PAD)).astype(np.float32)).cuda()
    X[:, Ln.K_IN:] = 0.0
    X = X.bfloat16()
    T = torch.from_numpy(rng.standard_normal((3000, 3)).astype(np.float32)).cuda()
    rows = torch.from_numpy(rng.integers(0, 3000, batch).astype(np.int32)).cuda()
    got = []
    for separate in (False, True):
        if separate:
            monkeypatch.setenv("CUBE_MLP_MMA_SYNC", "1")
        net = Ln.ShellNet(Ln.flatten(p), batch_cap=batch)
        loss = torch.zeros(1, device="cuda")
        net.train_step(X, T, rows, batch, 1e-3, loss)
        net.train_step(X, T, rows, batch, 1e-3, loss)  # the gradients of the first step are gone
        torch.cuda.synchronize()
        got.append((Ln.unflatten(net.grads().astype(np.float64)), net.params(), float(loss.item())))
        net.close()
    monkeypatch.delenv("CUBE_MLP_MMA_SYNC")
    (g, w, l), (gr, wr, lr) = got
    tol = 8 * np.sqrt(batch) * 2.0 ** -24
    # the second step's weights differ by the first update's rounding, which BF16 rarely turns into one unit
    # (2^-8 of a weight): 1e-3 of the gradients covers a few of those among 43779 weights
    for k in g:
        assert np.linalg.norm(g[k] - gr[k]) <= (tol + 1e-3) * np.linalg.norm(gr[k]), k
    assert abs(l - lr) <= 1e-4 * lr
    # an Adam update is at most about lr per parameter and step
    assert np.max(np.abs(w - wr)) <= 4e-3
    assert np.linalg.norm(w - wr) <= 1e-4 * np.linalg.norm(wr)
