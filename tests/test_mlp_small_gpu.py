"""The learned shell on boxes with fewer deposit bricks than multiprocessors: the density goes by particle there (no work
list), and the kick is still scale times the network's output on the features, on both sides of the line."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIXPI = float(np.float32(6 * np.pi))


@pytest.mark.parametrize("ng,kernels", [(32, 5), (80, 5), (96, 6)])  # 8, 125 and 216 bricks
def test_small_boxes(gpu, ng, kernels):
    import torch
    from cube2_b200 import ic
    from cube2_b200 import learned as Ln
    from cube2_b200.kick import FineKick
    from cube2_b200.layout import Layout, build_image
    L = Layout(ng=ng, nnt=1, nns=1, ratio_cs=4, ngb=4, app=0.1)
    img = build_image(*ic.uniform_random(ng ** 3, float(ng), 7), L)
    rho, idx, xp, vp = Ln.device_image(img, gpu)
    X = Ln.features(L, rho, idx, xp, img.n_used)
    torch.cuda.synchronize()
    net = Ln.ShellNet(Ln.init_params(4), batch_cap=4096)
    Y = torch.zeros((img.n_used, 3), device=gpu)
    v = vp.clone()
    torch.cuda.synchronize()
    net.forward(X, img.n_used, Y)
    before = FineKick.launch_count()
    net.kick(rho, idx, xp, img.n_used, v, 0.5, SIXPI, 1.0)
    # cell table, list, density (by particle one kernel, by bricks two), table of stencil rows, network
    assert FineKick.launch_count() - before == kernels
    torch.cuda.synchronize()
    own = torch.as_tensor(img.active, device=gpu)
    d, want = (v - vp).reshape(-1, 3)[own].double(), (0.5 * Ln.kick_coef(SIXPI, 1.0) * Y)[own].double()
    assert float((d - want).pow(2).sum().sqrt() / want.pow(2).sum().sqrt()) < 2e-3
    net.close()
