"""The learned shell's kick where device memory does not hold its table of stencil rows (8 bytes a fine cell): it reads the
density itself and gives the same velocities, the network's BF16 inputs being the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIXPI = float(np.float32(6 * np.pi))


def test_kick_without_memory_for_the_table(gpu):
    import torch
    from cube2_b200 import ic
    from cube2_b200 import learned as Ln
    from cube2_b200.kick import FineKick
    from cube2_b200.layout import Layout, build_image
    L = Layout(ng=256, nnt=2, nns=1, ratio_cs=4, ngb=4, app=0.1)
    pos, vel = ic.uniform_random(200000, 256.0, 5)
    img = build_image(pos, vel, L)
    rho, idx, xp, vp0 = Ln.device_image(img, gpu)
    net = Ln.ShellNet(Ln.init_params(4), batch_cap=16)
    FineKick.finalize()  # the shell's buffers go ...
    Ln.features(L, rho, idx, xp, img.n_used)  # ... and all but the table come back
    a, b = vp0.clone(), vp0.clone()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    table = 8 * L.ng ** 3
    held = torch.empty(torch.cuda.mem_get_info()[0] - 3 * table // 4, dtype=torch.uint8, device=gpu)
    free = torch.cuda.mem_get_info()[0]
    assert free < table
    net.kick(rho, idx, xp, img.n_used, a, 1.0, SIXPI, 1.0)
    assert torch.cuda.mem_get_info()[0] > free - table // 4  # no table
    del held
    torch.cuda.empty_cache()
    net.kick(rho, idx, xp, img.n_used, b, 1.0, SIXPI, 1.0)
    d = (b - vp0).double()
    assert float(d.pow(2).sum()) > 0
    # the density's float sums over bricks may turn single BF16 inputs
    assert float((a - b).double().pow(2).sum().sqrt() / d.pow(2).sum().sqrt()) < 1e-3
    net.close()
