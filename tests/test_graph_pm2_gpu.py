"""A captured kick keeps its buffers when PM1, PM2 and the learned shell run on the same layout in between: none of
them moves what a graph of the kick reads and writes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIXPI = float(np.float32(6 * np.pi))


def test_replay_after_other_layers(gpu):
    import torch
    from cube2_b200 import ic
    from cube2_b200 import learned as Ln
    from cube2_b200 import longrange as LR
    from cube2_b200.kick import CUBE_PM3_PERIODIC, FineKick
    from cube2_b200.layout import RATIO_SF, Layout, apm3_table, build_image, ixyz3_table
    L = Layout(ng=64, nnt=2, nns=1, ratio_cs=4, ngb=4, app=0.1)
    img = build_image(*ic.lognormal_poisson(64, 1.5, 4100)[:2], L)
    rho, idx, xp, vp0 = Ln.device_image(img, gpu)
    tabs = (np.arange(1, L.ns3 + 1, dtype=np.int32), np.full(L.ns3, 2, np.int32), ixyz3_table(L), apm3_table(4.0),
            RATIO_SF.copy())
    FineKick.finalize()  # the buffers are then the kick's own size
    fk = FineKick(L, pm3_mode=CUBE_PM3_PERIODIC, apm3f=4.0)
    vp, out = vp0.clone(), torch.zeros(8, device=gpu)
    torch.cuda.synchronize()
    graph = fk.kick_graph(rho, idx, xp, img.n_used, vp, out, *tabs, 1.0, SIXPI, 1.0)
    s = torch.cuda.Stream()
    graph.launch(s)
    torch.cuda.synchronize()
    want = (vp - vp0).double()
    net = Ln.ShellNet(Ln.init_params(4), batch_cap=16)
    shell = vp0.clone()
    torch.cuda.synchronize()
    net.kick(rho, idx, xp, img.n_used, shell, 0.5, SIXPI, 1.0)
    LR.pm1_force(img, 3.5, 1.0, SIXPI, 1.0, pm3_mode=CUBE_PM3_PERIODIC)
    LR.pm2_force(img, 3.5, 14.0, 1.0, SIXPI, 1.0, pm3_mode=CUBE_PM3_PERIODIC)
    vp.copy_(vp0)
    torch.cuda.synchronize()
    graph.launch(s)
    torch.cuda.synchronize()
    assert int(out[5:6].view(torch.int32)) == 0
    d = (vp - vp0).double()
    assert float((d - want).pow(2).sum().sqrt() / want.pow(2).sum().sqrt()) < 1e-6
    graph.close()
    net.close()
