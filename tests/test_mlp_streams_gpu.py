"""The learned shell's kick and the fine-scale kick of the same image on two streams at once, as a program runs them
that compares both velocities afterwards (cube_learned_fallback): each call has the mesh jobs and the deposit work list
of its own mesh, so neither changes the other's result.

Sums that go through float atomics differ by their order: 2^-24 of partial sums that cancel to a fraction of
themselves, 1e-6 of the kick here; work on the other mesh's jobs is off by the kick itself.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIXPI = float(np.float32(6 * np.pi))


def _rel_rms(a, b):
    return float((a - b).double().pow(2).sum().sqrt() / b.double().pow(2).sum().sqrt())


def test_shell_and_kick_on_two_streams(gpu):
    import torch
    from cube2_b200 import ic
    from cube2_b200 import learned as Ln
    from cube2_b200.kick import CUBE_PM3_PERIODIC, FineKick
    from cube2_b200.layout import RATIO_SF, Layout, apm3_table, build_image, ixyz3_table
    L = Layout(ng=96, nnt=2, nns=1, ratio_cs=4, ngb=4, app=0.1)
    img = build_image(*ic.lognormal_poisson(96, 1.5, 4200)[:2], L)
    rho, idx, xp, vp0 = Ln.device_image(img, gpu)
    fk = FineKick(L, pm3_mode=CUBE_PM3_PERIODIC, apm3f=4.0)
    tabs = (np.arange(1, L.ns3 + 1, dtype=np.int32), np.full(L.ns3, 2, np.int32), ixyz3_table(L), apm3_table(4.0),
            RATIO_SF.copy())
    net = Ln.ShellNet(Ln.init_params(4), batch_cap=16)
    out = torch.zeros(8, device=gpu)

    def kick(stream):
        v = vp0.clone()
        torch.cuda.synchronize()
        fk.kick_fine_device(rho, idx, xp, img.n_used, v, out, *tabs, 1.0, SIXPI, 1.0, stream=stream)
        return v

    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    want_kick = kick(a)
    torch.cuda.synchronize()
    f2 = out[:2].clone()
    want_shell = vp0.clone()
    torch.cuda.synchronize()
    net.kick(rho, idx, xp, img.n_used, want_shell, 0.5, SIXPI, 1.0, stream=b)
    torch.cuda.synchronize()
    for _ in range(8):
        shell = vp0.clone()
        v = kick(a)  # still running when the shell starts
        net.kick(rho, idx, xp, img.n_used, shell, 0.5, SIXPI, 1.0, stream=b)
        torch.cuda.synchronize()
        assert int(out[5:6].view(torch.int32)) == 0
        assert _rel_rms(v - vp0, want_kick - vp0) < 1e-6
        assert torch.allclose(out[:2], f2, rtol=1e-5)
        assert _rel_rms(shell - vp0, want_shell - vp0) < 1e-3  # BF16 inputs: a density's last bit can turn one
    net.close()
