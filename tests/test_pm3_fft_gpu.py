"""The potential's transforms (rows, columns, Green step, ghost points) at every mesh side they take, against FP64
transforms of the same density: the kick of a few particles, some of them at the box's faces and corners."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIXPI = float(np.float32(6 * np.pi))
ALPHA = float(np.float32(4.0) / np.float32(3.0))
OFF, WGT = (-2, -1, 1, 2), ((ALPHA - 1) / 4, -ALPHA / 2, ALPHA / 2, (1 - ALPHA) / 4)  # kick.f90:545-568


def _truth(pos, ng, n, G):
    """FP64: TSC deposit, potential, force difference, TSC gather.  Returns the force and the potential's rms."""
    import torch
    m = torch.as_tensor(pos * (n / ng), device="cuda")
    f = torch.floor(m)
    l = m - f
    w = torch.stack([(1 - l) ** 2 / 2, 1 - (1 - l) ** 2 / 2 - l ** 2 / 2, l ** 2 / 2], 0)  # [3, particle, axis]
    i = torch.stack([f - 1, f, f + 1], 0).long() % n
    phi = torch.zeros(n * n * n, dtype=torch.float64, device="cuda")
    pts = [(i[a, :, 0], i[b, :, 1], i[c, :, 2], w[a, :, 0] * w[b, :, 1] * w[c, :, 2])
           for a in range(3) for b in range(3) for c in range(3)]
    for x, y, z, t in pts:
        phi.index_add_(0, (z * n + y) * n + x, t)
    k = torch.fft.rfftn(phi.view(n, n, n))
    k *= torch.as_tensor(G, device="cuda")
    phi = torch.fft.irfftn(k, s=(n, n, n))
    del k
    F = torch.zeros(len(pos), 3, dtype=torch.float64, device="cuda")
    for x, y, z, t in pts:
        for o, q in zip(OFF, WGT):
            F[:, 0] += t * q * phi[z, y, (x + o) % n]
            F[:, 1] += t * q * phi[z, (y + o) % n, x]
            F[:, 2] += t * q * phi[(z + o) % n, y, x]
    return F.cpu().numpy(), float(phi.pow(2).mean().sqrt())


@pytest.mark.parametrize("n,nnt", [(64, 1), (80, 1), (96, 2), (128, 2), (144, 3), (160, 2), (192, 2), (240, 2), (256, 1),
                                   (288, 2), (320, 1), (384, 2), (480, 2), (512, 2), (576, 2), (640, 2), (768, 2),
                                   (960, 2), (1024, 2)])
def test_transforms_of_every_side(gpu, n, nnt):
    from cube2_b200.kick import CUBE_PM3_PERIODIC, FineKick, green_table
    from cube2_b200.layout import RATIO_SF, Layout, build_image, ixyz3_table
    from cube2_b200.workloads import physical_positions
    ng = n // 2
    rng = np.random.default_rng(n)
    edge = np.array([[x, y, z] for x in (0.2, ng - 0.2) for y in (0.3, ng - 0.3) for z in (0.1, ng - 0.1)])
    pos = np.concatenate([ng * rng.random((1000, 3)), edge, 2 + rng.random((200, 3)), ng - rng.random((200, 3))])
    L = Layout(ng=ng, nnt=nnt, nns=1, ratio_cs=4, ngb=4, app=0.1)
    img = build_image(pos, np.zeros(pos.shape, np.float32), L)
    fk = FineKick(L, pm3_mode=CUBE_PM3_PERIODIC, apm3f=4.0)
    vp, _, _, _ = fk.c_pm3_force_kernel(img, np.arange(1, L.ns3 + 1, dtype=np.int32), np.full(L.ns3, 2, np.int32),
                                        ixyz3_table(L), RATIO_SF, 1.0, SIXPI, 1.0)
    F, phi = _truth(physical_positions(img), ng, n, green_table(n, 4.0, 0.0, 0.5))
    got = np.empty((len(pos), 3))
    got[img.pid[img.active]] = vp[img.active]  # the coefficient a_mid dt / (6 pi) is 1
    rms = np.sqrt(np.mean(F ** 2))
    # Error of FP32 transforms: 2^-24 of the potential's rms a butterfly level, 2 * 3 log2 n levels, adding as their
    # root; through the difference (weights of norm < 1).  Three times that, and 2e-6 for the 27-point sums.
    tol = 3 * 2.0 ** -24 * np.sqrt(6 * np.log2(n)) * phi / rms + 2e-6
    err = np.sqrt(np.mean((got - F) ** 2)) / rms
    print(n, err, tol)
    assert err < tol
