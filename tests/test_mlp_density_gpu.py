"""The learned shell's CIC density, read through the BF16 inputs it ends in: log(1 + rho) of a cell turns to the
neighbouring BF16 value where the density's error passes a rounding boundary, so the turned cells measure
that error far below BF16's own.  Their squared difference may be twice that of sums of FP32 weights in FP32, of which a
few cells in 10^5 turn, plus eight cells near rho = 1 (one unit of BF16 is 2^-8 there): the spread of counts of
about twenty."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cic(pos, ng, dtype):
    import torch
    x = pos - 0.5
    i = torch.floor(x)
    f = (x - i).to(dtype)
    i = i.long()
    rho = torch.zeros(ng ** 3, dtype=dtype, device=pos.device)
    for c in range(8):
        d = [(c >> a) & 1 for a in range(3)]
        w = [f[:, a] if d[a] else 1 - f[:, a] for a in range(3)]
        X, Y, Z = [(i[:, a] + d[a]) % ng for a in range(3)]
        rho.index_add_(0, (Z * ng + Y) * ng + X, w[0] * w[1] * w[2])
    return rho


@pytest.mark.parametrize("field", ["uniform", "clustered"])
def test_density_is_as_close_as_sums_in_fp32(gpu, field):
    import torch
    from cube2_b200 import ic
    from cube2_b200 import learned as Ln
    from cube2_b200.layout import Layout, build_image
    from cube2_b200.workloads import physical_positions
    ng = 128
    L = Layout(ng=ng, nnt=2, nns=1, ratio_cs=4, ngb=4, app=0.1)
    pos, vel = ic.uniform_random(ng ** 3, float(ng), 7) if field == "uniform" else ic.lognormal_poisson(ng, 1.0, 4001)[:2]
    img = build_image(pos, vel, L)
    rho, idx, xp, _ = Ln.device_image(img, gpu)
    X = Ln.features(L, rho, idx, xp, img.n_used)
    torch.cuda.synchronize()  # the library has its own stream
    X = X[torch.as_tensor(img.active, device=gpu)]
    at = torch.as_tensor(physical_positions(img), device=gpu)
    mine = torch.full((ng ** 3,), -1.0, dtype=torch.bfloat16, device=gpu)
    p = torch.empty_like(at)
    p[:] = at[torch.as_tensor(img.pid[img.active].astype(np.int64), device=gpu)]  # in the inputs' order
    i0 = torch.floor(p - 0.5).long()
    for k in range(64):
        X3, Y3, Z3 = (i0[:, 0] + k % 4 - 1) % ng, (i0[:, 1] + k // 4 % 4 - 1) % ng, (i0[:, 2] + k // 16 - 1) % ng
        mine[(Z3 * ng + Y3) * ng + X3] = X[:, k]
    mine = mine.float()
    seen = mine >= 0
    assert int(seen.sum()) > 0.8 * ng ** 3
    want = torch.log1p(_cic(at, ng, torch.float64)).bfloat16().float()
    fp32 = torch.log1p(_cic(at, ng, torch.float32)).bfloat16().float()
    off, off32 = [float((x - want)[seen].double().pow(2).sum()) for x in (mine, fp32)]
    print(field, int((mine != want)[seen].sum()), int((fp32 != want)[seen].sum()), off, off32)
    assert off <= 2 * off32 + 8 * 2.0 ** -16
