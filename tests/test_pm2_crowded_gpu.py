"""PM2 on a crowded brick: its deposit goes by the work list, which splits the brick's particles over several blocks; on
meshes of few bricks it goes by coarse cell."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIXPI = float(np.float32(6 * np.pi))


def _image():
    from cube2_b200 import ic
    from cube2_b200.layout import Layout, build_image
    L = Layout(ng=64, nnt=2, nns=2, ratio_cs=4, ngb=4, app=0.1)
    rng = np.random.default_rng(21)
    pos, _ = ic.uniform_random(3000, 64.0, 13)
    pos = np.concatenate([pos, [41.0, 9.0, 13.0] + 2 * rng.random((40000, 3)), [2.5, 2.5, 2.5] + rng.random((2500, 3))])
    return build_image(pos, np.zeros(pos.shape, np.float32), L)


def test_few_bricks(gpu):
    from cube2_b200 import ic
    from cube2_b200 import longrange as LR
    from cube2_b200.kick import FineKick
    from cube2_b200.layout import Layout, build_image
    from oracle import oracle as O
    L = Layout(ng=32, nnt=1, nns=2, ratio_cs=4, ngb=4, app=0.1)
    img = build_image(*ic.uniform_random(3000, 32.0, 13), L)
    before = FineKick.launch_count()
    vp, _, _ = LR.pm2_force(img, 3.5, 14.0, 1.0, SIXPI, 1.0)
    assert FineKick.launch_count() - before == 5  # no work list
    act = img.active
    d = (vp - img.vp)[act].astype(np.float64)
    r = O.pm2(img, 3.5, 14.0, 1.0, SIXPI, 1.0)["dv"][act]
    assert np.sqrt(np.sum((d - r) ** 2) / np.sum(r ** 2)) < 1e-5


def test_crowded_brick(gpu):
    from cube2_b200 import longrange as LR
    from cube2_b200.kick import FineKick
    from oracle import oracle as O
    img = _image()
    before = FineKick.launch_count()
    vp, f2, vmax = LR.pm2_force(img, 3.5, 14.0, 1.0, SIXPI, 1.0)
    # cell table, work list, deposit, Green multiply (40^3 meshes: cuFFT), force, gather
    assert FineKick.launch_count() - before == 6
    ref = O.pm2(img, 3.5, 14.0, 1.0, SIXPI, 1.0)
    act = img.active
    d, r = vp[act].astype(np.float64), ref["vp"][act].astype(np.float64)
    assert np.sqrt(np.sum((d - r) ** 2) / np.sum(r ** 2)) < 1e-5
    assert np.all(vp[~act] == img.vp[~act])
    assert abs(f2 - ref["f2max"]) <= 1e-5 * ref["f2max"]


def test_particle_number_below_the_counts(gpu):
    """PM2 takes its particles from the cells' counts: a smaller n_used, for which the work list is too short, changes
    nothing but the split of the crowded bricks."""
    import torch
    from cube2_b200 import learned as Ln
    from cube2_b200.kick import CUBE_PM3_SUBTILE, FineKick, lib
    img = _image()
    rho, idx, xp, vp0 = Ln.device_image(img, gpu)
    FineKick(img.layout, pm3_mode=CUBE_PM3_SUBTILE).configure()
    f2, vmax = ctypes.c_float(), (ctypes.c_float * 3)()

    def call(n):
        vp = vp0.clone()
        torch.cuda.synchronize()  # the library has its own stream
        p = [ctypes.c_void_p(t.data_ptr()) for t in (rho, idx, xp)]
        f = [ctypes.c_float(x) for x in (1.0, SIXPI, 1.0, 3.5, 14.0)]
        assert lib().cube_pm2_force_device(*p, ctypes.c_int64(n), ctypes.c_void_p(vp.data_ptr()), *f,
                                           ctypes.byref(f2), vmax, None) == 0
        torch.cuda.synchronize()
        return vp.double()
    want, got = call(img.n_used), call(1000)
    assert float((got - want).pow(2).sum()) <= 1e-12 * float(want.pow(2).sum())
