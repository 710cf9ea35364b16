"""cube_pp_work_stats describes the work list of the last PP kick, whatever else ran since: a kick without PP, PM1 and
PM2 leave it as it is, the next PP kick replaces it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIXPI = float(np.float32(6 * np.pi))


def test_work_stats_outlive_kicks_without_pp(gpu):
    from cube2_b200 import ic
    from cube2_b200 import kick as K
    from cube2_b200 import longrange as LR
    from cube2_b200.layout import RATIO_SF, Layout, apm3_table, build_image, ixyz3_table
    L = Layout(ng=64, nnt=2, nns=1, ratio_cs=4, ngb=4, app=0.1)
    img = build_image(*ic.lognormal_poisson(64, 1.5, 4100)[:2], L)
    few = build_image(*ic.uniform_random(500, 64.0, 3), L)
    fk = K.FineKick(L, pm3_mode=K.CUBE_PM3_PERIODIC, apm3f=4.0)
    isort, ires, ix = np.arange(1, L.ns3 + 1, dtype=np.int32), np.full(L.ns3, 2, np.int32), ixyz3_table(L)
    fk.c_pp_force_kernel(img, isort, ires, ix, apm3_table(4.0), RATIO_SF, 1.0, SIXPI, 1.0)
    want = K.pp_work_stats()
    assert want["items"] > 0 and want["max_ni"] > 0
    fk.c_pm3_force_kernel(img, isort, ires, ix, RATIO_SF, 1.0, SIXPI, 1.0)
    assert K.pp_work_stats() == want
    LR.pm1_force(img, 3.5, 1.0, SIXPI, 1.0, pm3_mode=K.CUBE_PM3_PERIODIC)
    assert K.pp_work_stats() == want
    fk.c_pp_force_kernel(few, isort, ires, ix, apm3_table(4.0), RATIO_SF, 1.0, SIXPI, 1.0)
    assert 0 < K.pp_work_stats()["items"] <= 500
