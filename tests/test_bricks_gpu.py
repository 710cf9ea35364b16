"""The PM3 brick kernels where their geometry is ragged: tiles that are no whole number of bricks (one to five
coarse cells of a brick's two), buffered subtile meshes of 1 to 4 coarse cells at levels whose bricks
hold two cells, one, or none (level 4 takes the unbricked kernels), a tile buffer of more than one
cell, and small meshes.  Against the restatement, which sums in FP64: FP32 meshes and transforms
of these sizes differ from it by a few 1e-7 of the rms, the bar is the 1e-5 of the other PM3 tests.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIXPI = float(np.float32(6 * np.pi))
TOL = 1e-5


def _rel_rms(a, b):
    return float(np.sqrt(np.sum((a - b) ** 2) / np.sum(b ** 2)))


def _image(ng, nnt, nns, ngb=4, n=4000):
    from cube2_b200.layout import Layout, build_image
    rng = np.random.default_rng(ng + nnt)
    L = Layout(ng=ng, nnt=nnt, nns=nns, ratio_cs=4, ngb=ngb, app=0.1)
    pos = np.concatenate([ng * rng.random((n, 3)), np.mod(ng - 0.3 * rng.random((n // 4, 3)), ng)])  # a clump at the corner
    return build_image(pos, (0.05 * rng.standard_normal(pos.shape)).astype(np.float32), L)


def _compare(img, vp, f2, vmax, ref):
    act = img.active
    assert np.array_equal(vp[~act], img.vp[~act])
    assert _rel_rms((vp - img.vp)[act].astype(np.float64), (ref["vp"] - img.vp)[act].astype(np.float64)) < TOL
    assert abs(f2 - ref["f2max"]) <= 1e-5 * ref["f2max"]
    np.testing.assert_allclose(vmax, ref["vmax"], rtol=1e-5)


@pytest.mark.parametrize("ng,nnt", [(12, 1), (20, 1), (24, 2), (36, 3), (40, 2)])
def test_periodic_ragged_tiles(gpu, ng, nnt):
    from cube2_b200.kick import CUBE_PM3_PERIODIC, FineKick
    from cube2_b200.layout import RATIO_SF, ixyz3_table
    from oracle import oracle as O
    img = _image(ng, nnt, 1)
    L = img.layout
    fk = FineKick(L, pm3_mode=CUBE_PM3_PERIODIC, apm3f=4.0)
    vp, f2, vmax, _ = fk.c_pm3_force_kernel(img, np.arange(1, L.ns3 + 1, dtype=np.int32), np.full(L.ns3, 2, np.int32),
                                            ixyz3_table(L), RATIO_SF, 1.0, SIXPI, 1.0)
    _compare(img, vp, f2, vmax, O.pm3_periodic(img, 2, O.green(2 * ng, 4.0, 0.0, 0.5), 1.0, SIXPI, 1.0))


@pytest.mark.parametrize("ng,nnt,nns,ngb", [(8, 2, 1, 4), (16, 2, 2, 4), (24, 1, 2, 4), (24, 2, 1, 8), (32, 2, 1, 4)])
def test_subtile_ragged_meshes(gpu, ng, nnt, nns, ngb):
    from cube2_b200.kick import CUBE_PM3_SUBTILE, FineKick
    from cube2_b200.layout import RATIO_SF, ixyz3_table
    from oracle import oracle as O
    img = _image(ng, nnt, nns, ngb)
    L = img.layout
    ires = np.array([2 + q % 3 for q in range(L.ns3)], np.int32)
    greens = {}
    for lev in sorted(set(ires.tolist())):
        rsf = int(RATIO_SF[lev - 1])
        greens[lev] = O.green((L.ntt + 2) * 4 * rsf, 3.5, 3.5 * rsf, 1.0 / rsf)
    fk = FineKick(L, pm3_mode=CUBE_PM3_SUBTILE)
    isort, ix = np.arange(1, L.ns3 + 1, dtype=np.int32), ixyz3_table(L)
    vp, f2, vmax, _ = fk.c_pm3_force_kernel(img, isort, ires, ix, RATIO_SF, 1.0, SIXPI, 1.0, greens=greens)
    _compare(img, vp, f2, vmax, O.pm3_subtile(img, ires, ix, RATIO_SF, greens, 1.0, SIXPI, 1.0))
