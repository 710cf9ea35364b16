"""The pair-list PP kernel at the sizes where its decomposition changes, against the FP64 pair sum of
oracle/pp_direct.py.

Item sizes around the powers of two that set a particle's replicas, chunks and their remainders; stencils that
fit one batch of candidates and that need several; PP ranges of one to three cells; pairs inside the
softening length, on top of one another and at the edge of the range.  The FP32 force of a
particle sums at most a few thousand terms of one law, each within about 1e-6 of its FP64 value, and
its decoded positions are exact, so 2e-6 of the rms force bounds the rms error.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIXPI = float(np.float32(6 * np.pi))


def _kick(pos, ng, apm3f, app, shape):
    """(FP32 PP velocity change, FP64 force) of every particle of one periodic tile."""
    from cube2_b200 import kick as K
    from cube2_b200.layout import RATIO_SF, Layout, apm3_table, build_image, ixyz3_table
    from cube2_b200.workloads import physical_positions
    from oracle.pp_direct import pp_forces
    L = Layout(ng=ng, nnt=1, nns=1, ratio_cs=4, ngb=4, app=app)
    img = build_image(pos, np.zeros_like(pos, np.float32), L)
    fk = K.FineKick(L, pm3_mode=K.CUBE_PM3_PERIODIC)
    try:
        K.pp_set_shape(shape)
        vp, f2, _, _, _ = fk.c_pp_force_kernel(img, np.ones(1, np.int32), np.full(1, 2, np.int32), ixyz3_table(L),
                                               apm3_table(apm3f), RATIO_SF, 1.0, SIXPI, 1.0)
    finally:
        K.pp_set_shape(-1)
    dv = np.zeros((pos.shape[0], 3))
    dv[img.pid[img.active]] = vp[img.active]
    kick = float(np.float32(np.float32(SIXPI) / np.float32(6.0))) / np.pi
    want = kick * pp_forces(physical_positions(img), ng, float(np.float32(app)),
                            np.full(pos.shape[0], float(apm3_table(apm3f)[1])))
    return dv, want, f2


def _check(pos, ng, apm3f=4.0, app=0.1, shape=0):
    dv, want, f2 = _kick(pos, ng, apm3f, app, shape)
    scale = np.sqrt(np.mean(np.sum(want ** 2, axis=1)))
    assert scale > 0
    assert np.sqrt(np.mean(np.sum((dv - want) ** 2, axis=1))) <= 2e-6 * scale
    top = float(np.max(np.sum((want / 1.0) ** 2, axis=1)))
    assert abs(f2 - top) <= 2e-5 * top


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 8, 9, 12, 15, 16, 17, 31, 33])
def test_particles_per_cell(gpu, n):
    """Every other PP cell (2 fine cells a side) along x holds n particles: items of n (or chunks of 16 and the rest)."""
    rng = np.random.default_rng(n)
    c = np.stack(np.meshgrid(np.arange(0, 8, 2), np.arange(8), np.arange(8), indexing="ij"), -1).reshape(-1, 1, 3)
    pos = (2 * (c + rng.random((c.shape[0], n, 3)))).reshape(-1, 3)
    _check(pos, 16)


@pytest.mark.parametrize("shape", [0, 4, 5, 6])
@pytest.mark.parametrize("dense", [40, 400, 3000])
def test_crowded_stencils(gpu, dense, shape):
    """A clump in one corner of a cell, with sparse cells around: one batch of candidates up to dozens."""
    rng = np.random.default_rng(dense)
    pos = np.concatenate([8.0 + 0.9 * rng.random((dense, 3)), 16 * rng.random((2000, 3))])
    _check(pos, 16, shape=shape)


@pytest.mark.parametrize("apm3f,app", [(4.0, 0.0), (3.5, 0.1), (2.0, 0.1), (1.0, 0.3), (0.5, 0.05)])
def test_ranges_and_softening(gpu, apm3f, app):
    """Ranges of 2, 1.75, 1, 0.5 and 0.25 fine cells, without softening and with much of it."""
    rng = np.random.default_rng(7)
    pos = np.concatenate([16 * rng.random((4000, 3)), 4.0 + 0.5 * rng.random((200, 3))])
    _check(pos, 16, apm3f, app)


def test_coincident_and_edge_pairs(gpu):
    """Particles on top of one another and pairs just inside and outside the range."""
    rng = np.random.default_rng(9)
    a = 16 * rng.random((300, 3))
    r = np.repeat([1.999, 2.0, 2.001, 0.0999, 0.1001], 60)[:, None]
    u = rng.standard_normal((300, 3))
    b = a + r * u / np.linalg.norm(u, axis=1, keepdims=True)
    _check(np.mod(np.concatenate([a, a[:40], b]), 16), 16)
