"""Exciton solves whose numbers lie far from 1: couplings far below the diagonal, and whole problems taken by a
power of two. Energies, and with V2DOH (W proportional to 1 / EZ) the kernel, scale by that power exactly, so the
oracle is the same problem at scale 1, or the diagonal where the couplings are below its rounding. Tolerances: a
backward error of N eps |H|, taken 20 times as for the band reduction elsewhere; strengths sum to |h|^2 to 1e-12
per N terms."""
import numpy as np
import pytest

from wantibexos_b200 import synth, wtbgpu

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def mesh(m, n1, n2):
    a1, a2, a3 = m.rlat
    s = 2.0 * float(np.float32(np.pi)) / abs(a1 @ np.cross(a2, a3))
    b1, b2 = s * np.cross(a2, a3), s * np.cross(a3, a1)
    i, j = np.meshgrid(np.arange(n1), np.arange(n2), indexing="ij")
    return (b1 / n1 * i[..., None] + b2 / n2 * j[..., None]).reshape(-1, 3)


def build(ctx, n1, n2, energy, coupling, nv=1, nc=1):
    """The model's energies times 2^energy, its couplings times 2^coupling."""
    m = synth.config_model("c1")
    m.hre[:], m.him[:] = np.ldexp(m.hre, energy), np.ldexp(m.him, energy)
    m.efermi = float(np.ldexp(m.efermi, energy))
    m.scs = float(np.ldexp(m.scs, energy))
    ctx.set_model(m)
    ctx.bands(mesh(m, n1, n2), nv, nc, want_vectors=False)
    h = ctx.velocity(0.05)
    ctx.bse_build(wtbgpu.coulomb_params("V2DOH", [n1, n2, 1], 1e-3, [1, 1, 1], 0.0, float(np.ldexp(1.0, -coupling)), 0.0,
                                        0.0))
    return h


@pytest.mark.parametrize("coupling", [-200, -260, -350, -400, -480])
@pytest.mark.parametrize("n1,n2", [(17, 2), (16, 8), (43, 3)])
def test_couplings_far_below_the_diagonal(n1, n2, coupling, gpu_ctx):
    ctx = gpu_ctx
    h = build(ctx, n1, n2, 0, coupling)
    diag = np.sort(np.diag(ctx.bse_get_matrix()).real)
    W, act = ctx.bse_solve(True, True)
    assert np.abs(W - diag).max() <= 20 * len(W) * EPS * np.abs(diag).max()
    for col, v in ((0, 0), (1, 1), (2, 2), (6, 3), (7, 4)):
        norm = (np.abs(h[:, v]) ** 2).sum()
        assert abs(act[:, col].sum() - norm) <= 1e-12 * len(W) * norm + 1e-14


@pytest.mark.parametrize("scale", [-420, -340, -250, 250, 340, 420])
@pytest.mark.parametrize("n1,n2", [(17, 2), (16, 8)])
def test_whole_problem_scaled(n1, n2, scale, gpu_ctx):
    ctx = gpu_ctx
    build(ctx, n1, n2, 0, 0)
    W0, _ = ctx.bse_solve(want_act=False)
    build(ctx, n1, n2, scale, scale)
    W, _ = ctx.bse_solve(want_act=False)
    assert np.abs(np.ldexp(W, -scale) - W0).max() <= 20 * len(W) * EPS * np.abs(W0).max()
