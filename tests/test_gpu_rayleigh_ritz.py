"""The Rayleigh-Ritz eigensolver over its range: blocks of 8 to 40 vectors (problems of 8 to 80, one and two
rows a lane, one to three vectors a warp), and levels that come in equal pairs. The oracle is the dense solve.
Tolerances: a residual r moves a level by at most r (and by r^2 over the distance to the others, below 1e-9,
where they are apart), vectors orthonormal to 1e-10 as the block is kept."""
import numpy as np
import pytest

from wantibexos_b200 import synth, wtbgpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs", [False, True])
@pytest.mark.parametrize("nb", [8, 16, 24, 32, 40])
def test_lowest_against_dense(nb, pairs, gpu_ctx):
    ctx, n = gpu_ctx, 9
    m = synth.config_model("c1")
    if pairs:
        h = synth.make_gapped_model(4, 2, (-1.5, 0.3), (1.5, 0.3), 31)
        m = synth.make_gapped_model(8, 2, (-1.5, 0.3), (1.5, 0.3), 32)
        m.hre[:], m.him[:] = np.kron(h.hre, np.eye(2)), np.kron(h.him, np.eye(2))
    a1, a2, a3 = m.rlat
    s = 2.0 * float(np.float32(np.pi)) / abs(a1 @ np.cross(a2, a3))
    b1, b2 = s * np.cross(a2, a3), s * np.cross(a3, a1)
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    c = wtbgpu.coulomb_params("V2DRK", [n, n, 1], 1e-3, [1, 1, 1], 1.0, 1.0, 0.0, 40.0)
    ctx.set_model(m)
    ctx.bands((b1 / n * i[..., None] + b2 / n * j[..., None]).reshape(-1, 3), 2, 2, want_vectors=False)
    ctx.velocity(0.05, want=False)
    ctx.bse_build(c)
    nev = nb - 4
    W, act, X, it, res = ctx.bse_davidson(nev, nb=nb, tol=1e-7, want_vectors=True)
    H = ctx.bse_get_matrix()
    H = np.triu(H) + np.triu(H, 1).conj().T
    Wd, _ = ctx.bse_solve(False, False)
    assert res < 1e-7
    assert np.abs(W - Wd[:nev]).max() < (1e-7 if pairs else 1e-9)
    assert np.abs(X.conj().T @ X - np.eye(nev)).max() < 1e-10
    assert np.linalg.norm(H @ X - X * W[None], axis=0).max() < 2e-7
