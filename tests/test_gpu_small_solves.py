"""The smallest dense solves, around the size below which all vectors come from inverse iteration (N = 16): levels,
strengths and vectors, also of a model with every level in pairs. The oracle is LAPACK on the matrix that the library
built; N eps |H| is below 1e-13, taken 100 times; the strengths sum to |h|^2 to 1e-12 per N terms."""
import numpy as np
import pytest
import scipy.linalg as sla

from wantibexos_b200 import synth, wtbgpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs", [False, True])
@pytest.mark.parametrize("n", [2, 3, 7, 15, 16, 17])
def test_small_solves(n, pairs, gpu_ctx):
    ctx, m, nb = gpu_ctx, synth.config_model("c1"), 1
    if pairs:
        h = synth.make_gapped_model(4, 2, (-1.5, 0.3), (1.5, 0.3), 31)
        m, nb = synth.make_gapped_model(8, 2, (-1.5, 0.3), (1.5, 0.3), 32), 2
        m.hre[:], m.him[:] = np.kron(h.hre, np.eye(2)), np.kron(h.him, np.eye(2))
        n = max(1, n // 4)
    a1, a2, a3 = m.rlat
    b1 = 2.0 * float(np.float32(np.pi)) / abs(a1 @ np.cross(a2, a3)) * np.cross(a2, a3)
    ctx.set_model(m)
    ctx.bands(b1 / n * np.arange(n)[:, None], nb, nb, want_vectors=False)
    v = ctx.velocity(0.05)
    ctx.bse_build(wtbgpu.coulomb_params("V2DRK", [n, 1, 1], 1e-3, [1, 1, 1], 1.0, 1.0, 0.0, 40.0))
    U = np.triu(ctx.bse_get_matrix())
    H = U + np.triu(U, 1).conj().T
    N = len(H)
    W, act = ctx.bse_solve(True, True)
    assert np.abs(W - sla.eigvalsh(H)).max() < 1e-11
    for col, x in ((0, 0), (1, 1), (2, 2), (6, 3), (7, 4)):
        norm = (np.abs(v[:, x]) ** 2).sum()
        assert abs(act[:, col].sum() - norm) <= 1e-12 * N * norm + 1e-14
    A = ctx.bse_eigvecs(1, N)
    assert np.abs(H @ A - A * W[None]).max() < 1e-11
    assert np.abs(A.conj().T @ A - np.eye(N)).max() < 1e-11
