"""Exciton vectors where the back-transforms change form: groups of 32 sweeps with a ragged last one, one to
four chunks of eight vectors, one 32-row tile a CTA against several (from about 4800 rows), and levels that
come in equal pairs. The vectors are held to the matrix that the library built: residual 20 N eps |H|,
orthonormal to 20 N eps."""
import numpy as np
import pytest

from wantibexos_b200 import synth, wtbgpu

pytestmark = pytest.mark.gpu


def check(ctx, m, n1, n2, nv, nc, nev):
    N = n1 * n2 * nv * nc
    a1, a2, a3 = m.rlat
    s = 2.0 * float(np.float32(np.pi)) / abs(a1 @ np.cross(a2, a3))
    b1, b2 = s * np.cross(a2, a3), s * np.cross(a3, a1)
    i, j = np.meshgrid(np.arange(n1), np.arange(n2), indexing="ij")
    c = wtbgpu.coulomb_params("V2DRK", [n1, n2, 1], 1e-3, [1, 1, 1], 1.0, 1.0, 0.0, 40.0)
    ctx.set_model(m)
    ctx.bands((b1 / n1 * i[..., None] + b2 / n2 * j[..., None]).reshape(-1, 3), nv, nc, want_vectors=False)
    ctx.velocity(0.05, want=False)
    ctx.bse_build(c)
    U = np.triu(ctx.bse_get_matrix())
    H = U + np.triu(U, 1).conj().T
    W, _ = ctx.bse_solve(False, False)
    tol = 20 * N * np.finfo(float).eps
    for n0, n1_ in nev:
        A = ctx.bse_eigvecs(n0, n1_)
        assert np.linalg.norm(H @ A - A * W[None, n0 - 1:n1_], axis=0).max() <= tol * np.abs(W).max()
        assert np.abs(A.conj().T @ A - np.eye(A.shape[1])).max() <= tol
        assert np.all(A[-1].imag == 0.0) and np.all(A[-1].real >= 0.0)


@pytest.mark.parametrize("n1,n2", [(34, 1), (65, 1), (97, 1), (33, 32), (70, 70)])
def test_vectors(n1, n2, gpu_ctx):
    N = n1 * n2
    check(gpu_ctx, synth.config_model("c1"), n1, n2, 1, 1, [(1, 1), (2, 9), (N - 7, N), (1, min(N, 33))])


def test_vectors_of_pairs(gpu_ctx):
    h = synth.make_gapped_model(4, 2, (-1.5, 0.3), (1.5, 0.3), 31)
    p = synth.make_gapped_model(8, 2, (-1.5, 0.3), (1.5, 0.3), 32)
    p.hre[:], p.him[:] = np.kron(h.hre, np.eye(2)), np.kron(h.him, np.eye(2))
    check(gpu_ctx, p, 7, 5, 2, 2, [(1, 8), (2, 3), (3, 20)])
