"""Stage 1 in the forms that large matrices take, at small sizes: look-ahead groups of four and of three panels (panel
counts of every remainder, so that the last group has one to four), and every panel factored by the whole grid. The
oracle is the one-stage reduction of the same matrix. N eps |H| is below 1.5e-11 eV at N = 3135; the norm of h is kept
to 1e-12 per N terms; vectors to 1e-11 as in the tests of the chase. Two runs give the same bits, and so do a Q point
alone and in a group."""
import numpy as np
import pytest

from wantibexos_b200 import synth, wtbgpu

pytestmark = pytest.mark.gpu

MODEL = synth.config_model("c1")


def mesh(n1, n2):
    a1, a2, a3 = MODEL.rlat
    s = 2.0 * float(np.float32(np.pi)) / abs(a1 @ np.cross(a2, a3))
    b1, b2 = s * np.cross(a2, a3), s * np.cross(a3, a1)
    i, j = np.meshgrid(np.arange(n1), np.arange(n2), indexing="ij")
    return (b1 / n1 * i[..., None] + b2 / n2 * j[..., None]).reshape(-1, 3), b1


@pytest.mark.parametrize("mode", [4, 5])
@pytest.mark.parametrize("n1,n2", [(34, 1), (33, 2), (43, 3), (12, 12), (163, 1), (15, 13), (16, 16), (33, 32), (50, 48),
                                   (57, 55)])
def test_large_forms_against_one_stage(n1, n2, mode, gpu_ctx):
    ctx, N = gpu_ctx, n1 * n2
    k, _ = mesh(n1, n2)
    c = wtbgpu.coulomb_params("V2DRK", [n1, n2, 1], 1e-3, [1, 1, 1], 1.0, 1.0, 0.0, 40.0)
    ctx.set_model(MODEL)
    ctx.bands(k, 1, 1, want_vectors=False)
    h = ctx.velocity(0.05)
    out = []
    try:
        for md in (1, mode, mode):
            ctx.set_reduction(md)
            ctx.bse_build(c)
            if N < 300 and md == 1:
                U = np.triu(ctx.bse_get_matrix())
                H = U + np.triu(U, 1).conj().T
            out.append(ctx.bse_solve(True, True))
        A = ctx.bse_eigvecs(1, min(N, 32))
    finally:
        ctx.set_reduction(0)
    assert np.abs(out[0][0] - out[1][0]).max() < 3e-11
    assert np.array_equal(out[1][0], out[2][0]) and np.array_equal(out[1][1], out[2][1])
    for col, v in ((0, 0), (1, 1), (2, 2), (6, 3), (7, 4)):
        norm = (np.abs(h[:, v]) ** 2).sum()
        assert abs(out[1][1][:, col].sum() - norm) <= 1e-12 * N * norm + 1e-14
    if N < 300:
        assert np.abs(H @ A - A * out[1][0][None, :A.shape[1]]).max() < 1e-11
    assert np.abs(A.conj().T @ A - np.eye(A.shape[1])).max() < 1e-11


@pytest.mark.parametrize("mode", [4, 5])
def test_large_forms_in_a_group_of_q(mode, gpu_ctx):
    ctx, (n1, n2) = gpu_ctx, (23, 7)
    k, b1 = mesh(n1, n2)
    c = wtbgpu.coulomb_params("V2DRK", [n1, n2, 1], 1e-3, [1, 1, 1], 1.0, 1.0, 0.0, 40.0)
    q = np.array([[0.0, *(0.03 * i * b1)] for i in range(5)])
    ctx.set_model(MODEL)
    ctx.set_reduction(mode)
    try:
        ctx.bands(k, 1, 1, want_vectors=False)
        W, _ = ctx.bse_q_batch([k + x[1:] for x in q], q, c)
        for i in range(len(q)):
            assert np.array_equal(W[i], ctx.bse_q_eigenvalues(k + q[i, 1:], q[i], c))
    finally:
        ctx.set_reduction(0)
