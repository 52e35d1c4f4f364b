"""Band -> tridiagonal (bulge chasing) at the edges of its blocks: dimensions around multiples of the
band width 32, down to the smallest the two-stage reduction takes, with five, ten (temperature) and no
velocity vectors, and several bands in one launch. The oracle is LAPACK's ZHEEV on the matrix that the
library built. Tolerances: a backward error of N eps |H| (N <= 225, |H| < 10 eV) is below 5e-13 eV,
taken 20 times; strengths are sums over vectors that are accurate to that error over the level
distance, so only their sum (the norm of h, 1e-12 relative per N terms) is held tightly."""
import numpy as np
import pytest
import scipy.linalg as sla

from wantibexos_b200 import synth, wtbgpu

pytestmark = pytest.mark.gpu

MODEL = synth.config_model("c1")
PI32 = float(np.float32(np.pi))


def mesh(n1, n2):
    a1, a2, a3 = MODEL.rlat
    s = 2.0 * PI32 / abs(a1 @ np.cross(a2, a3))
    b1, b2 = s * np.cross(a2, a3), s * np.cross(a3, a1)
    i, j = np.meshgrid(np.arange(n1), np.arange(n2), indexing="ij")
    return (b1 / n1 * i[..., None] + b2 / n2 * j[..., None]).reshape(-1, 3), b1


@pytest.mark.parametrize("n1,n2", [(17, 2), (9, 7), (8, 8), (13, 5), (12, 8), (97, 1), (16, 8), (43, 3), (23, 7), (15, 15)])
@pytest.mark.parametrize("temp", [None, 300.0])
def test_chase_against_lapack(n1, n2, temp, gpu_ctx):
    ctx, N = gpu_ctx, n1 * n2
    k, _ = mesh(n1, n2)
    c = wtbgpu.coulomb_params("V2DRK", [n1, n2, 1], 1e-3, [1, 1, 1], 1.0, 1.0, 0.0, 40.0)
    ctx.set_model(MODEL)
    ctx.set_temperature(temp is not None, temp or 0.0)
    ctx.set_reduction(2)
    try:
        ctx.bands(k, 1, 1, want_vectors=False)
        h = ctx.velocity(0.05)
        ctx.bse_build(c)
        U = np.triu(ctx.bse_get_matrix())
        H = U + np.triu(U, 1).conj().T
        W, act = ctx.bse_solve(True, True)
        A = ctx.bse_eigvecs(1, min(N, 32))
    finally:
        ctx.set_reduction(0)
        ctx.set_temperature(False)
    ref = sla.eigvalsh(H)
    assert np.abs(W - ref).max() < 1e-11
    if temp is None:
        for col, v in ((0, 0), (1, 1), (2, 2), (6, 3), (7, 4)):
            norm = (np.abs(h[:, v]) ** 2).sum()
            assert abs(act[:, col].sum() - norm) <= 1e-12 * N * norm + 1e-14
    # the stored reflectors: eigenvectors through the back-transform
    assert np.abs(H @ A - A * W[None, :A.shape[1]]).max() < 1e-11
    assert np.abs(A.conj().T @ A - np.eye(A.shape[1])).max() < 1e-11


@pytest.mark.parametrize("n1,n2,nq", [(17, 2, 3), (13, 5, 2), (15, 15, 5)])
def test_several_bands_in_one_launch(n1, n2, nq, gpu_ctx):
    ctx = gpu_ctx
    k, b1 = mesh(n1, n2)
    c = wtbgpu.coulomb_params("V2DRK", [n1, n2, 1], 1e-3, [1, 1, 1], 1.0, 1.0, 0.0, 40.0)
    q = np.array([[0.0, *(0.03 * i * b1)] for i in range(nq)])
    ctx.set_model(MODEL)
    ctx.set_reduction(2)
    try:
        ctx.bands(k, 1, 1, want_vectors=False)
        W, _ = ctx.bse_q_batch([k + x[1:] for x in q], q, c)
        for i in range(nq):
            ctx.bse_build_q(k + q[i, 1:], q[i], c)
            U = np.triu(ctx.bse_get_matrix())
            assert np.abs(W[i] - sla.eigvalsh(U + np.triu(U, 1).conj().T)).max() < 1e-11
    finally:
        ctx.set_reduction(0)


@pytest.mark.parametrize("n1,n2", [(544, 1), (545, 1), (33, 32), (46, 46), (57, 55), (56, 56), (59, 57)])
def test_panels_against_one_stage(n1, n2, gpu_ctx):
    """Panel QR on one cluster: dimensions where the CTA count and the rows per thread change, and
    (3192, 3363) where the first panels are too long for a cluster. N eps |H| is below 1.5e-11 eV."""
    ctx, N = gpu_ctx, n1 * n2
    k, _ = mesh(n1, n2)
    c = wtbgpu.coulomb_params("V2DRK", [n1, n2, 1], 1e-3, [1, 1, 1], 1.0, 1.0, 0.0, 40.0)
    ctx.set_model(MODEL)
    ctx.bands(k, 1, 1, want_vectors=False)
    h = ctx.velocity(0.05)
    out = []
    try:
        for mode in (1, 2):
            ctx.set_reduction(mode)
            ctx.bse_build(c)
            out.append(ctx.bse_solve(True, True))
    finally:
        ctx.set_reduction(0)
    (W1, a1), (W2, a2) = out
    assert np.abs(W1 - W2).max() < 3e-11
    for col, v in ((0, 0), (1, 1), (2, 2), (6, 3), (7, 4)):
        norm = (np.abs(h[:, v]) ** 2).sum()
        assert abs(a2[:, col].sum() - norm) <= 1e-12 * N * norm + 1e-14
        assert abs(a1[:, col].sum() - norm) <= 1e-12 * N * norm + 1e-14
