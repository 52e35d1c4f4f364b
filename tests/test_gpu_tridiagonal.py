"""Eigenvalues and strengths of the tridiagonal form at the edges of its tiles (32 and 128 rows, blocks of
eight rows, warps of 32 vectors), and with levels that coincide: pairs equal to rounding, and pairs split by
less than the cluster distance. The oracle is LAPACK on the matrix that the library built. Tolerances: a
backward error d = 20 N eps |H| moves a level by d and turns a vector by d over its distance D to the
others, which changes the strength (summed over levels closer than 1e-6) by at most 4 |h|^2 d / D."""
import numpy as np
import pytest
import scipy.linalg as sla

from wantibexos_b200 import synth, wtbgpu

pytestmark = pytest.mark.gpu


def mesh(m, n1, n2):
    a1, a2, a3 = m.rlat
    s = 2.0 * float(np.float32(np.pi)) / abs(a1 @ np.cross(a2, a3))
    b1, b2 = s * np.cross(a2, a3), s * np.cross(a3, a1)
    i, j = np.meshgrid(np.arange(n1), np.arange(n2), indexing="ij")
    return (b1 / n1 * i[..., None] + b2 / n2 * j[..., None]).reshape(-1, 3)


def check(ctx, m, n1, n2, nv, nc):
    c = wtbgpu.coulomb_params("V2DRK", [n1, n2, 1], 1e-3, [1, 1, 1], 1.0, 1.0, 0.0, 40.0)
    ctx.set_model(m)
    ctx.bands(mesh(m, n1, n2), nv, nc, want_vectors=False)
    h = ctx.velocity(0.05)
    ctx.bse_build(c)
    U = np.triu(ctx.bse_get_matrix())
    H = U + np.triu(U, 1).conj().T
    W, act = ctx.bse_solve(True, True)
    N = len(W)
    ref, V = sla.eigh(H)
    d = 20 * N * np.finfo(float).eps * np.abs(ref).max()
    assert np.abs(W - ref).max() <= d
    first = np.flatnonzero(np.diff(ref, prepend=-np.inf) > 1e-6)
    last = np.append(first[1:], N) - 1
    below = np.diff(ref, prepend=-np.inf)[first]
    above = np.append(below[1:], np.inf)
    D = np.minimum(below, above)
    for col, v in ((0, 0), (1, 1), (2, 2), (6, 3), (7, 4)):
        want = np.abs(V.T @ h[:, v]) ** 2
        got = np.add.reduceat(act[:, col], first)
        norm = (np.abs(h[:, v]) ** 2).sum()
        assert np.all(np.abs(got - np.add.reduceat(want, first)) <= 4 * norm * d / D + 1e-14 * norm)
    return W, first, last


@pytest.mark.parametrize("n1,n2", [(2, 1), (7, 1), (8, 1), (9, 1), (31, 1), (32, 1), (11, 3), (13, 5), (127, 1),
                                   (16, 8), (43, 3), (16, 16), (257, 1)])
@pytest.mark.parametrize("reduction", [0, 1])
def test_sizes(n1, n2, reduction, gpu_ctx):
    gpu_ctx.set_reduction(reduction)
    try:
        check(gpu_ctx, synth.config_model("c1"), n1, n2, 1, 1)
    finally:
        gpu_ctx.set_reduction(0)


@pytest.mark.parametrize("split", [0.0, 1e-10, 3e-8])
def test_pairs(split, gpu_ctx):
    """Two copies of a model, its on-site levels changed by up to split: every exciton comes in groups of four,
    of levels equal to rounding (inverse iteration makes them), or about that distance apart."""
    h = synth.make_gapped_model(4, 2, (-1.5, 0.3), (1.5, 0.3), 31)
    p = synth.make_gapped_model(8, 2, (-1.5, 0.3), (1.5, 0.3), 32)
    assert np.array_equal(h.rvec, p.rvec)
    p.hre[:], p.him[:] = np.kron(h.hre, np.eye(2)), np.kron(h.him, np.eye(2))
    i0 = int(np.flatnonzero((p.rvec == 0).all(axis=1))[0])
    p.hre[i0] += np.diag(split * np.random.default_rng(3).uniform(0.0, 1.0, 8))
    W, first, last = check(gpu_ctx, p, 6, 5, 2, 2)
    assert len(first) <= len(W) // 2 + 1
