"""Per-k diagonalisation at the edges of its block sizes and work areas: band counts around one, two, four
and eight warps a k-point, odd ones (a round then leaves one index out), the largest in shared memory and
in global memory; few k-points and more than the device holds at once, ragged against the 32 x 32 tiles of
the vectors' layout. The oracle is LAPACK's ZHEEV on H(k). Tolerances: Jacobi leaves a backward error of a
few w eps |H| per sweep, ten sweeps at most: 50 w eps |H|."""
import numpy as np
import pytest

from oracle import wtb_oracle as O
from wantibexos_b200 import synth

pytestmark = pytest.mark.gpu


def check(ctx, m, kpt, some):
    e, v, no = ctx.eigsys(kpt)
    for k in some:
        H = O.hk(m, kpt[k])
        er, _, nr = O.eigsys(m, kpt[k])
        tol = 50 * m.w * np.finfo(float).eps * max(np.abs(er).max(), 1e-300)
        V = v[k].T                                   # columns
        assert no[k] == nr
        assert np.abs(e[k] - er).max() <= tol
        assert np.linalg.norm(H @ V - V * e[k][None], axis=0).max() <= 2 * tol
        assert np.abs(V.conj().T @ V - np.eye(m.w)).max() <= 50 * m.w * np.finfo(float).eps
        assert np.all(V[0].imag == 0.0)              # the gauge of ZHEEV('V', 'L')
    return e, v


@pytest.mark.parametrize("w", [1, 2, 3, 7, 8, 9, 16, 17, 31, 32, 33, 40, 77, 79, 80])
@pytest.mark.parametrize("nk", [1, 33, 700])
def test_eigsys_against_lapack(w, nk, gpu_ctx):
    m = synth.make_hex_model(w, 1, (-1.5, 0.3), (1.5, 0.3), 900 + w)
    kpt = np.random.default_rng(nk).uniform(-1.5, 1.5, (nk, 3))
    gpu_ctx.set_model(m)
    e, v = check(gpu_ctx, m, kpt, sorted({0, nk // 2, nk - 2 if nk > 1 else 0, nk - 1}))
    # the band window of the exciton path holds the same numbers
    nocp = gpu_ctx.eigsys(kpt, want_vectors=False)[2]
    if w >= 2 and (nocp == nocp[0]).all() and 0 < nocp[0] < w:
        eb, vb, nb, _ = gpu_ctx.bands(kpt, 1, 1)
        assert np.array_equal(nb, nocp)
        n0 = nocp[0]
        assert np.array_equal(eb, e[:, n0 - 1:n0 + 1]) and np.array_equal(vb, v[:, n0 - 1:n0 + 1])


@pytest.mark.parametrize("w", [2, 9, 24])
def test_diagonal_and_degenerate(w, gpu_ctx):
    """Nothing to rotate, and levels that coincide: H(k) = diag, exact; then all levels in pairs."""
    m = synth.make_hex_model(w, 1, (-1.5, 0.3), (1.5, 0.3), 7, hop_scale=0.0, h0_scale=0.0)
    kpt = np.random.default_rng(1).uniform(-1, 1, (5, 3))
    gpu_ctx.set_model(m)
    e, _, _ = gpu_ctx.eigsys(kpt)
    i0 = int(np.flatnonzero((m.rvec == 0).all(axis=1))[0])
    assert np.array_equal(e, np.broadcast_to(np.sort(np.diag(m.hre[i0])), e.shape))
    p = synth.make_hex_model(2 * w, 1, (-1.5, 0.3), (1.5, 0.3), 8)
    h = synth.make_hex_model(w, 1, (-1.5, 0.3), (1.5, 0.3), 8)
    p.hre[:], p.him[:] = np.kron(h.hre, np.eye(2)), np.kron(h.him, np.eye(2))
    gpu_ctx.set_model(p)
    check(gpu_ctx, p, kpt, range(5))


def test_vectors_in_several_pieces(gpu_ctx):
    """3000 k-points of 60 bands: 173 MB of vectors, copied in two ranges of the component."""
    m = synth.make_hex_model(60, 1, (-1.5, 0.3), (1.5, 0.3), 11)
    kpt = np.random.default_rng(2).uniform(-1.5, 1.5, (3000, 3))
    gpu_ctx.set_model(m)
    check(gpu_ctx, m, kpt, [0, 1499, 2998, 2999])
