"""Q points side by side: four at a time (N up to 3104), two (above), more and fewer points than lanes, against
each point by itself: the sums do not depend on what runs beside them, so the energies are the same bits."""
import numpy as np
import pytest

from wantibexos_b200 import synth, wtbgpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nv,nc,nq", [(6, 2, 2, 2), (6, 2, 2, 3), (12, 2, 2, 9), (13, 2, 2, 2), (13, 2, 2, 5), (29, 2, 2, 3)])
def test_q_points_side_by_side(n, nv, nc, nq, gpu_ctx):
    ctx, m = gpu_ctx, synth.config_model("c1")
    a1, a2, a3 = m.rlat
    s = 2.0 * float(np.float32(np.pi)) / abs(a1 @ np.cross(a2, a3))
    b1, b2 = s * np.cross(a2, a3), s * np.cross(a3, a1)
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    k = (b1 / n * i[..., None] + b2 / n * j[..., None]).reshape(-1, 3)
    c = wtbgpu.coulomb_params("V2DRK", [n, n, 1], 1e-3, [1, 1, 1], 1.0, 1.0, 0.0, 40.0)
    q = np.array([[0.03 * i * np.linalg.norm(b1), *(0.03 * i * b1)] for i in range(nq)])
    ctx.set_model(m)
    ctx.bands(k, nv, nc, want_vectors=False)
    for _ in range(2):   # buffers made, then kept
        W, _ = ctx.bse_q_batch([k + x[1:] for x in q], q, c)
    for x, w in zip(q, W):
        assert np.array_equal(w, ctx.bse_q_batch([k + x[1:]], x[None], c)[0][0])
