"""Dense -> band where the products around the panels change form: the last panels of a matrix (1, 16 and 17
rows and more), the 16-row tiles, one tile a CTA against several (from about 2400 rows), the first and the
second panel of a look-ahead group, an odd and an even number of panels. The oracle is the one-stage
reduction of the same matrix. N eps |H| is below 1e-11 eV; the norm of h is kept to 1e-12 per N terms."""
import numpy as np
import pytest

from wantibexos_b200 import synth, wtbgpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1,n2", [(34, 1), (48, 1), (49, 1), (64, 1), (65, 1), (9, 9), (97, 1), (16, 8), (43, 3), (49, 49),
                                   (50, 48), (80, 31)])
def test_stage1_against_one_stage(n1, n2, gpu_ctx):
    ctx, m, N = gpu_ctx, synth.config_model("c1"), n1 * n2
    a1, a2, a3 = m.rlat
    s = 2.0 * float(np.float32(np.pi)) / abs(a1 @ np.cross(a2, a3))
    b1, b2 = s * np.cross(a2, a3), s * np.cross(a3, a1)
    i, j = np.meshgrid(np.arange(n1), np.arange(n2), indexing="ij")
    c = wtbgpu.coulomb_params("V2DRK", [n1, n2, 1], 1e-3, [1, 1, 1], 1.0, 1.0, 0.0, 40.0)
    ctx.set_model(m)
    ctx.bands((b1 / n1 * i[..., None] + b2 / n2 * j[..., None]).reshape(-1, 3), 1, 1, want_vectors=False)
    h = ctx.velocity(0.05)
    out = []
    try:
        for mode in (1, 2, 2):
            ctx.set_reduction(mode)
            ctx.bse_build(c)
            out.append(ctx.bse_solve(True, True))
    finally:
        ctx.set_reduction(0)
    assert np.abs(out[0][0] - out[1][0]).max() < 2e-11
    assert np.array_equal(out[1][0], out[2][0]) and np.array_equal(out[1][1], out[2][1])   # no sum depends on timing
    for col, v in ((0, 0), (1, 1), (2, 2), (6, 3), (7, 4)):
        norm = (np.abs(h[:, v]) ** 2).sum()
        assert abs(out[1][1][:, col].sum() - norm) <= 1e-12 * N * norm + 1e-14
