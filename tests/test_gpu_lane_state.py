"""Q points side by side in one context: a Q that fails in the middle of a group leaves the context as it was, so the
next call gives the bits of the one before; and with the temperature form on, every Q has the bits of a call of its
own. The split-BF16 form adds its FP32 partial sums in no fixed order, so two calls of one Q differ as well: there the
levels agree to 64 roundings of FP32 at the size of the matrix."""
import numpy as np
import pytest

from wantibexos_b200 import synth, wtbgpu

pytestmark = pytest.mark.gpu

MODEL = synth.config_model("c1")
N1 = 12


def setup(ctx):
    a1, a2, a3 = MODEL.rlat
    s = 2.0 * float(np.float32(np.pi)) / abs(a1 @ np.cross(a2, a3))
    b1, b2 = s * np.cross(a2, a3), s * np.cross(a3, a1)
    i, j = np.meshgrid(np.arange(N1), np.arange(N1), indexing="ij")
    k = (b1 / N1 * i[..., None] + b2 / N1 * j[..., None]).reshape(-1, 3)
    q = np.array([[0.0, *(0.03 * i * b1)] for i in range(7)])
    c = wtbgpu.coulomb_params("V2DRK", [N1, N1, 1], 1e-3, [1, 1, 1], 1.0, 1.0, 0.0, 40.0)
    ctx.set_model(MODEL)
    ctx.bands(k, 2, 2, want_vectors=False)
    return k, q, [k + x[1:] for x in q], c


@pytest.mark.parametrize("bad", [0, 1, 3, 6])
def test_a_q_that_fails_leaves_the_context_right(bad, gpu_ctx):
    k, q, kq, c = setup(gpu_ctx)
    W, _ = gpu_ctx.bse_q_batch(kq, q, c)
    broken = [x.copy() for x in kq]
    broken[bad][5] = np.nan
    with pytest.raises(wtbgpu.WtbgError) as err:
        gpu_ctx.bse_q_batch(broken, q, c)
    assert err.value.status == -7
    assert np.array_equal(gpu_ctx.bse_q_batch(kq, q, c)[0], W)
    gpu_ctx.velocity(0.05, want=False)
    gpu_ctx.bse_build(c)
    assert np.abs(gpu_ctx.bse_solve(False, False)[0] - W[0]).max() < 1e-11   # Q = 0: the same matrix up to rounding


@pytest.mark.parametrize("form", ["temperature", "bf16x3"])
def test_forms_side_by_side(form, gpu_ctx):
    try:
        if form == "temperature":
            gpu_ctx.set_temperature(True, 300.0)
        else:
            gpu_ctx.set_precision(1)
        _, q, kq, c = setup(gpu_ctx)
        W, _ = gpu_ctx.bse_q_batch(kq, q, c)
        for i in range(len(q)):
            one = gpu_ctx.bse_q_eigenvalues(kq[i], q[i], c)
            tol = 0.0 if form == "temperature" else 64 * np.finfo(np.float32).eps / 2 * np.abs(one).max()
            assert np.abs(W[i] - one).max() <= tol, i
    finally:
        gpu_ctx.set_temperature(False)
        gpu_ctx.set_precision(0)
