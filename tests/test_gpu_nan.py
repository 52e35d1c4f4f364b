"""Numbers that are none: a k-point that is NaN gives NaN levels (or the status of a k-point without empty states) and
leaves the others alone, in every block size and both work areas of the per-k solver; a kernel of NaN or infinite
elements goes through the dense solve, and the next solve gives the bits of the one before."""
import numpy as np
import pytest

from wantibexos_b200 import synth, wtbgpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [1, 2, 3, 8, 17, 33, 90])
def test_nan_k_point(w, gpu_ctx):
    m = synth.make_hex_model(w, 1, (-1.5, 0.3), (1.5, 0.3), 900 + w)
    kpt = np.random.default_rng(w).uniform(-1.5, 1.5, (5, 3))
    gpu_ctx.set_model(m)
    e, v, no = gpu_ctx.eigsys(kpt)
    bad = kpt.copy()
    bad[2, 0] = np.nan
    e1, v1, no1 = gpu_ctx.eigsys(bad)
    rest = [0, 1, 3, 4]
    assert np.isnan(e1[2]).all() and no1[2] == w
    assert np.array_equal(e1[rest], e[rest]) and np.array_equal(v1[rest], v[rest]) and np.array_equal(no1[rest], no[rest])
    if w >= 2:
        with pytest.raises(wtbgpu.WtbgError) as err:
            gpu_ctx.bands(bad, 1, 1)
        assert err.value.status in (-7, -6)   # no empty state, or (a k-point before it) too few in the window


@pytest.mark.parametrize("r0", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("n1,n2", [(17, 2), (16, 8), (43, 3)])
def test_kernel_that_is_no_number(n1, n2, r0, gpu_ctx):
    ctx, m = gpu_ctx, synth.config_model("c1")
    a1, a2, a3 = m.rlat
    s = 2.0 * float(np.float32(np.pi)) / abs(a1 @ np.cross(a2, a3))
    b1, b2 = s * np.cross(a2, a3), s * np.cross(a3, a1)
    i, j = np.meshgrid(np.arange(n1), np.arange(n2), indexing="ij")
    ctx.set_model(m)
    ctx.bands((b1 / n1 * i[..., None] + b2 / n2 * j[..., None]).reshape(-1, 3), 1, 1, want_vectors=False)
    ctx.velocity(0.05, want=False)

    def solve(r):
        ctx.bse_build(wtbgpu.coulomb_params("V2DRK", [n1, n2, 1], 1e-3, [1, 1, 1], 1.0, 1.0, 0.0, r))
        W, act = ctx.bse_solve(True, True)
        return W, act, ctx.bse_eigvecs(1, 3)

    before = solve(40.0)
    solve(r0)
    for a, b in zip(solve(40.0), before):
        assert np.array_equal(a, b)
