"""Lowest and highest states of a problem whose energies lie far from 1: all of it times a power of two (with V2DOH
the kernel scales as 1 / EZ). The oracle is the dense solve of the same matrix. Tolerance: a residual r moves a level
by at most r, the tolerance that the solver was given. The preconditioner's clamp is 0.05 eV, so far below that the
iteration is unpreconditioned, which a block of 8 does not converge with in 200 steps: the top states from scale 1 up."""
import numpy as np
import pytest

from wantibexos_b200 import synth, wtbgpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [-180, -130, 0, 130, 180])
def test_states_of_a_scaled_problem(scale, gpu_ctx):
    ctx, n = gpu_ctx, 9
    m = synth.config_model("c1")
    m.hre[:], m.him[:] = np.ldexp(m.hre, scale), np.ldexp(m.him, scale)
    a1, a2, a3 = m.rlat
    s = 2.0 * float(np.float32(np.pi)) / abs(a1 @ np.cross(a2, a3))
    b1, b2 = s * np.cross(a2, a3), s * np.cross(a3, a1)
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    ctx.set_model(m)
    ctx.bands((b1 / n * i[..., None] + b2 / n * j[..., None]).reshape(-1, 3), 2, 2, want_vectors=False)
    ctx.bse_build(wtbgpu.coulomb_params("V2DOH", [n, n, 1], 1e-3, [1, 1, 1], 0.0, float(np.ldexp(1.0, -scale)), 0.0, 0.0))
    tol = float(np.ldexp(1e-7, scale))
    low = ctx.bse_davidson(6, nb=16, tol=tol, want_act=False)[0]
    top = ctx.bse_davidson(2, nb=8, largest=True, tol=tol, want_act=False)[0] if scale >= 0 else None
    W, _ = ctx.bse_solve(want_act=False)
    assert np.abs(low - W[:6]).max() <= tol
    assert top is None or np.abs(np.sort(top) - W[-2:]).max() <= tol
