"""The imaginary part of H(k)'s diagonal is not read (as by ZHEEV), whatever its size: the same bits with it and
without, on a path through both work areas of the per-k solver."""
import numpy as np
import pytest

from wantibexos_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [3, 24, 90])
def test_imaginary_onsite_terms_do_not_enter(w, gpu_ctx):
    m = synth.make_hex_model(w, 1, (-1.5, 0.3), (1.5, 0.3), 900 + w)
    kpt = np.random.default_rng(w).uniform(-1.5, 1.5, (9, 3))
    i0 = int(np.flatnonzero((m.rvec == 0).all(axis=1))[0])
    m.him[i0][np.diag_indices(w)] = 0.0
    gpu_ctx.set_model(m)
    e, v, no = gpu_ctx.eigsys(kpt)
    m.him[i0][np.diag_indices(w)] = np.random.default_rng(1).uniform(1e16, 1e17, w)
    gpu_ctx.set_model(m)
    e1, v1, no1 = gpu_ctx.eigsys(kpt)
    assert np.array_equal(no, no1) and np.array_equal(e, e1) and np.array_equal(v, v1)
