"""Host threads with a context each whose models need different amounts of shared memory: the per-k kernels, the
kernel build and the block solver of one must not lower the limits that the other's launches need. The same bits as
alone."""
import threading

import numpy as np
import pytest

from wantibexos_b200 import synth, wtbgpu

pytestmark = pytest.mark.gpu


def work(ctx, m, n, nv, nev, nb):
    a1, a2, a3 = m.rlat
    s = 2.0 * float(np.float32(np.pi)) / abs(a1 @ np.cross(a2, a3))
    b1, b2 = s * np.cross(a2, a3), s * np.cross(a3, a1)
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    k = (b1 / n * i[..., None] + b2 / n * j[..., None]).reshape(-1, 3)
    ctx.set_model(m)
    e, v, _ = ctx.eigsys(k)
    b = ctx.berry(k)
    o = ctx.sp_optbz(k, nv, nv, 0.05)
    ctx.bands(k, nv, nv, want_vectors=False)
    h = ctx.velocity(0.05)
    ctx.bse_build(wtbgpu.coulomb_params("V2DRK", [n, n, 1], 1e-3, [1, 1, 1], 1.0, 1.0, 0.0, 40.0))
    H = ctx.bse_get_matrix()
    W = ctx.bse_davidson(nev, nb=nb, tol=1e-6, want_act=False)[0]
    return e, v, b, o, h, H, W


def test_models_of_different_sizes_side_by_side():
    cases = [(synth.make_gapped_model(4, 2, (-1.5, 0.3), (1.5, 0.3), 31), 4, 1, 2, 8),
             (synth.make_gapped_model(40, 4, (-1.5, 0.3), (1.5, 0.3), 65), 5, 4, 24, 40)]
    ctxs = [wtbgpu.Context(0) for _ in cases]
    alone = [work(c, *a) for c, a in zip(ctxs, cases)]
    failed = []

    def many(c, a, want):
        try:
            for _ in range(60):
                for x, y in zip(work(c, *a), want):
                    assert np.array_equal(x, y)
        except BaseException as e:   # handed to the test's own thread
            failed.append(e)

    ts = [threading.Thread(target=many, args=a) for a in zip(ctxs, cases, alone)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for c in ctxs:
        c.close()
    assert not failed, failed
