"""Host threads with a context each on one device, all in the two-stage reduction, its Q groups and the exciton
vectors, whose grids wait for all their CTAs: every result carries the bits that the context gives alone."""
import threading

import numpy as np
import pytest

from wantibexos_b200 import synth, wtbgpu

pytestmark = pytest.mark.gpu

MODEL = synth.config_model("c1")


def work(ctx, n1, n2, nv, nc):
    a1, a2, a3 = MODEL.rlat
    s = 2.0 * float(np.float32(np.pi)) / abs(a1 @ np.cross(a2, a3))
    b1, b2 = s * np.cross(a2, a3), s * np.cross(a3, a1)
    i, j = np.meshgrid(np.arange(n1), np.arange(n2), indexing="ij")
    k = (b1 / n1 * i[..., None] + b2 / n2 * j[..., None]).reshape(-1, 3)
    q = np.array([[0.0, *(0.03 * i * b1)] for i in range(5)])
    c = wtbgpu.coulomb_params("V2DRK", [n1, n2, 1], 1e-3, [1, 1, 1], 1.0, 1.0, 0.0, 40.0)
    ctx.set_model(MODEL)
    ctx.bands(k, nv, nc, want_vectors=False)
    ctx.velocity(0.05, want=False)
    ctx.bse_build(c)
    W, act = ctx.bse_solve(True, True)
    A = ctx.bse_eigvecs(1, 8)
    Wq, _ = ctx.bse_q_batch([k + x[1:] for x in q], q, c)
    return W, act, A, Wq


def test_contexts_of_one_device_at_work_together():
    sizes = [(12, 12, 2, 2), (17, 13, 1, 2), (9, 4, 1, 1)]
    ctxs = [wtbgpu.Context(0) for _ in sizes]
    alone = [work(c, *s) for c, s in zip(ctxs, sizes)]
    failed = []

    def many(c, s, want):
        try:
            for _ in range(8):
                for a, b in zip(work(c, *s), want):
                    assert np.array_equal(a, b)
        except BaseException as e:   # handed to the test's own thread
            failed.append(e)

    ts = [threading.Thread(target=many, args=a) for a in zip(ctxs, sizes, alone)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for c in ctxs:
        c.close()
    assert not failed, failed
