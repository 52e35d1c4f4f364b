"""Q points side by side keep a matrix and panel buffers each in the context: the memory is given back with the next
model, and a call after that, and after a larger solve, gives the same bits."""
import numpy as np
import pytest

from wantibexos_b200 import synth, wtbgpu

pytestmark = pytest.mark.gpu


def test_lane_memory_is_given_back(gpu_ctx):
    torch = pytest.importorskip("torch")
    m = synth.config_model("c1")
    a1, a2, a3 = m.rlat
    s = 2.0 * float(np.float32(np.pi)) / abs(a1 @ np.cross(a2, a3))
    b1, b2 = s * np.cross(a2, a3), s * np.cross(a3, a1)

    def mesh(n):
        i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
        return (b1 / n * i[..., None] + b2 / n * j[..., None]).reshape(-1, 3)

    def coul(n):
        return wtbgpu.coulomb_params("V2DRK", [n, n, 1], 1e-3, [1, 1, 1], 1.0, 1.0, 0.0, 40.0)

    n = 18   # N = 1296
    N = n * n * 4
    q = np.array([[0.0, *(0.03 * i * b1)] for i in range(6)])
    kq = [mesh(n) + x[1:] for x in q]
    ctx = wtbgpu.Context(0)

    def path():
        ctx.set_model(m)
        ctx.bands(mesh(n), 2, 2, want_vectors=False)
        return ctx.bse_q_batch(kq, q, coul(n))[0]

    W = path()
    held = torch.cuda.mem_get_info(0)[0]
    ctx.set_model(m)
    assert torch.cuda.mem_get_info(0)[0] - held >= 3 * N * N * 16
    assert np.array_equal(path(), W)
    ctx.bands(mesh(26), 2, 2, want_vectors=False)   # N = 2704
    ctx.velocity(0.05, want=False)
    ctx.bse_build(coul(26))
    ctx.bse_solve(False, False)
    assert np.array_equal(path(), W)
    ctx.close()
