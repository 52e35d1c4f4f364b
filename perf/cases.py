"""Workloads of the exciton and optics path, each through the entry points a program calls.

listed() names the cases, draw() gives further ones of the same ranges, prepare() makes what a
program holds before the call (a Context with its Wannier model, the k-mesh, the interaction),
run() is one pass and exact() the same result from plain NumPy/Torch in 64 bits. Kinds:

  spectrum   one BSE deck: bands on the k-mesh, velocities, single-particle table, exciton
             kernel, dense solve with oscillator strengths, broadened eps(omega) of the excitons
             and of the independent particles
  path       exciton band structure: the eigenvalues of the kernel at every centre-of-mass
             momentum of a path (bands of the k-mesh, then all Q in one call)
  lowest     the fast form: block Davidson for the lowest excitons and the highest one, then
             eps(omega) by the Haydock recursion, both on the tensor-core product
  waves      dense solve, then the exciton wave functions of the lowest states
  eigsys     every band and vector on a k-mesh or path (band structure and DOS tools)
  berry      Berry curvature on a k-mesh

The sizes are those of this repository's configurations and tests: 8 to 40 orbitals, exciton
dimensions from a hundred to 14400, seeded synthetic hexagonal models.
"""
import math

import numpy as np
import torch

from wantibexos_b200 import synth, wtbgpu

PI32 = float(np.float32(np.pi))

# orbitals -> (shells of cells, onsite centre and half-width below / above the gap)
MODELS = {8: (3, 1.5, 0.3), 16: (4, 1.5, 0.3), 24: (5, 1.8, 0.4), 40: (4, 1.5, 0.3)}


def listed():
    return [
        # band structure along a path of k-points for a plot: the smallest call, launch latency
        {"name": "bands_path_w8", "kind": "eigsys", "w": 8, "n1": 61, "n2": 1},
        # the smallest deck of the repository (12x12 mesh, N = 576): a first look at a material
        {"name": "spectrum_576", "kind": "spectrum", "w": 8, "n1": 12, "n2": 12, "nv": 2, "nc": 2, "full": False,
         "temp": -1.0, "r0": 40.0, "numbse": 1001},
        # an odd mesh with the full dielectric tensor and circular polarisation
        {"name": "spectrum_odd_1292", "kind": "spectrum", "w": 8, "n1": 17, "n2": 19, "nv": 2, "nc": 2, "full": True,
         "temp": -1.0, "r0": 40.0, "numbse": 2001},
        # the temperature BSE at a usual convergence-test mesh
        {"name": "spectrum_temp_2304", "kind": "spectrum", "w": 16, "n1": 24, "n2": 24, "nv": 2, "nc": 2, "full": False,
         "temp": 300.0, "r0": 35.0, "numbse": 2001},
        # a wide band window on a coarse odd mesh
        {"name": "spectrum_3600", "kind": "spectrum", "w": 24, "n1": 15, "n2": 15, "nv": 4, "nc": 4, "full": True,
         "temp": -1.0, "r0": 30.0, "numbse": 2001},
        # a production spectrum on a converged 60x60 mesh: the largest dense solve here
        {"name": "spectrum_14400", "kind": "spectrum", "w": 16, "n1": 60, "n2": 60, "nv": 2, "nc": 2, "full": False,
         "temp": -1.0, "r0": 35.0, "numbse": 2001},
        # exciton band structure at a coarse mesh: many small eigenproblems
        {"name": "path_576", "kind": "path", "w": 8, "n1": 12, "n2": 12, "nv": 2, "nc": 2, "nq": 12, "r0": 40.0},
        # exciton band structure at the production mesh (a part of the 64-point path)
        {"name": "path_8100", "kind": "path", "w": 16, "n1": 30, "n2": 30, "nv": 3, "nc": 3, "nq": 3, "r0": 35.0},
        # lowest excitons and spectrum without the dense solve, the sweep's size
        {"name": "lowest_14400", "kind": "lowest", "w": 16, "n1": 60, "n2": 60, "nv": 2, "nc": 2, "nev": 32,
         "r0": 35.0, "numbse": 2001},
        # exciton wave functions of the lowest states (BSE_WF)
        {"name": "waves_2916", "kind": "waves", "w": 8, "n1": 27, "n2": 27, "nv": 2, "nc": 2, "nev": 8, "r0": 40.0},
        # every band of a large unit cell on a mesh (DOS)
        {"name": "eigsys_w40", "kind": "eigsys", "w": 40, "n1": 36, "n2": 36},
        # Berry curvature over the zone
        {"name": "berry_w24", "kind": "berry", "w": 24, "n1": 48, "n2": 48},
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spectrum", "spectrum", "spectrum", "path", "path", "lowest", "waves", "eigsys", "berry"])
    w = rng.choice([8, 16, 24])
    case = {"kind": kind, "w": w}
    if kind in ("eigsys", "berry"):
        if kind == "eigsys":
            case["w"] = rng.choice([8, 16, 24, 40])
        n1 = _between(rng, 4, 48)
        case.update(n1=n1, n2=max(1, n1 + rng.randint(-3, 3)))
        return case
    nv, nc = rng.randint(1, 4), rng.randint(1, 4)
    if w == 8:
        nv, nc = min(nv, 2), min(nc, 2)
    top = {"spectrum": 12000, "path": 8100, "lowest": 14400, "waves": 5000}[kind]
    size = _between(rng, 600 if kind == "lowest" else 140, top)
    n1 = max(4, int(math.sqrt(size / (nv * nc))))
    n2 = max(4, n1 + rng.randint(-2, 2))
    while n1 * n2 * nv * nc > top:
        n2 -= 1
    case.update(n1=n1, n2=n2, nv=nv, nc=nc, r0=float(rng.randint(10, 60)))
    size = n1 * n2 * nv * nc
    if kind == "spectrum":
        case.update(full=rng.random() < 0.4, temp=rng.choice([-1.0, -1.0, 300.0]), numbse=rng.choice([501, 1001, 2001]))
    elif kind == "path":
        case["nq"] = rng.randint(2, max(2, min(12, int(16000 / size))))
    elif kind == "lowest":
        case.update(nev=rng.choice([8, 16, 32]), numbse=rng.choice([1001, 2001]))
    else:
        case["nev"] = rng.randint(1, 12)
    return case


# ------------------------------------------------------------------------------ inputs
def _model(case, seed):
    shells, centre, half = MODELS[case["w"]]
    return synth.make_gapped_model(case["w"], shells, (-centre, half), (centre, half), 64 * int(seed) + 1)


def _recvec(rlat):
    a1, a2, a3 = rlat
    v23, v31, v12 = np.cross(a2, a3), np.cross(a3, a1), np.cross(a1, a2)
    s = (2.0 * PI32) / abs(a1 @ v23)
    return s * v23, s * v31, s * v12


def _mesh(case, rlat):
    b1, b2, _ = _recvec(rlat)
    i, j = np.meshgrid(np.arange(case["n1"]), np.arange(case["n2"]), indexing="ij")
    return ((b1 / case["n1"]) * i[..., None] + (b2 / case["n2"]) * j[..., None]).reshape(-1, 3)


def _momenta(case, rlat):
    """nq points from Gamma towards M, (distance, qx, qy, qz) per row; the first is Q = 0."""
    b1 = _recvec(rlat)[0]
    t = np.arange(case["nq"]) / 21.0
    q = 0.5 * t[:, None] * b1[None, :]
    return np.concatenate([t[:, None], q], axis=1)


def _ngrid(case):
    return [case["n1"], case["n2"], 1]


def _volume(rlat):
    return abs(np.cross(rlat[0], rlat[1]) @ rlat[2])


CSHIFT, EMAX = 0.05, 6.0


def prepare(case, seed):
    model = _model(case, seed)
    ctx = wtbgpu.Context(0)
    ctx.set_model(model)
    state = {"case": dict(case), "ctx": ctx, "kpt": _mesh(case, model.rlat), "vol": _volume(model.rlat)}
    kind = case["kind"]
    if kind not in ("eigsys", "berry"):
        state["coul"] = wtbgpu.coulomb_params("V2DRK", _ngrid(case), 1e-3, [1.0] * 3, 1.0, 1.0, 0.0, case["r0"])
    if kind == "spectrum" and case["temp"] >= 0.0:
        ctx.set_temperature(True, case["temp"])
    if kind == "path":
        state["q"] = _momenta(case, model.rlat)
        state["kq"] = [state["kpt"] + q[None, 1:] for q in state["q"]]
    if kind == "lowest":
        ctx.set_fast_product(1)
    return state


# ------------------------------------------------------------------------------ one pass
def run(state):
    case, ctx, kpt = state["case"], state["ctx"], state["kpt"]
    kind = case["kind"]
    if kind == "eigsys":
        e, v, nocp = ctx.eigsys(kpt)
        return {"e": e, "v": v, "nocp": nocp}
    if kind == "berry":
        return {"b": ctx.berry(kpt)}
    nv, nc = case["nv"], case["nc"]
    if kind == "path":
        ctx.bands(kpt, nv, nc, want_vectors=False)
        W, _ = ctx.bse_q_batch(state["kq"], state["q"], state["coul"])
        return {"W": W}
    e, _, nocp, gap = ctx.bands(kpt, nv, nc, want_vectors=False)
    ctx.velocity(CSHIFT, want=False)
    if kind == "spectrum":
        full = case["full"]
        sp = ctx.sp_table()
        ctx.bse_build(state["coul"])
        W, act = ctx.bse_solve(full, full)
        grid = (_ngrid(case), state["vol"], 0.0, EMAX, float(case["numbse"]), CSHIFT, True, 2.0)
        omega, eps = ctx.spectrum(W, act[:, :6], *grid)
        _, eps_sp = ctx.spectrum(sp[:, 6], sp[:, 7:13], *grid)
        return {"e": e, "nocp": nocp, "gap": gap, "sp": sp, "W": W, "act": act, "omega": omega, "eps": eps,
                "eps_sp": eps_sp}
    ctx.bse_build(state["coul"])
    if kind == "waves":
        W, act = ctx.bse_solve(False, False)
        return {"W": W, "act": act, "A": ctx.bse_eigvecs(1, case["nev"])}
    nev = case["nev"]
    W = ctx.bse_davidson(nev, nb=nev + 8, tol=1e-6, want_act=False)[0]
    top = ctx.bse_davidson(1, nb=8, largest=True, tol=1e-3, want_act=False)[0][0]
    omega, eps = ctx.bse_spectrum_fast(150, W[0], top, _ngrid(case), state["vol"], 0.0, EMAX, float(case["numbse"]),
                                       CSHIFT, True, 2.0)
    return {"e": e, "nocp": nocp, "gap": gap, "W": W, "omega": omega, "eps": eps}


def work(case):
    """Bytes and FP64 operations the path cannot do without: each input read once, each result
    written once; the kernel matrix of the excitons counts as written and read once."""
    shells = MODELS[case["w"]][0]
    cells, w, nk = 1 + 3 * shells * (shells + 1), case["w"], case["n1"] * case["n2"]
    bands = {"bytes": 16.0 * cells * w * w + 24.0 * nk, "flops": nk * (8.0 * cells * w * w / 2 + 25.0 * w ** 3)}
    kind = case["kind"]
    if kind == "eigsys":
        bands["bytes"] += nk * (16.0 * w * w + 8.0 * w + 4.0)
        return bands
    if kind == "berry":
        return {"bytes": bands["bytes"] + 48.0 * nk, "flops": bands["flops"] + nk * (24.0 * cells * w * w + 9.0 * w ** 3)}
    N = float(nk * case["nv"] * case["nc"])
    matrix = 16.0 * N * N / 2
    if kind == "path":
        nq = case["nq"]
        return {"bytes": bands["bytes"] * (1 + nq) + nq * (2 * matrix + 8.0 * N),
                "flops": bands["flops"] * (1 + nq) + nq * (16.0 / 3.0) * N ** 3}
    bands["flops"] += nk * 24.0 * cells * w * w
    if kind == "lowest":
        # the least a subspace method reads: the matrix once to apply it to the block, once per chain
        return {"bytes": bands["bytes"] + 5 * matrix, "flops": bands["flops"] + 8.0 * N * N * (case["nev"] + 3)}
    if kind == "waves":
        n = case["nev"]
        return {"bytes": bands["bytes"] + 2 * matrix + 16.0 * N * n, "flops": bands["flops"] + (16.0 / 3.0) * N ** 3
                + 16.0 * N * N * n}
    return {"bytes": bands["bytes"] + 2 * matrix + N * (8 * 9 + 60) + 100.0 * case["numbse"],
            "flops": bands["flops"] + (16.0 / 3.0) * N ** 3 + 30.0 * N * N + 60.0 * N * case["numbse"]}


# ------------------------------------------------------------------------------ 64-bit result
def _phases(R, k):
    kr = (k[0] * R[:, 0] + k[1] * R[:, 1]) + k[2] * R[:, 2]
    kr = kr.astype(np.float32).astype(np.float64)      # the phase is evaluated in single precision
    return np.cos(kr) + 1j * np.sin(kr)


def _cells(model):
    r, L = model.rvec.astype(np.float64), model.rlat
    return np.stack([(r[:, 0] * L[0, c] + r[:, 1] * L[1, c]) + r[:, 2] * L[2, c] for c in range(3)], axis=1)


def _bands64(model, kpt):
    """Energies (nk, w), vectors (nk, band, component) with a real first component, states below zero."""
    R, H = _cells(model), model.hre + 1j * model.him
    P = np.array([_phases(R, k) for k in kpt])
    Hk = np.tensordot(P, H, axes=(1, 0))
    e, V = np.linalg.eigh(Hk, UPLO="L")
    U = np.swapaxes(V, 1, 2)
    first = U[:, :, :1]
    mag = np.abs(first)
    U = U * np.where(mag > 0, np.conj(first) / np.where(mag > 0, mag, 1.0), 1.0)
    nocp = np.array([int(np.argmax(x > 0.0)) if (x > 0.0).any() else x.size for x in e])
    return e, U, nocp


def _gradient64(model, kpt):
    """dH/dk_a at every k, (3, nk, w, w); the onsite terms of the home cell do not enter."""
    R, H = _cells(model), (model.hre + 1j * model.him).copy()
    home = np.where((model.rvec == 0).all(axis=1))[0]
    for i in home:
        H[i][np.diag_indices(model.w)] = 0.0
    P = np.array([_phases(R, k) for k in kpt])
    R32 = R.astype(np.float32).astype(np.float64)
    return np.stack([np.tensordot(P * (1j * R32[:, a])[None, :], H, axes=(1, 0)) for a in range(3)])


def _window(e, U, nocp, nv, nc):
    idx = nocp[:, None] + np.arange(-nv, nc)[None, :]
    return np.take_along_axis(e, idx, 1), np.take_along_axis(U, idx[:, :, None], 1)


def _velocity64(model, kpt, eb, Ub, nv):
    G = _gradient64(model, kpt)
    de = eb[:, nv:, None] - eb[:, None, :nv]
    eta = float(np.float32(CSHIFT))
    h = np.einsum("kcm,akmn,kvn->akcv", Ub[:, nv:].conj(), G, Ub[:, :nv]) * (de / (de * de + eta * eta))
    h = h.reshape(3, -1)
    s = float(np.float32(1.0 / np.sqrt(np.float32(2.0))))
    return np.concatenate([h, [(h[0] + 1j * h[1]) * s, (h[0] - 1j * h[1]) * s]])


CIC = float(-np.float32(0.0904756) * np.float32(1000.0))


def _screened(case, rlat, dk):
    """Rytova-Keldysh W(q) per cell for unit dielectric constants (dk: (..., 3))."""
    area = np.linalg.norm(np.cross(rlat[0], rlat[1]))
    q = np.sqrt((dk ** 2).sum(-1))
    safe = np.where(q < 1e-3, 1.0, q)
    v = CIC / (case["n1"] * case["n2"] * area) / (1.0 + case["r0"] * safe) / safe
    return np.where(q < 1e-3, 0.0, v)


def _kernel64(case, model, kpt, eb, Ub, nv, nc, ebc=None, Ubc=None, q=None, occ=None):
    """The Hermitian exciton kernel, basis (k, c, v) with v fastest; conduction states at k + q."""
    ebc = eb if ebc is None else ebc
    Ubc = Ub if Ubc is None else Ubc
    nk = len(kpt)
    N = nk * nc * nv
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = lambda x: torch.as_tensor(np.ascontiguousarray(x), device=dev)  # noqa: E731
    C, V = t(Ubc[:, nv:]), t(Ub[:, :nv])
    W = t(_screened(case, model.rlat, kpt[:, None, :] - kpt[None, :, :]))
    oc = torch.einsum("kcm,ldm->kcld", C.conj(), C)
    ov = torch.einsum("kvm,lum->kvlu", V.conj(), V)
    H = (W[:, None, None, :, None, None] * oc[:, :, None, :, :, None] * ov[:, None, :, :, None, :]).reshape(N, N)
    if q is not None and np.linalg.norm(q) > 0.0:
        vq = float(_screened(case, model.rlat, np.asarray(q)))
        ex = torch.einsum("kcm,kvm->kcv", C.conj(), V).reshape(N)
        H = H - vq * ex[:, None] * ex.conj()[None, :]
    if occ is not None:      # the interaction of a pair is scaled by the occupation of its smaller index
        i = torch.arange(N, device=dev)
        H = H * t(occ)[torch.minimum(i[:, None], i[None, :])]
    de = (ebc[:, nv:, None] - eb[:, None, :nv]).reshape(N)
    H.diagonal().add_(t(de))
    return H


def _epsilon64(case, rlat, E, F, numbse):
    n = E.size
    eta = 10.0 * (E[-1] - E[0]) / n + CSHIFT
    c = float(np.float32(180.90)) / (float(np.float32(case["n1"] * case["n2"])) * _volume(rlat))
    om = EMAX * np.arange(numbse) / (numbse - 1.0)
    d = om[:, None] - E[None, :]
    den = d * d + eta * eta
    re = ((-d / den) @ F) * c + np.array([1.0, 1.0, 1.0, 0.0, 0.0, 0.0])[None, :]
    im = ((eta / den) @ F) * c
    edge = E[0] - float(np.float32(0.15))
    if edge > 0.0:
        first = max(1, int((om <= edge).sum()))
        shift = im[first] if first < numbse else np.zeros(6)
        im[first:] = np.maximum(im[first:] - shift, 0.0)
        im[:first] = 0.0
    return om, np.stack([2.0 * re, 2.0 * im], axis=1).astype(np.float32)


def _strengths(z, f, full):
    """|A^T h| products xx, yy, zz, xy, xz, yz, sp, sm; z = A^T h, f = A^T (h occupation), (5, N) each."""
    re = lambda a, b: (z[a] * f[b].conj()).real  # noqa: E731
    zero = np.zeros(z.shape[1])
    pairs = [(0, 0), (1, 1), (2, 2)] + ([(0, 1), (0, 2), (1, 2), (3, 3), (4, 4)] if full else [])
    cols = [re(a, b) for a, b in pairs]
    return np.stack(cols + [zero] * (8 - len(cols)), axis=1)


def exact(case, seed):
    model = _model(case, seed)
    kpt = _mesh(case, model.rlat)
    kind = case["kind"]
    e, U, nocp = _bands64(model, kpt)
    if kind == "eigsys":
        return {"e": e, "v": U, "nocp": nocp.astype(np.int32)}
    if kind == "berry":
        gamma, tol = float(np.float32(0.001)), float(np.float32(0.0001))
        G = _gradient64(model, kpt)
        T = np.einsum("knm,akml,kil->akni", U.conj(), G, U, optimize=True)
        d = e[:, :, None] - e[:, None, :]
        n = np.arange(model.w)
        on = (n[None, :, None] < nocp[:, None, None]) & (n[None, None, :] >= nocp[:, None, None]) & (np.abs(d) >= tol)
        wgt = np.where(on, -2.0 / (d * d + gamma * gamma), 0.0)
        return {"b": np.stack([(wgt * T[a] * T[b].conj()).imag.sum((1, 2)) for a, b in
                               ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))], axis=1)}
    nv, nc = case["nv"], case["nc"]
    N = len(kpt) * nv * nc
    if N > 3600:      # the dense eigenproblem in 64 bits takes too long here
        return None
    eb, Ub = _window(e, U, nocp, nv, nc)
    if kind == "path":
        out = []
        for q in _momenta(case, model.rlat):
            eq, Uq, nq = _bands64(model, kpt + q[None, 1:])
            ebq, Ubq = _window(eq, Uq, nq, nv, nc)
            H = _kernel64(case, model, kpt, eb, Ub, nv, nc, ebq, Ubq, q[1:])
            out.append(torch.linalg.eigvalsh(H).cpu().numpy())
        return {"W": np.array(out)}
    gap = float((eb[:, nv] - eb[:, nv - 1]).min())
    if kind == "lowest":
        W = torch.linalg.eigvalsh(_kernel64(case, model, kpt, eb, Ub, nv, nc)).cpu().numpy()
        return {"e": eb, "nocp": nocp.astype(np.int32), "gap": gap, "W": W[:case["nev"]], "omega": None, "eps": None}
    occ = None
    if kind == "spectrum" and case["temp"] >= 0.0:
        beta = 1.0 / (float(np.float32(8.617330350e-5)) * case["temp"])
        fermi = 1.0 / (np.exp(np.minimum(eb * beta, 700.0)) + 1.0)
        occ = (fermi[:, None, :nv] - fermi[:, nv:, None]).reshape(N)
    W, A = torch.linalg.eigh(_kernel64(case, model, kpt, eb, Ub, nv, nc, occ=occ))
    W, A = W.cpu().numpy(), A.cpu().numpy()
    h = _velocity64(model, kpt, eb, Ub, nv)
    z = h @ A
    f = z if occ is None else (h * occ[None, :]) @ A
    if kind == "waves":
        A = A[:, :case["nev"]]
        A = A * (np.conj(A[-1]) / np.abs(A[-1]))[None, :]
        return {"W": W, "act": _strengths(z, f, False), "A": A}
    act = _strengths(z, f, case["full"])
    om, eps = _epsilon64(case, model.rlat, W, act[:, :6], case["numbse"])
    return {"e": eb, "nocp": nocp.astype(np.int32), "gap": gap, "sp": None, "W": W, "act": act, "omega": om, "eps": eps,
            "eps_sp": None}
