"""The calls whose time this repository tracks, over the range of sizes, forms and solvers that it serves.

Every time-step case restarts a simulation from a state in host memory, as a host program or a
resumed run does: it gives the context U, p, phi and the constitutive fields, takes the steps and reads
the new U, p, phi, theta and tau back.  The states start from rest with a seeded lognormal
conformation, so no eigenvalue is degenerate.  The `ldu` cases are the lduMatrix::solver seam (host
matrix in, solution out) and the `correct` cases the constitutiveEq::correct() seam.
"""
import dataclasses
import math

import numpy as np
import torch

from rheotool_gb300 import abi
from rheotool_gb300.batch import BatchContext
from rheotool_gb300.case import Fields, SolverControl, cavity_case, contraction_case, periodic_channel_case
from rheotool_gb300.mesh import cavity_mesh, contraction_mesh, periodic_channel_mesh
from rheotool_gb300.runtime import ConstitutiveEq, Context, LduSolver

MODEL_KW = {"Oldroyd-BLog": {}, "GiesekusLog": {"alpha": 0.1}, "FENE-PLog": {"L2": 100.0},
            "PTTLog": {"epsilon": 0.25}}


def listed():
    return [
        # the smallest flow case a user runs: a coarse cavity, FP64, where launches and latency count
        dict(name="cavity32_fp64", kind="cavity", n=32, precision="fp64", model="Oldroyd-BLog", steps=2),
        # a 2-D cavity of an odd side in the mixed form, the size of one served request
        dict(name="cavity129_mixed", kind="cavity", n=129, precision="mixed", model="GiesekusLog", steps=4),
        # the 126,675-cell sample of the 4:1 contraction in the reference's precision
        dict(name="contraction127k_fp64", kind="contraction", nx_up=67, nx_down=66, ny_in=25, ny_out=13, nz=25,
             precision="fp64", model="GiesekusLog", steps=1),
        # the headline: the 1,000,000-cell 4:1 contraction in the reference's precision
        dict(name="contraction1m_fp64", kind="contraction", nx_up=134, nx_down=132, ny_in=50, ny_out=25, nz=50,
             precision="fp64", model="GiesekusLog", steps=1),
        # the same case in the mixed form
        dict(name="contraction1m_mixed", kind="contraction", nx_up=134, nx_down=132, ny_in=50, ny_out=25, nz=50,
             precision="mixed", model="GiesekusLog", steps=2),
        # a small 3-D request of the serving loop, in the mixed form
        dict(name="contraction38k_mixed", kind="contraction", nx_up=45, nx_down=44, ny_in=17, ny_out=8, nz=17,
             precision="mixed", model="GiesekusLog", steps=4),
        # a periodic (cyclic) PTT channel in the mixed form, the precision sweep's case at an eighth of its cells
        dict(name="periodic500k_mixed", kind="periodic", nx=200, ny=50, nz=50, precision="mixed", model="PTTLog",
             steps=1),
        # an OpenFOAM case as its polyMesh gives it, without box structure: the 2-D contraction tutorial's size
        dict(name="polymesh7k_fp64", kind="polymesh", nx=60, ny=20, precision="fp64", model="Oldroyd-BLog",
             solver="PBiCGStab", steps=1),
        # a parametric sweep of independent cavities of uneven size, stepped together
        dict(name="batch96_mixed", kind="batch", cases=96, n_min=32, n_max=128, steps=2),
        # the lduMatrix::solver seam: one pressure-like system, PCG with DIC
        dict(name="ldu_pcg_164k", kind="ldu", nx=96, ny=50, nz=45, solver="PCG", nc=1),
        # the same seam for a momentum-like system: three components, PBiCGStab with DILU
        dict(name="ldu_pbicgstab_46k", kind="ldu", nx=61, ny=40, nz=25, solver="PBiCGStab", nc=3),
        # the constitutiveEq::correct() seam alone, as a solver that keeps its own momentum equation calls it
        dict(name="correct250k_fp64", kind="correct", nx=125, ny=50, nz=40, precision="fp64", model="GiesekusLog"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["cavity", "contraction", "contraction", "periodic", "polymesh", "batch", "ldu", "ldu",
                       "correct"])
    precision = rng.choice(["fp64", "mixed"])
    model = rng.choice(["Oldroyd-BLog", "GiesekusLog", "FENE-PLog", "PTTLog"])
    if kind == "cavity":
        return dict(kind=kind, n=_log_int(rng, 16, 192), precision=precision, model=model, steps=rng.randint(1, 4))
    if kind == "contraction":   # 16k .. 1M cells, the serving loop's range
        f = (_log_int(rng, 16_000, 1_000_000) / 1e6) ** (1 / 3)
        return dict(kind=kind, nx_up=round(134 * f), nx_down=round(132 * f), ny_in=round(50 * f),
                    ny_out=round(25 * f), nz=round(50 * f), precision=precision, model=model, steps=1)
    if kind == "periodic":
        f = (_log_int(rng, 30_000, 500_000) / 5e5) ** (1 / 3)
        return dict(kind=kind, nx=round(200 * f), ny=round(50 * f), nz=round(50 * f), precision=precision,
                    model=rng.choice(["Oldroyd-BLog", "PTTLog"]), steps=1)
    if kind == "polymesh":
        nx = _log_int(rng, 24, 120)
        return dict(kind=kind, nx=nx, ny=max(8, nx // 3), precision=precision, model=model,
                    solver=rng.choice(["PBiCGStab", "PBiCG"]), steps=1)
    if kind == "batch":
        n_min = rng.randint(24, 64)
        return dict(kind=kind, cases=_log_int(rng, 4, 96), n_min=n_min, n_max=n_min + rng.randint(0, 64), steps=1)
    nx, ny, nz = _log_int(rng, 16, 160), _log_int(rng, 12, 80), _log_int(rng, 8, 60)
    if kind == "ldu":
        solver = rng.choice(["PCG", "PBiCGStab"])
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, solver=solver, nc=1 if solver == "PCG" else rng.choice([1, 3]))
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=precision, model=rng.choice(["Oldroyd-BLog", "GiesekusLog",
                                                                                       "PTTLog"]))


# ---------------------------------------------------------------------------
_meshes = {}


def _mesh(key, make):
    """One mesh of each size: a program builds its mesh once and keeps it."""
    if key not in _meshes:
        if sum(m.nCells for m in _meshes.values()) > 4_000_000:
            _meshes.clear()
        _meshes[key] = make()
    return _meshes[key]


def _lognormal(n, rng, sigma=0.1, planar=False):
    """theta = Q diag(sigma z) Q^T of a random rotation Q (about z alone in a plane flow), with its
    eigenvalues' exp (ascending) and eigenvectors (columns), and A = exp(theta) as xx xy xz yy yz zz."""
    mu = np.sort(sigma * rng.standard_normal((n, 3)), axis=1)
    q = rng.standard_normal((n, 4))
    if planar:
        q[:, 1:3] = 0.0
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    w, x, y, z = q.T
    R = np.empty((n, 3, 3))
    R[:, 0, 0], R[:, 0, 1], R[:, 0, 2] = 1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)
    R[:, 1, 0], R[:, 1, 1], R[:, 1, 2] = 2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)
    R[:, 2, 0], R[:, 2, 1], R[:, 2, 2] = 2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)

    def back(d):
        return np.stack([(R[:, i] * d * R[:, j]).sum(1) for i, j in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))],
                        axis=1)

    ev = np.exp(mu)
    return back(mu), ev, np.ascontiguousarray(R.reshape(n, 9)), back(ev)


def _conformation(f, model, rng, planar):
    """Gives the fields a lognormal conformation and the tau of it (the Oldroyd-B relation, as a start)."""
    f.theta, f.eigVals, f.eigVecs, A = _lognormal(f.theta.shape[0], rng, planar=planar)
    f.tau = model.etaP / model.lambda_ * (A - np.array([1.0, 0, 0, 1, 0, 1]))


def _case(c):
    kw = MODEL_KW.get(c.get("model"), {})
    k = c["kind"]
    if k == "cavity":
        case = cavity_case(c["n"], model=c["model"], mesh=_mesh((k, c["n"]), lambda: cavity_mesh(c["n"])), **kw)
    elif k == "contraction":
        dims = {d: c[d] for d in ("nx_up", "nx_down", "ny_in", "ny_out", "nz")}
        kw = {"alpha": 0.0, **kw}
        case = contraction_case(_mesh((k, *dims.values()), lambda: contraction_mesh(**dims)), model=c["model"], **kw)
    elif k == "polymesh":
        mesh = _mesh((k, c["nx"], c["ny"]), lambda: dataclasses.replace(
            contraction_mesh(c["nx"], c["nx"], 2 * c["ny"], c["ny"], two_d=True), shape=None, cellIJK=None))
        kw = {"alpha": 0.0, **kw}
        case = contraction_case(mesh, model=c["model"], dt=2e-3, **kw)
        case.solverU = SolverControl(c["solver"], "DILU", 1e-10)
        case.solverTheta = SolverControl(c["solver"], "DILU", 1e-10)
    else:
        dims = (c["nx"], c["ny"], c["nz"])
        case = periodic_channel_case(_mesh(("periodic", *dims), lambda: periodic_channel_mesh(*dims)),
                                     model=c["model"], **kw)
    case.precision = abi.RT_PREC_MIXED if c["precision"] == "mixed" else abi.RT_PREC_FP64
    return case


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "ldu":
        return _prepare_ldu(case, rng)
    if kind == "batch":
        return _prepare_batch(case, rng)
    cs = _case(case)
    ctx = Context()
    if kind == "correct":
        eq = ConstitutiveEq.New("const", cs, ctx)
    else:
        ctx.setup_case(cs)
    f = ctx.fields()   # the boundary values of the case
    if kind in ("periodic", "correct"):   # the laminar profile and its fluxes, with a seeded perturbation
        m = cs.mesh
        f.U[:, 0] = 1.5 * (1.0 - m.C[:, 1] ** 2) * (1.0 + 0.01 * rng.standard_normal(m.nCells))
        Uf = m.w[:, None] * (f.U[m.owner] - f.U[m.neighbour]) + f.U[m.neighbour]
        f.phi = (m.Sf * Uf).sum(1)
    _conformation(f, cs.model, rng, planar=kind in ("cavity", "polymesh"))
    if kind == "correct":
        ctx.set_fields(f)
        return dict(kind=kind, ctx=ctx, eq=eq, f=f)
    return dict(kind=kind, ctx=ctx, f=f, steps=case["steps"])


def _prepare_batch(c, rng):
    cases = []
    pick = np.random.default_rng(1000 * c["cases"] + c["n_min"])   # the sweep is the case's, its state the seed's
    for _ in range(c["cases"]):   # side, model, Wi and beta of each cavity
        n = int(pick.integers(c["n_min"], c["n_max"] + 1))
        model = ("Oldroyd-BLog", "GiesekusLog", "FENE-PLog")[int(pick.integers(0, 3))]
        cs = cavity_case(n, model=model, Wi=float(np.exp(pick.uniform(np.log(0.1), np.log(4.0)))),
                         beta=float(pick.uniform(0.1, 0.9)), mesh=_mesh(("cavity", n), lambda: cavity_mesh(n)),
                         **MODEL_KW[model])
        cs.precision = abi.RT_PREC_MIXED
        cases.append(cs)
    b = BatchContext(cases)
    f = b.ctx.fields()
    f.theta, f.eigVals, f.eigVecs, A = _lognormal(b.nCells, rng, planar=True)
    scale = np.repeat([cs.model.etaP / cs.model.lambda_ for cs in cases], np.diff(b.cellStart))
    f.tau = scale[:, None] * (A - np.array([1.0, 0, 0, 1, 0, 1]))
    return dict(kind="batch", ctx=b.ctx, batch=b, f=f, steps=c["steps"])


def _prepare_ldu(c, rng):
    dims = (c["nx"], c["ny"], c["nz"])
    m = _mesh(("ldu", *dims), lambda: contraction_mesh(dims[0] // 2, dims[0] - dims[0] // 2, dims[1] - 2 * (dims[1] // 4),
                                                       dims[1] // 4, dims[2]))
    ctx = Context()
    ctx.upload_mesh(m)
    N, nc = m.nCells, c["nc"]
    o, n = m.owner, m.neighbour
    # a laplacian with a lognormal cell coefficient (1/A of a momentum equation varies as much)
    k = np.exp(0.3 * rng.standard_normal(N))
    up = m.deltaCoeffs * m.magSf * (m.w * (k[o] - k[n]) + k[n])
    lo = up.copy()
    diag = -(np.bincount(o, up, N) + np.bincount(n, lo, N))
    bnd = np.bincount(m.bCell, m.bmagSf * m.bDelta, N)
    if c["solver"] == "PCG":   # the pressure equation: fixed at the outlet faces alone
        out = m.patch("outlet")
        s = slice(out.start, out.start + out.size)
        diag -= np.bincount(m.bCell[s], m.bmagSf[s] * m.bDelta[s], N)
    else:   # the momentum equation: ddt, walls, and upwind convection by a random flux
        flux = m.magSf * rng.standard_normal(m.nFaces)
        up, lo = -up + np.minimum(flux, 0.0), -lo - np.maximum(flux, 0.0)
        diag = -(np.bincount(o, up, N) + np.bincount(n, lo, N)) + bnd + m.V / 5e-3
    b = rng.standard_normal((nc, N)) * m.V
    ctl = SolverControl(c["solver"], "DIC" if c["solver"] == "PCG" else "DILU", 1e-10, maxIter=2000)
    return dict(kind="ldu", ctx=ctx, solver=LduSolver.New("x", ctl, ctx), diag=diag, up=up, lo=lo, b=b, mesh=m)


def run(state):
    ctx = state["ctx"]
    if state["kind"] == "ldu":
        psi = np.zeros_like(state["b"])
        state["solver"].solve(state["diag"], state["up"], state["lo"], psi, state["b"])
        return {"psi": psi}
    m, f = ctx.mesh, state["f"]
    N = m.nCells
    if state["kind"] == "correct":
        ctx.set_field(abi.RT_FIELD_THETA, f.theta, f.thetab)
        ctx.set_field(abi.RT_FIELD_EIGVALS, f.eigVals)
        ctx.set_field(abi.RT_FIELD_EIGVECS, f.eigVecs)
        state["eq"].correct()
        return {"theta": ctx.get_field(abi.RT_FIELD_THETA, (N, 6))[0], "tau": state["eq"].tau()}
    ctx.set_fields(f)
    if state["kind"] == "batch":
        state["batch"].step(state["steps"])
    else:
        ctx.step(state["steps"])
    return {"U": ctx.get_field(abi.RT_FIELD_U, (N, 3))[0], "p": ctx.get_field(abi.RT_FIELD_P, (N,))[0],
            "phi": ctx.get_field(abi.RT_FIELD_PHI, (m.nFaces,))[0],
            "theta": ctx.get_field(abi.RT_FIELD_THETA, (N, 6))[0], "tau": ctx.get_field(abi.RT_FIELD_TAU, (N, 6))[0]}


def _cells(c):
    k = c["kind"]
    if k == "cavity":
        return c["n"] ** 2
    if k == "contraction":
        return c["nz"] * (c["nx_up"] * (c["ny_in"] + 2 * c["ny_out"]) + c["nx_down"] * c["ny_in"])
    if k == "polymesh":
        return c["nx"] * 6 * c["ny"]
    if k == "batch":
        return c["cases"] * ((c["n_min"] + c["n_max"]) / 2) ** 2
    if k == "ldu":
        q, h = c["ny"] // 4, c["nx"] // 2
        return c["nz"] * (h * c["ny"] + (c["nx"] - h) * (c["ny"] - 2 * q))
    return c["nx"] * c["ny"] * c["nz"]


def work(case):
    """Each host field in and out once (FP64), and each step's state, matrix geometry and face data once."""
    N, k = _cells(case), case["kind"]
    faces = 2 if k in ("cavity", "polymesh", "batch") else 3   # internal faces a cell
    if k == "ldu":
        nc = case["nc"]
        return {"bytes": N * 8.0 * (1 + 2 * faces + 2 * nc), "flops": N * nc * (1.0 + 4 * faces)}
    if k == "correct":
        return {"bytes": N * 8.0 * (18 + 12 + 3 + 2 * faces), "flops": N * 1000.0}
    geometry = 8.0 * (1 + faces * 6)
    return {"bytes": N * (8.0 * (28 + faces + 16 + faces) + case["steps"] * (2 * 8.0 * (28 + faces) + geometry)),
            "flops": N * case["steps"] * 1500.0}


def exact(case, seed):
    """The solution of the `ldu` systems, by conjugate gradients (Jacobi; on A x = b, or on A^T A x = A^T b
    where A is not symmetric) and iterative refinement in 64 bits.  A time step and a correct() are None:
    their outputs are the iterates of a whole discretisation, which nothing plain gives."""
    if case["kind"] != "ldu":
        return None
    s = prepare(case, seed)
    m, dev = s["mesh"], "cuda" if torch.cuda.is_available() else "cpu"
    N = m.nCells
    t = {k: torch.tensor(np.ascontiguousarray(s[k]), device=dev) for k in ("diag", "up", "lo", "b")}
    o, n = (torch.tensor(a.astype(np.int64), device=dev) for a in (m.owner, m.neighbour))
    idx = torch.arange(N, device=dev)

    def csr(up, lo):
        return torch.sparse_coo_tensor(torch.stack([torch.cat([idx, o, n]), torch.cat([idx, n, o])]),
                                       torch.cat([t["diag"], up, lo]), (N, N)).to_sparse_csr()

    A = csr(t["up"], t["lo"])
    AT = A if case["solver"] == "PCG" else csr(t["lo"], t["up"])
    sym = case["solver"] == "PCG"
    d = t["diag"] if sym else t["diag"] ** 2
    if not sym:
        for i, v in ((o, t["lo"]), (n, t["up"])):   # the columns' sums of squares
            d = d.index_add(0, i, v * v)
    d = d[:, None]

    def op(x):
        return A @ x if sym else AT @ (A @ x)

    b = t["b"].T.contiguous()
    x = torch.zeros_like(b)
    for _ in range(4):   # refinement: each round solves for the residual of the last
        r = b - A @ x
        r = r if sym else AT @ r
        e, p, rz, r0 = torch.zeros_like(r), None, None, r.norm()
        for it in range(1500):
            z = r / d
            new = (r * z).sum(0)
            p = z if p is None else z + (new / rz) * p
            rz = new
            q = op(p)
            a = rz / (p * q).sum(0)
            e, r = e + a * p, r - a * q
            if it % 50 == 49 and not bool(r.norm() > 1e-11 * r0):
                break
        x = x + e
    return {"psi": x.T.contiguous()}
