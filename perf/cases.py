"""Workloads of the library as its users run them, for timing and for comparing results.

Every case goes through ressim_gb300.api (the host binding of include/rsg.h):
the sparse matrix and its solvers on a user's own system, the mesh and its
transmissibilities, and the simulator's time step, adjoint and ensemble step.
Grid sizes lie between the smallest ensemble member (32 x 32 x 8) and the
128 x 128 x 32 two-phase grid, ragged ones included; fluids, wells and fields
are those of ressim_gb300.workloads.

A time step starts from a state kept with save_state, one step into the run,
so every pass does the same step; solver tolerances are tight enough for
solutions of different roundings to agree to well below 1e-9.
"""
import numpy as np
import torch

from ressim_gb300 import abi, api
from ressim_gb300 import workloads as W

TIGHT = 1e-12  # relative residual of the linear systems


def listed():
    return [
        # CompRowMatrix.mult, host vectors in and out: the smallest call of the matrix interface
        {"name": "mult 32x32x8", "kind": "mult", "ni": 32, "nj": 32, "nk": 8},
        # the 2D single-phase potential problem (64 x 64, MPFA-O, CG + ILU(0)): assemble, lock, factor, solve
        {"name": "potential 64x64 CG ILU", "kind": "potential", "ni": 64, "nj": 64},
        # a host program's own pressure matrix, new values each Newton iteration: upload, factor, solve in FP64
        {"name": "solve 64x64x16 BiCGstab ILU", "kind": "solve", "method": "bicgstab", "ni": 64, "nj": 64, "nk": 16},
        # the same at the largest grid with the mixed-precision solver
        {"name": "solve 128x128x32 mixed ILU", "kind": "solve", "method": "mixed", "ni": 128, "nj": 128, "nk": 32},
        # AMG setup and solve: FP64 GMRES around FP32 BiCGstab with the FP32 hierarchy
        {"name": "solve 40x36x12 mixed AMG", "kind": "amg", "ni": 40, "nj": 36, "nk": 12},
        # a mesh with its geometry and MPFA-O transmissibilities, read back
        {"name": "mpfa 64x64x16", "kind": "mpfa", "ni": 64, "nj": 64, "nk": 16},
        # time steps of the two-phase five-spot: smallest ensemble member, largest ensemble member, a ragged grid
        {"name": "step 32x32x8 FP64", "kind": "step", "mixed": False, "ni": 32, "nj": 32, "nk": 8},
        {"name": "step 96x96x24 FP64", "kind": "step", "mixed": False, "ni": 96, "nj": 96, "nk": 24},
        {"name": "step 75x61x19 mixed", "kind": "step", "mixed": True, "ni": 75, "nj": 61, "nk": 19},
        # Peng-Robinson line drive: flash, four components, mixed-precision pressure solve
        {"name": "compositional 32x32x8 mixed", "kind": "compositional", "mixed": True, "ni": 32, "nj": 32, "nk": 8},
        # recorded forward run and discrete adjoint on the sub-grid of the gradient checks
        {"name": "adjoint 32x32x8", "kind": "adjoint", "ni": 32, "nj": 32, "nk": 8},
        # uneven two-phase members stepped together, one launch per Newton iteration
        {"name": "ensemble of 6 mixed", "kind": "ensemble", "members": 6, "grids": 7},
    ]


def _size(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["mult", "potential", "solve", "solve", "amg", "mpfa", "step", "step", "step", "compositional",
                       "adjoint", "ensemble"])
    if kind == "potential":
        return {"kind": kind, "ni": _size(rng, 48, 160), "nj": _size(rng, 48, 160)}
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(3, 6), "grids": rng.randint(1, 10 ** 6)}
    hi = {"mult": (128, 128, 32), "solve": (112, 112, 28), "amg": (44, 40, 13), "mpfa": (96, 96, 24),
          "step": (96, 96, 24), "compositional": (40, 40, 10), "adjoint": (36, 36, 9)}[kind]
    lo = (24, 24, 8) if kind == "amg" else (32, 32, 8)
    case = {"kind": kind}
    for axis, a, b in zip(("ni", "nj", "nk"), lo, hi):
        case[axis] = _size(rng, a, b)
    if kind == "solve":
        case["method"] = rng.choice(["bicgstab", "mixed"])
    if kind in ("step", "compositional"):
        case["mixed"] = rng.random() < 0.5
    return case


# ------------------------------------------------- a host program's matrix ---
def _smooth_field(shape, corr, generator, device):
    """A smooth random field on a periodic grid: mean 0, standard deviation 1."""
    noise = torch.randn(shape, generator=generator, dtype=torch.float64).to(device)
    lam = 1.0
    for axis, s in enumerate(shape):
        f = torch.fft.fftfreq(s, dtype=torch.float64, device=device) * 2 * np.pi
        view = [1] * len(shape)
        view[axis] = s
        lam = lam * torch.exp(-(f * corr) ** 2 / 4).reshape(view)
    g = torch.fft.ifftn(torch.fft.fftn(noise) * lam).real
    return (g - g.mean()) / g.std()


def _pressure_matrix(ni, nj, nk, seed):
    """(row_ptr, col, val) of a pressure system on the 27-point pattern in
    natural order: lognormal permeability (standard deviation 1 in log10,
    correlation length 8 cells, a tenth of it vertically), weak corner and
    edge couplings with an unsymmetric part as upstream weighting leaves it,
    and an accumulation term."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = torch.Generator().manual_seed(seed)
    K = 10.0 ** _smooth_field((nk, nj, ni), 8.0, g, dev)
    n = ni * nj * nk
    idx = torch.arange(n, device=dev).reshape(nk, nj, ni)
    skew = torch.randn((nk, nj, ni), generator=g, dtype=torch.float64).to(dev).mul_(0.05)
    cols = torch.full((27, nk, nj, ni), -1, dtype=torch.int64, device=dev)
    vals = torch.zeros((27, nk, nj, ni), dtype=torch.float64, device=dev)
    for e in range(27):
        dk, dj, di = e // 9 - 1, e // 3 % 3 - 1, e % 3 - 1
        if e == 13:
            continue
        here = tuple(slice(max(0, -d), s - max(0, d)) for d, s in zip((dk, dj, di), (nk, nj, ni)))
        there = tuple(slice(max(0, d), s - max(0, -d)) for d, s in zip((dk, dj, di), (nk, nj, ni)))
        w = {1: 1.0, 2: 0.08, 3: 0.02}[abs(dk) + abs(dj) + abs(di)] * (0.1 if dk else 1.0)
        t = w * 2 * K[here] * K[there] / (K[here] + K[there])
        cols[(e,) + here] = idx[there]
        vals[(e,) + here] = -t * (1 + skew[here] * (di - dj))
    diag = -vals.sum(0)
    vals[13] = diag + 2e-3 * diag.mean()
    cols[13] = idx
    cols, vals = cols.reshape(27, n).T, vals.reshape(27, n).T
    keep = cols >= 0
    rp = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    rp[1:] = torch.cumsum(keep.sum(1), 0)
    return (rp.to(torch.int32).cpu().numpy(), cols[keep].to(torch.int32).cpu().numpy(), vals[keep].cpu().numpy())


def _times(rp, col, val, x):
    """A x in 64 bits (torch)."""
    A = torch.sparse_csr_tensor(torch.from_numpy(rp).long(), torch.from_numpy(col).long(), torch.from_numpy(val),
                                (len(rp) - 1, len(rp) - 1))
    return (A @ torch.from_numpy(x)).numpy()


def _vector(n, seed):
    return np.random.Generator(np.random.PCG64(seed)).standard_normal(n)


# ---------------------------------------------------------------- prepare ---
def _spec(mixed, **kw):
    spec = W.runspec(method=abi.FGMRES_MIXED if mixed else abi.BICGSTAB, precond=abi.PC_ILU, stop_rule=1, **kw)
    spec.truncate_negative_moles = 1  # some fields overshoot in a few cells of the explicit molar update
    return spec


def _two_phase(ctx, ni, nj, nk, seed, **kw):
    case = W.two_phase_case(ni=ni, nj=nj, nk=nk, seed=seed)
    keep = abi.Keep()
    srcs = W.build_sources(keep, case)
    mesh = api.Mesh(ctx, 3, ni, nj, nk, case["perm"], coords=case["nodes"])
    mesh.compute_mpfa()
    sim = api.Discretisation(ctx, mesh, W.two_phase_fluid(keep), W.corey(), case["porosity"], case["compaction"],
                             srcs, W.build_initial(case), _spec(**kw))
    return {"ctx": ctx, "sim": sim, "mesh": mesh, "dt": case["dt"], "producer": case["producer"],
            "keep": (keep, srcs, case)}


def _kept(st):
    """One step into the run (the pattern's plans exist), then the state every pass starts from."""
    st["sim"].step(st["dt"])
    st["sim"].save_state()
    return st


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        members = []
        for m, (ni, nj, nk) in enumerate(W.ensemble_sizes(case["members"], case["grids"], (32, 32, 8), (56, 56, 14))):
            members.append(_kept(_two_phase(api.Context(0), ni, nj, nk, seed + 100 * m, mixed=False)))
        return {"kind": kind, "members": members, "sims": [m["sim"] for m in members],
                "dts": [m["dt"] for m in members]}
    ctx = api.Context(0)
    ni, nj, nk = case["ni"], case["nj"], case.get("nk", 1)
    if kind in ("mult", "solve", "amg"):
        rp, col, val = _pressure_matrix(ni, nj, nk, seed)
        n = len(rp) - 1
        x = _vector(n, seed)
        st = {"kind": kind, "ctx": ctx, "A": api.CompRowMatrix(ctx, n, rp, col, val), "x": x, "val": val}
        if kind != "mult":
            st["b"], st["x0"] = _times(rp, col, val, x), np.zeros(n)
            cls = api.BiCGstab if case.get("method") == "bicgstab" else api.MixedFGMRES
            st["solver"] = cls(ctx, abi.PC_AMG if kind == "amg" else abi.PC_ILU, rtol=TIGHT, max_iter=5000)
            st["solver"].set_matrix(st["A"])  # the pattern's plans, as in a program past its first iteration
        return st
    if kind == "potential":
        c = W.potential_case(ni=ni, nj=nj, seed=seed)
        mesh = api.Mesh(ctx, 2, ni, nj, 0, c["perm"])
        mesh.compute_mpfa()
        rp, col = mesh.pattern(1)
        A = api.CompRowMatrix(ctx, len(rp) - 1, rp, col)
        b = W.potential_rhs(c)
        st = {"kind": kind, "ctx": ctx, "mesh": mesh, "A": A, "b": b, "fixed": c["dirichlet_cells"],
              "solver": api.CG(ctx, abi.PC_ILU, rtol=TIGHT)}
        mesh.assemble_potential(A)
        A.zero_rows(1.0, st["fixed"])
        st["solver"].set_matrix(A)
        return st
    if kind == "mpfa":
        c = W.two_phase_case(ni=ni, nj=nj, nk=nk, seed=seed)
        return {"kind": kind, "ctx": ctx, "dims": (ni, nj, nk), "perm": c["perm"], "nodes": c["nodes"]}
    if kind == "compositional":
        c = W.compositional_case(ni, nj, nk, seed=seed, dt=2000.0)
        keep = abi.Keep()
        fluid = W.compositional_fluid(keep)
        srcs = W.build_compositional_sources(keep, c, fluid.nc)
        mesh = api.Mesh(ctx, 3, ni, nj, nk, c["perm"], coords=c["nodes"])
        mesh.compute_mpfa()
        sim = api.Discretisation(ctx, mesh, fluid, W.corey(), c["porosity"], c["compaction"], srcs,
                                 W.build_compositional_initial(c, fluid.nc), _spec(case["mixed"]))
        return _kept({"kind": kind, "ctx": ctx, "sim": sim, "mesh": mesh, "dt": c["dt"], "keep": (keep, srcs, c)})
    if kind == "adjoint":
        st = _two_phase(ctx, ni, nj, nk, seed, mixed=False, rtol=1e-13, atol=1e-24, ptol=1e-11, max_newton=30)
        st["dt"] /= 4  # a short step: no cell reaches the truncation, which has no derivative
    else:
        st = _two_phase(ctx, ni, nj, nk, seed, mixed=case["mixed"])
    st["kind"] = kind
    return _kept(st)


# -------------------------------------------------------------------- run ---
def run(state):
    kind = state["kind"]
    if kind == "mult":
        return state["A"].mult(state["x"])
    if kind in ("solve", "amg"):
        A, solver = state["A"], state["solver"]
        A.set_values(state["val"])
        solver.set_matrix(A)
        return solver.solve(A, state["b"], state["x0"])
    if kind == "potential":
        A, solver = state["A"], state["solver"]
        state["mesh"].assemble_potential(A)
        A.zero_rows(1.0, state["fixed"])
        solver.set_matrix(A)
        x = solver.solve(A, state["b"], state["b"])
        return {"p": x, "flux": state["mesh"].connection_flux(x)}
    if kind == "mpfa":
        mesh = api.Mesh(state["ctx"], 3, *state["dims"], state["perm"], coords=state["nodes"])
        mesh.compute_mpfa()
        ptr, el, t = mesh.transmissibilities()
        centers, volumes = mesh.geometry()
        mesh.release()
        return {"ptr": ptr, "el": el, "t": t, "centers": centers, "volumes": volumes}
    if kind == "ensemble":
        for s in state["sims"]:
            s.restore_state()
        _, statuses = api.ensemble_step_batched(state["sims"], state["dts"], precision=1)
        if statuses.any():
            raise RuntimeError("an ensemble member failed: %s" % statuses)
        return [dict(zip(("p", "N", "S"), s.state())) for s in state["sims"]]
    sim = state["sim"]
    sim.restore_state()
    if kind == "adjoint":
        J, _ = sim.forward([state["dt"]] * 2, 1, state["producer"], [0.0, 1.0])
        grad, dp0, dN0, _ = sim.backward(rtol=1e-13)
        return {"J": J, "grad": grad, "dp0": dp0, "dN0": dN0}
    sim.step(state["dt"])
    return dict(zip(("p", "N", "S"), sim.state()))


# ------------------------------------------------------------------- work ---
def work(case):
    """Bytes and operations of one pass.  A Krylov iteration reads the matrix
    (value and column) and both factors and about ten vectors per
    application of each; iterations and Newton iterations per pass are the
    usual ones of these systems (BiCGstab and the inner BiCGstab apply
    matrix and factors twice an iteration)."""
    kind = case["kind"]
    if kind == "ensemble":
        grids = W.ensemble_sizes(case["members"], case["grids"], (32, 32, 8), (56, 56, 14))
        parts = [work({"kind": "step", "mixed": True, "ni": i, "nj": j, "nk": k}) for i, j, k in grids]
        return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts)}
    ni, nj, nk = case["ni"], case["nj"], case.get("nk", 1)
    n = ni * nj * nk
    nnz = (3 * ni - 2) * (3 * nj - 2) * (3 * nk - 2 if nk > 1 else 1)
    if kind == "mult":
        return {"bytes": 12 * nnz + 20 * n, "flops": 2 * nnz}
    if kind == "mpfa":
        # corner points, tensors, geometry in and out; about twelve connections' local systems per corner point
        return {"bytes": 24 * n + 48 * n + 32 * n + 12 * 54 * n, "flops": 12 ** 3 * 2 * n}
    entry = 8 if case.get("mixed") or case.get("method") == "mixed" or kind == "amg" else 12
    applies = {"potential": 80, "solve": 150, "amg": 60, "step": 300, "compositional": 60, "adjoint": 1200}[kind]
    return {"bytes": applies * (2 * entry * nnz + 80 * n) + 600 * n, "flops": applies * 4 * nnz + 1000 * n}


# ------------------------------------------------------------------ exact ---
def exact(case, seed):
    """The product in 64 bits; for a solve, the vector its right-hand side was made from."""
    if case["kind"] not in ("mult", "solve", "amg"):
        return None  # a whole mesh or simulator: no short 64-bit restatement
    rp, col, val = _pressure_matrix(case["ni"], case["nj"], case.get("nk", 1), seed)
    x = _vector(len(rp) - 1, seed)
    return _times(rp, col, val, x) if case["kind"] == "mult" else x
