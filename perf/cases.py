"""The work that a user of this framework has it do, as timed cases: the
condensation and reconstruction of one device, of a batch of devices and of
host buffers, and the Newton solves built on them, from the smallest meshes
to the largest of the benchmark configurations.

A case is a dict of plain values; ``listed()`` gives the fixed ones,
``draw(rng)`` one more of the same ranges, ``prepare`` the solvers, states and
buffers that a user's program holds, ``run`` one pass through the public entry
points, ``work`` the bytes and operations that a pass cannot do without and
``exact`` the condensed systems in plain 64-bit torch.
"""

import functools
import math

import numpy as np
import torch

from ddhdg_b200 import _lib, workloads
from ddhdg_b200.batch import CondenseBatch
from ddhdg_b200.functions import EV, KB, Q
from ddhdg_b200.problem import DDFluxType
from ddhdg_b200.solver import NPSolver

LENGTH_SCALE = 1e-6  # mesh unit of the diodes, metres


def listed():
    return [
        # one Newton step's local work on a 1D device: launch latency
        dict(name="condense_1d_m64_k2", kind="condense", dim=1, m=64, k=2, flux=0),
        # the small 2D diode (32 x 32 cells, degree 1) of the first configuration
        dict(name="condense_2d_m32_k1", kind="condense", dim=2, m=32, k=1, flux=0),
        # the headline workload: 256 x 256 cells, degree 2
        dict(name="condense_2d_m256_k2", kind="condense", dim=2, m=256, k=2, flux=0),
        # the highest degree in 2D, on an odd mesh
        dict(name="condense_2d_m101_k3", kind="condense", dim=2, m=101, k=3, flux=0),
        # a 3D degree-1 device, on an odd mesh
        dict(name="condense_3d_m31_k1", kind="condense", dim=3, m=31, k=1, flux=0),
        # the largest local systems (3D, degree 2), with the upwinded flux
        dict(name="condense_3d_m9_k2", kind="condense", dim=3, m=9, k=2, flux=2),
        # independent 2D diodes of mixed sizes and degrees, one launch per step
        dict(name="batch_2d_n12", kind="batch", n=12, lo=16, hi=128),
        # the same step for a host program that keeps its vectors in host memory
        dict(name="host_2d_m160_k2", kind="host", dim=2, m=160, k=2, flux=0),
        # a whole small solve: equilibrium, then the solve at a bias
        dict(name="solve_2d_m32_k1", kind="solve", dim=2, m=32, k=1, bias=0.3, mixed=False),
        # one point of the bias sweep on the 256 x 256 degree-2 diode
        dict(name="newton_2d_m256_k2", kind="newton", dim=2, m=256, k=2, bias=0.05, mixed=False),
        # one bias point of a 3D device, mixed-precision condensation
        dict(name="newton_3d_m14_k1_mixed", kind="newton", dim=3, m=14, k=1, bias=0.2, mixed=True),
        # the serving loop's step: requests of different sizes advanced together
        dict(name="serve_2d_n6", kind="serve", n=6, lo=32, hi=96, bias=0.3, mixed=True),
    ]


def _spread(rng, lo, hi):
    """A whole number in lo..hi, uniform over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


# largest mesh per side of the condensation cases, by (dim, degree)
_CONDENSE_MAX = {(1, 1): 4096, (1, 2): 4096, (1, 3): 4096, (2, 1): 256, (2, 2): 256, (2, 3): 101, (3, 1): 31,
                 (3, 2): 9}


def draw(rng):
    kind = rng.choice(["condense", "condense", "condense", "batch", "host", "solve", "newton", "newton", "serve"])
    if kind == "condense":
        dim, k = rng.choice([(1, 1), (1, 2), (1, 3), (2, 1), (2, 2), (2, 2), (2, 3), (3, 1), (3, 2)])
        hi = _CONDENSE_MAX[dim, k]
        lo = {1: 16, 2: 8, 3: 4}[dim]
        return dict(kind=kind, dim=dim, m=_spread(rng, lo, hi), k=k, flux=rng.choice([0, 0, 0, 2]))
    if kind == "batch":
        return dict(kind=kind, n=rng.randint(3, 12), lo=16, hi=rng.randint(32, 128))
    if kind == "host":
        return dict(kind=kind, dim=2, m=_spread(rng, 16, 160), k=rng.choice([1, 2]), flux=0)
    if kind == "solve":
        return dict(kind=kind, dim=2, m=_spread(rng, 32, 96), k=1, bias=rng.choice([0.1, 0.2, 0.3]), mixed=False)
    if kind == "newton":
        if rng.random() < 0.3:
            return dict(kind=kind, dim=3, m=rng.randint(8, 14), k=1, bias=0.2, mixed=rng.choice([True, False]))
        return dict(kind=kind, dim=2, m=_spread(rng, 32, 200), k=rng.choice([1, 2]), bias=rng.choice([0.05, 0.2]),
                    mixed=rng.choice([True, False]))
    return dict(kind=kind, n=rng.randint(2, 6), lo=32, hi=rng.randint(48, 96), bias=rng.choice([0.1, 0.3]),
                mixed=rng.choice([True, False]))


# ------------------------------------------------------------------ devices
def _devices(case, seed):
    """The devices of a case: mesh and degree from the case, doping level and
    junction position from the seed (batches: sizes and degrees spread over
    the case's range in a fixed order, so that every seed costs the same)."""
    rng = np.random.default_rng(seed)
    n = case.get("n", 1)
    newton = case["kind"] in ("solve", "newton", "serve")
    out = []
    for i in range(n):
        if n > 1:
            t = (i * 0.6180339887498949) % 1.0
            m = int(round(case["lo"] + t * (case["hi"] - case["lo"])))
            k = 1 + i % (2 if newton else 3)
            dim = 2
        else:
            dim, m, k = case["dim"], case["m"], case["k"]
        N = float(10 ** (rng.uniform(22.5, 23.0) if newton else rng.uniform(21.0, 24.0)))
        xj = float(rng.uniform(0.45, 0.55) if newton else rng.uniform(0.3, 0.7))
        out.append(dict(dim=dim, m=m, k=k, N=N, xj=xj, flux=case.get("flux", 0), mixed=bool(case.get("mixed"))))
    return out


def _solver(d):
    precision = 1 if d["mixed"] and 3 * (d["k"] + 1) ** d["dim"] <= 32 else 0
    pb, prm, adim = workloads.diode(dim=d["dim"], m=d["m"], k=d["k"], N_D=d["N"], N_A=d["N"], x_j=d["xj"],
                                    flux=DDFluxType(d["flux"]), precision=precision)
    prm.consistent_drift_jacobian = True
    prm.consistent_recombination_jacobian = True
    return NPSolver(pb, prm, adim), pb


def _lobatto(k):
    return {1: [0.0, 1.0], 2: [0.0, 0.5, 1.0],
            3: [0.0, 0.5 - 0.1 * math.sqrt(5.0), 0.5 + 0.1 * math.sqrt(5.0), 1.0]}[k]


def _face_layout(dim, m):
    """Face index of every cell's faces [cells, 2 dim] and the face count:
    faces axis by axis, lexicographic, the low side first."""
    idx = np.arange(m ** dim)
    ci = np.stack([(idx // m ** a) % m for a in range(dim)], 1)
    faces = np.zeros((m ** dim, 2 * dim), dtype=np.int64)
    off = 0
    for a in range(dim):
        ext = [m + (b == a) for b in range(dim)]
        for side in (0, 1):
            fi = ci.copy()
            fi[:, a] += side
            stride, f = 1, np.zeros(len(idx), dtype=np.int64)
            for b in range(dim):
                f += fi[:, b] * stride
                stride *= ext[b]
            faces[:, 2 * a + side] = off + f
        off += int(np.prod(ext))
    return ci, faces, off


def _state(d, seed):
    """A Newton iterate near equilibrium: a smooth potential step across the
    junction, its Boltzmann densities and fluxes, and relative noise; with a
    trace update of the size of a Newton step.  Rescaled units."""
    dim, m, k, N, xj = d["dim"], d["m"], d["k"], d["N"], d["xj"]
    rng = np.random.default_rng([seed, m, k, dim])
    g = workloads.GAAS
    ut = KB * g["T"] / Q
    Vn, Vp = workloads.lcn_potential(N), workloads.lcn_potential(-N)
    nodes = np.array(_lobatto(k))

    def fields(x):
        w = 0.05
        th = np.tanh((x - xj) / w)
        V = Vn + (Vp - Vn) * 0.5 * (1 + th)
        dV = (Vp - Vn) * 0.5 * (1 - th * th) / w
        n = g["Nc"] * np.exp((V - g["Ec"]) / ut) / N
        p = g["Nv"] * np.exp((g["Ev"] - V) / ut) / N
        return (V, n, p), (-dV, -n * dV / ut, p * dV / ut)

    nb, nf, F = (k + 1) ** dim, (k + 1) ** (dim - 1), 2 * dim
    ci, faces, nfaces = _face_layout(dim, m)
    ref = nodes[np.arange(nb) % (k + 1)]
    val, flux = fields((ci[:, :1] + ref[None]) / m)
    cell = np.zeros((m ** dim, 3, dim + 1, nb))
    for c in range(3):
        cell[:, c, dim] = val[c]
        cell[:, c, 0] = flux[c]
    trace = np.zeros((nfaces, 3, nf))
    for f in range(F):
        fr = np.zeros(nf)
        if f // 2 == 0:
            fr[:] = f % 2
        else:
            r = np.arange(nf)
            for t in range(dim - 1):
                if (f // 2 + 1 + t) % dim == 0:
                    fr = nodes[r % (k + 1)]
                r = r // (k + 1)
        v, _ = fields((ci[:, :1] + fr[None]) / m)
        for c in range(3):
            trace[faces[:, f], c] = v[c]
    cell *= 1 + 1e-3 * rng.standard_normal(cell.shape)
    trace *= 1 + 1e-3 * rng.standard_normal(trace.shape)
    upd = 1e-3 * trace * rng.standard_normal(trace.shape)
    return cell.reshape(m ** dim, -1), trace, upd


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    devs = _devices(case, seed)
    kind = case["kind"]
    if kind in ("condense", "host", "batch"):
        solvers, upds = [], []
        for i, d in enumerate(devs):
            s, _ = _solver(d)
            cell, trace, upd = _state(d, seed + 7919 * i)
            s.set_state(cell, trace)
            solvers.append(s)
            upds.append(torch.as_tensor(upd.reshape(-1), device=s.device))
        if kind == "condense":
            return dict(kind=kind, solver=solvers[0], upd=upds[0])
        if kind == "batch":
            b = CondenseBatch(solvers)
            for dst, src in zip(b.update_trace, upds):
                dst.copy_(src)
            return dict(kind=kind, batch=b)
        s = solvers[0]
        nc, Nt = s.ncells, s.sizes().Nt
        dev = dict(dtype=torch.float64, device=s.device)
        return dict(kind=kind, solver=s, cell=s.cell_state.cpu().pin_memory(),
                    trace=s.trace_state.cpu().pin_memory(), upd=upds[0].cpu().pin_memory(),
                    out=torch.empty(nc * s.Nc_all, dtype=torch.float64).pin_memory(),
                    tt=torch.empty(nc, Nt, Nt, **dev), rhs=torch.empty(nc, Nt, **dev),
                    dflag=torch.empty(nc, Nt, dtype=torch.int32, device=s.device), dval=torch.empty(nc, Nt, **dev))
    solvers, problems, starts = [], [], []
    for d in devs:
        s, pb = _solver(d)
        if kind != "solve":
            s.compute_thermodynamic_equilibrium()
            starts.append((s.cell_state.clone(), s.trace_state.clone()))
        solvers.append(s)
        problems.append(pb)
    st = dict(kind=kind, solvers=solvers, problems=problems, starts=starts, bias=case["bias"])
    if kind == "serve":
        st["batch"] = CondenseBatch(solvers)
    return st


# ---------------------------------------------------------------------- run
def run(state):
    kind = state["kind"]
    if kind == "condense":
        s = state["solver"]
        tt, rhs, dflag, dval = s.assemble_condense()
        return tt, rhs, dflag, dval, s.reconstruct(state["upd"])
    if kind == "batch":
        b = state["batch"]
        b.condense()
        b.reconstruct()
        return [(b.tt[i], b.rhs[i], b.dflag[i], b.dval[i], b.update_cell[i]) for i in range(len(b.tt))]
    if kind == "host":
        s = state["solver"]
        sp = s._sp()
        _lib.check(s.L.ddhdg_assemble_condense_host(
            s._ctx, state["cell"].data_ptr(), state["trace"].data_ptr(), 0, state["tt"].data_ptr(),
            state["rhs"].data_ptr(), state["dflag"].data_ptr(), state["dval"].data_ptr(), sp),
            "assemble_condense_host")
        _lib.check(s.L.ddhdg_reconstruct_host(s._ctx, state["upd"].data_ptr(), 0, state["out"].data_ptr(), sp),
                   "reconstruct_host")
        return (state["tt"], state["rhs"], state["dflag"], state["dval"],
                state["out"].view(s.ncells, s.Nc_all))
    if kind == "solve":
        s, pb = state["solvers"][0], state["problems"][0]
        s.cell_state.zero_()
        s.trace_state.zero_()
        workloads.set_bias(pb, 0.0)
        s.update_boundary_tables()
        s.compute_thermodynamic_equilibrium()
        workloads.set_bias(pb, state["bias"])
        s.update_boundary_tables()
        s.run()
        return s.cell_state.clone(), s.trace_state.clone()
    for s, pb, start in zip(state["solvers"], state["problems"], state["starts"]):
        s.cell_state.copy_(start[0])
        s.trace_state.copy_(start[1])
        workloads.set_bias(pb, state["bias"])
        s.update_boundary_tables()
    if kind == "newton":
        s = state["solvers"][0]
        s.run()
        return s.cell_state.clone(), s.trace_state.clone()
    # the serving loop: batched Newton steps until every request has converged
    b = state["batch"]
    done = np.zeros(len(state["solvers"]), dtype=bool)
    for _ in range(30):
        norms, status = b.newton_step(1.0)
        if any(status):
            raise RuntimeError(f"batched Newton step failed: {status}")
        upd, cur = norms[:, :2].max(1), norms[:, 2:].max(1)
        done |= (upd < 1e-10) | (upd < 1e-10 * cur)
        if done.all():
            break
    return [(s.cell_state.clone(), s.trace_state.clone()) for s in state["solvers"]]


# --------------------------------------------------------------------- work
def _condense_work(dim, m, k):
    """Bytes and operations of one condensation and one reconstruction: the
    state in, the condensed block, right-hand side, flags and the cell update
    out; the scalar system's assembly, LU, solves and Schur product."""
    nb, nf, F = (k + 1) ** dim, (k + 1) ** (dim - 1), 2 * dim
    Ns, Nt, Nc = 3 * nb, F * 3 * nf, 3 * (dim + 1) * nb
    cells, faces = m ** dim, dim * (m + 1) * m ** (dim - 1)
    by = cells * 8 * (Nc + Nt * Nt + 2 * Nt + Nc) + cells * 4 * Nt + faces * 8 * 6 * nf
    fq = F * nf
    asm = 7 * 2 * nb * nb * (nb * (1 + dim) + fq) + 5 * 2 * nb * F * nf * (nb * dim + fq)
    fl = asm + 2 * Ns ** 3 / 3 + 2 * Ns * Ns * (1 + Nt) + 2 * Nt * Nt * Ns + 2 * Ns * Nt + 2 * (Nc - Ns) * (nb + F * nf)
    return by, cells * fl


def _trace_work(dim, m, k, comps):
    """Operations of a nested-dissection LU solve of the trace system: the
    grid bisected along its longest axis, each separator eliminated densely
    against the boundary of its box."""
    nd = comps * (k + 1) ** (dim - 1)

    @functools.lru_cache(maxsize=None)
    def box(ext, bnd):  # bnd: (low, high) of every axis on the physical boundary
        vol = math.prod(ext)
        if vol == 1:
            e = sum(sum(b) for b in bnd) * nd
            return _front(e, 2 * dim * nd - e)
        s = max(range(dim), key=lambda a: (ext[a], -a))
        e = vol // ext[s] * nd
        kept = sum(vol // ext[a] * ((not bnd[a][0]) + (not bnd[a][1])) for a in range(dim)) * nd
        lo = ext[s] // 2
        a = box(ext[:s] + (lo,) + ext[s + 1:], bnd[:s] + ((bnd[s][0], False),) + bnd[s + 1:])
        b = box(ext[:s] + (ext[s] - lo,) + ext[s + 1:], bnd[:s] + ((False, bnd[s][1]),) + bnd[s + 1:])
        return a + b + _front(e, kept)

    def _front(e, kept):
        return 2 * e ** 3 / 3 + 2 * e * e * (kept + 1) + 2 * e * kept * (kept + 1)

    return box((m,) * dim, ((True, True),) * dim)


def work(case):
    by = fl = 0.0
    for d in _devices(case, 0):
        b, f = _condense_work(d["dim"], d["m"], d["k"])
        if case["kind"] in ("solve", "newton", "serve"):
            # about five Newton steps; states in and out once
            f = 5 * (f + _trace_work(d["dim"], d["m"], d["k"], 3))
            if case["kind"] == "solve":
                f += 5 * _trace_work(d["dim"], d["m"], d["k"], 1)
            nb, nf = (d["k"] + 1) ** d["dim"], (d["k"] + 1) ** (d["dim"] - 1)
            faces = d["dim"] * (d["m"] + 1) * d["m"] ** (d["dim"] - 1)
            b = 16 * (d["m"] ** d["dim"] * 3 * (d["dim"] + 1) * nb + faces * 3 * nf)
        by += b
        fl += f
    return {"bytes": int(by), "flops": int(fl)}


# -------------------------------------------------------------------- exact
def exact(case, seed):
    if case["kind"] not in ("condense", "host", "batch"):
        return None  # a whole Newton solve: minutes in plain torch
    out = []
    for i, d in enumerate(_devices(case, seed)):
        out.append(_exact_device(d, *_state(d, seed + 7919 * i)))
    return out if case["kind"] == "batch" else out[0]


def _tables(dim, k, h):
    """Tensor-product Lagrange bases on the Gauss-Lobatto nodes and the
    (k+1)-point Gauss rule, on a cell of side h and on its faces."""
    nodes = np.array(_lobatto(k))
    gx, gw = np.polynomial.legendre.leggauss(k + 1)
    gx, gw = 0.5 * (gx + 1), 0.5 * gw
    polys = []
    for i in range(k + 1):
        p = np.poly1d([1.0])
        for j in range(k + 1):
            if j != i:
                p = p * np.poly1d([1.0, -nodes[j]]) / (nodes[i] - nodes[j])
        polys.append(p)
    val = lambda x: np.array([[p(xx) for p in polys] for xx in np.atleast_1d(x)])  # noqa: E731
    der = lambda x: np.array([[p.deriv()(xx) for p in polys] for xx in np.atleast_1d(x)])  # noqa: E731

    def tensor(mats):  # axis 0 fastest, in points and in nodes
        r = np.ones((1, 1))
        for mt in mats:
            r = np.kron(mt, r)
        return r

    B, D1 = val(gx), der(gx) / h
    nb, nf = (k + 1) ** dim, (k + 1) ** (dim - 1)
    T = {"phi": tensor([B] * dim),
         "grad": np.stack([tensor([D1 if a == s else B for a in range(dim)]) for s in range(dim)], 1),
         "wc": tensor([gw[:, None]] * dim)[:, 0] * h ** dim}
    wf = tensor([gw[:, None]] * (dim - 1))[:, 0]
    T["xi"] = tensor([B] * (dim - 1))
    T["wf"] = wf * h ** (dim - 1)
    phif = np.zeros((2 * dim, nf, nb))
    for f in range(2 * dim):
        a, side = divmod(f, 2)
        tang = [(a + 1 + t) % dim for t in range(dim - 1)]
        for q in range(nf):
            x = np.zeros(dim)
            x[a] = side
            r = q
            for t in tang:
                x[t] = gx[r % (k + 1)]
                r //= k + 1
            phif[f, q] = tensor([val(x[b]) for b in range(dim)])[0]
    T["phif"] = phif
    mass = T["phi"].T @ (T["wc"][:, None] * T["phi"])
    sg = np.array([-1.0, 1.0] * dim)
    G = np.einsum("qe,qsc,q->sce", T["phi"], T["grad"], T["wc"])
    CW = np.zeros((dim, nb, 2 * dim, nf))
    for f in range(2 * dim):
        CW[f // 2, :, f] = sg[f] * np.einsum("qm,qc,q->cm", T["xi"], phif[f], T["wf"])
    T["P"] = np.linalg.solve(mass[None], G)
    T["Q"] = np.linalg.solve(mass[None], CW.reshape(dim, nb, -1)).reshape(CW.shape)
    T["PWc"] = np.einsum("sce,qc->qse", T["P"], T["phi"])
    T["QWc"] = np.einsum("scfm,qc->qsfm", T["Q"], T["phi"])
    ax = np.arange(2 * dim) // 2
    T["PWf"] = np.einsum("f,fce,fqc->fqe", sg, T["P"][ax], phif)
    T["QWf"] = np.einsum("f,fcgm,fqc->fqgm", sg, T["Q"][ax], phif)
    T["proj"] = np.linalg.solve(T["xi"].T @ (wf[:, None] * T["xi"]), T["xi"].T * wf)
    T["sg"] = sg
    return T


def _exact_device(d, cell, trace, upd):
    """Condensed system and cell update of every cell: the flux unknowns
    eliminated with the cell mass matrix, the scalar system (V, n, p) solved
    for the residual and for every trace dof."""
    dim, m, k, N, xj = d["dim"], d["m"], d["k"], d["N"], d["xj"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    h = 1.0 / m
    nb, nf, F = (k + 1) ** dim, (k + 1) ** (dim - 1), 2 * dim
    T = {a: torch.as_tensor(v, dtype=torch.float64, device=dev) for a, v in _tables(dim, k, h).items()}
    ci, faces, _ = _face_layout(dim, m)
    g = workloads.GAAS
    Vres, ut, L = 1.0, KB * g["T"] / Q, LENGTH_SCALE  # the temperature magnitude Q / KB makes the unit of V one volt
    eps = g["eps_r"] * 8.85418781762e-12 / (L * L * Q * Q * N / Q)
    mu = (0.0, g["mu_n"], g["mu_p"])
    rec_rescale = Q * N / (L * L * Q)
    ni = math.sqrt(g["Nc"] * g["Nv"] * math.exp((g["Ev"] - g["Ec"]) * EV / (KB * g["T"]))) / N
    srh = 1e-9
    gx = 0.5 * (np.polynomial.legendre.leggauss(k + 1)[0] + 1)
    xq = (ci[:, :1] + gx[np.arange(nb) % (k + 1)][None]) * h
    dop = np.where(xj - xq > 0, 1.0, -1.0)
    bcV, bcD = [None] * 2, [None] * 2
    for side, dp in ((0, N), (1, -N)):
        V = workloads.lcn_potential(dp)
        bcV[side] = V / Vres
        bcD[side] = (g["Nc"] * math.exp((Q * V - g["Ec"] * EV) / (KB * g["T"])) / N,
                     g["Nv"] * math.exp((-Q * V + g["Ev"] * EV) / (KB * g["T"])) / N)
    res = ([], [], [], [], [])
    step = max(1, int(2e8 / ((3 * nb) * (1 + 2 * F * 3 * nf) * 8 + (F * 3 * nf) ** 2 * 8)))
    for c0 in range(0, m ** dim, step):
        sl = slice(c0, min(m ** dim, c0 + step))
        to = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
        u = to(cell[sl]).view(-1, 3, dim + 1, nb)
        lam, dl = to(trace[faces[sl]]), to(upd[faces[sl]])
        lam, dl = lam.view(-1, F, 3, nf).transpose(1, 2), dl.view(-1, F, 3, nf).transpose(1, 2)  # [B, 3, F, nf]
        W, uS = u[:, :, :dim], u[:, :, dim]
        o = _exact_cells(T, dim, nb, nf, F, u, W, uS, lam, dl, to(dop[sl]), ci[sl], m, eps, mu, ut, rec_rescale, ni,
                         srh, N, d["flux"], bcV, bcD)
        for r, x in zip(res, o):
            r.append(x.cpu())
    return tuple(torch.cat(r) for r in res)


def _exact_cells(T, dim, nb, nf, F, u, W, uS, lam, dl, dop, ci, m, eps, mu, ut, rec_rescale, ni, srh, N, flux, bcV,
                 bcD):
    E = torch.einsum
    B = u.shape[0]
    z = lambda *s: torch.zeros(B, *s, dtype=torch.float64, device=u.device)  # noqa: E731
    ax = torch.arange(F, device=u.device) // 2
    c0, W0 = E("qa,bca->bcq", T["phi"], uS), E("qa,bcsa->bcsq", T["phi"], W)
    c0f = E("fqa,bca->bcfq", T["phif"], uS)
    W0n = E("f,fqa,bcfa->bcfq", T["sg"], T["phif"], W[:, :, ax])
    tr0 = E("qm,bcfm->bcfq", T["xi"], lam)
    n0, p0 = c0[:, 1], c0[:, 2]
    num, den = n0 * p0 - ni * ni, srh * (n0 + ni) + srh * (p0 + ni)
    r = num * N / den / rec_rescale
    drn = (p0 / den - num * srh / den ** 2) / rec_rescale * N
    drp = (n0 / den - num * srh / den ** 2) / rec_rescale * N
    Wres = E("sce,bke->bksc", T["P"], uS) - E("scfm,bkfm->bksc", T["Q"], lam) - W
    Wrc = E("qc,bksc->bksq", T["phi"], Wres)
    Wrf = E("f,fqc,bkfc->bkfq", T["sg"], T["phif"], Wres[:, :, ax])
    E0n = W0n[:, 0]
    one = torch.ones_like(E0n)
    side = one if flux == 0 else torch.where(E0n > 0, one, 0 * one)  # 1: the cell's density in the drift flux
    al, ka, be = z(3, 3, nb), z(3, 3, nb), z(3, 3, dim, nb)
    ga, rh, tw = z(3, 3, F, nf), z(3, 3, F, nf), z(3, 3, F, nf)
    ctc, ctd, tcs, ttc, rr = (z(3, F, nf) for _ in range(5))
    r0, r1, rf = z(3, nb), z(3, dim, nb), z(3, F, nf)
    ka[:, 0, 0] = -eps
    al[:, 0, 1], al[:, 0, 2] = 1.0, -1.0
    ga[:, 0, 0], rh[:, 0, 0], tw[:, 0, 0] = 1.0, eps, -eps
    ctc[:, 0] = tcs[:, 0] = ttc[:, 0] = -1.0
    rr[:, 0] = -eps * E0n - c0f[:, 0] + tr0[:, 0]
    rf[:, 0] = tr0[:, 0] - eps * E0n - c0f[:, 0]
    r0[:, 0] = dop + p0 - n0
    r1[:, 0] = eps * W0[:, 0]
    for b, s in ((1, 1.0), (2, -1.0)):
        cb = (n0, p0)[b - 1]
        cst = side * c0f[:, b] + (1 - side) * tr0[:, b]
        drift = s * mu[b] * E0n
        al[:, b, 1], al[:, b, 2] = -drn, -drp
        ka[:, b, 0] = -s * cb * mu[b]
        ka[:, b, b] = ut * mu[b]
        be[:, b, b] = -s * mu[b] * W0[:, 0]
        rh[:, b, 0], tw[:, b, 0] = s * mu[b] * cst, -s * mu[b] * cst
        ga[:, b, b] = side * drift - 1.0
        rh[:, b, b], tw[:, b, b] = -ut * mu[b], ut * mu[b]
        ctc[:, b] = 1.0
        ctd[:, b] = (1 - side) * drift
        tcs[:, b] = -side * drift + 1.0
        ttc[:, b] = 1.0 + ctd[:, b]
        J = drift * cst - ut * mu[b] * W0n[:, b]
        rr[:, b] = -J + c0f[:, b] - tr0[:, b]
        rf[:, b] = -tr0[:, b] - J + c0f[:, b]
        r0[:, b] = r
        r1[:, b] = s * cb[:, None] * mu[b] * W0[:, 0] - ut * mu[b] * W0[:, b]
    r1 = r1 - E("bcpq,bpsq->bcsq", ka, Wrc)
    rf = rf - E("bcpfq,bpfq->bcfq", rh, Wrf)
    TLc, TLg, TLf = T["wc"][:, None] * T["phi"], T["wc"][:, None, None] * T["grad"], T["wf"][:, None] * T["phif"]
    S = E("bcpq,qa,qe->bcape", al, TLc, T["phi"]) + E("bcpsq,qsa,qe->bcape", be, TLg, T["phi"]) \
        + E("bcpq,qae->bcape", ka, E("qsa,qse->qae", TLg, T["PWc"])) \
        + E("bcpfq,fqae->bcape", ga, E("fqa,fqe->fqae", TLf, T["phif"])) \
        + E("bcpfq,fqae->bcape", rh, E("fqa,fqe->fqae", TLf, T["PWf"]))
    R0 = E("qa,bcq->bca", TLc, r0) + E("qsa,bcsq->bca", TLg, r1) + E("fqa,bcfq->bca", TLf, rf)
    Rt = -E("bcpq,qafm->bcafpm", ka, E("qsa,qsfm->qafm", TLg, T["QWc"])) \
        - E("bcpgq,gqafm->bcafpm", rh, E("gqa,gqfm->gqafm", TLf, T["QWf"]))
    face = E("fqa,qm->fqam", TLf, T["xi"])
    Rd = Rt.clone()
    for b in range(3):
        Rt[:, b, :, :, b] += E("bfq,fqam->bafm", ctc[:, b], face)
        Rd[:, b, :, :, b] += E("bfq,fqam->bafm", ctc[:, b] + ctd[:, b], face)
    Ns, Nt = 3 * nb, F * 3 * nf
    Sm = S.reshape(B, Ns, Ns)
    Rm = torch.cat([R0.reshape(B, Ns, 1), Rt.reshape(B, Ns, Nt), Rd.reshape(B, Ns, Nt)], 2)
    sc = Sm.abs().amax(2, keepdim=True)
    Y = torch.linalg.solve(Sm / sc, Rm / sc)
    Y0, Yt, Yd = Y[:, :, 0], Y[:, :, 1:1 + Nt], Y[:, :, 1 + Nt:]
    # Dirichlet data on the contacts (x faces of the device)
    flag, g = z(F, 3, nf), z(F, 3, nf)
    cx = torch.as_tensor(ci[:, 0], device=u.device)
    for f, on in ((0, cx == 0), (1, cx == m - 1)):
        for b in range(3):
            bc = bcV[f] if b == 0 else bcD[f][b - 1]
            gv = E("mq,bq->bm", T["proj"], bc - tr0[:, b, f])
            flag[:, f, b] = on.double()[:, None]
            g[:, f, b] = torch.where(on[:, None], gv, 0 * gv)
    gt, ft = g.reshape(B, Nt), flag.reshape(B, Nt)
    Yc0 = Y0 - E("bst,bt->bs", Yd, gt)
    wx = T["wf"][:, None] * T["xi"]
    Tc = z(F, 3, nf, 3, nb)
    Tq = E("qm,bcpfq,fqgn->bfcmgpn", wx, tw, T["QWf"])
    for p in range(3):
        Tc[:, :, :, :, p] = E("qm,bcfq,fqe->bfcme", wx, tw[:, :, p], T["PWf"])
    for b in range(3):
        Tc[:, :, b, :, b] += E("qm,bfq,fqe->bfme", wx, tcs[:, b], T["phif"])
        for f in range(F):
            Tq[:, f, b, :, f, b] += E("qm,bq,qn->bmn", wx, ttc[:, b, f], T["xi"])
    H = Wrf - E("fqgn,bgpn->bpfq", T["QWf"], g)
    rZ = E("qm,bcfq->bfcm", wx, rr + E("bcpfq,bpfq->bcfq", tw, H))
    Tm = Tc.reshape(B, Nt, Ns)
    rhs = (E("bts,bs->bt", Tm, Yc0) + rZ.reshape(B, Nt)) * (1 - ft)
    tt = (Tm @ Yd + Tq.reshape(B, Nt, Nt)) * (1 - ft)[:, :, None] * (1 - ft)[:, None, :]
    du = Y0 - E("bst,bt->bs", Yt, dl.transpose(1, 2).reshape(B, Nt))
    out = z(3, dim + 1, nb)
    du = du.view(B, 3, nb)
    out[:, :, dim] = du
    out[:, :, :dim] = E("sce,bke->bksc", T["P"], uS + du) - E("scfm,bkfm->bksc", T["Q"], lam + dl) - W
    return tt, rhs, flag.reshape(B, Nt).to(torch.int32), gt, out.reshape(B, -1)
