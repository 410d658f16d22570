"""What the speed of this engine is measured on.

Each case is work that a user of the engine has it do, through its public
entry points: a sweep (`Solver.sweep`, the whole path: Green's tables, fill,
LU and solve, de-embedding) and the stages that a program also calls by
themselves (`Greens`, `Solver.impedance`, `dense_solve`). Meshes are
the workloads of `mom25d_gb300/workloads.py`; their cell size sets the number
of unknowns. The frequencies (and the matrices of the dense solves) are made
from the seed.

What a sweep returns is held in 32 bits here (S and gamma in complex64, the
impedances in float32), because that is what it has: the Nelder-Mead wave fit
behind S stops anywhere in a flat valley of its objective, and mom25d's own S
moves by 8e-9 to 6e-8 when the fit's inputs are multiplied by 1 + 1e-15
(tests/golden/fit_floor.npz, tests/conftest.py fit_floor); the mixed path's
S is specified to 1e-5. The stages return what they compute: complex128.
"""

import math

import numpy as np
import torch

import mom25d_gb300 as G
from mom25d_gb300 import workloads
from mom25d_gb300.solver import Greens, Solver, dense_solve, tabulation_radii

GHz = 1e9

# workload: band [GHz] and range of max_cell [mm] that a user meshes it with
WORKLOADS = {
    "line": ((2.0, 9.0), (0.25, 0.7)),
    "shunt_via": ((3.0, 9.0), (0.15, 0.5)),
    "stripline": ((2.0, 10.0), (0.1, 0.4)),
    "tee": ((1.0, 10.0), (0.17, 0.7)),
    "bandpass": ((1.0, 12.0), (0.24, 0.6)),
    "via": ((1.0, 20.0), (0.16, 0.5)),
    "lpf": ((0.5, 8.0), (0.35, 1.0)),
}
MAX_N = 5943  # the largest listed mesh


def listed():
    return [
        # the Green's tables of one frequency alone: what a sweep of a layered stack begins each point
        # with, and what a program that fills elsewhere asks for (the smallest call)
        dict(name="greens_via", kind="greens", workload="via", cell=0.2),
        # one frequency of a short line with the default precision: a quick look at one small structure
        dict(name="line_point_fp64", kind="sweep", workload="line", cell=0.5, precision="fp64", nf=1, workers=1),
        # one frequency of the open-stub tee (N = 1085) in mixed precision: latency of a small point, as an
        # optimiser's objective calls it
        dict(name="tee_point_mixed", kind="sweep", workload="tee", cell=0.5, precision="mixed", nf=1, workers=1),
        # a short sweep of the tee with the default precision, four points in flight
        dict(name="tee_sweep_fp64", kind="sweep", workload="tee", cell=0.5, precision="fp64", nf=8, workers=4),
        # a sweep of the two-layer via transition (N = 3789): vias, two metal levels, eight points in flight
        dict(name="via_sweep_mixed", kind="sweep", workload="via", cell=0.2, precision="mixed", nf=8, workers=8),
        # one point of the low-pass filter (N = 5943, the engine's headline mesh) alone
        dict(name="lpf_point_mixed", kind="sweep", workload="lpf", cell=0.35, precision="mixed", nf=1, workers=1),
        # the headline sweep: the same filter, eight points in flight
        dict(name="lpf_sweep_mixed", kind="sweep", workload="lpf", cell=0.35, precision="mixed", nf=16, workers=8),
        # the same filter's point with the default precision (the largest)
        dict(name="lpf_point_fp64", kind="sweep", workload="lpf", cell=0.35, precision="fp64", nf=1, workers=1),
        # one point of a band-pass filter (N = 2434) with the compressed operator (method="hmatrix")
        dict(name="bandpass_point_hmatrix", kind="sweep", workload="bandpass", cell=0.46, precision="hmatrix", nf=1,
             workers=1),
        # the impedance matrix of the band-pass filter as a host array (mom25d's assemble): the fill by itself
        dict(name="impedance_fp64", kind="impedance", workload="bandpass", cell=0.46, precision="fp64"),
        # mom25d's _dense_solve on host arrays: a ragged order with two port columns in fp64, and a larger one
        # with four columns by the complex64 LU with refinement
        dict(name="solve_fp64", kind="solve", n=1543, nrhs=2, precision="fp64"),
        dict(name="solve_mixed", kind="solve", n=4001, nrhs=4, precision="mixed"),
    ]


def _mesh(case):
    lay, stack, mkw, _ = workloads.BUILDERS[case["workload"]](G, **({"k": 4} if case["workload"] == "bandpass" else {}))
    mkw = dict(mkw, max_cell=case["cell"] * 1e-3)
    return lay.mesh(**mkw), stack


def draw(rng):
    def log(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    kind = rng.choice(("sweep", "sweep", "sweep", "solve", "impedance", "greens"))
    if kind == "solve":
        precision = rng.choice(("fp64", "mixed"))
        return dict(kind=kind, n=int(log(150, 5000 if precision == "mixed" else 3000)), nrhs=rng.randint(1, 8),
                    precision=precision)
    workload = rng.choice(sorted(WORKLOADS))
    lo, hi = WORKLOADS[workload][1]
    case = dict(kind=kind, workload=workload, cell=round(log(lo, hi), 3))
    if kind == "greens":
        return case
    n = _mesh(case)[0].n_unknowns
    while n > (3000 if kind == "impedance" else MAX_N):
        case["cell"] = round(min(hi, case["cell"] * 1.15), 3)
        n = _mesh(case)[0].n_unknowns
    if kind == "impedance":
        return dict(case, precision="fp64")
    # the compressed operator is for the larger meshes
    compressed = ("hmatrix",) if 800 < n < 3500 and workload in ("tee", "bandpass", "lpf") else ()
    case["precision"] = rng.choice(("fp64", "mixed", "mixed") + compressed)
    if case["precision"] == "hmatrix":
        return dict(case, nf=1, workers=1)
    # an fp64 point costs about as much as ten mixed ones: the whole stays below the largest listed case
    cap = (0.5 if case["precision"] == "fp64" else 12) * (MAX_N / n) ** 2
    nf = max(1, min(int(log(1, 17)), int(cap)))
    return dict(case, nf=nf, workers=rng.choice((1, 4, 8)) if nf > 1 else 1)


def _solver(case):
    mesh, stack = _mesh(case)
    if case.get("precision") == "hmatrix":
        return Solver(mesh, stack, verbose=False, method="hmatrix")
    return Solver(mesh, stack, verbose=False, precision=case.get("precision", "fp64"))


def _freqs(case, seed, nf):
    """nf frequencies across the workload's band, one in each of nf equal parts of it."""
    f0, f1 = WORKLOADS[case["workload"]][0]
    u = (np.arange(nf) + np.random.default_rng(seed).uniform(0.05, 0.95, nf)) / nf
    return (f0 + (f1 - f0) * u) * GHz


def _matrix(case, seed):
    """Z and B of a dense solve: the potentials between n cells of a
    seeded strip layout over a ground plane, e^{-jkR}/R less the image's, as
    the entries of a moment-method matrix fall off and oscillate, with cells
    of uneven size and conductor loss on the diagonal; B: one 1 V gap across
    a few cells per column."""
    n, nrhs = case["n"], case["nrhs"]
    rng = np.random.default_rng(seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    side = math.sqrt(n)
    p = torch.tensor(rng.uniform(0, 1, (n, 2)) * (2.0 * side, 0.5 * side), device=dev)
    a = torch.tensor(rng.uniform(0.2, 0.4, n), device=dev)
    d2 = (p[:, None, 0] - p[None, :, 0]) ** 2 + (p[:, None, 1] - p[None, :, 1]) ** 2
    s2 = a[:, None] * a[None, :]
    R, Ri = torch.sqrt(d2 + s2), torch.sqrt(d2 + s2 + 9.0)
    k = 2 * math.pi / (0.8 * side)
    Z = torch.complex(torch.cos(k * R) / R - torch.cos(k * Ri) / Ri, torch.sin(k * Ri) / Ri - torch.sin(k * R) / R)
    Z = 1j * Z + torch.diag(torch.full((n,), 0.05, dtype=torch.complex128, device=dev))
    B = np.zeros((n, nrhs), complex)
    for c in range(nrhs):
        B[rng.choice(n, min(n, 12), replace=False), c] = rng.choice((-1.0, 1.0), min(n, 12))
    return Z.cpu().numpy(), B


def prepare(case, seed):
    if case["kind"] == "solve":
        Z, B = _matrix(case, seed)
        return dict(case=case, Z=Z, B=B)
    sol = _solver(case)
    f = _freqs(case, seed, case.get("nf", 1))
    # the tables' radii: the grid of the band's upper end, as a program that compares tables of several
    # frequencies asks for them (Greens(rho=))
    st = sol.stack
    kref = 2 * math.pi * WORKLOADS[case["workload"]][0][1] * GHz / G.C0 * math.sqrt(max(d.eps_r for d in st.layers))
    rho = tabulation_radii(sol.rho_max, 2 * math.pi / kref, min(d.t for d in st.layers))
    return dict(case=case, solver=sol, f=f, rho=rho)


def run(state):
    case = state["case"]
    if case["kind"] == "solve":
        return dense_solve(state["Z"], state["B"], precision=case["precision"])
    sol, f = state["solver"], state["f"]
    if case["kind"] == "greens":
        g = Greens(sol, float(f[0]), rho=state["rho"])
        S, c, coef = g.tables()
        g.close()
        return dict(S=S, lead=c, coef=coef)
    if case["kind"] == "impedance":
        return sol.impedance(float(f[0]))
    r = sol.sweep(f, workers=case["workers"])
    return dict(S=r.S.astype(np.complex64), gamma=r.gamma.astype(np.complex64), z0=r.z0.astype(np.float32),
                z0_line=r.z0_line.astype(np.complex64), fit_residual=r.fit_residual.astype(np.float32))


def work(case):
    if case["kind"] == "solve":
        n, m = case["n"], case["nrhs"]
        return dict(bytes=16.0 * n * n + 32.0 * n * m, flops=8.0 / 3 * n ** 3 + 8.0 * n * n * m)
    mesh, stack = _mesh(case)
    n, nt = mesh.n_unknowns, len(mesh.tris)
    if case["kind"] == "greens":
        # tables of 3 kernels per level pair at some 300 radii, each an integral over some 1500 path
        # nodes of one Bessel function and a complex multiply-add per kernel
        lv = len(mesh.layer_names) ** 2
        return dict(bytes=300.0 * lv * (3 + 12) * 16, flops=300.0 * 1500 * (30 + 24 * lv))
    # seven test points per triangle pair at the least, some 50 operations each (distance, interval,
    # two complex cubics, the sums)
    fill = 350.0 * nt * nt
    if case["kind"] == "impedance":
        return dict(bytes=16.0 * n * n, flops=fill)
    elem = 16 if case["precision"] == "fp64" else 8
    if case["precision"] == "hmatrix":
        # the near field filled and read once per iteration is what the compressed method saves: its
        # memory is counted once, its operations as a fifth of the dense fill's
        return dict(bytes=0.3 * 16.0 * n * n, flops=0.3 * fill)
    nf = case["nf"]
    return dict(bytes=2.0 * elem * n * n * nf, flops=(fill + 8.0 / 3 * n ** 3 + 16.0 * n * n) * nf)


def exact(case, seed):
    if case["kind"] != "solve" or case["n"] > 5000:
        return None  # the moment-method path has no independent form that is quick enough here
    Z, B = _matrix(case, seed)
    return np.linalg.solve(Z, B)
