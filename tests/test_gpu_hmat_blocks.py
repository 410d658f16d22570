"""The compressed operator's preconditioner blocks where the caller's lists
leave parts of a block out (diag_kernel in csrc/hmatrix.cu)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def operator(monkeypatch=None, edit=None, cell=0.35, **kw):
    import mom25d_gb300 as G
    from mom25d_gb300 import hmatrix, workloads
    from mom25d_gb300.solver import Solver

    lay, sub, mkw, _ = workloads.line(G, length=4e-3, cell=cell * 1e-3)
    sol = Solver(lay.mesh(**mkw), sub, verbose=False)
    if edit:
        make = hmatrix.Plan

        def plan(*a):
            P = make(*a)
            edit(P)
            return P

        monkeypatch.setattr(hmatrix, "Plan", plan)
    return sol, hmatrix.HMatrix(sol, **kw)


@pytest.mark.parametrize("kept", ["diagonal", "all but the corners"])
def test_leaf_pairs_left_out_are_zero(gpu, monkeypatch, kept):
    """Leaf pairs that no item of a block names are zero in it, at the first
    assembly and at the next: the same preconditioner, the same solution."""

    def edit(P):
        it, off, out, ioff = P.pc_items, P.pc_item_off, [], [0]
        for k in range(P.npc):
            b = it[off[k]:off[k + 1]]
            gap = abs(b[:, 1] - b[:, 2])
            b = b[gap == 0] if kept == "diagonal" else b[gap < gap.max()]
            out.append(b)
            ioff.append(ioff[-1] + len(b))
        assert ioff[-1] < len(it)
        P.pc_items, P.pc_item_off = np.concatenate(out), np.array(ioff, np.int64)

    sol, hop = operator(monkeypatch, edit, prec_block=100, leaf=24)
    assert hop.plan.npc >= 2
    B = sol.port_excitations().astype(complex)
    g = sol.greens(5e9)
    zs = complex(sol.surface_impedance(5e9))
    out = []
    for _ in range(3):
        hop.assemble(g, zs)
        out.append((hop.solve(B, rtol=1e-10), hop.stats["gmres_iterations"]))
    for X, its in out[1:]:
        assert its == out[0][1] and np.array_equal(X, out[0][0])
    hop.close()
    sol.close()
