"""The compressed operator's plans for the meshes on which
test_gpu_hmat_prec.py takes the preconditioner for the operator's inverse."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length,cell", [(2.0, 0.7), (3.0, 0.6), (4.0, 0.5), (4.0, 0.35), (5.0, 0.34)])
def test_plans_of_one_block(gpu, length, cell):
    """With eta = 0 and room for every unknown the plan is one block, as the tests of its inverse take it."""
    import mom25d_gb300 as G
    from mom25d_gb300 import workloads
    from mom25d_gb300.hmatrix import Plan
    from mom25d_gb300.solver import Solver

    lay, sub, mkw, _ = workloads.line(G, length=length * 1e-3, cell=cell * 1e-3)
    sol = Solver(lay.mesh(**mkw), sub, verbose=False)
    sol.geometry()
    P = Plan(sol.mesh, sol.zl, sol._blocks_host, eta=0.0, prec_block=min(sol.mesh.n_unknowns, 1024), overlap=False)
    assert P.npc == 1 and P.prec_sizes[0] == sol.mesh.n_unknowns
    sol.close()
