"""The compressed operator's preconditioner blocks (the gj_* kernels in
csrc/hmatrix.cu) at sizes around their panels of 16 columns and tiles of 64,
through the solve that uses them: with one block over all unknowns the
preconditioner is the operator's own inverse in complex64."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length,cell", [(2.0, 0.7), (3.0, 0.6), (4.0, 0.5), (4.0, 0.35), (5.0, 0.34)])
def test_one_block_is_the_inverse(gpu, length, cell):
    import mom25d_gb300 as G
    from mom25d_gb300 import workloads
    from mom25d_gb300.hmatrix import HMatrix
    from mom25d_gb300.solver import Solver

    lay, sub, mkw, _ = workloads.line(G, length=length * 1e-3, cell=cell * 1e-3)
    mesh = lay.mesh(**mkw)
    n = mesh.n_unknowns
    sol = Solver(mesh, sub, verbose=False)
    f = 5e9
    # eta = 0: no far blocks, every leaf pair near, so the block holds the whole matrix
    hop = HMatrix(sol, eta=0.0, prec_block=min(n, 1024), overlap=False)
    if hop.plan.npc != 1:
        pytest.skip("more than one block")
    g = sol.greens(f)
    hop.assemble(g, complex(sol.surface_impedance(f)))
    B = sol.port_excitations().astype(complex)
    X = hop.solve(B, rtol=1e-10)
    # right-preconditioned by an inverse good to e = cond(W Z W) 2^-24 the residual falls by e a step: the
    # scaled matrix of this line has a condition number below 1e5, so e < 1e-2 and five steps reach 1e-10
    assert max(hop.stats["gmres_iterations"]) <= 6, hop.stats["gmres_iterations"]
    Z = sol.impedance(f)
    assert np.linalg.norm(Z @ X - B) <= 1e-8 * np.linalg.norm(B)
    hop.close()
    sol.close()
