"""What a handle of the compressed operator holds on the device (csrc/hmatrix.cu)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_memory_of_a_handle(gpu):
    """A handle keeps its operator and the blocks' inverses; what only an assembly needs is not held beside them."""
    import torch

    import mom25d_gb300 as G
    from mom25d_gb300 import workloads
    from mom25d_gb300.hmatrix import HMatrix
    from mom25d_gb300.solver import Solver

    lay, sub, mkw, _ = workloads.BUILDERS["bandpass"](G, k=4)
    sol = Solver(lay.mesh(**dict(mkw, max_cell=0.46e-3)), sub, verbose=False)
    sol.geometry()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    hop = HMatrix(sol)
    torch.cuda.synchronize()
    held = before - torch.cuda.mem_get_info()[0]
    P = hop.plan
    inverses = 8 * int((P.prec_sizes.astype(np.int64) ** 2).sum())
    near = int((P.near_arr[:, 1].astype(np.int64) * P.near_arr[:, 3]).sum())
    m, n = P.far_arr[:, 1].astype(np.int64), P.far_arr[:, 3].astype(np.int64)
    kcap = np.minimum(np.maximum(2, np.minimum(m, n) // 3), 96)
    terms = int((kcap * (m + n))[np.minimum(m, n) > 64].sum())
    # near blocks and low-rank terms in complex128 and in double-float; half of the inverses for all lists and vectors
    assert inverses > 32 << 20
    assert held <= 32 * (near + terms) + inverses + inverses // 2, (held, near, terms, inverses)
    hop.close()
    sol.close()
