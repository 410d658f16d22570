"""The wave fit (fit_kernel in csrc/deembed.cu) for port groups of one to
four ports and more or fewer than 32 cuts per feed, against the oracle's fit
of the same cut currents and voltages."""

import numpy as np
import pytest
from conftest import gamma_floor

from oracle import sweep as O

pytestmark = pytest.mark.gpu

mm = 1e-3


def layout(nports, feed):
    import mom25d_gb300 as G

    W = 1.137 * mm
    lay = G.Layout()
    for k in range(max(1, nports // 2)):  # parallel lines, fed at one or both ends
        y = 2 * k * W
        lay.add_rect(0, y - W / 2, 4 * mm, y + W / 2)
        lay.add_port(f"A{k}", (0, y), "-x", W, feed)
        if nports > 1:
            lay.add_port(f"B{k}", (4 * mm, y), "+x", W, feed)
    return lay, G.Substrate(eps_r=3.55, h=0.508 * mm, tand=0.0027, sigma=5.8e7)


@pytest.mark.parametrize("nports,feed,cell", [(1, 8 * mm, 0.5 * mm), (2, 14 * mm, 0.2 * mm), (4, 8 * mm, 0.5 * mm),
                                              (4, 14 * mm, 0.25 * mm)])
def test_fit_groups(gpu, nports, feed, cell):
    from mom25d_gb300.solver import Solver

    lay, sub = layout(nports, feed)
    sol = Solver(lay.mesh(max_cell=cell, edge_cell=0.15 * mm), sub, verbose=False)
    assert len(sol.groups) == 1 and len(sol.ports) == nports
    f = 5e9
    S, z0, gamma, z0_line, res, _, _ = sol.point(f)
    _, _, I, V = sol.last_deembed()
    off = np.r_[0, np.cumsum([pm.s.size for pm in sol.pm])]
    datasets = [(sol.pm[p].s, I[off[p]:off[p + 1], e], V[off[p]:off[p + 1], e])
                for p in range(nports) for e in range(nports)]
    b0 = float(sol.beta0(f)[0])
    g, z, coefs, r = O.fit_waves([d[0] for d in datasets], [d[1] for d in datasets], [d[2] for d in datasets],
                                 1e-3 * b0 + 1j * b0)
    # the same search on the same data ends within the flat valley in which the fit's floor was measured
    assert np.all(np.abs(gamma - g) <= 3 * gamma_floor() * abs(g))
    assert np.all(np.abs(z0_line - z) <= 3 * gamma_floor() * abs(z))
    # gamma off by d |gamma| moves the fitted waves by at most d (beta s) of their size, beta s of a few
    # radians over the feed, and at a minimum the squared residual by the square of that
    assert np.all(np.abs(res**2 - r**2) <= (10 * 3 * gamma_floor())**2)
    sol.close()
