"""The Sommerfeld integral radius by radius (csrc/greens.cu): a radius's
value does not depend on the radii tabulated with it, arguments beyond the
end of the J0 tables among them."""

import numpy as np
import pytest
from test_gpu_greens_tables import create

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kmax,im,krmax,rmax,n", [(100.0, 10.0, 200.0, 0.01, 5), (600.0, 200.0, 4e4, 0.03, 33),
                                                  (900.0, 25.0, 4.2e5, 0.04, 96), (9000.0, 25.0, 2e6, 0.04, 65)])
def test_radius_alone(gpu, kmax, im, krmax, rmax, n):
    from mom25d_gb300 import engine as E

    rng = np.random.default_rng(n)
    kc = np.sort(rng.uniform(1.0, kmax, 300)) + 1j * im * rng.uniform(0.1, 1, 300)
    kr = np.sort(rng.uniform(0.5 * kmax + 400, krmax + kmax + 400, 1500))
    wc, wr = rng.uniform(0.5, 1, kc.size) + 0.1j, rng.uniform(0.5, 1, kr.size)
    rho = np.concatenate([[0.0], np.sort(rng.uniform(0, rmax, n - 1))])
    ctx = E.Context(0)
    res = create(ctx, kc, wc, kr, wr, rho)[0]
    for part in (slice(0, 4), slice(n // 2, None), slice(0, None, 3)):
        if rho[part].size >= 4:
            assert np.array_equal(create(ctx, kc, wc, kr, wr, rho[part])[0], res[part]), part
    ctx.close()
