"""Pivots whose squares leave the range of their type: the LU's panel
(csrc/lu_panel.cu) divides by them as by any other."""

import numpy as np
import pytest
from test_gpu_lu_paths import factors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [7, 65, 129, 300])
@pytest.mark.parametrize("dtype,scale", [(np.complex128, 2.0**600), (np.complex128, 2.0**-600),
                                         (np.complex64, 2.0**70), (np.complex64, 2.0**-70)])
def test_pivots_of_unusual_size(gpu, n, dtype, scale):
    """Scaling by a power of two scales U and leaves L and the pivots as they are, bit for bit."""
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))).astype(dtype)
    F, ipiv = factors(A)
    G, gpiv = factors(A * dtype(scale))
    assert np.array_equal(ipiv, gpiv)
    assert np.array_equal(np.tril(F, -1), np.tril(G, -1))
    assert np.array_equal(np.triu(F) * dtype(scale), np.triu(G))
