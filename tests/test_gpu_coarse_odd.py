"""The coarse kernel's 1024-thread form (2D, coupled or variable viscosity, an odd
bottom level of more than 1024 cells) against the per-level launches
(fhd_ctx_set_coarse 0): equal bit for bit.  A single odd level on either side of
1024 cells, with more cells than threads, and one below even levels."""
import numpy as np
import pytest

from tests.test_gpu_coarse import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("visc", [-1, 2, -2, 3, -3])
@pytest.mark.parametrize("n", [[31, 33], [25, 41], [45, 63], [66, 70], [34, 61]])
def test_odd_bottoms(cuda, n, visc, precision):
    phi1, x1, n1 = _run(cuda, 2, n, visc, {}, 1, precision)
    phi0, x0, n0 = _run(cuda, 2, n, visc, {}, 0, precision)
    for a, b in zip(phi1 + x1, phi0 + x0):
        assert np.array_equal(a, b)
    assert n1 < n0
