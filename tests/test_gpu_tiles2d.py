"""The 2D tile smoothers (one or two red-black smooths per launch) against the
colour-by-colour sweeps (fhd_ctx_set_fused 0): the same expression on the same
operands in the same colour order, so equal bit for bit in both precisions.
The shapes cover tiles that do not divide the level, extents below one tile
in each direction (the tile wraps around more than once), and smooth counts
that leave the unknowns in the other buffer."""
import numpy as np
import pytest

import lowmachfhd_b200 as L
from tests import problems as P
from tests.test_gpu_parity import dev, host, zeros

pytestmark = pytest.mark.gpu

# (n, smooths down, smooths up): finest levels above the single-CTA coarse end
CASES = [([256, 128], 2, 2), ([120, 112], 2, 2), ([130, 98], 3, 2), ([4, 4096], 2, 1), ([4096, 4], 1, 2),
         ([62, 202], 4, 3), ([514, 22], 1, 1), ([12, 1000], 2, 2)]


def _run(cuda, n, down, up, precision, fused, seed=191):
    pb = P.problem(2, n, 1, dx=1.0, seed=seed)
    rng = np.random.default_rng(seed)
    alpha = [1.0 + 0.2 * rng.random(pb.nc) for _ in range(2)]
    phi0, _ = P.random_stokes(2, n, seed=seed + 3)
    rhs, _ = P.random_stokes(2, n, seed=seed + 1)
    b_u, b_p = P.random_stokes(2, n, seed=seed + 2)
    params = L.default_params(stag_mg_nsmooths_down=down, stag_mg_nsmooths_up=up, mg_nsmooths_down=down,
                              mg_nsmooths_up=up)
    with L.StokesSolver(2, n, 1.0, 1, params=params, precision=precision) as s:
        s.set_fused(fused)
        s.set_tune(0)
        coef = (dev(alpha, cuda), dev(pb.beta, cuda), dev(pb.beta_ed, cuda), dev(pb.gamma, cuda))
        phi = dev(phi0, cuda)  # a start that is not zero
        s.stag_mg_solver(*coef, 0.7, phi, dev(rhs, cuda))
        x_u, x_p = zeros(pb.nc, 2, cuda), zeros(pb.nc, 1, cuda)[0]
        s.apply_precon(dev(b_u, cuda), dev(b_p, cuda), x_u, x_p, *coef, 1.5)
        return host(phi) + host(x_u) + [host(x_p)], s.kernel_launches


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n,down,up", CASES)
def test_tiles_equal_colour_sweeps(cuda, n, down, up, precision):
    a, na = _run(cuda, n, down, up, precision, -1)
    b, nb = _run(cuda, n, down, up, precision, 0)
    assert na < nb
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
