"""The z-march smoothers (one or two red-black smooths per launch) against the
colour-by-colour sweeps (fhd_ctx_set_fused 0) on the same inputs.  Both
evaluate the same expression on the same operands in the same colour order,
so they agree bit for bit in both precisions; the shapes cover tiles that do
not divide the level, rows that wrap inside one tile and rows cut into
several, short z-runs, and smooth counts that leave the unknowns in the other
buffer."""
import numpy as np
import pytest

import lowmachfhd_b200 as L
from tests import problems as P
from tests.test_gpu_parity import dev, host, zeros

pytestmark = pytest.mark.gpu

# (n, smooths down, smooths up): finest levels above the single-CTA coarse end
CASES = [([40, 40, 40], 2, 2), ([72, 24, 56], 2, 2), ([34, 30, 26], 3, 2), ([130, 18, 22], 1, 2), ([20, 70, 66], 2, 1),
         ([96, 64, 32], 4, 1), ([28, 28, 28], 1, 1), ([256, 32, 16], 2, 2)]


def _run(cuda, n, down, up, precision, fused, seed=91):
    pb = P.problem(3, n, 1, dx=1.0, seed=seed)
    rng = np.random.default_rng(seed)
    alpha = [1.0 + 0.2 * rng.random(pb.nc) for _ in range(3)]
    phi0, _ = P.random_stokes(3, n, seed=seed + 3)
    rhs, _ = P.random_stokes(3, n, seed=seed + 1)
    b_u, b_p = P.random_stokes(3, n, seed=seed + 2)
    params = L.default_params(stag_mg_nsmooths_down=down, stag_mg_nsmooths_up=up, mg_nsmooths_down=down,
                              mg_nsmooths_up=up)
    with L.StokesSolver(3, n, 1.0, 1, params=params, precision=precision) as s:
        s.set_fused(fused)
        s.set_tune(0)
        coef = (dev(alpha, cuda), dev(pb.beta, cuda), dev(pb.beta_ed, cuda), dev(pb.gamma, cuda))
        phi = dev(phi0, cuda)  # a start that is not zero
        s.stag_mg_solver(*coef, 0.7, phi, dev(rhs, cuda))
        x_u, x_p = zeros(pb.nc, 3, cuda), zeros(pb.nc, 1, cuda)[0]
        s.apply_precon(dev(b_u, cuda), dev(b_p, cuda), x_u, x_p, *coef, 1.5)
        return host(phi) + host(x_u) + [host(x_p)], s.kernel_launches


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n,down,up", CASES)
def test_march_equals_colour_sweeps(cuda, n, down, up, precision):
    a, na = _run(cuda, n, down, up, precision, -1)
    b, nb = _run(cuda, n, down, up, precision, 0)
    assert na < nb
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
