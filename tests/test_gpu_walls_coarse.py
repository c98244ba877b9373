"""The single-block coarse end of the staggered V-cycle on walled domains
against the per-level launches (fhd_ctx_set_coarse 0): the same expressions in
the same order, so equal bit for bit in FP64; and both against the oracle at
the tolerance of the wall tests.  The shapes have even and odd bottoms, odd
extents between walls (in place) and across a periodic direction (two passes),
and every kind of wall at each end."""
import numpy as np
import pytest

import lowmachfhd_b200 as L
import oracle as O
from tests import problems as P
from tests.test_gpu_parity import dev, host, zeros
from tests.test_gpu_walls import NS, PE, SL, periodic_afterwards, solver, wall_rhs  # noqa: F401

pytestmark = pytest.mark.gpu

CASES = [
    (2, [64, 48], [PE, NS, PE], [PE, SL, PE]),
    (2, [40, 24], [SL, NS, PE], [NS, SL, PE]),
    (2, [128, 128], [NS, PE, PE], [NS, PE, PE]),
    (2, [15, 9], [PE, NS, PE], [PE, NS, PE]),
    (2, [15, 9], [NS, SL, PE], [NS, SL, PE]),
    (3, [32, 16, 24], [PE, PE, NS], [PE, PE, SL]),
    (3, [12, 20, 8], [NS, SL, NS], [SL, SL, NS]),
    (3, [40, 24, 40], [PE, NS, PE], [PE, NS, PE]),
    (3, [5, 7, 9], [SL, PE, NS], [SL, PE, NS]),
]


@pytest.mark.parametrize("dim,n,bc_lo,bc_hi", CASES)
def test_walls_coarse_end(cuda, dim, n, bc_lo, bc_hi):
    rng = np.random.default_rng(61)
    pb = P.problem(dim, n, 1, dx=1.0, seed=62)
    alpha = [1.0 + 0.2 * rng.random(pb.nc) for _ in range(dim)]
    b_u, b_p = wall_rhs(dim, n, bc_lo, 63, 1.5)
    out = []
    for coarse in (1, 0):
        with solver(dim, n, bc_lo, bc_hi) as s:
            s.set_coarse(coarse)
            coef = (dev(alpha, cuda), dev(pb.beta, cuda), dev(pb.beta_ed, cuda), dev(pb.gamma, cuda))
            x_u, x_p = zeros(pb.nc, dim, cuda), zeros(pb.nc, 1, cuda)[0]
            s.apply_precon(dev(b_u, cuda), dev(b_p, cuda), x_u, x_p, *coef, 1.5)
            phi = zeros(pb.nc, dim, cuda)
            s.stag_mg_solver(*coef, 1.5, phi, dev(b_u, cuda))
            out.append((host(x_u) + [host(x_p)] + host(phi), s.kernel_launches))
    for a, b in zip(out[0][0], out[1][0]):
        assert np.array_equal(a, b)
    assert out[0][1] < out[1][1]
    O.set_walls(bc_lo, bc_hi)
    opb = O.Problem(dim, n, 1.0, 1, alpha, pb.beta, pb.beta_ed, pb.gamma)
    ref = O.stag_mg_solver(opb, O.default_params(), 1.5, b_u)
    assert P.rel_inf(out[0][0][dim + 1:], ref) < 1e-12
