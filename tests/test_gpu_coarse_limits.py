"""Where the staggered coarse end begins in 2D.  Levels of uncoupled variable
viscosity (visc_type -1) in FP32 enter the single-block kernel up to 4096 cells,
levels of the other viscosity types and precisions up to 2400: a
stag_mg_solver call whose finest level enters it launches what the call on half
the extents launches, and the preparation of one more level.  The results agree with the per-level launches at the tolerance of
test_coarse_kernel_mixed."""
import pytest

import lowmachfhd_b200 as L
from tests import problems as P
from tests.test_gpu_parity import dev, host, zeros

pytestmark = pytest.mark.gpu


def _solve(cuda, n, visc, precision, coarse=1):
    pb = P.problem(2, n, visc, dx=1.0, seed=41)
    rhs, _ = P.random_stokes(2, n, seed=42)
    with L.StokesSolver(2, n, 1.0, visc, params=L.default_params(), precision=precision) as s:
        s.set_coarse(coarse)
        s.set_tune(0)
        phi = zeros(pb.nc, 2, cuda)
        s.stag_mg_solver(dev(pb.alpha_fc, cuda), dev(pb.beta, cuda), dev(pb.beta_ed, cuda), dev(pb.gamma, cuda), 0.7,
                         phi, dev(rhs, cuda))
        return host(phi), s.kernel_launches


@pytest.mark.parametrize("n,visc,precision,enters", [
    ([64, 64], -1, "mixed", True), ([48, 64], -1, "mixed", True), ([64, 66], -1, "mixed", False),
    ([56, 56], -1, "fp64", False), ([64, 64], -2, "mixed", False), ([64, 64], 2, "mixed", False),
    ([48, 48], -2, "mixed", True), ([40, 56], 3, "fp64", True),
])
def test_two_dimensional_limit(cuda, n, visc, precision, enters):
    a, na = _solve(cuda, n, visc, precision)
    b, _ = _solve(cuda, n, visc, precision, coarse=0)
    assert P.rel_inf(a, b) < 1e-5
    # one level less, all of it in the kernel; one more level is prepared by
    # five launches (cell and edge viscosities, gamma, alpha, pressure
    # coefficients)
    _, base = _solve(cuda, [m // 2 for m in n], visc, precision)
    assert (na == base + 5) == enters
