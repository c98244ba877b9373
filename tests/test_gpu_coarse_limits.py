"""Where the coarse end of the V-cycles begins in 2D.

Levels that smooth by colour launches enter the single-block kernel as soon as
they fit when the call's launches are issued one by one: a stag_mg_solver call
whose finest level enters launches what the call on half the extents launches, and
the preparation of one more level.  In GMRES, whose preconditioner is replayed as a
graph, levels above 2400 cells (visc_type -1 in FP32: 4096) go by launches.
Levels of constant viscosity smooth on tiles and go by launches above 2400 cells
either way.  The routes agree bit for bit."""
import numpy as np
import pytest

import lowmachfhd_b200 as L
from tests import problems as P
from tests.test_gpu_parity import dev, host, zeros

pytestmark = pytest.mark.gpu


def _solver(n, visc, precision, **kw):
    return L.StokesSolver(2, n, 1.0, visc, params=L.default_params(**kw), precision=precision)


def _problem(cuda, n, visc):
    pb = P.problem(2, n, visc, dx=1.0, seed=41)
    rhs, b_p = P.random_stokes(2, n, seed=42)
    return pb, rhs, b_p, (dev(pb.alpha_fc, cuda), dev(pb.beta, cuda), dev(pb.beta_ed, cuda), dev(pb.gamma, cuda))


def _stag(cuda, n, visc, precision, coarse=1, fused=-1):
    pb, rhs, _, coef = _problem(cuda, n, visc)
    with _solver(n, visc, precision) as s:
        s.set_coarse(coarse)
        s.set_fused(fused)
        s.set_tune(0)
        phi = zeros(pb.nc, 2, cuda)
        s.stag_mg_solver(*coef, 0.7, phi, dev(rhs, cuda))
        return host(phi), s.kernel_launches


@pytest.mark.parametrize("n,visc,precision,fused,enters", [
    ([64, 64], -1, "mixed", -1, True), ([64, 64], -2, "mixed", -1, True), ([64, 64], 2, "mixed", -1, True),
    ([48, 64], 3, "fp64", -1, True), ([56, 56], -3, "fp64", -1, True), ([64, 64], 1, "mixed", 0, True),
    ([64, 64], 1, "mixed", -1, False), ([48, 64], 1, "fp64", -1, False), ([48, 48], 1, "mixed", -1, True),
    ([96, 112], 2, "mixed", -1, False),  # does not fit
])
def test_single_calls(cuda, n, visc, precision, fused, enters):
    a, na = _stag(cuda, n, visc, precision, fused=fused)
    b, _ = _stag(cuda, n, visc, precision, coarse=0, fused=fused)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    # one level less, all of it in the kernel; one more level is prepared by
    # five launches (cell and edge viscosities, gamma, alpha, pressure
    # coefficients)
    _, base = _stag(cuda, [m // 2 for m in n], visc, precision, fused=fused)
    assert (na == base + 5) == enters


@pytest.mark.parametrize("n,visc,precision,launches", [
    ([64, 64], -1, "mixed", False), ([48, 64], -1, "mixed", False), ([64, 66], -1, "mixed", True),
    ([56, 56], -1, "fp64", True), ([64, 64], -2, "mixed", True), ([64, 64], 2, "mixed", True),
    ([48, 48], -2, "mixed", False), ([40, 56], 3, "fp64", False),
])
def test_solves(cuda, n, visc, precision, launches):
    """one GMRES iteration with the preconditioner as a graph and without"""
    pb, rhs, b_p, coef = _problem(cuda, n, visc)
    out = []
    for graphs in (1, 0):
        with _solver(n, visc, precision, gmres_max_inner=1, gmres_max_outer=1) as s:
            s.set_graphs(graphs)
            s.set_tune(0)
            x_u, x_p = zeros(pb.nc, 2, cuda), zeros(pb.nc, 1, cuda)[0]
            s.gmres(dev(rhs, cuda), dev(b_p, cuda), x_u, x_p, *coef, 0.7)
            out.append((host(x_u) + [host(x_p)], s.kernel_launches))
    for x, y in zip(out[0][0], out[1][0]):
        assert np.array_equal(x, y)
    assert (out[0][1] > out[1][1]) == launches
