"""The two-pass orthogonalisation of GMRES (all products in one pass, the
triangular solve that turns them into modified Gram-Schmidt coefficients, the
update in a second) against the oracle's vector-by-vector modified
Gram-Schmidt: restart lengths below, at and beyond the vectors one launch
takes (6), fields that do not fill a block and ones with a remainder.  The
coefficients agree but for rounding, so the iteration counts are equal and the
solutions agree to the 1e-10 of the other solver tests."""
import numpy as np
import pytest

import lowmachfhd_b200 as L
import oracle as O
from tests import problems as P
from tests.test_gpu_parity import dev, host, zeros

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n", [(2, [8, 6]), (2, [96, 80]), (3, [12, 20, 8])])
@pytest.mark.parametrize("m", [1, 2, 6, 7, 13, 30])
def test_gmres_restart_lengths(cuda, dim, n, m):
    pb = P.problem(dim, n, -1, dx=1.0, seed=51)
    b_u, b_p = P.random_stokes(dim, n, seed=52)
    # one smooth per multigrid level: a weaker preconditioner, so that the
    # long restarts fill
    kw = dict(gmres_rel_tol=1e-9, gmres_max_inner=m, gmres_max_outer=200, gmres_max_iter=400, stag_mg_nsmooths_down=1,
              stag_mg_nsmooths_up=0, stag_mg_nsmooths_bottom=1, mg_nsmooths_down=1, mg_nsmooths_up=0)
    rc, ref_u, ref_p, _, st_ref = O.gmres(pb, O.default_params(**kw), 2.0, b_u, b_p)
    with L.StokesSolver(dim, n, 1.0, -1, params=L.default_params(**kw)) as s:
        x_u, x_p = zeros(pb.nc, dim, cuda), zeros(pb.nc, 1, cuda)[0]
        status, _, st = s.gmres(dev(b_u, cuda), dev(b_p, cuda), x_u, x_p, dev(pb.alpha_fc, cuda), dev(pb.beta, cuda),
                                dev(pb.beta_ed, cuda), dev(pb.gamma, cuda), 2.0)
    assert status == rc
    assert st["total_iters"] == st_ref.total_iters
    assert P.rel_inf(host(x_u), ref_u) < 1e-10
    assert P.rel_inf([host([x_p])[0]], [ref_p]) < 1e-10
