"""The stochastic momentum flux divergence for every number of noise fields it
takes (one and two run unrolled kernels, three and four the general one), on
boxes below and across a thread block, against the oracle at the tolerance of
test_stochastic_m_fluxdiv."""
import numpy as np
import pytest

import lowmachfhd_b200 as L
import oracle as O
from tests import problems as P
from tests.test_gpu_parity import dev, host, zeros

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rngs", [1, 2, 3, 4])
@pytest.mark.parametrize("dim,n", [(2, [3, 5]), (2, [65, 33]), (3, [2, 3, 5]), (3, [33, 9, 4])])
def test_noise_fields(cuda, dim, n, n_rngs):
    nc = P.nc_of(dim, n)
    rng = np.random.default_rng(18)
    eta, T = 1 + rng.random(nc), 1 + rng.random(nc)
    eta_ed, T_ed = O.average_cc_to_edge(dim, n, eta), O.average_cc_to_edge(dim, n, T)
    W_cc, W_ed = P.stochastic_fields(dim, n, seed=19, n_rngs=n_rngs, symmetric=False)
    wts = [0.5, -0.25, 1.5, 0.125][:n_rngs]
    kw = dict(k_B=2.0, variance_coef_mom=1.0, dV=0.125, stoch_stress_form=0, filtering_width=0)
    ref = O.stochastic_m_fluxdiv(dim, n, 0.5, O.StochParams(**kw), eta, eta_ed, T, T_ed, 0.1, wts, W_cc, W_ed)
    with L.StokesSolver(dim, n, 0.5, 1) as s:
        f = zeros(nc, dim, cuda)
        s.stochastic_m_fluxdiv(L.StochParams(**kw), f, False, dev(eta, cuda), dev(eta_ed, cuda), dev(T, cuda),
                               dev(T_ed, cuda), 0.1, wts, dev(W_cc, cuda), dev(W_ed, cuda))
    assert P.rel_inf(host(f), ref) < 1e-13
