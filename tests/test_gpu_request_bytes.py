"""The bytes the server reserves for a request against what a context that runs
the same step allocates (fhd_ctx_device_bytes) plus the request's state and
noise: never less, and more by no more than the fixed reserve, the autotuner's
scratch (3 dim arrays of the finest level) and four multigrid words per cell (the
estimate's coarser levels, which an odd extent does not have: 26 arrays of 1/7 of
the cells in 3D)."""
import math

import pytest
import torch

import lowmachfhd_b200 as L
from tests.test_gpu_parity import zeros

pytestmark = pytest.mark.gpu

CASES = [(3, [64, 48, 64], 1, 1, "mixed", {}), (3, [64, 48, 32], 3, 1, "mixed", {}), (3, [32, 40, 48], 2, 1, "fp64", {}),
         (2, [256, 192], 1, 1, "mixed", {}), (2, [128, 256], 2, -1, "fp64", {}), (3, [33, 48, 31], 1, 1, "mixed", {}),
         (3, [48, 48, 48], 1, -2, "mixed", dict(gmres_max_inner=9)), (3, [32, 32, 32], 1, 1, "fp64",
                                                                     dict(visc_schur_approx=1, stag_mg_smoother=0,
                                                                          stag_mg_omega=0.6))]


@pytest.mark.parametrize("dim,n,ns,visc,precision,kw", CASES)
def test_reserved_bytes_cover_a_request(cuda, dim, n, ns, visc, precision, kw):
    nc, nE = math.prod(n), 1 if dim == 2 else 3
    params = L.default_params(gmres_max_iter=1, **kw)
    prec = L.FHD_PREC_MIXED if precision == "mixed" else L.FHD_PREC_FP64
    mp = L.mixture_params([1.0, 2.0, 3.0][:ns], [0.01] * (ns * (ns - 1) // 2), rhobar=[1.0] * ns) if ns > 1 else None
    one = torch.ones(nc, dtype=torch.float64, device=cuda)
    u, rho, pi = zeros(nc, dim, cuda), [one / ns for _ in range(ns)], zeros(nc, 1, cuda)[0]
    W = lambda k: zeros(nc, k, cuda)
    sp = L.StochParams(k_B=1e-4, variance_coef_mom=1.0, dV=1.0, stoch_stress_form=1, filtering_width=0)
    with L.StokesSolver(dim, n, 1.0, visc, params=params, precision=precision) as s:
        s.advance_timestep_overdamped(sp, mp, 0.1, u, rho, pi, one, [one] * nE, zeros(nc, 1, cuda)[0], one, [one] * nE,
                                      W(2 * dim), W(4 * nE), W(2 * dim * ns) if ns > 1 else None)
        held = s.device_bytes
    held += 8 * nc * (dim + 2 * ns + 4 + 2 * nE)  # velocity, densities and fluxes, pi, eta, kappa, T, edges
    held += 8 * nc * (2 * dim + 2 * nE + (2 * dim * ns if ns > 1 else 0))
    kwr = dict(mix=mp) if ns > 1 else {}
    est = L.Server.request_bytes(L.make_request(dim=dim, n_cells=n, nspecies=ns, visc_type=visc, precision=prec,
                                                params=params, **kwr))
    over = est - (64 << 20) - held
    word = 4 if precision == "mixed" else 8
    scratch = 3 * dim * word * nc
    # (the scalar arrays of a context, below 1 MiB, lie in the fixed reserve)
    assert scratch - (1 << 20) <= over <= scratch + 4 * word * nc
