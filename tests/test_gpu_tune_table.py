"""What one context puts into the process-wide plan table must serve every
context of the same level shapes.  A first context meets a shape with the tuner
on under conditions of its own -- colour launches asked for
(fhd_ctx_set_fused 0), or level-0 arrays left by the call before that are not
aligned to pairs -- and a default context of that shape then smooths as the
fixed rules do where the tiles or the march apply: one launch per smooths, so
as many launches as with the tuner off.  The shapes are tuned by no other
test."""
import numpy as np
import pytest
import torch

import lowmachfhd_b200 as L
from tests import problems as P
from tests.test_gpu_parity import dev, host, zeros

pytestmark = pytest.mark.gpu


def _offset(arrs, cuda):
    """device copies that begin 8 bytes past a 16-byte boundary"""
    out = []
    for a in arrs:
        t = torch.empty(a.size + 1, dtype=torch.float64, device=cuda)
        t[1:].copy_(torch.from_numpy(np.ascontiguousarray(a)))
        out.append(t[1:])
    return out


def _solver(n, precision):
    return L.StokesSolver(len(n), n, 1.0, 1, params=L.default_params(), precision=precision)


def _data(cuda, n):
    dim = len(n)
    pb = P.problem(dim, n, 1, dx=1.0, seed=31)
    rhs, b_p = P.random_stokes(dim, n, seed=32)
    coef = (dev(pb.alpha_fc, cuda), dev(pb.beta, cuda), dev(pb.beta_ed, cuda), dev(pb.gamma, cuda))
    return dim, pb, rhs, b_p, coef


def _precon(s, cuda, dim, pb, rhs, b_p, coef):
    x_u, x_p = zeros(pb.nc, dim, cuda), zeros(pb.nc, 1, cuda)[0]
    l0 = s.kernel_launches
    s.apply_precon(dev(rhs, cuda), dev(b_p, cuda), x_u, x_p, *coef, 1.5)
    return host(x_u) + [host(x_p)], s.kernel_launches - l0


def _after(cuda, precision, D, n):
    """a default context and one with the tuner off: results and launches (3D:
    of the staggered multigrid; 3D pressure levels have no tiles and keep the
    plan that was timed)"""
    dim, pb, rhs, b_p, coef = D
    out = []
    for tune in (-1, 0):
        with _solver(n, precision) as s:
            s.set_tune(tune)
            phi = zeros(pb.nc, dim, cuda)
            s.stag_mg_solver(*coef, 1.5, phi, dev(rhs, cuda))
            na = s.kernel_launches
            x, nb = _precon(s, cuda, *D)
            out.append((host(phi) + x, (na, nb) if dim == 2 else na))
    assert out[0][1] == out[1][1]
    for x, y in zip(out[0][0], out[1][0]):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("precision,n", [("mixed", [136, 168]), ("fp64", [152, 88]), ("fp64", [56, 40, 72])])
def test_colour_launches_do_not_decide_for_others(cuda, precision, n):
    D = _data(cuda, n)
    with _solver(n, precision) as s:
        s.set_fused(0)
        s.set_tune(1)
        _precon(s, cuda, *D)
    _after(cuda, precision, D, n)


@pytest.mark.parametrize("n", [[104, 184], [44, 36, 52]])
def test_unaligned_arrays_do_not_decide_for_others(cuda, n):
    D = _data(cuda, n)
    dim, pb, rhs, b_p, coef = D
    with _solver(n, "fp64") as s:
        s.set_tune(0)
        # the multigrid's level 0 keeps these arrays until the next call
        s.stag_mg_solver(*coef, 1.5, _offset([np.zeros(pb.nc)] * dim, cuda), _offset(rhs, cuda))
        s.set_tune(1)
        _precon(s, cuda, *D)
    _after(cuda, "fp64", D, n)
