"""Branches of the single-block coarse kernels that ordinary hierarchies do not
reach, against the per-level launches (fhd_ctx_set_coarse 0): equal bit for bit
in FP64, at test_coarse_kernel_mixed's tolerance in FP32.

Pressure coefficients that do not fit beside the unknowns (read from global
memory by every sweep) belong to a bottom level only, which enters the kernel
whatever its cells: extents that mg_minwidth or an odd number leaves
uncoarsened.  Rows of more x-pairs than the block has threads need an extent
above 1024 in a level of few cells."""
import numpy as np
import pytest
import torch

import lowmachfhd_b200 as L
from tests import problems as P
from tests.test_gpu_coarse import _run
from tests.test_gpu_parity import dev, host, zeros
from tests.test_gpu_walls import NS, PE, SL, periodic_afterwards, solver, wall_rhs  # noqa: F401

pytestmark = pytest.mark.gpu

CAP = 200 * 1024  # unknowns, right-hand sides and scratch of one kernel


def _equal(a, b, precision):
    for x, y in zip(a, b):
        if precision == "fp64":
            assert np.array_equal(x, y)
        else:
            assert P.rel_inf([x], [y]) < 1e-5


# one staggered and one pressure level each: even and odd, 2D and 3D
@pytest.mark.parametrize("dim,n,minwidth,precision", [
    (3, [24, 16, 20], 16, "fp64"), (3, [24, 24, 24], 16, "mixed"), (3, [19, 21, 19], 2, "fp64"),
    (2, [90, 94], 64, "fp64"), (2, [91, 93], 2, "fp64"),
])
def test_pressure_coefficients_in_global_memory(cuda, dim, n, minwidth, precision):
    nc, w = int(np.prod(n)), 8 if precision == "fp64" else 4
    even = all(m % 2 == 0 for m in n)
    optin = torch.cuda.get_device_properties(cuda).shared_memory_per_block_optin
    assert 3 * nc * w <= CAP and ((2 if even else 3) + dim) * nc * w > optin
    # the staggered level does not fit: only the pressure level's launches
    # become one
    assert 3 * dim * nc * w > CAP
    kw = dict(mg_minwidth=minwidth, stag_mg_minwidth=minwidth)
    phi1, x1, n1 = _run(cuda, dim, n, 1, kw, 1, precision)
    phi0, x0, n0 = _run(cuda, dim, n, 1, kw, 0, precision)
    _equal(phi1 + x1, phi0 + x0, precision)
    assert n1 < n0


@pytest.mark.parametrize("dim,n,precision", [(2, [1100, 2], "fp64"), (2, [1100, 2], "mixed"),
                                             (3, [1030, 2, 2], "mixed")])
def test_rows_longer_than_the_block(cuda, dim, n, precision):
    assert n[0] // 2 > 512 and 3 * dim * np.prod(n) * (8 if precision == "fp64" else 4) <= CAP
    phi1, x1, n1 = _run(cuda, dim, n, 1, {}, 1, precision)
    phi0, x0, n0 = _run(cuda, dim, n, 1, {}, 0, precision)
    _equal(phi1 + x1, phi0 + x0, precision)
    assert n1 + 2 < n0  # both multigrids


@pytest.mark.parametrize("bc_lo,bc_hi", [([PE, NS, PE], [PE, SL, PE]), ([NS, PE, PE], [SL, PE, PE])])
def test_rows_longer_than_the_block_between_walls(cuda, bc_lo, bc_hi):
    dim, n = 2, [1100, 2]
    pb = P.problem(dim, n, 1, dx=1.0, seed=72)
    alpha = [1.0 + 0.2 * np.random.default_rng(71).random(pb.nc) for _ in range(dim)]
    b_u, b_p = wall_rhs(dim, n, bc_lo, 73, 1.5)
    out = []
    for coarse in (1, 0):
        with solver(dim, n, bc_lo, bc_hi) as s:
            s.set_coarse(coarse)
            x_u, x_p = zeros(pb.nc, dim, cuda), zeros(pb.nc, 1, cuda)[0]
            s.apply_precon(dev(b_u, cuda), dev(b_p, cuda), x_u, x_p, dev(alpha, cuda), dev(pb.beta, cuda),
                           dev(pb.beta_ed, cuda), dev(pb.gamma, cuda), 1.5)
            out.append((host(x_u) + [host(x_p)], s.kernel_launches))
    _equal(out[0][0], out[1][0], "fp64")
    assert out[0][1] < out[1][1]
