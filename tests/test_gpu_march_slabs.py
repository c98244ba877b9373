"""Thin slabs of many cells, on which the z-march works on several times the
cells that it stores: the fixed rules leave the most extreme to the colour
launches, and the autotuner times the march against the other plans and keeps
the faster.  Whatever runs equals the colour launches bit for bit."""
import numpy as np
import pytest

import lowmachfhd_b200 as L
from tests import problems as P
from tests.test_gpu_parity import dev, host, zeros

pytestmark = pytest.mark.gpu


def _run(cuda, n, precision, tune, fused=-1):
    pb = P.problem(3, n, 1, dx=1.0, seed=91)
    rhs, _ = P.random_stokes(3, n, seed=92)
    with L.StokesSolver(3, n, 1.0, 1, params=L.default_params(), precision=precision) as s:
        s.set_tune(tune)
        s.set_fused(fused)
        phi = zeros(pb.nc, 3, cuda)
        s.stag_mg_solver(dev(pb.alpha_fc, cuda), dev(pb.beta, cuda), dev(pb.beta_ed, cuda), dev(pb.gamma, cuda), 0.7,
                         phi, dev(rhs, cuda))
        return host(phi), s.kernel_launches, s.tune_info("stag", 0)


# pairs worked on for each stored: 5.1 (rules: colours; timed), 4.4 (FP32 4.0),
# 3.1 (rules: march; not timed)
@pytest.mark.parametrize("n,precision,colours", [([1024, 128, 6], "fp64", True), ([512, 256, 6], "fp64", True),
                                                 ([512, 192, 12], "fp64", False), ([512, 256, 10], "mixed", False)])
def test_slabs(cuda, n, precision, colours):
    ref, n0, _ = _run(cuda, n, precision, 0, fused=0)
    a, na, _ = _run(cuda, n, precision, 0)
    b, _, info = _run(cuda, n, precision, 1)
    assert (na == n0) == colours
    assert info["pair_us"] > 0 and info["kind"] in ("tiled", "colour")
    for x, y, z in zip(ref, a, b):
        assert np.array_equal(x, y) and np.array_equal(x, z)
