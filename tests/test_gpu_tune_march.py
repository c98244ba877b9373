"""The z-march and the 2D tiles through the plan path: forced by the index one
past a level's candidate list (fhd_ctx_set_tune 2 + ncand) and taken from an
imported table line with that index.  Equal bit for bit to the colour launches
(forced index 0) in both precisions.  An imported plan of the finest level
leaves the launches of the fixed rules; the forced index takes the first
candidate, colour launches, on coarser levels with shorter lists."""
import numpy as np
import pytest
import torch

import lowmachfhd_b200 as L
from tests import problems as P
from tests.test_gpu_parity import dev, host, zeros

pytestmark = pytest.mark.gpu


def _run(cuda, n, precision, tune):
    dim = len(n)
    pb = P.problem(dim, n, 1, dx=1.0, seed=81)
    rhs, b_p = P.random_stokes(dim, n, seed=82)
    with L.StokesSolver(dim, n, 1.0, 1, params=L.default_params(), precision=precision) as s:
        s.set_tune(tune)
        coef = (dev(pb.alpha_fc, cuda), dev(pb.beta, cuda), dev(pb.beta_ed, cuda), dev(pb.gamma, cuda))
        phi = zeros(pb.nc, dim, cuda)
        s.stag_mg_solver(*coef, 0.7, phi, dev(rhs, cuda))
        ns = s.kernel_launches
        x_u, x_p = zeros(pb.nc, dim, cuda), zeros(pb.nc, 1, cuda)[0]
        s.apply_precon(dev(rhs, cuda), dev(b_p, cuda), x_u, x_p, *coef, 1.5)
        which = ["stag"] if dim == 3 else ["stag", "cc"]  # (3D pressure levels have no tiles)
        return host(phi) + host(x_u) + [host(x_p)], ns, [s.tune_info(w, 0) for w in which]


def _check(cuda, n, precision, out, launches, info, cands, forced):
    ref, nr, _ = _run(cuda, n, precision, 0)
    col, nc, _ = _run(cuda, n, precision, 2)  # colour launches, the first candidate, on every level
    assert launches < nc
    assert launches == nr or forced
    for x, y, z in zip(out, ref, col):
        assert np.array_equal(x, z) and np.array_equal(y, z)
    for i, c in zip(info, cands):
        assert i["kind"] == "tiled" and i["candidates"] == c and i["pair_us"] == 0
        assert i["shape"][4] > 0


CASES = [([64, 32, 40], "mixed"), ([64, 32, 40], "fp64"), ([112, 120], "mixed"), ([112, 120], "fp64")]


@pytest.mark.parametrize("n,precision", CASES)
def test_forced_index_past_the_list(cuda, n, precision):
    dim = len(n)
    cands = [len(L.tune_candidates(w, dim, n, precision, 1)) for w in ("stag", "cc")[: 4 - dim]]
    assert len(set(cands)) == 1
    out, launches, info = _run(cuda, n, precision, 2 + cands[0])
    _check(cuda, n, precision, out, launches, info, cands, True)


@pytest.mark.parametrize("n,precision", [([72, 24, 40], "mixed"), ([120, 136], "fp64")])  # tuned by no other test
def test_imported_index_past_the_list(cuda, n, precision):
    dim = len(n)
    pr = torch.cuda.get_device_properties(cuda)
    cands, lines = [], []
    for w in ("stag", "cc")[: 4 - dim]:
        cands.append(len(L.tune_candidates(w, dim, n, precision, 1)))
        key = L.tune_key(w, dim, n, precision, 1, sms=pr.multi_processor_count,
                         smem_optin=pr.shared_memory_per_block_optin,
                         smem_sm=pr.shared_memory_per_multiprocessor, device=cuda.index or 0)
        lines.append(f"{key} {cands[-1]}\n")
    assert L.tune_import("".join(lines)) == len(lines)
    out, launches, info = _run(cuda, n, precision, -1)
    _check(cuda, n, precision, out, launches, info, cands, False)
