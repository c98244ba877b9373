"""fhd_ctx_tune_info of the plans that run whole smooths in one launch: the 2D
tiles of both multigrids and the 3D march.  Every level of either hierarchy is
asked, with fewer staggered than pressure levels too (stag_mg_minwidth above
mg_minwidth), and the shape is the one that the kernels launch: the interior
of a tile of two smooths (56 x 16 cells, 256 threads), or the march's tile."""
import pytest

import lowmachfhd_b200 as L
from tests import problems as P
from tests.test_gpu_parity import dev, zeros

pytestmark = pytest.mark.gpu


def _plans(cuda, dim, n, precision, **kw):
    pb = P.problem(dim, n, 1, dx=1.0, seed=5)
    b_u, b_p = P.random_stokes(dim, n, seed=6)
    with L.StokesSolver(dim, n, 1.0, 1, params=L.default_params(**kw), precision=precision) as s:
        x_u, x_p = zeros(pb.nc, dim, cuda), zeros(pb.nc, 1, cuda)[0]
        s.apply_precon(dev(b_u, cuda), dev(b_p, cuda), x_u, x_p, dev(pb.alpha_fc, cuda), dev(pb.beta, cuda),
                       dev(pb.beta_ed, cuda), dev(pb.gamma, cuda), 1.5)
        out = {}
        for which in ("stag", "cc"):
            out[which] = []
            for level in range(32):
                try:
                    out[which].append(s.tune_info(which, level))
                except L.FhdError:
                    break
    return out


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("kw", [{}, dict(stag_mg_minwidth=128), dict(stag_mg_minwidth=256)])
def test_tiles_report_their_shape(cuda, precision, kw):
    plans = _plans(cuda, 2, [256, 256], precision, **kw)
    if kw:
        assert len(plans["stag"]) < 3 <= len(plans["cc"])
    # pressure levels of 256^2, 128^2 and 64^2 go by launches
    assert [p["kind"] for p in plans["cc"][:4]] == ["tiled"] * 3 + ["rules"]
    assert plans["stag"][0]["kind"] == "tiled"
    for p in plans["stag"] + plans["cc"]:
        if p["kind"] == "tiled":
            assert p["shape"] == [56, 16, 1, 1, 256]


def test_march_reports_its_shape(cuda):
    plans = _plans(cuda, 3, [64, 32, 48], "mixed")
    p = plans["stag"][0]
    assert p["kind"] == "tiled"
    x, y, zruns, per_sm, threads = p["shape"]
    assert 0 < x <= 64 and 0 < y <= 32 and zruns >= 1 and per_sm == 1
    assert threads % 32 == 0 and threads >= x // 2 * y
