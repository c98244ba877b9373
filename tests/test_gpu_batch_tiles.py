"""The batched solver's tile smoothers on boxes whose packed fields begin at
odd offsets (an odd box before them: pairs are loaded as scalars), extents
below and across a tile, and smooth counts that end in either buffer, against
single-box solves (which the oracle tests cover) at the tolerance of
test_gpu_batch: the same iterations, solutions within 1e-10."""
import pytest

from tests import problems as P
from tests.test_gpu_batch import batched, rhs, single

pytestmark = pytest.mark.gpu

SIZES = [(15, 21), (128, 96), (4, 1600), (35, 9), (200, 72), (144, 144)]
ETAS = [1.0, 2.5, 0.7, 3.0, 1.2, 4.0]


@pytest.mark.parametrize("down,up", [(2, 2), (1, 2), (3, 1), (1, 1), (2, 3), (4, 4)])
def test_batched_tiles_equal_single_box(cuda, down, up):
    params = dict(gmres_rel_tol=1e-9, stag_mg_nsmooths_down=down, stag_mg_nsmooths_up=up, mg_nsmooths_down=down,
                  mg_nsmooths_up=up)
    bs = rhs(SIZES, 70)
    _, xs, stats, _ = batched(cuda, SIZES, ETAS, bs, "fp64", 2.0, params)
    for k, (nx, ny) in enumerate(SIZES):
        st1, x1, s1 = single(cuda, nx, ny, ETAS[k], bs[k], "fp64", 2.0, params)
        assert stats[k]["total_iters"] == s1["total_iters"], k
        assert stats[k]["status"] == st1
        assert P.rel_inf(xs[k][:2], x1[:2]) < 1e-10, k
        assert P.rel_inf(xs[k][2:], x1[2:]) < 1e-10, k
