"""A vector's energy has the same bits alone and with others in one call, on SELL and row-group systems:
one, several and more than all of the blocks whose partial sums order it (needs a B200)."""
import numpy as np
import pytest

import solidfem_b200 as sf
from tests.helpers import mg_options, product_model
from tests.test_zz_no_alloc import energy_products

pytestmark = pytest.mark.gpu


def check(study, counts):
    xs = np.random.default_rng(1).standard_normal((8, study.report()["free_dofs"]))
    alone = [energy_products(study, xs[k:k + 1]) for k in range(8)]
    for count in counts:
        ys, es = energy_products(study, xs[:count])
        for k in range(count):
            assert np.array_equal(ys[k].view(np.uint64), alone[k][0][0].view(np.uint64)), (count, k)
            assert es[k].view(np.uint64) == alone[k][1][0].view(np.uint64), (count, k)


@pytest.mark.parametrize("sell", [1, 0])
@pytest.mark.parametrize("div", [(1, 1, 1), (12, 3, 3), (30, 7, 6), (45, 8, 8)])
def test_every_count(div, sell):
    _, model = product_model((10.0, 1.0, 1.0), div, 200000.0, 0.3)
    check(sf.StaticStudy.new(model, mg_options(sf.Precision.DOUBLE, sell_min_rows=sell)), range(1, 9))


def test_warps_of_several_slices():
    _, model = product_model((100.0, 100.0, 0.8), (120, 120, 2), 2000.0, 0.35)
    study = sf.StaticStudy.new(model)
    assert study.report()["free_dofs"] // 3 > 1024 * 8 * 32  # more slices than warps of the most blocks
    check(study, (2, 3, 4, 6, 8))
