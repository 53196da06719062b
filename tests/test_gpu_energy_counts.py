"""sf_study_energy_products over every vector count on SELL and row-group systems, whose kernels are
chosen by the count: one vector, up to four in one walk, five to eight in two (needs a B200)."""
import numpy as np
import pytest

import solidfem_b200 as sf
from tests.helpers import mg_options, product_model
from tests.test_zz_no_alloc import check_against_system_multiply, energy_products

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", range(1, 9))
@pytest.mark.parametrize("sell", [1, 0])
@pytest.mark.parametrize("div", [(1, 1, 1), (12, 3, 3), (30, 7, 6)])  # under one slice or block; ragged last ones
def test_every_count(div, sell, count):
    _, model = product_model((10.0, 1.0, 1.0), div, 200000.0, 0.3)
    study = sf.StaticStudy.new(model, mg_options(sf.Precision.DOUBLE, sell_min_rows=sell))
    xs = np.random.default_rng(count).standard_normal((count, study.report()["free_dofs"]))
    check_against_system_multiply(study, xs, *energy_products(study, xs))


def test_more_slices_than_partial_slots():
    """Two slices a block in two groups: past 4096 blocks each block walks several pairs."""
    _, model = product_model((100.0, 100.0, 0.8), (120, 120, 2), 2000.0, 0.35)
    study = sf.StaticStudy.new(model)
    assert study.report()["free_dofs"] // 3 > 4096 * 64
    xs = np.random.default_rng(3).standard_normal((7, study.report()["free_dofs"]))
    check_against_system_multiply(study, xs, *energy_products(study, xs))
