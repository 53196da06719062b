"""Coarse matrices of levels with few blocks (six threads a block) and with many (one): both the
oracle's to the bit (needs a B200)."""
import numpy as np
import pytest

import solidfem_b200 as sf
from tests.helpers import mg_options, oracle_study, product_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,div,many", [((10.0, 2.0, 2.0), (20, 6, 6), False),
                                           ((100.0, 100.0, 0.8), (30, 30, 2), True)])
def test_coarse_matrices_are_bit_exact(oracle, size, div, many):
    _, model = product_model(size, div, 70000.0, 0.33)
    study = sf.StaticStudy.new(model, mg_options(sf.Precision.DOUBLE, coarse_dofs=1000))
    ref = oracle_study(oracle, size, div, 70000.0, 0.33, oracle.default_options(coarse_dofs=1000, precision=oracle.DOUBLE))
    mine, theirs = study.levels(), ref.levels()
    assert len(mine) == len(theirs) >= 2
    assert (len(theirs[1]["columns"]) > 32768) == many
    for a, b in zip(mine, theirs):
        for name in ("starts", "columns"):
            assert np.array_equal(a[name], b[name]), name
        assert np.array_equal(a["values"].view(np.uint64), b["values"].view(np.uint64))
