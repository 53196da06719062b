"""The power iteration's norm, a serial sum done in parallel in chunks of 256 terms and 32 chunks at
a time, at sizes around both: lambda_max must equal the oracle's to the bit (needs a B200)."""
import pytest

import solidfem_b200 as sf
from tests.helpers import mg_options, oracle_study, product_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("div", [(1, 1, 1), (16, 1, 1), (13, 4, 4), (14, 4, 4), (24, 6, 5)])  # 54 ... 20,592 unknowns
def test_largest_eigenvalue_is_bit_exact(oracle, div):
    size, E, nu = (10.0, 1.0, 1.0), 70000.0, 0.33
    _, model = product_model(size, div, E, nu)
    study = sf.StaticStudy.new(model, mg_options(sf.Precision.DOUBLE, coarse_dofs=1000))
    ref = oracle_study(oracle, size, div, E, nu, oracle.default_options(coarse_dofs=1000, precision=oracle.DOUBLE))
    assert [lv["lambda_max"] for lv in study.levels()] == [lv["lambda_max"] for lv in ref.levels()]
