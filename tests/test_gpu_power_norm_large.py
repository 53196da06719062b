"""The power iteration's norm with more chunks than threads in the block that scans them (needs a
B200): lambda_max must equal the oracle's to the bit."""
import pytest

import solidfem_b200 as sf
from tests.helpers import mg_options, oracle_study, product_model

pytestmark = pytest.mark.gpu


def test_largest_eigenvalue_is_bit_exact(oracle):
    size, div, E, nu = (10.0, 2.0, 2.0), (36, 10, 10), 70000.0, 0.33  # 95,256 unknowns, 373 chunks
    _, model = product_model(size, div, E, nu)
    study = sf.StaticStudy.new(model, mg_options(sf.Precision.DOUBLE, coarse_dofs=1000))
    ref = oracle_study(oracle, size, div, E, nu, oracle.default_options(coarse_dofs=1000, precision=oracle.DOUBLE))
    assert [lv["lambda_max"] for lv in study.levels()] == [lv["lambda_max"] for lv in ref.levels()]
