"""The coarsest level's explicit inverse, built in panels of 32 columns, at sizes around its tiles:
a study whose finest level is factored, against a host restatement of the same sums (needs a B200)."""
import numpy as np
import pytest

import solidfem_b200 as sf
from tests.helpers import mg_options, product_model

pytestmark = pytest.mark.gpu


def host_inverse(a):
    """Cholesky, L^-1 and L^-T L^-1, every entry's terms in ascending order."""
    n = len(a)
    low, x = np.tril(a), np.eye(n)
    for k in range(n):
        d = np.sqrt(low[k, k])
        x[k] /= d
        below = low[k + 1:, k] / d
        low[k + 1:, k + 1:] -= np.outer(below, below)
        x[k + 1:] -= np.outer(below, x[k])
    inverse = np.zeros((n, n))
    for k in range(n):
        inverse += np.outer(x[k], x[k])
    return inverse


@pytest.mark.parametrize("div", [(1, 1, 1), (2, 1, 1), (6, 2, 2), (16, 1, 1)])  # n = 54, 108, 900, 864 = 27 x 32
def test_explicit_inverse(div):
    _, model = product_model((10.0, 1.0, 1.0), div, 200000.0, 0.3)
    study = sf.StaticStudy.new(model, mg_options(sf.Precision.DOUBLE, coarse_dofs=3000))
    starts, cols, vals = study.matrix()
    n = len(starts) - 1
    a = np.zeros((n, n))
    a[np.repeat(np.arange(n), np.diff(starts).astype(np.int64)), cols] = vals
    r = np.random.default_rng(n).standard_normal(n)
    inverse = host_inverse(a)
    # The inverses are equal; both products with r round n terms of each row, in their own order.
    bound = 2 * n * np.finfo(float).eps * (np.abs(inverse) @ np.abs(r))
    assert np.all(np.abs(study.precondition(r) - inverse @ r) <= bound)
