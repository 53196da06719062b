"""Raw systems become 3x3 block rows on the device: rows of every length and overlap, unknown counts
that leave the last block row two, one or no padding rows, with and without entries in the padded
diagonal block's columns (needs a B200)."""
import numpy as np
import pytest

import solidfem_b200 as sf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 127, 386, 1000])
@pytest.mark.parametrize("density", [0.0, 0.02, 0.6])
def test_solution_of_any_sparsity(n, density):
    rng = np.random.default_rng(n)
    a = np.where(rng.random((n, n)) < density, rng.standard_normal((n, n)), 0.0)
    a = np.triu(a, 1)
    a = a + a.T
    a[np.arange(n), np.arange(n)] = np.abs(a).sum(1) + rng.uniform(1.0, 2.0, n)  # diagonally dominant by >= 1
    rows, cols = np.nonzero(a)
    starts = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.uint64)
    b = rng.standard_normal(n)
    system = sf.System(starts, cols.astype(np.uint32), a[rows, cols], b,
                       sf.StudyOptions(pcg=sf.PcgOptions(tolerance=1e-12)))
    assert system.solve().kind == sf.Outcome.CONVERGED
    # ||x - x*||_inf <= ||A^-1||_inf ||r||_inf with ||A^-1||_inf <= 1 (dominance) and ||r|| <= 1.01e-12 ||b||,
    # or the rounding floor of the true residual, n eps |A| |x|
    x = system.estimate()
    floor = n * np.finfo(float).eps * np.linalg.norm(np.abs(a) @ np.abs(x))
    assert np.abs(x - np.linalg.solve(a, b)).max() <= 2.0 * max(1.01e-12 * np.linalg.norm(b), floor)
