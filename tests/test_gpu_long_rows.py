"""Raw systems with a few long rows among short ones: block rows merged 32 scalar entries of a row at
a time, and the product's lanes chosen by the longest row (needs a B200)."""
import numpy as np
import pytest

import solidfem_b200 as sf

pytestmark = pytest.mark.gpu


def chain_with_long_rows(n, long, width, rng):
    """A chain whose `long` rows (and columns) couple to the chain in `width` places, as dense triples
    and dominant by 1 or more."""
    rows, cols = [np.arange(n - 1)], [np.arange(1, n)]
    for r in long:
        other = rng.choice(np.delete(np.arange(n), r), min(width, n - 1), replace=False)
        rows.append(np.minimum(r, other))
        cols.append(np.maximum(r, other))
    pairs = np.unique(np.concatenate(rows).astype(np.int64) * n + np.concatenate(cols))
    i, j = pairs // n, pairs % n
    v = rng.standard_normal(len(i))
    weight = np.zeros(n)
    np.add.at(weight, i, np.abs(v))
    np.add.at(weight, j, np.abs(v))
    d = np.arange(n)
    i, j = np.concatenate([d, i, j]), np.concatenate([d, j, i])
    v = np.concatenate([weight + rng.uniform(1.0, 2.0, n), v, v])
    order = np.lexsort((j, i))
    starts = np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n))]).astype(np.uint64)
    return i[order], j[order], v[order], starts


@pytest.mark.parametrize("n,long,width", [
    (100, [50], 99), (101, [100], 100), (102, [0, 101], 101),           # full rows, with 2, 1 and no padding rows
    (386, [7], 29), (386, [7], 30), (386, [7, 8], 31), (386, [6, 8], 62), (386, [6, 7, 8], 64),  # around 32 and 64
    (3000, [1500], 1000),                                                # more than 256 blocks among 1,000 rows
    (30000, [3, 29999], 1000),                                           # among 10,000
    (30000, [11], 29999),                                                # too long a row to stage
])
def test_solution(n, long, width):
    rng = np.random.default_rng(n + width)
    i, j, v, starts = chain_with_long_rows(n, long, width, rng)
    b = rng.standard_normal(n)
    system = sf.System(starts, j.astype(np.uint32), v, b, sf.StudyOptions(pcg=sf.PcgOptions(tolerance=1e-12)))
    assert system.solve().kind == sf.Outcome.CONVERGED
    x = system.estimate()
    # the converged solve's own test: the true residual is within the tolerance, or at the product's
    # rounding floor, (longest row) eps |A| |x|
    absolute = np.zeros(n)
    np.add.at(absolute, i, np.abs(v * x[j]))
    residual = b.copy()
    np.subtract.at(residual, i, v * x[j])
    floor = (width + 3) * np.finfo(float).eps * np.linalg.norm(absolute)
    assert np.linalg.norm(residual) <= 1.01e-12 * np.linalg.norm(b) + 2.0 * floor
