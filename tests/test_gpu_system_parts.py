"""A raw system of more scalar entries than cross to the device at once (4,194,304): its block rows are
made in parts (needs a B200)."""
import numpy as np
import pytest

import solidfem_b200 as sf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [300001, 600000])  # 5.1 and 10.2 million entries: two and three parts
def test_solution(n):
    rng = np.random.default_rng(n)
    i, j, v = [], [], []
    for k in (1, 2, 4, 7, 50, 301, 1000, n - 2):
        a = np.arange(n - k)
        w = rng.standard_normal(n - k)
        i += [a, a + k]
        j += [a + k, a]
        v += [w, w]
    weight = np.zeros(n)
    for a, w in zip(i, v):
        np.add.at(weight, a, np.abs(w))
    i, j = np.concatenate([np.arange(n)] + i), np.concatenate([np.arange(n)] + j)
    v = np.concatenate([weight + rng.uniform(1.0, 2.0, n)] + v)  # dominant by 1 or more
    order = np.lexsort((j, i))
    i, j, v = i[order], j[order], v[order]
    assert len(v) > 4194304
    starts = np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n))]).astype(np.uint64)
    b = rng.standard_normal(n)
    system = sf.System(starts, j.astype(np.uint32), v, b, sf.StudyOptions(pcg=sf.PcgOptions(tolerance=1e-10)))
    assert system.solve().kind == sf.Outcome.CONVERGED
    residual = b - np.bincount(i, weights=v * system.estimate()[j], minlength=n)
    # the converged solve's own test: the true relative residual is within the tolerance
    assert np.linalg.norm(residual) <= 1.01e-10 * np.linalg.norm(b)
