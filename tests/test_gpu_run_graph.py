"""A small solver replays four iterations as one graph once that pays; stepping one iteration at a
time never does. Both must give the same bits, iteration counts and ends, past convergence and past
an iteration cap that is no multiple of four (needs a B200)."""
import numpy as np
import pytest

import solidfem_b200 as sf
from tests.helpers import mg_options, product_model

pytestmark = pytest.mark.gpu


def end_of(advance):
    try:
        outcome = advance()
        return outcome.kind, outcome.progress.iteration, outcome.progress.relative_residual
    except sf.SolidfemError as e:
        return e.status


def by_ones(solver):
    while (outcome := solver.step(1)).kind == sf.Outcome.RUNNING:
        pass
    return outcome


def resident(div, precision, cap):
    _, model = product_model((10.0, 1.0, 1.0), div, 200000.0, 0.3)
    options = mg_options(precision, coarse_dofs=1500)
    options.pcg.max_iterations = cap
    return sf.StaticStudy.new(model, options)


@pytest.mark.parametrize("cap", [None, 17])
@pytest.mark.parametrize("precision", [sf.Precision.MIXED, sf.Precision.DOUBLE])
@pytest.mark.parametrize("div", [(12, 3, 3), (60, 9, 9)])  # the second near the most unknowns of such a solver
def test_studies(div, precision, cap):
    whole, single = resident(div, precision, cap), resident(div, precision, cap)
    n = whole.report()["free_dofs"]
    rng = np.random.default_rng(n)
    warm = rng.standard_normal(n)
    ran = 0
    while ran < 16 * whole.device_timing()["launches_per_iteration"]:  # what the longer graph is made after
        whole.resolve(warm)
        end_of(whole.solve)
        ran += whole.progress().iteration
    load = rng.standard_normal(n)
    for solver in (whole, single):
        solver.resolve(load)
    assert end_of(whole.solve) == end_of(lambda: by_ones(single))
    assert np.array_equal(whole.displacements().view(np.uint64), single.displacements().view(np.uint64))


@pytest.mark.parametrize("cap", [None, 101])
@pytest.mark.parametrize("n", [300, 4001])
def test_raw_systems(n, cap):
    i = np.arange(n)
    rows = np.concatenate([i, i[1:], i[:-1]])
    cols = np.concatenate([i, i[:-1], i[1:]])
    vals = np.concatenate([np.full(n, 2.0 + 1e-3), np.full(2 * n - 2, -1.0)])
    order = np.lexsort((cols, rows))
    starts = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.uint64)
    b = np.random.default_rng(n).standard_normal(n)

    def system():
        return sf.System(starts, cols[order].astype(np.uint32), vals[order], b,
                         sf.StudyOptions(pcg=sf.PcgOptions(tolerance=1e-12, max_iterations=cap)))

    whole, single = system(), system()
    ends = end_of(whole.solve), end_of(lambda: by_ones(single))
    assert ends[0] == ends[1]
    assert np.array_equal(whole.estimate().view(np.uint64), single.estimate().view(np.uint64))
