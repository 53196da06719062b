"""Point records of a finished recovery cross in chunks put together in buffers of their own or, from
524,288 points on (and when those are not to be had), in memory that the patch fits have done with, so
the results can be read again (needs a B200)."""
import numpy as np
import pytest

import solidfem_b200 as sf
from tests.helpers import mg_options, product_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quadrature", [sf.Quadrature.FOUR_POINT, sf.Quadrature.FOURTEEN_POINT])
@pytest.mark.parametrize("div", [(1, 1, 1), (12, 3, 3), (30, 16, 13)])  # the last: 149,760 and 524,160 points
def test_results_read_twice(div, quadrature):
    _, model = product_model((10.0, 1.0, 1.0), div, 200000.0, 0.3)
    model.set_quadrature(quadrature)
    check(sf.StaticStudy.new(model, mg_options(sf.Precision.MIXED, coarse_dofs=1500)))


def test_results_read_twice_from_many_points():
    _, model = product_model((10.0, 1.0, 1.0), (30, 16, 14), 200000.0, 0.3)  # 564,480 points
    model.set_quadrature(sf.Quadrature.FOURTEEN_POINT)
    check(sf.StaticStudy.new(model, mg_options(sf.Precision.MIXED, coarse_dofs=1500)))


def check(study):
    assert study.solve().kind == sf.Outcome.CONVERGED
    first, again = study.solution(), study.solution()
    for name in ("displacements", "nodal_stress", "nodal_von_mises"):
        assert np.array_equal(getattr(first, name).view(np.uint64), getattr(again, name).view(np.uint64))
    records = first.point_stresses
    assert np.array_equal(records.view(np.uint8), again.point_stresses.view(np.uint8))
    n, points = len(records), len(records) // study.mesh.tet_count()
    assert np.array_equal(records["tet"], np.arange(n) // points)
    assert np.array_equal(records["point"], np.arange(n) % points)
    # each record's own parts belong together: von Mises from its stress (element.rs:186-189)
    s = records["stress"]
    a, b, c = s[:, 0] - s[:, 1], s[:, 1] - s[:, 2], s[:, 2] - s[:, 0]
    vm = np.sqrt(0.5 * (a * a + b * b + c * c) + 3.0 * (s[:, 3] ** 2 + s[:, 4] ** 2 + s[:, 5] ** 2))
    assert np.allclose(records["von_mises"], vm, rtol=1e-14)
