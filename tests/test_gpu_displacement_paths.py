"""Displacements of under 2,048 nodes are spread on the host, of more on the device: the same bits as
the recovery's own copy on both sides of the line, prescribed values included (needs a B200)."""
import numpy as np
import pytest

import solidfem_b200 as sf
from tests.helpers import mg_options, product_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("div", [(1, 1, 1), (12, 4, 4), (13, 4, 4), (20, 6, 6)])  # 27, 2,025, 2,187 and 6,929 nodes
def test_displacements_are_the_recoverys(div):
    mesh, model = product_model((10.0, 1.0, 1.0), div, 200000.0, 0.3)
    tip = int(np.argmax(mesh.nodes() @ [1.0, 0.1, 0.01]))
    model.prescribe_displacement(tip, 2, 1e-3)
    study = sf.StaticStudy.new(model, mg_options(sf.Precision.MIXED))
    assert study.solve().kind == sf.Outcome.CONVERGED
    d = study.displacements()
    assert d[tip, 2] == 1e-3
    assert np.all(d[np.abs(mesh.nodes()[:, 0]) < 1e-9] == 0.0)
    assert np.array_equal(d.view(np.uint64), study.solution().displacements.view(np.uint64))
