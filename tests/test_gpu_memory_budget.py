"""What a study holds on the device must not grow: it counts against its memory budget, and against
the server's. The budgets below were the smallest that took these studies before the recovery's
incidence was kept beside them (needs a B200)."""
import numpy as np
import pytest

import solidfem_b200 as sf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device", [None, 0])
@pytest.mark.parametrize("div,precision,budget", [
    ((12, 4, 4), sf.Precision.DOUBLE, 13595628), ((12, 4, 4), sf.Precision.MIXED, 15597244),
    ((20, 8, 8), sf.Precision.DOUBLE, 54484624), ((20, 8, 8), sf.Precision.MIXED, 61790112)])
def test_a_study_fits_the_budget_it_fitted(div, precision, budget, device):
    mesh = sf.box_tet_mesh((0, 0, 0), (10.0, 1.0, 1.0), div, device=device)
    nodes = mesh.nodes()
    model = sf.Model(mesh, sf.Material(200000.0, 0.3))
    model.fix_nodes(np.flatnonzero(np.abs(nodes[:, 0]) < 1e-9))
    model.add_nodal_force(int(np.argmax(nodes[:, 0])), (0.0, 0.0, 1.0))
    study = sf.StaticStudy.new(model, sf.StudyOptions(preconditioner=sf.MultigridOptions(precision=precision),
                                                      device_memory_budget=budget))
    assert study.solve().kind == sf.Outcome.CONVERGED
    assert np.array_equal(study.solution().displacements, study.displacements())
