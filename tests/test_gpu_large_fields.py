"""Fields of several megabytes come to the host in chunks, displacements of 16,384 nodes or more
spread on the device (needs a B200). The part is just over both limits: 18,081 nodes and 48,000
integration points (4.2 MB of point records, two chunks)."""
import numpy as np
import pytest

import solidfem_b200 as sf
from tests.helpers import mg_options, oracle_study, product_model
from tests.test_gpu_recovery import check_recovery_bits

pytestmark = pytest.mark.gpu

SIZE, DIV = (20.0, 10.0, 10.0), (20, 10, 10)


@pytest.fixture(scope="module")
def solved():
    mesh, model = product_model(SIZE, DIV, 200000.0, 0.3)
    study = sf.StaticStudy.new(model, mg_options(sf.Precision.MIXED, coarse_dofs=1500))
    assert study.solve().kind == sf.Outcome.CONVERGED
    return mesh, study


def test_displacements_solve_the_system(solved):
    mesh, study = solved
    d = study.displacements()
    fixed = np.abs(mesh.nodes()[:, 0]) < 1e-9
    assert np.all(d[fixed] == 0.0)
    u, rhs = d[~fixed].ravel(), study.rhs()
    # the converged solve's own test: the true relative residual is within the tolerance
    assert np.linalg.norm(rhs - study.system_multiply(u)) <= 1.01e-9 * np.linalg.norm(rhs)


def test_recovery_is_bit_exact(oracle, solved):
    _, study = solved
    ref = oracle_study(oracle, SIZE, DIV, 200000.0, 0.3, oracle.default_options(coarse_dofs=1500))
    sol = check_recovery_bits(oracle, study, ref)
    assert np.array_equal(sol.displacements, study.displacements())
    assert np.array_equal(sol.point_stresses["tet"], np.repeat(np.arange(12000), 4))
    assert np.array_equal(sol.point_stresses["point"], np.tile(np.arange(4), 12000))


def test_a_new_load_reaches_the_device(solved):
    _, study = solved
    load = np.random.default_rng(5).standard_normal(study.report()["free_dofs"])
    study.resolve(load)
    assert np.array_equal(study.rhs(), load)
    assert study.solve().kind == sf.Outcome.CONVERGED
    u = study.displacements().ravel()
    u = u[np.repeat(~(np.abs(study.mesh.nodes()[:, 0]) < 1e-9), 3)]
    assert np.linalg.norm(load - study.system_multiply(u)) <= 1.01e-9 * np.linalg.norm(load)
