"""Stress fields of parts with vertices of more elements than a warp has lanes (a ring of tets around an
axis, both of whose ends are in every one), and of 31 to 33: the oracle's to the bit (needs a B200)."""
import numpy as np
import pytest

import solidfem_b200 as sf
from tests.helpers import mg_options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device", [None, 0])
@pytest.mark.parametrize("around", [31, 32, 33, 45, 60])
def test_recovery_is_bit_exact(oracle, around, device):
    angle = 2.0 * np.pi * np.arange(around) / around
    rim = np.stack([np.cos(angle), np.sin(angle), np.zeros(around)], 1)
    positions = np.concatenate([[[0.0, 0.0, -0.5], [0.0, 0.0, 0.5]], rim])
    k = np.arange(around)
    tets = np.stack([np.zeros(around, int), 2 + k, 2 + (k + 1) % around, np.ones(around, int)], 1).astype(np.uint32)
    tets = tets[np.random.default_rng(around).permutation(around)]
    mesh = sf.Mesh.from_linear(positions, tets, device=device)
    omesh = oracle.Mesh.linear(positions, tets)
    nodes = mesh.nodes()
    assert np.array_equal(nodes, omesh.nodes())
    held = np.flatnonzero(np.abs(nodes[:, 0] - 1.0) + np.abs(nodes[:, 1]) < 0.8)
    pulled = int(np.argmin(nodes[:, 0]))
    model = sf.Model(mesh, sf.Material(1000.0, 0.3))
    model.fix_nodes(held)
    model.add_nodal_force(pulled, (-1.0, 0.5, 0.25))
    study = sf.StaticStudy.new(model, mg_options(sf.Precision.DOUBLE, coarse_dofs=3000))
    assert study.solve().kind == sf.Outcome.CONVERGED
    ref = oracle.Study(omesh, oracle.uniform(1000.0, 0.3), oracle.default_options(coarse_dofs=3000, precision=oracle.DOUBLE),
                       held, forces=[(pulled, (-1.0, 0.5, 0.25))])
    sol = study.solution()
    stress, von_mises = ref.recover_with(sol.displacements)
    assert np.array_equal(sol.nodal_stress.view(np.uint64), stress.view(np.uint64))
    assert np.array_equal(sol.nodal_von_mises.view(np.uint64), von_mises.view(np.uint64))
