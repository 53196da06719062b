"""Bodies of meshes generated on the device, found by a union-find over shared faces: a study must
refuse and accept what it does with the host's mesh (needs a B200)."""
import numpy as np
import pytest

import solidfem_b200 as sf

pytestmark = pytest.mark.gpu


def boxes(offsets, div):
    """Linear boxes side by side, each with vertices of its own."""
    box = sf.box_tet_mesh((0, 0, 0), (1.0, 1.0, 1.0), div)
    nodes, tets = box.nodes()[:box.vertex_count()], box.tets()[:, :4]
    return (np.concatenate([nodes + np.array([o, 0.0, 0.0]) for o in offsets]),
            np.concatenate([tets + i * len(nodes) for i in range(len(offsets))]))


def outcome(positions, tets, device, held_x):
    mesh = sf.Mesh.from_linear(positions, tets, device=device)
    nodes = mesh.nodes()
    model = sf.Model(mesh, sf.Material(1000.0, 0.3))
    model.fix_nodes(np.flatnonzero(np.isin(np.round(nodes[:, 0], 9), held_x)))
    model.add_nodal_force(int(np.argmax(nodes[:, 0])), (0.0, 0.0, 1.0))
    try:
        sf.StaticStudy.new(model)
    except sf.SolidfemError as e:
        return e.status, e.detail["tet"], e.detail["node"]
    return sf.Status.OK


@pytest.mark.parametrize("div", [(1, 1, 1), (7, 5, 6)])
@pytest.mark.parametrize("offsets,held_x", [
    ([0.0], [0.0]),                    # one body
    ([0.0, 2.0], [0.0, 2.0]),          # two, both held
    ([0.0, 2.0], [0.0]),               # the second free
    ([0.0, 2.0, 4.0], [2.0, 4.0]),     # the first free
])
def test_bodies_as_on_the_host(div, offsets, held_x):
    positions, tets = boxes(offsets, div)
    rng = np.random.default_rng(1)
    tets = tets[rng.permutation(len(tets))]  # bodies interleaved in element order
    assert outcome(positions, tets, 0, held_x) == outcome(positions, tets, None, held_x)


def test_boxes_that_share_only_an_edge_are_two_bodies():
    positions, tets = boxes([0.0], (2, 2, 2))
    mirror = positions * np.array([-1.0, 1.0, 1.0])
    far = mirror * np.array([1.0, -1.0, 1.0])  # two reflections keep the orientation
    shared = {tuple(p): i for i, p in enumerate(positions)}
    number = np.array([shared.get(tuple(p), len(positions) + i) for i, p in enumerate(far + 0.0)])
    used = np.unique(number)
    every = np.concatenate([positions, far])
    compact = {int(v): i for i, v in enumerate(np.unique(np.concatenate([np.arange(len(positions)), used])))}
    second = np.vectorize(lambda v: compact[int(number[v])])(tets)
    kept = np.array(sorted(compact))
    both = np.concatenate([tets, second])
    for held in ([1.0], [1.0, -1.0]):
        assert outcome(every[kept], both, 0, held) == outcome(every[kept], both, None, held)
