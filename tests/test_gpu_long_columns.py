"""A prolongator column too long for the device's sort (8,192 entries): its transpose is made on the
host (needs a B200). A hub with 1,000 leaves is the first aggregate; each leaf has ten outer nodes,
gathered by a node of their own, so 11,001 rows reach the hub's column."""
import numpy as np
import pytest

import solidfem_b200 as sf

pytestmark = pytest.mark.gpu

LEAVES, OUTER = 1000, 10


@pytest.mark.parametrize("precision", [sf.Precision.DOUBLE, sf.Precision.MIXED])
def test_star_of_stars(precision):
    rng = np.random.default_rng(5)

    def direction(n):
        d = rng.standard_normal((n, 3))
        return d / np.linalg.norm(d, axis=1)[:, None]

    leaf = 1 + np.arange(LEAVES)
    outer = 1 + LEAVES + np.arange(LEAVES * OUTER)
    gather = 1 + LEAVES + LEAVES * OUTER + np.arange(LEAVES)
    owner = np.repeat(np.arange(LEAVES), OUTER)
    at = np.zeros((gather[-1] + 1, 3))
    at[leaf] = direction(LEAVES)                                # every edge between 0.5 and 1.5 long:
    at[outer] = at[leaf][owner] + direction(LEAVES * OUTER)     # all neighbours are strong
    at[gather] = at[leaf] + 0.5 * direction(LEAVES)
    i = np.concatenate([np.zeros(LEAVES, int), leaf[owner], gather[owner]])
    j = np.concatenate([leaf, outer, outer])
    w = rng.uniform(0.5, 1.5, len(i))
    nodes = len(at)
    diagonal = np.full(nodes, 0.05)
    np.add.at(diagonal, i, w)
    np.add.at(diagonal, j, w)
    rows = np.concatenate([np.arange(nodes), i, j])
    cols = np.concatenate([np.arange(nodes), j, i])
    vals = np.concatenate([diagonal, -w, -w])
    order = np.lexsort((cols, rows))
    rows, cols, vals = rows[order], cols[order], vals[order]
    # each coupling times the identity, as whole 3x3 blocks
    starts = np.concatenate([[0], np.cumsum(np.repeat(3 * np.bincount(rows, minlength=nodes), 3))]).astype(np.uint64)
    first = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=nodes))])
    scalar_cols, scalar_vals = [], []
    for r in range(nodes):
        c, v = cols[first[r]:first[r + 1]], vals[first[r]:first[r + 1]]
        for p in range(3):
            scalar_cols.append((3 * c[:, None] + np.arange(3)).ravel())
            block = np.zeros((len(c), 3))
            block[:, p] = v
            scalar_vals.append(block.ravel())
    x, y, z = at.T
    o, l = np.zeros(nodes), np.ones(nodes)
    modes = np.stack([np.stack([l, o, o, o, z, -y], 1), np.stack([o, l, o, -z, o, x], 1),
                      np.stack([o, o, l, y, -x, o], 1)], 1)  # translations and rotations
    b = rng.standard_normal(3 * nodes)
    options = sf.StudyOptions(pcg=sf.PcgOptions(tolerance=1e-9, max_iterations=200),
                              preconditioner=sf.MultigridOptions(precision=precision, coarse_dofs=7000))
    system = sf.System(starts, np.concatenate(scalar_cols).astype(np.uint32), np.concatenate(scalar_vals), b, options,
                       near_null=modes.reshape(-1), positions=at)
    assert system.level_count() >= 2
    assert system.solve().kind == sf.Outcome.CONVERGED
    u = system.estimate().reshape(nodes, 3)
    residual = b.reshape(nodes, 3).copy()
    np.subtract.at(residual, rows, vals[:, None] * u[cols])
    # the converged solve's own test: the true relative residual is within the tolerance
    assert np.linalg.norm(residual) <= 1.01e-9 * np.linalg.norm(b)
