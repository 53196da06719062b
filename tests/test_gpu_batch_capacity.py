"""A batch of more blocks than the device holds walks several of them per block, also where their
partial sums order the dot products: every member must keep the bits of its solve alone (needs a B200)."""
import numpy as np
import pytest

import solidfem_b200 as sf
from tests.helpers import mg_options, product_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [sf.Precision.MIXED, sf.Precision.DOUBLE])
def test_large_batch_keeps_each_members_bits(precision):
    def studies():
        out = []
        for i in range(10):
            _, model = product_model((10.0, 1.0, 1.0), (18 + i % 3, 4, 4), 200000.0 / (i + 1), 0.3)
            out.append(sf.StaticStudy.new(model, mg_options(precision, coarse_dofs=1500, batchable=True)))
        return out

    alone = studies()
    for study in alone:
        assert study.solve().kind == sf.Outcome.CONVERGED
    together = studies()
    assert all(status == sf.Status.OK for _, status in sf.solve_batch(together))
    for a, b in zip(alone, together):
        assert np.array_equal(a.displacements().view(np.uint64), b.displacements().view(np.uint64))
