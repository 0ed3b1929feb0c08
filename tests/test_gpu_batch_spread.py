"""A batch with the library's own choice of what to spread over CTAs: few
instances (all of at least 10 qubits are spread), one instance alone, and many
equal ones (all run whole), against the single-instance adjoint."""
import numpy as np
import pytest

from spinoza_gb300 import adjoint, batch
from spinoza_gb300.core import State

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shapes,spread", [
    ([(9, 2), (10, 1), (12, 3), (14, 2)], 3),
    ([(13, 2)], 1),
    ([(10, 1)] * 9000, 0),  # more than four per CTA slot
])
def test_spread_by_cost_matches_the_single_adjoint(gpu, shapes, spread):
    made = {}
    insts = [made.setdefault((i % 3, s), batch.hea_instance(*s, 70 + i % 3)) for i, s in enumerate(shapes)]
    b = batch.Batch(insts)
    e, g = b.run()
    info = b.info()
    assert info["wide_in_kernel"] == spread and info["wide_separate"] == 0 and 1 <= info["tiles_per_item"] <= 64
    grads = b.split(g)
    for i in list(range(min(4, len(insts)))) + [len(insts) - 1]:
        n, ops, pidx, theta, terms = insts[i]
        e1, g1 = adjoint.adjoint_gradient(State(n), adjoint.set_params(ops, pidx, theta), pidx, terms)
        assert abs(e[i] - e1) < 1e-12 * max(1.0, abs(e1))
        np.testing.assert_allclose(grads[i], g1, atol=1e-11, rtol=0)
    assert np.array_equal(b.run()[1], g)  # the same bits again
