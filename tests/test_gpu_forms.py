"""Which form of the FP64 Jacobi PCG a plan's launches take, and that each form gives the
streamed one's bits where the tests of its own file do not reach."""
import numpy as np
import pytest

import femm_gpu_b200 as fg
from femm_gpu_b200 import meshes

pytestmark = pytest.mark.gpu


def same(a, b):
    for f in ("a", "b1", "b2", "flux"):
        assert np.array_equal(getattr(a, f), getattr(b, f), equal_nan=True), f
    for x, y in zip(a.info, b.info):
        assert (x.status, x.iterations, x.linear_iterations) == (y.status, y.iterations, y.linear_iterations)
        assert x.residual_l2 == y.residual_l2


@pytest.mark.parametrize("m, items, resident", [(8, 32, True), (10, 16, True), (10, 17, False), (10, 32, False),
                                                (11, 32, True), (12, 24, True)])
def test_few_ctas_with_many_items_are_left_to_the_streamed_form(gpu, m, items, resident):
    """Three CTAs are too few owners for 32 items' sums; one or two need none, four have 8 each."""
    model = meshes.square_nonlinear(m=m, seed=3)
    currents = meshes.seeded_currents(items, model.circuit_count, 15.0, seed=1)
    plans = [fg.Plan(model, streamed=s) for s in (False, True)]
    same(*[p.solve(currents) for p in plans])
    assert plans[0].pcg_shapes()[0]["resident"] == resident
