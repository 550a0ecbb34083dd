"""The window form of the FP64 Jacobi PCG (the SpMV's operand in a sliding window in shared
memory) against the streamed form: the same partition, operations and summation orders, so the
same bits.  The sizes are ones that the resident form does not fit: every item width, odd item
counts, q in shared memory and in global memory, rows wider than the eight entries read ahead,
odd and even iteration budgets (x is updated every other iteration), items that stop at
different iterations."""
import numpy as np
import pytest

import femm_gpu_b200 as fg
from femm_gpu_b200 import meshes

pytestmark = pytest.mark.gpu


def solve_both(model, currents, **options):
    opts = fg.production_options(**options)
    plans = [fg.Plan(model, streamed=s) for s in (False, True)]
    a, b = [p.solve(currents, options=opts) for p in plans]
    for f in ("a", "b1", "b2", "flux"):
        assert np.array_equal(getattr(a, f), getattr(b, f), equal_nan=True), f
    for x, y in zip(a.info, b.info):
        assert (x.status, x.iterations, x.linear_iterations) == (y.status, y.iterations, y.linear_iterations)
        assert x.residual_l2 == y.residual_l2
    return plans[0].pcg_shapes()[0], a


@pytest.mark.parametrize("m, items", [(560, 1), (500, 2), (400, 3), (300, 8), (354, 7), (420, 16), (250, 13)])
def test_squares_give_the_streamed_bits(gpu, m, items):
    model = meshes.square_nonlinear(m=m, seed=3)
    shape, r = solve_both(model, meshes.seeded_currents(items, model.circuit_count, 15.0, seed=items))
    assert not shape["resident"] and all(i.status == 0 for i in r.info)


@pytest.mark.parametrize("name, items", [("sector", 32), ("sector", 11), ("plunger", 32), ("plunger", 5)])
def test_unstructured_rows_give_the_streamed_bits(gpu, name, items):
    model = meshes.annular_sector() if name == "sector" else meshes.axisymmetric_plunger()
    currents = meshes.seeded_currents(items, model.circuit_count, 15.0, seed=items)
    currents[::3] *= 1e-3  # linear items beside saturated ones
    shape, _ = solve_both(model, currents)
    assert not shape["resident"]


@pytest.mark.parametrize("budget", [1, 2, 7, 8])
def test_iteration_budgets_give_the_streamed_bits(gpu, budget):
    model = meshes.square_nonlinear(m=354, seed=3)
    shape, _ = solve_both(model, meshes.seeded_currents(8, model.circuit_count, 15.0, seed=1), max_newton_iterations=2,
                          max_linear_iterations=budget, recover_nonconvergence=0)
    assert shape["window"]
