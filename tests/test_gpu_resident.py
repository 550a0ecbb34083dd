"""The resident form of the FP64 Jacobi PCG (a CTA's share of the system on chip, CTAs
exchanging messages) against the streamed form: the same partition, operations and summation
orders, so the same bits -- iterates, residuals, iteration counts and statuses.  The sizes
sit at the edges of the form: less than one row group, two, the last one with a row group per
SM and the first without (two row groups per CTA, an odd number of them, the operator's values
in shared memory or in L2, several steps per warp), and rows wider than the eight entries
gathered together."""
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


def solve_both(model, items, limit=15.0, **options):
    currents = meshes.seeded_currents(items, model.circuit_count, limit, seed=items)
    opts = fg.production_options(**options)
    res = [fg.Plan(model, streamed=s).solve(currents, options=opts) for s in (False, True)]
    same(*res)
    return res[0]


@pytest.mark.parametrize("m, items", [(4, 1), (23, 1), (24, 1), (24, 3), (46, 2), (64, 4), (65, 7), (64, 16),
                                      (65, 32), (138, 8), (139, 8),
                                      (250, 4), (100, 32), (130, 16), (390, 1), (270, 2)])
def test_squares_give_the_streamed_bits(gpu, m, items):
    r = solve_both(meshes.square_nonlinear(m=m, seed=3), items)
    assert all(s == 0 for s in r.status)


@pytest.mark.parametrize("model", [meshes.annular_sector(40, 60), meshes.axisymmetric_plunger(60, 121),
                                   meshes.sliding_band_machine(nr=40, nt=30, rotor_deg=7.3)],
                         ids=["antiperiodic", "axisymmetric", "wide_rows"])
def test_other_models_give_the_streamed_bits(gpu, model):
    assert all(s == 0 for s in solve_both(model, 3).status)


def test_wide_rows_that_leave_the_values_in_l2(gpu):
    """One row group per CTA whose entries do not fit beside the state: 20-entry ring rows."""
    r = solve_both(meshes.sliding_band_machine(80, 60), 8, max_newton_iterations=3, recover_nonconvergence=0)
    assert all(i.linear_iterations > 100 for i in r.info)


def test_exhausted_budget_and_inactive_items(gpu):
    model = meshes.square_nonlinear(m=40, seed=3)
    solve_both(model, 5, max_newton_iterations=2, max_linear_iterations=7, recover_nonconvergence=0)
    currents = meshes.seeded_currents(5, 3, 20.0, seed=1)
    currents[1] = np.nan  # refused before the solve: never active
    res = [fg.Plan(model, streamed=s).solve(currents) for s in (False, True)]
    same(*res)
    assert res[0].status[1] != 0 and res[0].status[0] == 0


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("tol, maxit", [(1e-10, 2000), (3e-16, 400), (1e-10, 0), (1e-10, 3)])
def test_linear_solves_give_the_streamed_bits(gpu, shared, tol, maxit):
    """Restarts from the true residual (a tolerance at the rounding level), budgets, zero and
    non-finite right-hand sides, an indefinite operator, and the dividing preconditioner."""
    model = meshes.square_nonlinear(m=30, seed=5)
    plans = [fg.Plan(model, streamed=s) for s in (False, True)]
    items = 6
    vals, _, _ = plans[0].assemble(np.zeros((items, plans[0].N)), np.ones((items, 3)), 0)
    rng = np.random.default_rng(11)
    rhs = rng.normal(size=(items, plans[0].rows))
    rhs[1] = 0.0
    rhs[2, 100] = np.nan
    vals = vals * (1.0 + 0.1 * np.arange(items))[:, None]
    if not shared:
        vals[3] *= -1.0
    for operator in (vals, vals * 1e-309):  # the second: subnormal values, 1/d overflows
        operator = operator[0] if shared else operator
        res = [p.pcg(operator, rhs, tol=tol, maxit=maxit, shared=shared) for p in plans]
        assert np.array_equal(res[0][0], res[1][0], equal_nan=True)
        for x, y in zip(res[0][1], res[1][1]):
            assert (x.status, x.iterations) == (y.status, y.iterations)
            assert x.residual_l2 == y.residual_l2 or (np.isnan(x.residual_l2) and np.isnan(y.residual_l2))


def test_tangents_give_the_streamed_bits(gpu):
    model = meshes.annular_sector(40, 60)
    plans = [fg.Plan(model, streamed=s) for s in (False, True)]
    base = plans[0].solve([[5.0, -3.0, 1.0]])
    directions = np.random.default_rng(2).normal(size=(5, 3))
    got = [p.solve_tangent(base.a[0], [5.0, -3.0, 1.0], directions) for p in plans]
    for x, y in zip(got[0][:4], got[1][:4]):
        assert np.array_equal(x, y)
    assert [i.iterations for i in got[0][4]] == [i.iterations for i in got[1][4]]
