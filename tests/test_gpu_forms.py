"""Which form of the FP64 Jacobi PCG a plan's launches take, and that each form gives the
streamed one's bits where the tests of its own file do not reach."""
import numpy as np
import pytest

import femm_gpu_b200 as fg
import oracle as O
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


def window_rows(plan, items):
    """Shared-memory bytes of the window form's ring and of q beside it, as the launch sizes them."""
    ro, col = plan.symbolic()[:2]
    bandwidth = int(np.abs(np.repeat(np.arange(plan.rows), np.diff(ro)) - col).max())
    kp = 1 << (items - 1).bit_length()
    step = 32 * min(kp, 2) // kp  # rows of a warp-step
    steps = -(-plan.rows // 32) * 32 // step
    groups = min(-(-steps // 16), 296)
    most = max(steps * min(groups, 2 * c + 2) // groups - steps * 2 * c // groups for c in range((groups + 1) // 2))
    return (2 * bandwidth + 4 * 16 * step) * kp * 8, most * step * kp * 8


MODELS = {"square30": lambda: meshes.square_nonlinear(m=30, seed=5), "square12": lambda: meshes.square_nonlinear(m=12, seed=5),
          "sector2400": lambda: meshes.annular_sector(40, 60), "sector": meshes.annular_sector,
          "plunger": meshes.axisymmetric_plunger,
          "wide_rows": lambda: meshes.sliding_band_machine(nr=40, nt=30, rotor_deg=7.3)}


@pytest.mark.parametrize("name, items", [
    ("square12", 1), ("square12", 13),  # one round, one CTA
    ("square30", 1), ("square30", 2), ("square30", 3), ("square30", 8), ("square30", 16), ("square30", 32),
    ("sector2400", 1), ("sector2400", 7),  # odd numbers of row groups: 5, 19
    ("wide_rows", 1), ("wide_rows", 2), ("wide_rows", 3), ("wide_rows", 5), ("wide_rows", 16),  # rows of 20 entries
    ("sector", 4), ("sector", 16), ("sector", 32), ("plunger", 1), ("plunger", 9), ("plunger", 32)])
def test_the_window_form_where_it_is_asked_for(gpu, name, items):
    model = MODELS[name]()
    plans = [fg.Plan(model, window=True), fg.Plan(model, streamed=True)]
    currents = meshes.seeded_currents(items, model.circuit_count, 15.0, seed=items)
    currents[::3] *= 1e-3  # linear items beside saturated ones
    options = fg.production_options(max_newton_iterations=6, recover_nonconvergence=0)
    same(*[p.solve(currents, options=options) for p in plans])
    assert plans[0].pcg_shapes()[0]["window"] and not plans[1].pcg_shapes()[0]["window"]
    ring, q = window_rows(plans[0], items)
    in_shared = ring + q <= 220 * 1024
    assert in_shared == (not (items == 32 and name in ("sector", "plunger")))  # both places are tried


@pytest.mark.parametrize("budget", [0, 1, 2, 7, 8])
def test_window_form_iteration_budgets(gpu, budget):
    model = MODELS["sector2400"]()
    plans = [fg.Plan(model, window=True), fg.Plan(model, streamed=True)]
    currents = meshes.seeded_currents(5, model.circuit_count, 15.0, seed=1)
    options = fg.production_options(max_newton_iterations=2, max_linear_iterations=budget, recover_nonconvergence=0)
    same(*[p.solve(currents, options=options) for p in plans])
    assert plans[0].pcg_shapes()[0]["window"]


def linear_systems(plan, items, shared):
    """Operators and right-hand sides with a zero one, one that is not finite and (an operator per
    item) an indefinite operator; then subnormal values, whose reciprocals overflow, so that the
    Jacobi step divides."""
    vals, _, _ = plan.assemble(np.zeros((1, plan.N)), np.ones((1, 3)), 0)
    rng = np.random.default_rng(11)
    rhs = rng.normal(size=(6, plan.rows))
    rhs[1] = 0.0
    rhs[2, 100] = np.nan
    vals = vals * (1.0 + 0.1 * np.arange(6))[:, None]
    if not shared:
        vals[3] *= -1.0
    for scale in (1.0, 1e-309):
        if items == 1:
            for i in range(4):
                yield scale * vals[i] if shared else scale * vals[i:i + 1], rhs[i:i + 1]
        else:
            yield scale * vals[0] if shared else scale * vals, rhs


# Systems of each form and of its variants: the window form (small, and with several rounds),
# two row groups per CTA with the values in shared memory and in L2, an odd number of groups, and
# one operator for all items.
@pytest.mark.parametrize("form, m, items, shared, grid", [
    ("window", 30, 6, False, 4), ("window", 30, 1, False, 1), ("window", 250, 6, False, 148),
    ("resident", 140, 6, False, 76), ("resident", 277, 1, False, 75), ("resident", 140, 6, True, 76),
    ("resident", 208, 6, True, 148), ("resident", 277, 1, True, 75)])
@pytest.mark.parametrize("tol, maxit", [(1e-10, 2000), (3e-16, 120), (1e-10, 0), (1e-10, 3)])
def test_linear_solves_give_the_streamed_bits(gpu, form, m, items, shared, grid, tol, maxit):
    """Restarts from the true residual (a tolerance at the rounding level), budgets, zero and
    non-finite right-hand sides, an indefinite operator, and the dividing preconditioner."""
    model = meshes.square_nonlinear(m=m, seed=5)
    plans = [fg.Plan(model, window=form == "window"), fg.Plan(model, streamed=True)]
    for operator, rhs in linear_systems(plans[0], items, shared):
        res = [p.pcg(operator, rhs, tol=tol, maxit=maxit, shared=shared) for p in plans]
        assert np.array_equal(res[0][0], res[1][0], equal_nan=True)
        for x, y in zip(res[0][1], res[1][1]):
            assert (x.status, x.iterations) == (y.status, y.iterations)
            assert x.residual_l2 == y.residual_l2 or (np.isnan(x.residual_l2) and np.isnan(y.residual_l2))
    assert plans[0].pcg_shapes()[0][form] and plans[0].last_timing().pcg_grid == grid


@pytest.mark.parametrize("streamed", [False, True])
def test_small_linear_solves_match_the_oracle(gpu, streamed):
    """The streamed form at sizes that a plan gives to the resident one, beside it."""
    model = meshes.square_nonlinear(m=30, seed=5)
    plan = fg.Plan(model, streamed=streamed)
    s = O.assemble(model, np.zeros(model.node_count), [3.0, -5.0, 8.0], 0)
    nan = s.rhs.copy()
    nan[17] = np.nan
    for values, rhs, tol, maxit in ((s.val, s.rhs, 1e-10, 2000), (s.val, s.rhs, 1e-10, 3), (s.val, s.rhs, 1e-10, 0),
                                    (s.val, 0.0 * s.rhs, 1e-10, 2000), (s.val, nan, 1e-10, 2000),
                                    (-s.val, s.rhs, 1e-10, 2000), (s.val, s.rhs, 1e-14, 2000)):
        system = O.csr_system(s.off, s.col, values, rhs)
        status, x, its, res = O.pcg(system, rhs=rhs, tol=tol, maxit=maxit)
        got, info = plan.pcg(values[None, :], rhs, tol=tol, maxit=maxit)
        assert info[0].status == status
        if status == 0:
            assert abs(info[0].iterations - its) <= 1 + its // 50
            assert np.linalg.norm(got[0] - x) <= 1e-6 * np.linalg.norm(x)
        if maxit in (0, 3):
            assert info[0].iterations == its == maxit
            assert abs(info[0].residual_l2 - res) <= 1e-9 * res
    assert plan.pcg_shapes()[0]["resident"] is not streamed


def test_streamed_launch_shapes_leave_results_bitwise_unchanged(gpu, monkeypatch):
    """The shapes that the autotuner chooses from on a plan that runs them: tuned, untuned, and in
    CTAs of 1024 threads."""
    model = meshes.square_nonlinear(m=60, seed=3)
    currents = meshes.seeded_currents(8, 3, 20.0, seed=13)
    tuned = fg.Plan(model, streamed=True)
    r = [tuned.solve(currents)]
    shape = tuned.pcg_shapes()[0]
    assert not shape["resident"] and not shape["window"] and shape["candidates"] == 5
    assert tuned.last_timing().pcg_block == shape["threads_per_block"]
    monkeypatch.setenv("FG_PCG_TUNE", "0")
    for block in ("512", "1024"):
        monkeypatch.setenv("FG_PCG_BLOCK", block)
        plan = fg.Plan(model, streamed=True)
        r.append(plan.solve(currents))
        assert plan.pcg_shapes() == [] and plan.last_timing().pcg_block == int(block)
    same(r[0], r[1])
    same(r[0], r[2])


@pytest.mark.parametrize("form", ["resident", "window"])
def test_the_reported_shape_is_the_one_that_runs(gpu, form):
    plan = fg.Plan(meshes.square_nonlinear(m=60, seed=3), window=form == "window")
    plan.solve(meshes.seeded_currents(8, 3, 20.0, seed=13))
    shape = plan.pcg_shapes()[0]
    assert shape[form] and shape["threads_per_block"] == plan.last_timing().pcg_block == 512
    assert not shape["value_ring"] and not shape["column_cache"] and shape["candidates"] == 5


@pytest.mark.parametrize("m, form, most", [(60, "resident", 5), (354, "window", 9)])
def test_trials_of_the_first_solve(gpu, m, form, most):
    """No warm-up where the times are only reported; no second trial of a candidate that was clearly
    behind in the first (five streamed shapes against the window form, a fifth faster)."""
    plan = fg.Plan(meshes.square_nonlinear(m=m, seed=3))
    currents = meshes.seeded_currents(8, 3, 20.0, seed=13)
    options = fg.production_options(max_newton_iterations=2, max_linear_iterations=100, recover_nonconvergence=0)
    launches = []
    for _ in range(2):
        plan.solve(currents, options=options)
        launches.append(plan.last_timing().kernel_launches)
    assert plan.pcg_shapes()[0][form] and 0 < launches[0] - launches[1] <= most
