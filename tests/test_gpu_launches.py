"""What a launch of the FP64 Jacobi PCG leaves alone: the launches of other plans (the kernels
and their attributes are shared by all threads of a process).
"""
import threading

import numpy as np
import pytest

import femm_gpu_b200 as fg
from femm_gpu_b200 import meshes

pytestmark = pytest.mark.gpu


def test_plans_of_different_sizes_solve_on_two_threads(gpu):
    """Two plans whose launches of one kernel need different amounts of shared memory, each
    owned by a thread: every call passes and answers as it does alone."""
    cases = []
    for m in (8, 40):
        model = meshes.square_nonlinear(m=m, seed=3)
        plan = fg.Plan(model)
        currents = meshes.seeded_currents(8, model.circuit_count, 15.0, seed=m)
        cases.append((plan, currents, plan.solve(currents)))
    stop, wrong = threading.Event(), []

    def work(plan, currents, alone, calls):
        try:
            while not stop.is_set() and calls != 0:
                r = plan.solve(currents)
                if not (np.array_equal(r.a, alone.a) and np.array_equal(r.flux, alone.flux)):
                    wrong.append("another answer")
                    break
                calls -= 1
        except fg.FgError as e:
            wrong.append(str(e))
        stop.set()

    threads = [threading.Thread(target=work, args=(*cases[0], -1)), threading.Thread(target=work, args=(*cases[1], 60))]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not wrong, wrong
