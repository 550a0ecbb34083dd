"""What a launch of the FP64 Jacobi PCG leaves alone: the launches of other plans (the kernels
and their attributes are shared by all threads of a process) and the caller's own CUDA error.
"""
import ctypes
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


def test_a_pending_error_of_the_caller_stays_pending(gpu):
    """A solve that passes neither reports nor clears an error the caller has yet to read."""
    n = 1_000_000  # beyond the forms that keep the system on chip
    ro = np.minimum(3 * np.arange(n + 1) - 1, 3 * n - 2).astype(np.int32)
    ro[0] = 0
    r = np.arange(n)
    col = np.stack([r - 1, r, r + 1], axis=1).ravel()
    val = np.tile([-1.0, 4.0, -1.0], n)
    keep = (col >= 0) & (col < n)
    col, val = col[keep].astype(np.int32), val[keep]
    rhs = np.ones((1, n))
    fg.csr_pcg(ro, col, val, np.full(n, 4.0), rhs, tol=1e-10, maxit=100)
    runtime = ctypes.CDLL("libcudart.so.12")
    runtime.cudaGetLastError()
    error = runtime.cudaSetDevice(1 << 20)  # refused by the runtime: no such device
    assert error != 0
    try:
        _, info = fg.csr_pcg(ro, col, val, np.full(n, 4.0), rhs, tol=1e-10, maxit=100)
        assert info[0].status == 0 and runtime.cudaPeekAtLastError() == error
    finally:
        runtime.cudaGetLastError()
