"""The benchmark's roofline counts the bytes of the PCG form that ran (CPU)."""
import sys

import pytest

from conftest import ROOT

if ROOT not in sys.path:
    sys.path.insert(0, ROOT)
import bench  # noqa: E402


class Shapes:
    def __init__(self, **form):
        self.form = form

    def pcg_shapes(self):
        return [{"items": 4, "precision": 0, "resident": False, "window": False},
                {"items": 8, "precision": 0, "resident": False, "window": False, **self.form}]


@pytest.mark.parametrize("plan, items, form", [(Shapes(window=True), 8, "window"), (Shapes(resident=True), 5, "resident"),
                                               (Shapes(), 8, "streamed"), (Shapes(window=True), 4, "streamed"),
                                               (Shapes(window=True), 32, "streamed")])
def test_the_form_that_ran(plan, items, form):
    assert bench.pcg_form(plan, items, 0) == form
    assert form in bench.PCG_KERNELS


def test_bytes_of_each_form():
    n, nnz = 249001, 1739017
    assert bench.pcg_bytes_per_item_iteration(n, nnz, 0, 0) == 8 * nnz + 104 * n
    assert bench.pcg_bytes_per_item_iteration(n, nnz, 0, 0, "window") == 8 * nnz + 72 * n
    assert bench.pcg_bytes_per_item_iteration(n, nnz, 0, 0, "resident") == 8 * n
    assert bench.pcg_bytes_per_item_iteration(n, nnz, 1, 32) == 4 * nnz + (52 + 128) * n
    assert bench.pcg_shared_bytes(n, nnz, "window") == 4 * nnz + 4 * (n + 1)
    # the measured traffic of each form is its own capture's
    streamed, window = [bench.traffic_per_cg_iteration("square500_items8", f) for f in ("streamed", "window")]
    assert streamed[0] == 258e6 and window[0] == 191e6 and streamed[1] != window[1]
    assert bench.traffic_per_cg_iteration("square500_items8", "resident") == (None, None)
