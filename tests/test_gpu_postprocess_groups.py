"""The device postprocess takes items in groups of one, two or four and adds the CTAs' sums in
its last CTA: every group size and remainder against the host form.

The force terms are summed in another order: with E terms the sums agree within E eps of the
sum of the terms' magnitudes, bounded here by that of the largest item's.  The air-gap samples
use the host's operation order and are equal.
"""
import numpy as np
import pytest

import femm_gpu_b200 as fg
from femm_gpu_b200 import meshes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case():
    model = meshes.annular_sector(40, 62)
    model.group = np.array([0, 10, 10, 3, 4, 5, 6], np.int32)
    plan = fg.Plan(model)
    mask = (np.hypot(model.xy[:, 0], model.xy[:, 1]) < 0.0455).astype(np.float64)
    post = fg.Postprocess(plan, selected_group=10, air_group=0, radius_m=0.0455,
                          angles_rad=np.radians([5.0, 44.0, 81.0]), mask=mask)
    currents = meshes.seeded_currents(9, 3, 15.0, seed=3)
    return post, plan.solve(currents, options=fg.production_options(max_newton_iterations=3,
                                                                    recover_nonconvergence=0))


def on_device(post, r, items):
    import torch

    dev = [torch.from_numpy(np.ascontiguousarray(x[items])).cuda() for x in (r.a, r.b1, r.b2)]
    torch.cuda.synchronize()
    return post.compute_device(len(items), *[x.data_ptr() for x in dev])


@pytest.mark.parametrize("count", [1, 2, 3, 4, 5, 8, 9])
def test_every_group_size_matches_the_host_form(gpu, case, count):
    post, r = case
    items = list(range(count))
    host = post.compute(r.a[items], r.b1[items], r.b2[items])
    scale = np.abs(host.force).max()
    for _ in range(2):  # the arrival counters are left as they were found
        dev = on_device(post, r, items)
        assert (dev.status == 0).all()
        assert np.abs(dev.force - host.force).max() <= 1e-11 * scale
        assert np.abs(dev.torque - host.torque).max() <= 1e-11 * np.abs(host.torque).max()
        assert np.array_equal(dev.radial_b, host.radial_b)


def test_a_field_that_is_not_finite_fails_its_item_only(gpu, case):
    post, r = case
    broken = type(r)(r.a.copy(), r.b1.copy(), r.b2.copy(), r.flux, r.info)
    outer = 7  # an element away from the mask's step: its products are zero when finite
    broken.b1[2, outer] = np.nan
    broken.b2[4, outer] = np.inf
    host = post.compute(broken.a[:6], broken.b1[:6], broken.b2[:6])
    dev = on_device(post, broken, list(range(6)))
    assert np.array_equal(dev.status, host.status) and (dev.status[[2, 4]] != 0).all()
    assert (np.delete(dev.status, [2, 4]) == 0).all()
