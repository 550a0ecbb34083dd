"""The warm start's network where there is no GPU (CPU)."""
import pytest

import femm_gpu_b200 as fg
from conftest import gpu_available
from femm_gpu_b200 import learned


@pytest.mark.skipif(gpu_available(), reason="a CUDA device is there")
def test_a_network_without_a_gpu_reports_the_allocation():
    with pytest.raises(fg.FgError) as e:
        learned.Mlp(4, 8, 3)
    assert fg.capi.STATUS_NAMES[e.value.status] == "GPU_ALLOCATION_FAILED"
