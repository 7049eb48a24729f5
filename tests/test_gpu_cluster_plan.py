"""The plan of 2 049 to 8 192 seeds by a cluster of CTAs, at the edges of its range and of its CTAs' parts."""
import numpy as np
import pytest

from test_gpu_small_plan import test_plan_offsets as check_plan_offsets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("idt", [np.int64, np.int32])
@pytest.mark.parametrize("replace", [0, 1])
@pytest.mark.parametrize("n", [2049, 2056, 2057, 4104, 8185, 8191, 8192, 8193])
def test_cluster_plan_offsets(n, replace, idt):
    check_plan_offsets(n, replace, idt)
