"""The largest of many keys decides the form of the relabel operator's table wherever it stands among them, against numpy."""
import numpy as np
import pytest
import torch

from gpu_util import Words, unique_relabel
from test_gpu_relabel_dense import slots
from test_gpu_relabel_paths import want

pytestmark = pytest.mark.gpu


# a sweep of the reading CTAs covers 2^19 keys, 1 024 each
@pytest.mark.parametrize("n", [1 << 19, (1 << 19) + 1, (1 << 20) + 700])
def test_one_large_key_anywhere(n):
    words = Words()
    rng = np.random.default_rng(n)
    line = 2 * slots(n)
    for at in (0, 255, 1023, 255 * 1024 + 256, 256 * 1024, 300 * 1024 + 700, 511 * 1024 + 1023, min(n - 1, 1 << 19), n - 1):
        keys = rng.integers(0, line, n)
        keys[at] = line
        ids = np.concatenate([keys[:3000], [line, line - 1, line + 1], rng.integers(0, line, 50)])
        u, lab = unique_relabel([torch.from_numpy(keys).cuda()], [torch.from_numpy(ids).cuda()], words)
        assert words.take_status() == 0
        wu, wl = want(keys, ids)
        assert np.array_equal(u, wu) and np.array_equal(lab, wl)
