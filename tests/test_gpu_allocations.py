"""Allocations of the operator layer where somebody looks at them: the fill of uninitialised memory that goes with
deterministic algorithms, and dispatch modes."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def table(ops):
    ct = torch.classes.dgs_classes.ChunkTensor([1000, 20], torch.float32, 1000 * 80)
    ct._CAPI_load_from_tensor(torch.randn(1000, 20))
    return ct


def test_deterministic_fill(table):
    idx = torch.arange(500, device="cuda")
    count = torch.tensor([123], device="cuda")
    torch.use_deterministic_algorithms(True)
    try:
        out = table._CAPI_index_counted(idx, count)
    finally:
        torch.use_deterministic_algorithms(False)
    assert not out[:123].isnan().any() and out[123:].isnan().all()  # rows past the count: the fill value


class Seen(TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.names = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.names.append(str(func))
        return func(*args, **(kwargs or {}))


def test_dispatch_mode_sees_the_output(table):
    idx = torch.arange(500, device="cuda")
    with Seen() as seen:
        out = table._CAPI_index(idx)
    assert out.shape == (500, 20) and any("aten.empty" in n for n in seen.names)
