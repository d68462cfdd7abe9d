"""Which clears go to the current GPU's stream, and which to the tensor library: shown with stand-ins for tensors and module."""
import pytest

from meshslice_b200 import _native


class _Tensor:
    def __init__(self, ptr, device, contiguous=True, block=7):
        self.is_cuda, self.device_index, self.contiguous, self.ptr, self.block = device is not None, device, contiguous, ptr, block
        self.cleared = 0

    def is_contiguous(self):
        return self.contiguous

    def get_device(self):
        return -1 if self.device_index is None else self.device_index

    def numel(self):
        return 16

    def element_size(self):
        return 4

    def data_ptr(self):
        return self.ptr

    def untyped_storage(self):
        return type("Storage", (), {"data_ptr": lambda _: self.block})()

    def zero_(self):
        self.cleared += 1


@pytest.fixture
def memsets(monkeypatch):
    calls = []
    gpu = type("Cuda", (), {"_cuda_getDevice": staticmethod(lambda: 0), "_cuda_getCurrentRawStream": staticmethod(lambda d: 100 + d)})
    monkeypatch.setattr(_native, "_cuda", gpu)
    monkeypatch.setattr(_native, "load", lambda: type("C", (), {"memset_zero": staticmethod(lambda *a: calls.append(a))}))
    return calls


@pytest.mark.parametrize("device,contiguous,here", [(0, True, True), (0, False, False), (1, True, False), (None, True, False)])
def test_a_clear_goes_to_the_tensors_own_device(memsets, device, contiguous, here):
    """A tensor of another GPU than the current one is cleared on its own device's stream, as ``Tensor.zero_`` does."""
    t = _Tensor(4096, device, contiguous)
    _native.zero_(t)
    assert memsets == ([(4096, 64, 100)] if here else []) and t.cleared == (0 if here else 1)


@pytest.mark.parametrize("device", [0, 1, None])
def test_two_clears_in_one_launch_are_the_current_gpus(memsets, device):
    a, b = _Tensor(4096, device), _Tensor(4160, device)
    _native.zero_both_(a, b)
    assert memsets == ([(4096, 128, 100)] if device == 0 else []) and (a.cleared, b.cleared) == ((0, 0) if device == 0 else (1, 1))
