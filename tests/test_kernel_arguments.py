"""What the functional layer hands to kernels that load 16 bytes at a time, seen on the CPU: tensors that say they are
on the GPU, and a library that records its arguments."""
import pytest
import torch

from multimesh_jax_b200.ops import kernels as K


class OnGpu(torch.Tensor):
    is_cuda = property(lambda self: True)


class Recorder:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *args: (self.calls.append((name, args)), 0)[1]


@pytest.mark.parametrize("offset", range(9))
def test_logits_that_start_anywhere_reach_the_loss_on_16_bytes(monkeypatch, offset):
    """A view of a flat buffer is contiguous whatever it starts on."""
    rows, V = 3, 16
    lib = Recorder()
    monkeypatch.setattr(K._lib, "load", lambda: lib)
    monkeypatch.setattr(K, "_stream", lambda: 0)
    flat = torch.randn(rows * V + 16).bfloat16()
    flat = flat[-flat.data_ptr() // 2 % 8:]
    logits = flat[offset:offset + rows * V].view(rows, V).as_subclass(OnGpu)
    assert logits.is_contiguous() and logits.data_ptr() % 16 == offset % 8 * 2
    K.cross_entropy_to(logits, torch.zeros(rows, dtype=torch.int64), 1.0)
    ((name, args),) = lib.calls
    assert args[0] % 16 == 0 and name == ("mm_cross_entropy_to" if offset % 8 == 0 else "mm_cross_entropy")
