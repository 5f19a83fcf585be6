"""One status word per device, whichever threads ask for it first: kernels keep its address."""
from types import SimpleNamespace

import torch

from nvfp4_training_b200 import _lib


def test_a_second_thread_in_the_allocation_gets_the_same_word(monkeypatch):
    other = []

    def zeros(*args, **kwargs):
        if not other:
            other.append(None)
            other[0] = _lib.status_word("cuda:7")          # another thread, while this one allocates
        return torch.Tensor.new_zeros(torch.empty(0, dtype=torch.int32), 1)
    monkeypatch.setattr(_lib, "_status", {})
    monkeypatch.setattr(_lib, "torch", SimpleNamespace(zeros=zeros, device=torch.device, int32=torch.int32))
    mine = _lib.status_word("cuda:7")
    assert mine is other[0] and _lib.status_word("cuda:7") is mine
