"""What the 32-bit product is told about its weights, without a GPU: a library that only notes its calls."""

import torch

from models_b200.kernels import ops
from models_b200.parts.linear import linear


class OnCard(torch.Tensor):
    is_cuda = True


class Noted:
    def __init__(self):
        self.ready = []

    def mb_gemm_f32(self, *args):
        self.ready.append(args[-2])
        return 0

    class mb_gemm_f32_scratch:
        def __new__(cls, m, k):
            return 0


def test_only_loaded_weights_are_read_ahead(monkeypatch):
    """A kernel starts its follower before it has written its result, so what an op is given as `w` may be read after the wait alone."""
    lib = Noted()
    monkeypatch.setattr(ops, "gemm32", lambda: lib)
    monkeypatch.setattr(ops, "_cuda", lambda *tensors: None)
    monkeypatch.setattr(ops, "_stream", lambda: None)
    a, w = torch.zeros(3, 64), torch.zeros(8, 64)
    ops.gemm_f32(a, w)
    ops.gemm_f32(a, w, True)
    assert lib.ready == [0, 0]
    linear(a.as_subclass(OnCard), w, torch.float32)
    assert lib.ready == [0, 0, 1]
