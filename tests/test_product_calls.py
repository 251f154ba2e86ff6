"""What the kernels' launchers are told and asked, without a GPU: libraries that only note and answer calls."""

import torch

from models_b200.kernels import build, ops
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
        def __new__(cls, *sizes):
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


def test_waits_that_gave_up_are_found_in_every_library(monkeypatch):
    class Library:
        def __init__(self, **statuses):
            for name, status in statuses.items():
                setattr(self, name, lambda status=status: status)

    libraries = {"/somewhere/libmb_a.so": Library(mb_gemm_f32_status=0, mb_gated_delta_chunks_status=1),
                 "/somewhere/libmb_b.so": Library(mb_gemm_tc_status=513), "/somewhere/libmb_c.so": Library()}
    monkeypatch.setattr(build, "_loaded", libraries)
    assert ops.waits_given_up() == {"libmb_a.so: mb_gated_delta_chunks_status": 1, "libmb_b.so: mb_gemm_tc_status": 513}
