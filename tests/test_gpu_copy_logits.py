"""Logits to memory of the caller's: pageable, pinned (copied to directly), and an address that host code must not touch, which
the runtime answers for."""
import ctypes as C

import numpy as np
import pytest
import torch

from spbitnet_b200 import synth
from spbitnet_b200.engine import DeviceModel, InferenceEngine

pytestmark = pytest.mark.gpu


def test_destinations():
    eng = InferenceEngine(DeviceModel(synth.random_model(synth.TINY, seed=3)))
    n = synth.TINY["vocab_size"]
    eng.forward(5)
    want = eng.logits()
    copy = eng._lib.spb_engine_copy_logits
    pinned = torch.full((n,), 9.0).pin_memory()
    assert copy(eng._h, C.c_void_p(pinned.data_ptr())) == 0 and (pinned.numpy() == want).all()
    for dst in (torch.full((n,), 9.0, device="cuda"), torch.full((n + 8,), 9.0, device="cuda")[8:]):
        if copy(eng._h, C.c_void_p(dst.data_ptr())) == 0:  # unified addressing: the runtime may take it
            torch.cuda.synchronize()
            assert (dst.cpu().numpy() == want).all()
    again = np.full(n + 1, 9.0, np.float32)
    assert copy(eng._h, C.c_void_p(again[1:].ctypes.data)) == 0
    assert (again[1:] == want).all() and again[0] == 9.0
