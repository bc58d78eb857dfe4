"""Replacing a matrix of an engine whose last token may still be running: the token that was enqueued multiplies on the old
matrix, the next one on the new, as in an engine that waits in between; and a prepared copy that is written again behind a
product that reads it."""
import ctypes as C

import numpy as np
import pytest
import torch

from spbitnet_b200 import kernels as K
from spbitnet_b200 import synth
from spbitnet_b200._lib import check
from spbitnet_b200.engine import DeviceModel, InferenceEngine

pytestmark = pytest.mark.gpu


def _forward(eng, token, wait):
    """One token; without `wait` the call returns as soon as it is enqueued."""
    check(eng._lib.spb_engine_forward(eng._h, token, None))
    if wait:
        eng.logits()


def _replace(eng, model):
    for l, layer in enumerate(model.layers):
        for i, t in enumerate(layer["linear"]):
            check(eng._lib.spb_engine_set_linear(eng._h, l, i, C.c_void_p(t["d_meta"].data_ptr()),
                                                 C.c_void_p(t["d_values"].data_ptr()), float(t["gamma"]), t["rows"], t["cols"],
                                                 t["meta_stride"], t["values_stride"]))


@pytest.mark.parametrize("prepared", [True, False])
def test_between_tokens(prepared):
    models = [DeviceModel(synth.random_model(synth.TINY, seed=s)) for s in (11, 12)]
    models[1].embed, models[1].final_norm, models[1].lm_head = models[0].embed, models[0].final_norm, models[0].lm_head
    got = []
    for wait in (True, False):
        eng = InferenceEngine(models[0])
        eng.set_prepared_weights(prepared)
        logits = []
        for step in range(6):
            _forward(eng, 7 * step + 1, wait)
            _forward(eng, 7 * step + 2, wait)
            _replace(eng, models[(step + 1) % 2])
            logits.append(eng.logits())
        got.append(np.stack(logits))
        eng.close()
    assert (got[0] == got[1]).all()
    assert not (got[0][0] == got[0][1]).all()


def test_prepared_copy_written_again():
    rows, cols = 6912, 2560
    mats = [synth.device_sparse_matrix(rows, cols, s) for s in (1, 2)]
    ms, vs = mats[0][0].shape[1], mats[0][1].shape[1]
    x = torch.randint(-127, 128, (cols,), device="cuda").to(torch.int8)
    want = []
    for meta, values in mats:
        y = torch.zeros(rows, dtype=torch.int32, device="cuda")
        K.sparse_ternary_gemv_gpu(meta, values, x, y, rows, cols, ms, vs)
        want.append(y)
    prep = K.prepare_weights(*mats[0], rows, cols, ms, vs)
    ys = [torch.zeros(rows, dtype=torch.int32, device="cuda") for _ in range(16)]
    for i, y in enumerate(ys):  # product and rewrite one behind the other on the stream
        K.prepared_gemv_gpu(prep, x, y, rows, cols)
        check(K.load().spb_prepare_weights(C.c_void_p(mats[(i + 1) % 2][0].data_ptr()), C.c_void_p(mats[(i + 1) % 2][1].data_ptr()),
                                           rows, cols, ms, vs, C.c_void_p(prep.data_ptr()),
                                           C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert all((y == want[i % 2]).all() for i, y in enumerate(ys))
