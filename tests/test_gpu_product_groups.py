"""The products of a layer that share their activations, as one launch of either form: prompts of a few tokens give the same
bits whichever form the library is told to take (the sums are integers), on widths where each of them is the chosen one."""
import numpy as np
import pytest

from spbitnet_b200 import kernels as K, synth
from spbitnet_b200.engine import DeviceModel, InferenceEngine
from spbitnet_b200.shard_engine import ShardEngine

pytestmark = pytest.mark.gpu

WIDE = dict(synth.TINY, hidden_size=1024, intermediate_size=2304, num_attention_heads=8, num_key_value_heads=2, head_dim=128,
            num_hidden_layers=2)  # v starts in the middle of the grid; row counts of 16 blocks and of 2 1/4 tiles
ODD = dict(synth.TINY, hidden_size=384, intermediate_size=640, num_attention_heads=6, num_key_value_heads=2, head_dim=64)


@pytest.mark.parametrize("cfg", [synth.TINY, WIDE, ODD], ids=["tiny", "wide", "odd"])
def test_forms_agree(cfg):
    model = DeviceModel(synth.random_model(cfg, seed=21))
    tokens = np.random.default_rng(3).integers(0, cfg["vocab_size"], 40).astype(np.int32)
    eng = InferenceEngine(model)
    for n in (2, 4, 5, 8, 9, 16, 17, 32, 40):
        got = []
        for variant in (1, 0, 3, 4):
            old = K.set_gemm_variant(variant)
            try:
                eng.close()
                eng = InferenceEngine(model)  # graphs hold the form they were captured with
                eng.prefill(tokens[:n])
                got.append(eng.logits())
            finally:
                K.set_gemm_variant(old)
        assert all((g == got[0]).all() for g in got[1:]), n
    before = K.gemm_tc_timeouts()
    for batch in (2, 8, 9):
        got = []
        for variant in (1, 0, 3, 4):
            old = K.set_gemm_variant(variant)
            try:
                e = ShardEngine(model, batch=batch)
                e.step(tokens[:batch])
                got.append(e.logits_rows())
            finally:
                K.set_gemm_variant(old)
        assert all((g == got[0]).all() for g in got[1:]), batch
    assert K.gemm_tc_timeouts() == before
