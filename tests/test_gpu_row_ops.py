"""Register-resident vector ops of a batch of rows: row lengths at the edges of one, two and four 16-byte pieces per thread,
multiples of 8 that fill no warp, and lengths the scalar forms take (no multiple of 8), through a batched prompt against the
CPU oracle (1e-2, the bound of the other prefill tests: one int8 step of a requantised activation) and against the same prompt
in two calls (same bits: the order of a row's sums does not depend on the batch)."""
import numpy as np
import pytest

import oracle
from spbitnet_b200 import synth
from spbitnet_b200.engine import DeviceModel, InferenceEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,inter,heads,kv_heads,head_dim",
                         [(8, 1024, 1, 1, 8), (1024, 1032, 2, 1, 72), (1032, 4096, 3, 3, 40), (4104, 8200, 4, 2, 128),
                          (260, 1036, 5, 1, 12), (264, 516, 2, 2, 132)])
def test_prompt_rows(hidden, inter, heads, kv_heads, head_dim):
    cfg = dict(synth.TINY, hidden_size=hidden, intermediate_size=inter, num_attention_heads=heads, num_key_value_heads=kv_heads,
               head_dim=head_dim, num_hidden_layers=2, vocab_size=300, max_position_embeddings=64)
    model = synth.random_model(cfg, seed=hidden)
    eng = InferenceEngine(DeviceModel(model))
    tokens = np.random.default_rng(inter).integers(0, cfg["vocab_size"], 19).astype(np.int32)
    eng.prefill(tokens)
    one = eng.logits()
    cpu = oracle.Engine(model)
    for t in tokens:
        ref = cpu.forward(int(t))
    assert np.abs(one - ref).max() < 1e-2
    eng.reset()
    eng.prefill(tokens[:7])
    eng.prefill(tokens[7:])
    assert (eng.logits() == one).all()
