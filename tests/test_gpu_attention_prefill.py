"""The prompt attention kernel at the edges of its tiles (16 tokens per warp, 64 positions per K/V tile, one to four token
tiles per block), against the token-serial step on the same engine: same logits within 1e-2, the bound of the other
prefill tests (one int8 step of a requantised activation)."""
import numpy as np
import pytest

from spbitnet_b200 import synth
from spbitnet_b200.engine import DeviceModel, InferenceEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(2, 2, 64), (4, 1, 128), (8, 1, 64), (6, 2, 128)])
def test_prompt_attention_matches_token_serial(heads, kv_heads, head_dim):
    cfg = dict(synth.TINY, num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=head_dim,
               max_position_embeddings=256)
    eng = InferenceEngine(DeviceModel(synth.random_model(cfg, seed=heads)))
    tokens = np.random.default_rng(head_dim).integers(0, cfg["vocab_size"], 200).astype(np.int32)
    serial = {}
    for i, t in enumerate(tokens[:196]):
        eng.forward(int(t))
        serial[i + 1] = eng.logits()
    for first, n in [(0, 1), (0, 15), (0, 17), (0, 64), (0, 65), (0, 129), (1, 16), (63, 2), (63, 64), (100, 33), (3, 193)]:
        eng.reset()
        if first:
            eng.prefill(tokens[:first])
        eng.prefill(tokens[first:first + n])
        assert np.abs(eng.logits() - serial[first + n]).max() < 1e-2, (first, n)
