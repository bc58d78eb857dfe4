"""reset() clears what a sequence has written, whatever wrote it and wherever it stopped: after sequences of several lengths (one
token, a batch, a batch and single tokens, the whole cache), the same short prompt gives the bits that a fresh engine gives, alone
and with a batch of sequences; and the logits handed out before stay as they were."""
import numpy as np
import pytest

from spbitnet_b200 import synth
from spbitnet_b200.engine import DeviceModel, InferenceEngine
from spbitnet_b200.shard_engine import ShardEngine

pytestmark = pytest.mark.gpu

ODD = dict(synth.TINY, num_attention_heads=3, num_key_value_heads=1, head_dim=40, max_position_embeddings=37)  # layers padded to 256 bytes


@pytest.mark.parametrize("cfg", [synth.TINY, ODD], ids=["tiny", "odd"])
def test_single_sequence(cfg):
    model = DeviceModel(synth.random_model(cfg, seed=5))
    tokens = np.random.default_rng(1).integers(0, cfg["vocab_size"], cfg["max_position_embeddings"]).astype(np.int32)

    def short(eng):
        out = []
        for t in tokens[:3]:
            eng.forward(int(t))
            out.append(eng.logits())
        return out

    want = short(InferenceEngine(model))
    eng = InferenceEngine(model)
    kept = []
    for n, singles in [(0, 1), (5, 0), (9, 4), (len(tokens), 0), (0, len(tokens))]:
        if n:
            eng.prefill(tokens[:n])
        for t in tokens[:singles]:
            eng.forward(int(t))
        eng.generate(tokens[:1], min(4, len(tokens) - eng.seq_len)) if eng.seq_len < len(tokens) else None
        eng.reset()
        assert eng.seq_len == 0
        kept += list(zip(short(eng), want))
        eng.reset()
    assert all((a == b).all() for a, b in kept)


def test_batch():
    cfg, batch = synth.TINY, 3
    model = DeviceModel(synth.random_model(cfg, seed=6))
    tokens = np.random.default_rng(2).integers(0, cfg["vocab_size"], (20, batch)).astype(np.int32)
    fresh, eng = ShardEngine(model, batch=batch), ShardEngine(model, batch=batch)
    fresh.step(tokens[0])
    for n in (1, 20, 7):
        for t in tokens[:n]:
            eng.step(t)
        eng.generate(tokens[:2], 3)
        eng.reset()
        eng.step(tokens[0])
        assert (eng.logits() == fresh.logits()).all()
        eng.reset()
