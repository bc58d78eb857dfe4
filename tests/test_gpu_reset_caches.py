"""reset() leaves the caches as a new engine has them, whatever wrote them and however far: read from the caches themselves, since
no logits depend on what lies past a sequence's position."""
import numpy as np
import pytest

from spbitnet_b200 import synth
from spbitnet_b200.engine import DeviceModel, InferenceEngine
from spbitnet_b200.shard_engine import ShardEngine

pytestmark = pytest.mark.gpu

ODD = dict(synth.TINY, num_attention_heads=3, num_key_value_heads=1, head_dim=40, max_position_embeddings=37)  # layers padded to 256 bytes
LONG = dict(synth.TINY, max_position_embeddings=1500)  # a prompt of several chunks


def _nonzeros(eng):
    count = getattr(eng._lib, "spb_debug_shard_engine_cache_nonzeros" if isinstance(eng, ShardEngine) else "spb_debug_engine_cache_nonzeros")
    got = [count(eng._h, v) for v in (0, 1)]
    assert min(got) >= 0
    return got


def _written(cfg, positions, batch=1):
    """What `positions` positions of every layer and sequence hold, give or take the values that come out as zero."""
    n = positions * cfg["num_key_value_heads"] * cfg["head_dim"] * cfg["num_hidden_layers"] * batch
    return lambda counts: all(0.9 * n < c <= n for c in counts)


@pytest.mark.parametrize("cfg", [synth.TINY, ODD, LONG], ids=["tiny", "odd", "long"])
def test_single_sequence(cfg):
    eng = InferenceEngine(DeviceModel(synth.random_model(cfg, seed=5)))
    limit = cfg["max_position_embeddings"]
    tokens = np.random.default_rng(1).integers(0, cfg["vocab_size"], limit).astype(np.int32)

    def forward(n):
        for t in tokens[:n]:
            eng.forward(int(t))

    def generate(n, chunk):
        old = eng.set_prefill_chunk(chunk)
        eng.generate(tokens[:n], 3)
        eng.set_prefill_chunk(old)

    assert _nonzeros(eng) == [0, 0]
    ways = [(lambda: forward(1), 1), (lambda: forward(7), 7), (lambda: eng.prefill(tokens[:9]), 9), (lambda: generate(5, 0), 7),
            (lambda: generate(5, 64), 7), (lambda: (eng.prefill(tokens[:6]), forward(4), eng.prefill(tokens[:5])), 15),
            (lambda: eng.prefill(tokens), limit), (lambda: (eng.prefill(tokens[:limit - 2]), forward(2)), limit)]
    for i, (write, positions) in enumerate(ways):
        write()
        assert _written(cfg, positions)(_nonzeros(eng)), i
        eng.reset()
        assert _nonzeros(eng) == [0, 0], i


@pytest.mark.parametrize("cfg", [synth.TINY, ODD], ids=["tiny", "odd"])
def test_batch(cfg):
    batch = 3
    eng = ShardEngine(DeviceModel(synth.random_model(cfg, seed=6)), batch=batch)
    tokens = np.random.default_rng(2).integers(0, cfg["vocab_size"], (20, batch)).astype(np.int32)
    assert _nonzeros(eng) == [0, 0]
    for n, generated in ((1, 0), (20, 0), (4, 5), (0, 6)):
        for t in tokens[:n]:
            eng.step(t)
        positions = n
        if generated:
            eng.generate(tokens[:2], generated)
            positions += 1 + generated
        assert _written(cfg, positions, batch)(_nonzeros(eng)), (n, generated)
        eng.reset()
        assert _nonzeros(eng) == [0, 0], (n, generated)
