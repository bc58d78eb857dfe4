"""Attention of a batched decode step at the edges of its tiles of 32 positions and of the groups of query heads it takes: the
logits of each sequence against the same sequence decoded alone (1e-2, one int8 step of a requantised activation)."""
import numpy as np
import pytest

from spbitnet_b200 import synth
from spbitnet_b200.engine import DeviceModel, InferenceEngine
from spbitnet_b200.shard_engine import ShardEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(2, 2, 64), (4, 1, 128), (8, 1, 64), (6, 2, 128), (4, 1, 32), (10, 1, 64)])
def test_each_sequence_alone(heads, kv_heads, head_dim):
    cfg = dict(synth.TINY, num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=head_dim, hidden_size=256,
               max_position_embeddings=128)
    model = DeviceModel(synth.random_model(cfg, seed=heads))
    steps, batch = 67, 3
    tokens = np.random.default_rng(head_dim).integers(0, cfg["vocab_size"], (steps, batch)).astype(np.int32)
    together, alone = ShardEngine(model, batch=batch), InferenceEngine(model)
    got = {}
    for i in range(steps):
        together.step(tokens[i])
        if i + 1 in (1, 2, 31, 32, 33, 64, 65, 67):
            got[i + 1] = together.logits().copy()
    for b in range(batch):
        alone.reset()
        for i in range(steps):
            alone.forward(int(tokens[i, b]))
            if i + 1 in got:
                assert np.abs(got[i + 1][b] - alone.logits()).max() < 1e-2, (b, i + 1)
