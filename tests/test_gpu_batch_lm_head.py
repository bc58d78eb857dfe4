"""The batched LM head at the edges of its tiles (256 rows, 64 columns, 16 vectors): the logits of one step of a batch equal
each sequence's own step, whose LM head is the single-vector kernel, to the rounding of fp32 sums of another order
(hidden terms of size |w x| <= 0.1 * 6, 2^-24 relative each: 2e-5)."""
import numpy as np
import pytest

from spbitnet_b200 import synth
from spbitnet_b200.engine import DeviceModel, InferenceEngine
from spbitnet_b200.shard_engine import ShardEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,vocab,batch", [(128, 256, 2), (256, 257, 16), (320, 511, 17), (256, 1001, 64), (64, 33, 33)])
def test_batched_logits_equal_single(hidden, vocab, batch):
    cfg = dict(synth.TINY, hidden_size=hidden, vocab_size=vocab, num_hidden_layers=0)  # embedding, final norm, LM head
    dm = DeviceModel(synth.random_model(cfg, seed=vocab))
    together, alone = ShardEngine(dm, batch=batch), InferenceEngine(dm)
    tokens = np.random.default_rng(batch).integers(0, vocab, batch).astype(np.int32)
    together.step(tokens)
    got = together.logits_rows()
    for b in range(batch):
        alone.reset()
        alone.forward(int(tokens[b]))
        assert np.abs(got[b] - alone.logits()).max() < 2e-5, b
