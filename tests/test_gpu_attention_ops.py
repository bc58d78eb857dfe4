"""The three attention ops of one token at the edges of their splits: positions per block and blocks per cluster of the output
(64, 128, 256), values per thread and the register limit of the softmax (128, 4096), positions per load of the scores; caches
off the 16-byte boundary take the scalar forms.  float64 references; the bounds are those of fp32 sums (1e-5) and of one half
rounding (2^-11 of the value)."""
import numpy as np
import pytest
import torch

from spbitnet_b200 import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(8, 2, 64), (20, 5, 128), (2, 2, 256), (3, 1, 40), (2, 1, 1536), (4, 2, 12)])
@pytest.mark.parametrize("seq_len", [1, 2, 33, 63, 64, 127, 128, 129, 255, 256, 700, 4096, 4099])
@pytest.mark.parametrize("off", [0, 1])
def test_against_float64(heads, kv_heads, head_dim, seq_len, off):
    if seq_len > 700 and head_dim > 256:
        pytest.skip("a cache of that size adds no edge")
    max_seq = seq_len + 3
    g = torch.Generator(device="cuda")
    g.manual_seed(seq_len + head_dim)
    def half(*shape):
        n = int(np.prod(shape))
        return torch.randn(n + 8, generator=g, device="cuda").half()[off:off + n].view(*shape)
    q, k, v = half(heads, head_dim), half(kv_heads, max_seq, head_dim), half(kv_heads, max_seq, head_dim)
    kv = torch.arange(heads, device="cuda") * kv_heads // heads
    scale = head_dim ** -0.5
    s = torch.full((heads, max_seq), 7.0, device="cuda")
    K.attention_scores_gpu(q, k, s, heads, kv_heads, head_dim, max_seq, seq_len, scale)
    want = torch.einsum("hd,hpd->hp", q.double(), k[kv, :seq_len].double()) * scale
    assert (s[:, :seq_len].double() - want).abs().max() < 1e-5 * max(1.0, want.abs().max().item())
    K.softmax_gpu(s, heads, max_seq, seq_len)
    prob = torch.softmax(want, 1)
    assert ((s[:, :seq_len].double() - prob).abs() < 4e-5 * prob).all()
    assert (s[:, seq_len:] == 7.0).all()
    out = torch.zeros((heads, head_dim), dtype=torch.float16, device="cuda")
    K.attention_output_gpu(s, v, out, heads, kv_heads, head_dim, max_seq, seq_len)
    ref = torch.einsum("hp,hpd->hd", s[:, :seq_len].double(), v[kv, :seq_len].double())
    assert ((out.double() - ref).abs() <= 2.0 ** -11 * ref.abs() + 1e-5).all()
