"""The prompt attention kernel's own output against float64: weights far below the row's largest, scores of both signs and
sizes, and values that are not finite, at positions a row sees and at ones it does not."""
import numpy as np
import pytest
import torch

from spbitnet_b200 import kernels as K

pytestmark = pytest.mark.gpu


def _run(q, k, v, first, scale):
    T, nh, hd = q.shape
    nkv, max_seq, _ = k.shape
    out = torch.full_like(q, 7.0)
    K.debug_prefill_attention(q, k, v, out, T, nh, nkv, hd, max_seq, scale, torch.tensor([first], dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    return out


def _exact(q, k, v, first, scale):
    """Row by row over the positions the row sees, float64."""
    T, nh, hd = q.shape
    group = nh // k.shape[0]
    out = torch.empty((T, nh, hd), dtype=torch.float64, device="cuda")
    kd, vd = k.double().repeat_interleave(group, 0), v.double().repeat_interleave(group, 0)
    for t in range(T):
        n = first + t + 1
        w = torch.softmax(torch.einsum("hd,hnd->hn", q[t].double(), kd[:, :n]) * scale, -1)
        out[t] = torch.einsum("hn,hnd->hd", w, vd[:, :n])
    return out


@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("bits", [13, 20, 26, 28])
def test_many_small_weights(head_dim, bits):
    """One position with nearly all of the weight and a value of zero, thousands with a weight of 2^-bits of it: their sum is
    the output.  Rounded to half (2^-11) it has to be right to 2^-11 + what 22 bits of each weight lose."""
    n, T, nh, nkv = 4000, 20, 4, 2
    scale = head_dim ** -0.5
    q = torch.zeros((T, nh, head_dim), dtype=torch.float16, device="cuda")
    k = torch.zeros((nkv, 4096, head_dim), dtype=torch.float16, device="cuda")
    v = torch.ones_like(k)
    q[..., 0] = 1.0
    k[:, 0, 0] = bits * np.log(2.0) / scale
    v[:, 0] = 0.0
    got, want = _run(q, k, v, n, scale).double(), _exact(q, k, v, n, scale)
    assert ((got - want).abs() <= 2.0 ** -10.9 * want + 2.0 ** -25).all()


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(3, 3, 64), (4, 1, 128), (8, 1, 64), (6, 2, 128)])
@pytest.mark.parametrize("spread", [0.2, 1.0, 6.0])
def test_random(heads, kv_heads, head_dim, spread):
    """2^-11 of the value for its rounding to half; sums of up to 700 fp32 products and weights with a relative error of 2^-20
    or so from the exponential of a score of up to 200 add 2^-18 of the largest value."""
    g = torch.Generator(device="cuda")
    g.manual_seed(heads)
    first, T = 601, 99
    q, k, v = ((s * torch.randn(shape, generator=g, device="cuda")).half()
               for s, shape in [(spread, (T, heads, head_dim)), (1.0, (kv_heads, 768, head_dim)), (1.0, (kv_heads, 768, head_dim))])
    scale = head_dim ** -0.5
    got, want = _run(q, k, v, first, scale).double(), _exact(q, k, v, first, scale)
    assert ((got - want).abs() <= 2.0 ** -10.9 * want.abs() + 2.0 ** -16).all()


def test_long_sequence_without_bias():
    """Equal weights over thousands of positive values: sums that a tensor core accumulates over the whole sequence come out low by
    a few 2^-16 (each addition is cut off, not rounded), enough to move one rounding to half in thirty.  Rounded once, an fp32
    result moves one in a few hundred."""
    heads, kv_heads, head_dim, T, first = 4, 2, 128, 32, 4000
    g = torch.Generator(device="cuda")
    g.manual_seed(9)
    q = 0.1 * torch.randn((T, heads, head_dim), generator=g, device="cuda").half()
    k = torch.randn((kv_heads, 4096, head_dim), generator=g, device="cuda").half()
    v = 1.0 + torch.rand((kv_heads, 4096, head_dim), generator=g, device="cuda").half()
    scale = head_dim ** -0.5
    got, want = _run(q, k, v, first, scale), _exact(q, k, v, first, scale)
    assert (got != want.half()).double().mean() < 0.01


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(2, 2, 64), (4, 1, 128), (6, 2, 128)])
@pytest.mark.parametrize("first", [0, 50, 130])
def test_values_that_are_not_finite(heads, kv_heads, head_dim, first):
    """Infinities and NaNs of V reach the rows that see their positions, in their dimension, and no others; a row that sees an
    infinity gets it and not the NaN that a zero weight, or a zero half of a weight, would make of it."""
    g = torch.Generator(device="cuda")
    g.manual_seed(first)
    T = 90
    q, k, v = (torch.randn(shape, generator=g, device="cuda").half()
               for shape in [(T, heads, head_dim), (kv_heads, 256, head_dim), (kv_heads, 256, head_dim)])
    v[:, first + 20, 3] = float("inf")
    v[0, first + 21, 5] = float("-inf")
    v[:, first + 41, 7] = float("nan")
    v[-1, first + 70, 3] = float("-inf")
    v[:, 220] = float("nan")  # past every row
    scale = head_dim ** -0.5
    got, want = _run(q, k, v, first, scale).double(), _exact(q, k, v, first, scale)
    assert torch.isfinite(want[:20]).all() and not torch.isfinite(want[-1]).all()
    assert (torch.isnan(got) == torch.isnan(want)).all()
    assert (got[torch.isinf(want)] == want[torch.isinf(want)]).all()
    ok = torch.isfinite(want)
    assert ((got[ok] - want[ok]).abs() <= 2.0 ** -10.9 * want[ok].abs() + 2.0 ** -16).all()


def test_keys_that_are_not_finite():
    """A NaN or an infinity of K changes the rows that see it only."""
    heads, kv_heads, head_dim, T, first = 4, 2, 64, 70, 10
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    q, k, v = (torch.randn(shape, generator=g, device="cuda").half()
               for shape in [(T, heads, head_dim), (kv_heads, 128, head_dim), (kv_heads, 128, head_dim)])
    scale = head_dim ** -0.5
    clean = _run(q, k, v, first, scale)
    for bad in (float("nan"), float("inf")):
        k2 = k.clone()
        k2[:, first + 33, 2] = bad
        got = _run(q, k2, v, first, scale)
        assert (got[:33] == clean[:33]).all()
        assert torch.isnan(got[33:]).any()
