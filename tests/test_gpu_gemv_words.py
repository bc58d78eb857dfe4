"""GEMV and BitLinear on widths, strides and alignments outside the 128-column kernels: exact against the oracle at the edges of
a 64-column unit, of a warp's 32 units and of the rows a block takes, with rows and activations off every boundary; and against
the reference's table for bitmaps that do not have two bits set."""
import numpy as np
import pytest
import torch

import oracle
from spbitnet_b200 import kernels as K, synth
from gpu_util import Guarded, dev

pytestmark = pytest.mark.gpu


def _offset(words, stride, off):
    """The rows of a word matrix `stride` words apart, the first one `off` words into its buffer."""
    rows, n = words.shape
    buf = np.zeros(off + rows * stride + 8, np.uint32)
    np.lib.stride_tricks.as_strided(buf[off:], (rows, n), (4 * stride, 4))[:] = words
    t = dev(buf)
    return t, t.data_ptr() + 4 * off


@pytest.mark.parametrize("rows,cols", [(1, 4), (3, 60), (5, 64), (7, 68), (300, 132), (2049, 2052), (3001, 3204), (640, 2560),
                                       (17, 16388), (9, 65536), (3, 65540), (9500, 516)])
@pytest.mark.parametrize("off", [0, 1])
def test_gemv_and_bitlinear(rows, cols, off):
    case = synth.gemv_case(rows, cols, seed=rows + cols)
    ms, vs = case["meta_stride"] + off, case["values_stride"] + off
    km, meta = _offset(case["meta"].reshape(rows, -1), ms, off)
    kv, values = _offset(case["values"].reshape(rows, -1), vs, off)
    xb = torch.zeros(cols + 16, dtype=torch.int8, device="cuda")
    xb[off:off + cols] = dev(case["x"])
    y = Guarded(rows * 4)
    K.sparse_ternary_gemv_gpu(meta, values, xb.data_ptr() + off, y.ptr, rows, cols, ms, vs)
    want = oracle.sparse_gemv(case["meta"], case["values"], case["x"], rows, cols, threads=4)
    assert (y.read(np.int32) == want).all()
    x = (np.random.default_rng(cols).standard_normal(cols) * 2).astype(np.float16)
    hb = torch.zeros(cols + 16, dtype=torch.float16, device="cuda")
    hb[off:off + cols] = dev(x)
    absmax = oracle.absmax_reduce(x)
    out = Guarded(rows * 2)
    K.fused_sparse_bitlinear_gpu(meta, values, hb.data_ptr() + 2 * off, out.ptr, dev(np.array([absmax], np.float32)), 0.03, rows,
                                 cols, ms, vs)
    want_h = oracle.fused_bitlinear(case["meta"], case["values"], x, absmax, 0.03, rows, cols)
    assert (out.read(np.float16).view(np.uint16) == want_h.view(np.uint16)).all()
    del km, kv


def test_bitmaps_without_two_bits_decode_as_the_table_has_them():
    rows, cols = 40, 68
    rng = np.random.default_rng(0)
    meta = rng.integers(0, 2**32, (rows, 3), dtype=np.uint64).astype(np.uint32)
    values = rng.integers(0, 2**32, (rows, 2), dtype=np.uint64).astype(np.uint32)
    x = rng.integers(-127, 128, cols).astype(np.int8)
    want = np.zeros(rows, np.int64)
    for g in range(cols // 4):
        b = (meta[:, g // 8] >> np.uint32(4 * (g % 8))) & 15
        s = (values[:, g // 16] >> np.uint32(2 * (g % 16))) & 3
        for r in range(rows):
            pos = [i for i in range(4) if (int(b[r]) >> i) & 1]
            p0, p1 = pos if len(pos) == 2 else (0, 0)
            want[r] += (-1 if s[r] & 1 else 1) * int(x[4 * g + p0]) + (-1 if s[r] & 2 else 1) * int(x[4 * g + p1])
    y = Guarded(rows * 4)
    K.sparse_ternary_gemv_gpu(dev(meta), dev(values), dev(x), y.ptr, rows, cols, 3, 2)
    assert (y.read(np.int32) == want).all()
