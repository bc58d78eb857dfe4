"""The tcgen05 product at the edges of its tiles and of its split: row and batch tails, one step of K and ranges that do not
divide over a cluster, widths that are no multiple of a word, unaligned operands.  Integer sums: exact."""
import numpy as np
import pytest
import torch

import oracle
from spbitnet_b200 import kernels as K, synth
from gpu_util import Guarded, dev

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def tcgen05_form():
    old = K.set_gemm_variant(3)
    before = K.gemm_tc_timeouts()
    yield
    K.set_gemm_variant(old)
    assert K.gemm_tc_timeouts() == before


@pytest.mark.parametrize("rows,cols,n", [(1, 4, 1), (128, 256, 16), (127, 512, 17), (129, 768, 1), (130, 2560, 15),
                                         (256, 16384, 3), (640, 2304, 65), (384, 6912, 200), (20, 28672, 24),
                                         (300, 272, 33), (301, 132, 40), (37, 3204, 129), (513, 1036, 257)])
def test_sums_and_scaled_half(rows, cols, n):
    case = synth.gemm_case(rows, cols, n, seed=rows * 31 + n)
    want = oracle.sparse_gemm(case["meta"], case["values"], case["X"], rows, cols)
    Y = Guarded(n * rows * 4)
    K.sparse_ternary_gemm_gpu(dev(case["meta"]), dev(case["values"]), dev(case["X"]), Y.ptr, rows, cols, n,
                              case["meta_stride"], case["values_stride"])
    assert (Y.read(np.int32).reshape(n, rows) == want).all()
    out, ws = Guarded(n * rows * 2), Guarded(n * rows * 4)
    K.sparse_bitlinear_gemm_gpu(dev(case["meta"]), dev(case["values"]), dev(case["X"]), out.ptr, dev(case["absmax"]), 0.05,
                                rows, cols, n, case["meta_stride"], case["values_stride"], acc_workspace=ws.ptr)
    wh = np.stack([oracle.dequantize(want[j], case["absmax"][j], np.float32(0.05)) for j in range(n)])
    assert (out.read(np.float16).reshape(n, rows).view(np.uint16) == wh.view(np.uint16)).all()


def test_unaligned_operands_and_padded_rows():
    rows, cols, n = 150, 640, 21
    case = synth.gemm_case(rows, cols, n, seed=4)
    want = oracle.sparse_gemm(case["meta"], case["values"], case["X"], rows, cols)
    ms, vs = case["meta_stride"], case["values_stride"]
    for pad_m, pad_v, shift in [(4, 2, 0), (1, 3, 0), (0, 0, 1), (12, 10, 3)]:
        meta = np.full((rows, ms + pad_m), 0xFFFFFFFF, np.uint32)  # the padding is never used
        values = np.full((rows, vs + pad_v), 0xFFFFFFFF, np.uint32)
        meta[:, :ms], values[:, :vs] = case["meta"], case["values"]
        x = torch.zeros(n * cols + 16, dtype=torch.int8, device="cuda")
        x[shift:shift + n * cols] = dev(case["X"]).flatten()
        Y = Guarded(n * rows * 4, align_offset=4 * shift)
        K.sparse_ternary_gemm_gpu(dev(meta), dev(values), x.data_ptr() + shift, Y.ptr, rows, cols, n, ms + pad_m, vs + pad_v)
        assert (Y.read(np.int32).reshape(n, rows) == want).all(), (pad_m, pad_v, shift)


@pytest.mark.parametrize("halves", [1, 2])
@pytest.mark.parametrize("rows,cols,n", [(1, 128, 1), (127, 384, 17), (129, 640, 200), (257, 1408, 33), (301, 3200, 260),
                                         (520, 4992, 16), (33, 65408, 5)])
def test_sign_rows_on_eight_byte_boundaries(rows, cols, n, halves):
    """Widths that are odd multiples of 128: tight sign rows are 8 bytes off the 16-byte boundaries every other row.  Tight rows,
    rows on 16-byte boundaries from a base that is not, and padding that must not be read."""
    case = synth.gemm_case(rows, cols, n, seed=rows + cols)
    want = oracle.sparse_gemm(case["meta"], case["values"], case["X"], rows, cols)
    wh = np.stack([oracle.dequantize(want[j], case["absmax"][j], np.float32(0.05)) for j in range(n)])
    ms, vs = case["meta_stride"], case["values_stride"]
    meta, x, absmax = dev(case["meta"]), dev(case["X"]), dev(case["absmax"])
    old = K.set_gemm_row_halves(halves)
    try:
        for stride, shift in [(vs, 0), (vs + 2, 2), (vs + 8, 0)]:
            flat = np.full(rows * stride + shift, 0xFFFFFFFF, np.uint32)
            flat[shift:].reshape(rows, stride)[:, :vs] = case["values"]
            values = dev(flat)
            Y = Guarded(n * rows * 4)
            K.sparse_ternary_gemm_gpu(meta, values.data_ptr() + 4 * shift, x, Y.ptr, rows, cols, n, ms, stride)
            assert (Y.read(np.int32).reshape(n, rows) == want).all(), (stride, shift)
            out, ws = Guarded(n * rows * 2), Guarded(n * rows * 4)
            K.sparse_bitlinear_gemm_gpu(meta, values.data_ptr() + 4 * shift, x, out.ptr, absmax, 0.05, rows, cols, n, ms, stride,
                                        acc_workspace=ws.ptr)
            assert (out.read(np.float16).reshape(n, rows).view(np.uint16) == wh.view(np.uint16)).all(), (stride, shift)
    finally:
        K.set_gemm_row_halves(old)


@pytest.mark.parametrize("rows,cols,n,pad", [(40, 68, 5, 0), (300, 132, 40, 0), (130, 272, 17, 2), (150, 640, 21, 1), (257, 1036, 33, 0)])
def test_bitmaps_without_two_bits_decode_as_the_table_has_them(rows, cols, n, pad):
    """Layouts outside whole 128-column rows: any bitmap, both signs on the first column where it has not two bits set."""
    rng = np.random.default_rng(rows)
    ms, vs = (cols // 4 + 7) // 8 + pad, (cols // 4 + 15) // 16 + pad
    if pad == 2:
        ms, vs = (ms + 3) // 4 * 4, (vs + 3) // 4 * 4  # tensor maps take these rows
    case = synth.gemm_case(rows, cols, n, seed=7)
    meta = np.zeros((rows, ms), np.uint32)
    values = rng.integers(0, 2**32, (rows, vs), dtype=np.uint64).astype(np.uint32)
    meta[:, :case["meta"].reshape(rows, -1).shape[1]] = case["meta"].reshape(rows, -1)
    for r in range(0, rows, 3):  # every third row: any bits in the row's own groups
        for g in range(cols // 4):
            meta[r, g // 8] = (int(meta[r, g // 8]) & ~(15 << (4 * (g % 8)))) | (int(rng.integers(0, 16)) << (4 * (g % 8)))
    x = rng.integers(-127, 128, (n, cols)).astype(np.int8)
    w = np.zeros((rows, cols), np.int64)
    g = np.arange(cols // 4)
    b = (meta[:, g // 8] >> (4 * (g % 8)).astype(np.uint32)) & 15
    s = (values[:, g // 16] >> (2 * (g % 16)).astype(np.uint32)) & 3
    for r in range(rows):
        for k in g:
            pos = [i for i in range(4) if (int(b[r, k]) >> i) & 1]
            p0, p1 = pos if len(pos) == 2 else (0, 0)
            w[r, 4 * k + p0] += -1 if s[r, k] & 1 else 1
            w[r, 4 * k + p1] += -1 if s[r, k] & 2 else 1
    Y = Guarded(n * rows * 4)
    K.sparse_ternary_gemm_gpu(dev(meta), dev(values), dev(x), Y.ptr, rows, cols, n, ms, vs)
    assert (Y.read(np.int32).reshape(n, rows) == x.astype(np.int64) @ w.T).all()
