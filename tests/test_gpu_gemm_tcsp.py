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
