"""Python mirror of the reference's kernel host wrappers (namespace spbitnet,
include/spbitnet/sparse_ternary_kernels.h and inference_kernels.h): same names, same
argument order, torch CUDA tensors in place of device pointers.  Every function forwards
to the C-ABI of libspbitnet_b200.so (through the CPython module `_calls`); errors raise SpbError instead of exiting.
"""
from __future__ import annotations

import ctypes as C

import torch

from . import _lib
from ._lib import check, load


class _Calls:
    """The kernel entry points: tensors, addresses, None and streams in, SpbError for a status other than 0.  Looked up at the
    first call of each: this module can be imported before the library is built."""

    def __getattr__(self, name):
        fn = getattr(_lib.calls(), name)
        setattr(self, name, fn)
        return fn


_c = _Calls()


def _p(t):
    if t is None:
        return C.c_void_p(0)
    if isinstance(t, int):
        return C.c_void_p(t)
    return C.c_void_p(t.data_ptr())


def _stream(stream):
    if stream is None:
        return C.c_void_p(torch.cuda.current_stream().cuda_stream)
    if isinstance(stream, int):
        return C.c_void_p(stream)
    return C.c_void_p(stream.cuda_stream)


def set_pdl(enabled: bool) -> bool:
    return bool(load().spb_set_pdl(int(enabled)))


def set_gemv_variant(variant: int) -> int:
    """0 automatic, 1 pair kernel, 2 per-group table kernel, 3 tcgen05 sparse kernel, 4 warp-level sparse MMA kernel."""
    return load().spb_set_gemv_variant(int(variant))


def set_gemm_variant(variant: int) -> int:
    """0 automatic, 1 SIMT form, 3 tcgen05 sparse form, 4 warp-level sparse MMA form where it applies, else 3."""
    return load().spb_set_gemm_variant(int(variant))


def set_gemm_row_halves(halves: int) -> int:
    """0 automatic, 1 / 2 weight-row halves per block of the tcgen05 product; returns the previous setting."""
    return load().spb_set_gemm_row_halves(int(halves))


def gemm_tc_timeouts() -> int:
    return load().spb_gemm_tc_timeouts()


def debug_bounded_wait_selftest(limit_cycles: int = 4000, stream=None) -> int:
    """Runs the library's bounded-wait self-test and returns its status code (SPB_E_TIMEOUT is the
    expected answer: the wait ran out, was counted, and the block returned)."""
    return load().spb_debug_bounded_wait_selftest(int(limit_cycles), _stream(stream))


def debug_grid_barrier_selftest(limit_cycles: int = 200000, stream=None) -> int:
    """Two blocks at a grid barrier of the persistent decode step that expects three arrivals: returns
    SPB_E_TIMEOUT when both bounded waits ran out, were counted and the kernel returned."""
    return load().spb_debug_grid_barrier_selftest(int(limit_cycles), _stream(stream))


def debug_prefill_attention(Q, K, V, out, T, num_heads, num_kv_heads, head_dim, max_seq_len, scale, d_pos, stream=None):
    """The prompt attention of InferenceEngine.prefill by itself (testing aid): Q and out (T, heads, head_dim) half, caches
    (kv heads, max_seq_len, head_dim) half, d_pos the first token's position (int32, device)."""
    check(load().spb_debug_prefill_attention(_p(Q), _p(K), _p(V), _p(out), T, num_heads, num_kv_heads, head_dim, max_seq_len,
                                             float(scale), _p(d_pos), _stream(stream)))


# ---- sparse_ternary_kernels.h ---------------------------------------------------------

def sparse_ternary_unpack_gpu(meta, values, out, rows, cols, meta_row_stride, values_row_stride, stream=None):
    _c.spb_sparse_ternary_unpack(meta, values, out, rows, cols, meta_row_stride, values_row_stride, stream)


def sparse_ternary_gemv_gpu(meta, values, x, y, rows, cols, meta_row_stride, values_row_stride, stream=None):
    _c.spb_sparse_ternary_gemv(meta, values, x, y, rows, cols, meta_row_stride, values_row_stride, stream)


def prepared_weights_bytes(rows, cols) -> int:
    return int(load().spb_prepared_weights_bytes(rows, cols))


def prepare_weights(meta, values, rows, cols, meta_row_stride, values_row_stride, stream=None):
    """Packed rows on the device -> the prepared form (a uint8 CUDA tensor) that prepared_gemv_gpu takes."""
    nbytes = prepared_weights_bytes(rows, cols)
    if nbytes == 0:
        raise ValueError(f"prepared weights: shape {rows}x{cols} not taken (cols must be a multiple of 256)")
    out = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    _c.spb_prepare_weights(meta, values, rows, cols, meta_row_stride, values_row_stride, out, stream)
    return out


def prepared_gemv_gpu(prepared, x, y, rows, cols, stream=None):
    _c.spb_prepared_gemv(prepared, x, y, rows, cols, stream)


def prepared_bitlinear_q8_gpu(prepared, xq, out_half, d_absmax, gamma, rows, cols, stream=None):
    _c.spb_prepared_bitlinear_q8(prepared, xq, out_half, d_absmax, gamma, rows, cols, stream)


class GemvWorkList:
    """A device-resident list of GEMVs for sparse_ternary_gemv_batch_gpu.  items: iterable of
    (meta, values, x, y, rows, cols, meta_row_stride, values_row_stride) with CUDA tensors (or
    device addresses) for the first four."""

    def __init__(self, items):
        import numpy as np
        from ._lib import GemvItem
        items = list(items)
        arr = (GemvItem * len(items))()
        for i, (meta, values, x, y, rows, cols, ms, vs) in enumerate(items):
            arr[i] = GemvItem(_p(meta).value, _p(values).value, _p(x).value, _p(y).value, rows, cols, ms, vs)
        check(load().spb_gemv_batch_check(arr, len(items)))
        self.n = len(items)
        self.max_rows = max((it[4] for it in items), default=0)
        self.max_cols = max((it[5] for it in items), default=0)
        raw = np.frombuffer(bytes(arr), dtype=np.uint8).copy() if items else np.zeros(1, np.uint8)
        self.d_items = torch.from_numpy(raw).cuda()
        self._keep = items  # keeps the tensors alive


def sparse_ternary_gemv_batch_gpu(work: GemvWorkList, stream=None):
    _c.spb_sparse_ternary_gemv_batch(work.d_items, work.n, work.max_rows, work.max_cols, stream)


def sparse_ternary_gemv_scaled_gpu(meta, values, x, y, y_acc, d_absmax, gamma, rows, cols, meta_row_stride,
                                   values_row_stride, stream=None):
    _c.spb_sparse_ternary_gemv_scaled(meta, values, x, y, y_acc, d_absmax, gamma, rows, cols, meta_row_stride,
                                      values_row_stride, stream)


def fused_sparse_bitlinear_gpu(meta, values, x, output, d_absmax, gamma, rows, cols, meta_row_stride,
                               values_row_stride, stream=None):
    _c.spb_fused_sparse_bitlinear(meta, values, x, output, d_absmax, gamma, rows, cols, meta_row_stride,
                                  values_row_stride, stream)


def sparse_bitlinear_q8_gpu(meta, values, xq, output, d_absmax, gamma, rows, cols, meta_row_stride,
                            values_row_stride, stream=None):
    _c.spb_sparse_bitlinear_q8(meta, values, xq, output, d_absmax, gamma, rows, cols, meta_row_stride,
                               values_row_stride, stream)


def sparse_ternary_gemm_gpu(meta, values, X, Y, rows, cols, n, meta_row_stride, values_row_stride, stream=None):
    _c.spb_sparse_ternary_gemm(meta, values, X, Y, rows, cols, n, meta_row_stride, values_row_stride, stream)


def sparse_bitlinear_gemm_gpu(meta, values, Xq, output, d_absmax, gamma, rows, cols, n, meta_row_stride,
                              values_row_stride, acc_workspace=None, stream=None):
    """BitLinear over n quantised activation rows (no counterpart in the reference, whose prefill is token-serial):
    output[j] = half(float(W @ Xq[j]) * (gamma * d_absmax[j] / 127)).  acc_workspace: n * rows int32, needed only by
    the forms without a fused epilogue."""
    _c.spb_sparse_bitlinear_gemm(meta, values, Xq, output, d_absmax, gamma, acc_workspace, rows, cols, n, meta_row_stride,
                                 values_row_stride, stream)


# ---- inference_kernels.h ----------------------------------------------------------------

def rms_norm_gpu(input, weight, output, size, eps, stream=None):
    _c.spb_rms_norm(input, weight, output, size, eps, stream)


def absmax_quantize_gpu(input, output, d_absmax, size, stream=None):
    _c.spb_absmax_quantize(input, output, d_absmax, size, stream)


def absmax_reduce_gpu(input, d_absmax, size, stream=None):
    _c.spb_absmax_reduce(input, d_absmax, size, stream)


def dequantize_gpu(input, output, d_absmax, gamma, size, stream=None):
    _c.spb_dequantize(input, output, d_absmax, gamma, size, stream)


def rope_gpu(vec, num_heads, head_dim, pos, theta, stream=None):
    _c.spb_rope(vec, num_heads, head_dim, pos, theta, stream)


def scatter_kv_gpu(src, cache, num_kv_heads, head_dim, max_seq_len, pos, stream=None):
    _c.spb_scatter_kv(src, cache, num_kv_heads, head_dim, max_seq_len, pos, stream)


def attention_scores_gpu(Q, K_cache, scores, num_heads, num_kv_heads, head_dim, max_seq_len, seq_len, scale,
                         stream=None):
    _c.spb_attention_scores(Q, K_cache, scores, num_heads, num_kv_heads, head_dim, max_seq_len, seq_len, scale, stream)


def softmax_gpu(scores, num_heads, max_seq_len, seq_len, stream=None):
    _c.spb_softmax(scores, num_heads, max_seq_len, seq_len, stream)


def attention_output_gpu(scores, V_cache, output, num_heads, num_kv_heads, head_dim, max_seq_len, seq_len,
                         stream=None):
    _c.spb_attention_output(scores, V_cache, output, num_heads, num_kv_heads, head_dim, max_seq_len, seq_len, stream)


def decode_attention_gpu(Q, K_cache, V_cache, output, num_heads, num_kv_heads, head_dim, max_seq_len, seq_len,
                         scale, stream=None):
    _c.spb_decode_attention(Q, K_cache, V_cache, output, num_heads, num_kv_heads, head_dim, max_seq_len, seq_len, scale,
                            stream)


def decode_attention_scratch_bytes(num_heads, head_dim, max_seq_len) -> int:
    return int(load().spb_decode_attention_scratch_bytes(num_heads, head_dim, max_seq_len))


def decode_attention_split_gpu(Q, K_cache, V_cache, output, num_heads, num_kv_heads, head_dim, max_seq_len, seq_len,
                               scale, scratch, stream=None):
    nbytes = scratch.numel() * scratch.element_size()
    _c.spb_decode_attention_split(Q, K_cache, V_cache, output, num_heads, num_kv_heads, head_dim, max_seq_len, seq_len,
                                  scale, scratch, nbytes, stream)


def relu2_mul_gpu(gate, up, output, size, stream=None):
    _c.spb_relu2_mul(gate, up, output, size, stream)


def relu2_mul_f32_gpu(gate, up, output, size, stream=None):
    _c.spb_relu2_mul_f32(gate, up, output, size, stream)


def rms_norm_f32in_gpu(input, weight, output, size, eps, stream=None):
    _c.spb_rms_norm_f32in(input, weight, output, size, eps, stream)


def float_to_half_gpu(input, output, size, stream=None):
    _c.spb_float_to_half(input, output, size, stream)


def residual_add_gpu(a, b, output, size, stream=None):
    _c.spb_residual_add(a, b, output, size, stream)


def half_gemv_gpu(W, x, y, rows, cols, stream=None):
    _c.spb_half_gemv(W, x, y, rows, cols, stream)


# ---- conversion on the GPU (no counterpart among the reference's GPU wrappers) -----------------

def prune_pack_gpu(weights, stream=None):
    """Magnitude 2:4 pruning + sign extraction + packing of a CUDA float32 matrix, byte-identical to
    python/convert_model.py (generate_24_mask, quantize_ternary_absmean, the zero-at-mask fix,
    pack_sparse_ternary).  Returns (meta, values, gamma): int32 CUDA tensors holding the uint32 words,
    and gamma = mean |w| accumulated in double precision."""
    import torch
    assert weights.is_cuda and weights.dtype == torch.float32 and weights.dim() == 2 and weights.stride(1) == 1
    rows, cols = weights.shape
    ms, vs = (cols // 4 + 7) // 8, (cols // 4 + 15) // 16
    meta = torch.empty((rows, ms), dtype=torch.int32, device=weights.device)  # every word of the tight rows is written
    values = torch.empty((rows, vs), dtype=torch.int32, device=weights.device)
    abs_sum = torch.zeros(1, dtype=torch.float64, device=weights.device)
    _c.spb_prune_pack_gpu(weights, rows, cols, weights.stride(0), meta, values, ms, vs, abs_sum, stream)
    gamma = float(abs_sum.item()) / max(1, rows * cols)
    return meta, values, gamma
