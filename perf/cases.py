"""The work that users of this framework have it do, as measurable cases.

Kinds (``case["kind"]``), each through the public Python entry points:

  gemv      one ternary matrix times one int8 vector, int32 sums (kernels.sparse_ternary_gemv_gpu)
  bitlinear absmax_reduce_gpu + fused_sparse_bitlinear_gpu on a half vector: one projection of a decode step as an
            engine that drives the kernels itself calls it
  gemm      one ternary matrix times n int8 rows: int32 sums (sparse_ternary_gemm_gpu) or the scaled half result
            (sparse_bitlinear_gemm_gpu)
  layer     one decoder layer for one token, op by op in the order of the reference's forward pass
  prefill   InferenceEngine: reset, a prompt as one batch, the last token's logits to the host
  chat      InferenceEngine: reset, a prompt, then tokens one at a time, the caller choosing each from the host logits
  batch     ShardEngine on one GPU: several sequences decoded in lock step, their logits to the host at the end
  convert   float weights to the packed format (kernels.prune_pack_gpu)
"""
import math

import torch

from spbitnet_b200 import kernels as K
from spbitnet_b200 import synth
from spbitnet_b200.engine import InferenceEngine
from spbitnet_b200.shard_engine import ShardEngine

# hidden, inter, heads, kv_heads, head_dim, vocab of the model shapes that the configurations and tests use
_MODELS = {
    "tiny": (256, 512, 4, 2, 64, 512),
    "small": (2048, 5632, 16, 4, 128, 32000),
    "2b": (2560, 6912, 20, 5, 128, 128256),
    "wide": (8192, 28672, 64, 8, 128, 128256),
}
_MAX_SEQ = 4096
_EPS, _THETA = 1e-5, 500000.0


def listed():
    return [
        # the smallest projection of the 2B-4T shape (k/v): a call is mostly latency
        {"name": "gemv_640x2560", "kind": "gemv", "rows": 640, "cols": 2560},
        # the largest matrix of the configurations (gate/up of the 70B shape), the packed rows streamed once
        {"name": "gemv_28672x8192", "kind": "gemv", "rows": 28672, "cols": 8192},
        # a projection whose sizes fit no tile: a pruned or odd model dimension
        {"name": "bitlinear_3001x3204", "kind": "bitlinear", "rows": 3001, "cols": 3204},
        # a small serving batch on one FFN matrix
        {"name": "gemm_6912x2560_n16", "kind": "gemm", "rows": 6912, "cols": 2560, "n": 16, "half": False},
        # a ragged batch of prompt rows through the FFN down projection, scaled half output
        {"name": "gemm_2560x6912_n200", "kind": "gemm", "rows": 2560, "cols": 6912, "n": 200, "half": True},
        # the largest product: a full chunk of rows through the largest matrix
        {"name": "gemm_28672x8192_n1024", "kind": "gemm", "rows": 28672, "cols": 8192, "n": 1024, "half": True},
        # the reference's host code on this library: one call per op, 700 tokens into a conversation
        {"name": "layer_2b_pos700", "kind": "layer", "model": "2b", "pos": 700},
        # the prompt lengths of a question and of a document
        {"name": "prefill_2b_128", "kind": "prefill", "model": "2b", "layers": 30, "prompt": 128},
        {"name": "prefill_2b_1800", "kind": "prefill", "model": "2b", "layers": 30, "prompt": 1800},
        # a chat turn with a sampler on the host
        {"name": "chat_2b_37_24", "kind": "chat", "model": "2b", "layers": 30, "prompt": 37, "tokens": 24},
        # serving many sequences of the wide shape (a few of its layers)
        {"name": "batch_wide_64", "kind": "batch", "model": "wide", "layers": 4, "batch": 64, "steps": 16},
        # converting a checkpoint matrix
        {"name": "convert_8192x8192", "kind": "convert", "rows": 8192, "cols": 8192},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """A matrix dimension: mostly a multiple of 256 as models have, now and then any multiple of four."""
    v = _log(rng, lo, hi)
    return max(256, v // 256 * 256) if rng.random() < 0.75 else max(4, v // 4 * 4)


def draw(rng):
    kind = rng.choice(["gemv", "bitlinear", "gemm", "gemm", "layer", "prefill", "chat", "batch", "convert"])
    if kind in ("gemv", "bitlinear"):
        return {"kind": kind, "rows": _log(rng, 256, 28672), "cols": _size(rng, 512, 8192)}
    if kind == "gemm":
        return {"kind": kind, "rows": _log(rng, 256, 28672), "cols": _size(rng, 512, 8192), "n": _log(rng, 2, 1024),
                "half": rng.random() < 0.5}
    if kind == "layer":
        return {"kind": kind, "model": rng.choice(["small", "2b"]), "pos": _log(rng, 8, 4000)}
    if kind in ("prefill", "chat"):
        model = rng.choice(["tiny", "small", "2b"])
        case = {"kind": kind, "model": model, "layers": rng.randint(2, 6 if model == "tiny" else 30)}
        if kind == "prefill":
            return dict(case, prompt=_log(rng, 4, 1800))
        return dict(case, prompt=_log(rng, 4, 900), tokens=rng.randint(4, 24))
    if kind == "batch":
        return {"kind": kind, "model": rng.choice(["2b", "wide"]), "layers": rng.randint(2, 4),
                "batch": _log(rng, 2, 64), "steps": rng.randint(4, 16)}
    return {"kind": kind, "rows": _log(rng, 256, 8192), "cols": _size(rng, 512, 8192)}


def _config(case):
    h, inter, nh, nkv, hd, vocab = _MODELS[case["model"]]
    return dict(hidden_size=h, num_hidden_layers=case.get("layers", 1), num_attention_heads=nh, num_key_value_heads=nkv,
                head_dim=hd, intermediate_size=inter, vocab_size=vocab, max_position_embeddings=_MAX_SEQ,
                rms_norm_eps=_EPS, rope_theta=_THETA)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _randint(g, lo, hi, shape, dtype):
    return torch.randint(lo, hi, shape, generator=g, device="cuda").to(dtype)


def _matrix(rows, cols, seed):
    """Packed rows of one ternary matrix; a width that is no multiple of 64 is converted from floats."""
    if cols % 64 == 0:
        return synth.device_sparse_matrix(rows, cols, seed)
    meta, values, _ = K.prune_pack_gpu(torch.randn((rows, cols), generator=_gen(seed), device="cuda"))
    return meta, values


def prepare(case, seed):
    kind, g = case["kind"], _gen(seed)
    s = {"kind": kind}
    if kind in ("gemv", "bitlinear", "gemm"):
        rows, cols = case["rows"], case["cols"]
        meta, values = _matrix(rows, cols, seed)
        n = case.get("n", 1)
        s.update(rows=rows, cols=cols, n=n, meta=meta, values=values, ms=meta.shape[1], vs=values.shape[1],
                 half=case.get("half", kind == "bitlinear"), gamma=1.0 / math.sqrt(cols))
        if kind == "bitlinear":
            s["x"] = torch.randn(cols, generator=g, device="cuda").half()
            s["absmax"] = torch.zeros(1, device="cuda")
        else:
            s["x"] = _randint(g, -127, 128, (n, cols), torch.int8)
            s["absmax"] = 0.5 + 3.5 * torch.rand(n, generator=g, device="cuda")
        s["y"] = torch.zeros((n, rows), dtype=torch.float16 if s["half"] else torch.int32, device="cuda")
        if kind == "gemm" and s["half"]:
            s["acc"] = torch.empty((n, rows), dtype=torch.int32, device="cuda")
    elif kind == "layer":
        cfg = _config(case)
        s.update(_layer_state(synth.DeviceRandomModel(cfg, seed=seed), cfg, case["pos"], g))
    elif kind in ("prefill", "chat"):
        cfg = _config(case)
        # one random layer, every further layer a device copy of it: each still streams its own bytes
        s["engine"] = InferenceEngine(synth.DeviceRandomModel(cfg, seed=seed, repeat_layer=True))
        s["prompt"] = _randint(g, 0, cfg["vocab_size"], (case["prompt"],), torch.int32).cpu().numpy()
        s["tokens"] = _randint(g, 0, cfg["vocab_size"], (case.get("tokens", 0),), torch.int32).tolist()
    elif kind == "batch":
        cfg = _config(case)
        s["engine"] = ShardEngine(synth.DeviceRandomModel(cfg, seed=seed, repeat_layer=True), batch=case["batch"])
        s["tokens"] = _randint(g, 0, cfg["vocab_size"], (case["steps"], case["batch"]), torch.int32).cpu().numpy()
    else:
        s["w"] = 0.02 * torch.randn((case["rows"], case["cols"]), generator=g, device="cuda")
    return s


def _layer_state(model, cfg, pos, g):
    """The buffers that a program keeps which drives the reference's forward pass op by op."""
    hd, nkv = cfg["head_dim"], cfg["num_key_value_heads"]
    q, kv = cfg["num_attention_heads"] * hd, nkv * hd

    def half(n):
        return torch.zeros(n, dtype=torch.float16, device="cuda")

    layer = model.layers[0]
    cache = [torch.zeros((nkv, _MAX_SEQ, hd), dtype=torch.float16, device="cuda") for _ in range(2)]
    for c in cache:
        c[:, :pos] = torch.randn((nkv, pos, hd), generator=g, device="cuda").half()
    return {"cfg": cfg, "pos": pos, "linear": layer["linear"], "norm": layer["norm"], "k_cache": cache[0],
            "v_cache": cache[1], "x_in": torch.randn(cfg["hidden_size"], generator=g, device="cuda").half(),
            "x": half(cfg["hidden_size"]), "normed": half(cfg["hidden_size"]), "q": half(q), "k": half(kv),
            "v": half(kv), "attn": half(q), "o": half(cfg["hidden_size"]), "gate": half(cfg["intermediate_size"]),
            "up": half(cfg["intermediate_size"]), "act": torch.zeros(cfg["intermediate_size"], device="cuda"),
            "ffn": half(cfg["intermediate_size"]), "down": half(cfg["hidden_size"]),
            "scores": torch.zeros((cfg["num_attention_heads"], _MAX_SEQ), device="cuda"),
            "absmax": torch.zeros(1, device="cuda")}


def _bitlinear(s, i, x, y):
    t = s["linear"][i]
    K.absmax_reduce_gpu(x, s["absmax"], t["cols"])
    K.fused_sparse_bitlinear_gpu(t["d_meta"], t["d_values"], x, y, s["absmax"], t["gamma"], t["rows"], t["cols"],
                                 t["meta_stride"], t["values_stride"])


def _run_layer(s):
    cfg, pos = s["cfg"], s["pos"]
    h, inter, hd = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"]
    nh, nkv = cfg["num_attention_heads"], cfg["num_key_value_heads"]
    K.rms_norm_gpu(s["x_in"], s["norm"][0], s["normed"], h, _EPS)
    _bitlinear(s, 0, s["normed"], s["q"])
    _bitlinear(s, 1, s["normed"], s["k"])
    _bitlinear(s, 2, s["normed"], s["v"])
    K.rope_gpu(s["q"], nh, hd, pos, _THETA)
    K.rope_gpu(s["k"], nkv, hd, pos, _THETA)
    K.scatter_kv_gpu(s["k"], s["k_cache"], nkv, hd, _MAX_SEQ, pos)
    K.scatter_kv_gpu(s["v"], s["v_cache"], nkv, hd, _MAX_SEQ, pos)
    K.attention_scores_gpu(s["q"], s["k_cache"], s["scores"], nh, nkv, hd, _MAX_SEQ, pos + 1, 1.0 / math.sqrt(hd))
    K.softmax_gpu(s["scores"], nh, _MAX_SEQ, pos + 1)
    K.attention_output_gpu(s["scores"], s["v_cache"], s["attn"], nh, nkv, hd, _MAX_SEQ, pos + 1)
    _bitlinear(s, 3, s["attn"], s["o"])
    K.rms_norm_gpu(s["o"], s["norm"][2], s["o"], h, _EPS)
    K.residual_add_gpu(s["x_in"], s["o"], s["x"], h)
    K.rms_norm_gpu(s["x"], s["norm"][1], s["normed"], h, _EPS)
    _bitlinear(s, 4, s["normed"], s["gate"])
    _bitlinear(s, 5, s["normed"], s["up"])
    K.relu2_mul_f32_gpu(s["gate"], s["up"], s["act"], inter)
    K.rms_norm_f32in_gpu(s["act"], s["norm"][3], s["ffn"], inter, _EPS)
    _bitlinear(s, 6, s["ffn"], s["down"])
    K.residual_add_gpu(s["x"], s["down"], s["x"], h)
    return {"x": s["x"], "k_cache": s["k_cache"], "v_cache": s["v_cache"]}


def run(s):
    kind = s["kind"]
    if kind == "gemv":
        K.sparse_ternary_gemv_gpu(s["meta"], s["values"], s["x"], s["y"], s["rows"], s["cols"], s["ms"], s["vs"])
        return s["y"]
    if kind == "bitlinear":
        K.absmax_reduce_gpu(s["x"], s["absmax"], s["cols"])
        K.fused_sparse_bitlinear_gpu(s["meta"], s["values"], s["x"], s["y"], s["absmax"], s["gamma"], s["rows"],
                                     s["cols"], s["ms"], s["vs"])
        return s["y"]
    if kind == "gemm" and s["half"]:
        K.sparse_bitlinear_gemm_gpu(s["meta"], s["values"], s["x"], s["y"], s["absmax"], s["gamma"], s["rows"],
                                    s["cols"], s["n"], s["ms"], s["vs"], acc_workspace=s["acc"])
        return s["y"]
    if kind == "gemm":
        K.sparse_ternary_gemm_gpu(s["meta"], s["values"], s["x"], s["y"], s["rows"], s["cols"], s["n"], s["ms"], s["vs"])
        return s["y"]
    if kind == "layer":
        return _run_layer(s)
    if kind == "convert":
        return K.prune_pack_gpu(s["w"])
    engine = s["engine"]
    engine.reset()
    if kind == "batch":
        for t in s["tokens"]:
            engine.step(t)
        return engine.logits_rows()
    engine.prefill(s["prompt"])
    logits = [engine.logits()]
    for t in s["tokens"]:
        engine.forward(t)
        logits.append(engine.logits())
    return logits


def work(case):
    """Bytes that have to cross HBM once and operations on the weights that are kept (two per multiply-add)."""
    kind = case["kind"]
    if kind == "convert":
        n = case["rows"] * case["cols"]
        return {"bytes": n * (4 + 0.1875), "flops": n}
    if kind in ("gemv", "bitlinear", "gemm"):
        rows, cols, n = case["rows"], case["cols"], case.get("n", 1)
        x = 2 if kind == "bitlinear" else 1
        y = 2 if case.get("half", kind == "bitlinear") else 4
        return {"bytes": 0.1875 * rows * cols + n * (x * cols + y * rows), "flops": rows * cols * n}
    cfg = _config(case)
    weights = sum(r * c for r, c in synth.linear_shapes(cfg)) * cfg["num_hidden_layers"]
    kv = 2 * cfg["num_key_value_heads"] * cfg["head_dim"] * cfg["num_hidden_layers"]  # values per position
    att = 4 * cfg["num_attention_heads"] * cfg["head_dim"] * cfg["num_hidden_layers"]  # operations per position pair
    head = cfg["vocab_size"] * cfg["hidden_size"]
    if kind == "layer":
        p = case["pos"] + 1
        return {"bytes": 0.1875 * weights + 2 * kv * p, "flops": weights + att * p}
    if kind == "batch":
        b, n = case["batch"], case["steps"]
        pairs = b * n * (n + 1) / 2
        return {"bytes": n * (0.1875 * weights + 2 * head) + 2 * kv * (b * n + pairs),
                "flops": b * n * (weights + 2 * head) + att * pairs}
    p, n = case["prompt"], case.get("tokens", 0)
    pairs = p * (p + 1) / 2 + n * p + n * (n + 1) / 2
    return {"bytes": (1 + n) * (0.1875 * weights + 2 * head) + 2 * kv * (2 * p + n * p + n * (n + 1) / 2),
            "flops": (p + n) * weights + (1 + n) * 2 * head + att * pairs}


def tolerance(case):
    kind = case["kind"]
    if kind == "convert":
        return {"rel": 1e-6}  # the packed words are whole numbers; gamma is a double sum
    if kind == "gemv" or (kind == "gemm" and not case["half"]):
        return "exact"
    if kind in ("bitlinear", "gemm"):
        return {"rel": 1e-3}  # half results of exact integer sums
    # half activations quantised to int8 at every projection: a sum formed in another order moves a rounded value, and
    # the layers after it carry the difference on.  The logits of one prompt as a batch and token by token, both
    # correct, differ by 3e-4 to 9e-3.
    return {"rel": 1e-2 if kind == "layer" else 2e-2}
