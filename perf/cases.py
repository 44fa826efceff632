"""The work that users of this framework have it do, as cases that can be timed and compared.

`listed()` names twelve of them, `draw(rng)` gives further ones of the same ranges. A case is run through the package's
public entry points only. Seven kinds:

* encoder    - a whole BERT encoder forward on packed sequences (what the encoder object is for): FP16 or INT8, base or
               large sizes, device tensors or host buffers, from one short query to a full batch;
* attention  - the fused attention alone, as the attention plugin calls it: fixed, packed or separate-tensor layout,
               FP16 (any length) or INT8 (up to 512 keys);
* interleaved - the INT8 operators of the CHW32-interleaved plugins: attention, then residual + LayerNorm with the
               pre-LayerNorm sum as a second output;
* skip_ln    - residual + bias + LayerNorm alone, FP32 / FP16 / INT8;
* embedding  - embedding + LayerNorm front end, fixed layout with the mask index or packed with the pre-LayerNorm sum,
               with or without the quantised copy;
* fc         - one fully connected layer with its epilogue;
* layer_fp32 - one encoder layer on FP32 tensors, operator by operator (the plugins' type_id 0).
"""
import numpy as np
import torch

import tensorrt_b200 as T
from tensorrt_b200 import synthetic

DEV = "cuda:0"
MODELS = {"base": (12, 768, 12, 3072), "large": (24, 1024, 16, 4096)}  # layers, hidden, heads, feed-forward width
VOCAB, POSITIONS, SEGMENTS = 30522, 512, 2
TYPES = {"fp32": torch.float32, "fp16": torch.float16, "int8": torch.int8}
SIZE = {"fp32": 4, "fp16": 2, "int8": 1}
ENCODER_FLOPS_MAX = 3.6e13  # of the largest listed encoder case


def listed():
    return [
        # one short question to a loaded model: what an interactive service waits for
        {"name": "encoder_base_fp16_one_query", "kind": "encoder", "model": "base", "dtype": "fp16", "batch": 1, "min_len": 37, "max_len": 37, "host": False},
        # a few ragged requests collected by a server, ids and results in host memory
        {"name": "encoder_large_int8_host_8", "kind": "encoder", "model": "large", "dtype": "int8", "batch": 8, "min_len": 32, "max_len": 384, "host": True},
        # a batch of short sentences with padding removed (classification, retrieval)
        {"name": "encoder_base_fp16_32", "kind": "encoder", "model": "base", "dtype": "fp16", "batch": 32, "min_len": 64, "max_len": 128, "host": False},
        # the throughput workload: full-length question answering in INT8
        {"name": "encoder_large_int8_64x384", "kind": "encoder", "model": "large", "dtype": "int8", "batch": 64, "min_len": 384, "max_len": 384, "host": False},
        # offline scoring of a ragged corpus in FP16
        {"name": "encoder_large_fp16_256", "kind": "encoder", "model": "large", "dtype": "fp16", "batch": 256, "min_len": 32, "max_len": 384, "host": False},
        # whole documents, longer than the encoder's position table: the attention operator in a user's own model
        {"name": "attention_fp16_documents", "kind": "attention", "dtype": "fp16", "layout": "packed", "heads": 16, "head_size": 64, "batch": 11, "min_len": 200, "max_len": 2000},
        # padded batch at the longest INT8 length, lengths through the mask index
        {"name": "attention_int8_fixed_512", "kind": "attention", "dtype": "int8", "layout": "fixed", "heads": 12, "head_size": 64, "batch": 24, "min_len": 256, "max_len": 512},
        # the interleaved INT8 plugins at a medium batch
        {"name": "interleaved_int8_256", "kind": "interleaved", "heads": 16, "head_size": 64, "batch": 37, "min_len": 100, "max_len": 256},
        # wide rows, bandwidth only
        {"name": "skip_ln_fp16_4096", "kind": "skip_ln", "dtype": "fp16", "hidden": 4096, "tokens": 32001, "bias": True},
        # front end of a padded INT8 network: hidden states, their quantised copy and the mask index
        {"name": "embedding_fixed_int8_64x384", "kind": "embedding", "layout": "fixed", "dtype": "fp16", "hidden": 1024, "batch": 64, "min_len": 32, "max_len": 384, "quantised": True},
        # last projection of an INT8 block whose output stays in FP16
        {"name": "fc_int8_to_fp16_5001", "kind": "fc", "dtype": "int8", "out": "fp16", "m": 5001, "n": 1024, "k": 4096, "gelu": False},
        # one layer at full precision, to check a quantised model against
        {"name": "layer_fp32_8x128", "kind": "layer_fp32", "hidden": 768, "heads": 12, "ffn": 3072, "batch": 8, "seqlen": 128},
    ]


def _log(rng, lo, hi):
    """A whole number, spread evenly over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))))


def _lengths_range(rng, longest):
    hi = _log(rng, 16, longest)
    return (hi if rng.random() < 0.3 else rng.randint(max(1, hi // 8), hi)), hi


def draw(rng):
    kind = rng.choice(["encoder", "encoder", "encoder", "attention", "attention", "interleaved", "skip_ln", "embedding", "fc", "layer_fp32"])
    if kind == "encoder":
        while True:
            lo, hi = _lengths_range(rng, 512)
            c = {"kind": kind, "model": rng.choice(["base", "large"]), "dtype": rng.choice(["fp16", "int8"]), "batch": _log(rng, 1, 256), "min_len": lo, "max_len": hi, "host": rng.random() < 0.25}
            if _encoder_flops(c, c["batch"] * hi, c["batch"] * hi * hi) <= ENCODER_FLOPS_MAX:
                return c
    if kind == "attention":
        layout = rng.choice(["fixed", "packed", "packed", "separate"])
        dtype = rng.choice(["fp16", "int8"])
        while True:
            lo, hi = _lengths_range(rng, 512 if dtype == "int8" or layout == "separate" else 2048)
            c = {"kind": kind, "dtype": dtype, "layout": layout, "heads": rng.choice([12, 16]), "head_size": rng.choice([64, 64, 64, 32]), "batch": _log(rng, 1, 128), "min_len": lo, "max_len": hi}
            if c["batch"] * c["heads"] * hi * hi <= 128 * 16 * 512 * 512 and c["batch"] * hi >= 64:
                return c
    if kind == "interleaved":
        lo, hi = _lengths_range(rng, 512)
        return {"kind": kind, "heads": rng.choice([12, 16]), "head_size": 64, "batch": _log(rng, 1, 128), "min_len": lo, "max_len": hi}
    if kind == "skip_ln":
        dtype, hidden = rng.choice(["fp16", "fp16", "int8", "int8", "fp32"]), rng.choice([384, 768, 768, 1024, 1024, 2048, 4096])
        return {"kind": kind, "dtype": dtype, "hidden": hidden, "tokens": _log(rng, 32, (1 << 28) // hidden), "bias": rng.random() < 0.7}
    if kind == "embedding":
        lo, hi = _lengths_range(rng, 512)
        return {"kind": kind, "layout": rng.choice(["fixed", "packed"]), "dtype": rng.choice(["fp16", "fp16", "fp16", "fp32"]), "hidden": rng.choice([768, 1024]), "batch": _log(rng, 1, 256), "min_len": lo, "max_len": hi, "quantised": rng.random() < 0.5}
    if kind == "fc":
        dtype = rng.choice(["fp16", "int8"])
        hidden = rng.choice([768, 1024])
        n, k = rng.choice([(3 * hidden, hidden), (hidden, hidden), (4 * hidden, hidden), (hidden, 4 * hidden)])
        return {"kind": kind, "dtype": dtype, "out": "fp16" if dtype == "fp16" else rng.choice(["int8", "int8", "fp16"]), "m": _log(rng, 1, 65536), "n": n, "k": k, "gelu": n == 4 * hidden and rng.random() < 0.7}
    hidden = rng.choice([768, 1024])
    return {"kind": kind, "hidden": hidden, "heads": hidden // 64, "ffn": 4 * hidden, "batch": _log(rng, 1, 16), "seqlen": _log(rng, 16, 256)}


def _lengths(case, seed):
    """Sequence lengths uniform in [min_len, max_len], the longest present: the same ones for a case, in an order of the seed."""
    g = np.random.default_rng([case["batch"], case["min_len"], case["max_len"]])
    n = g.integers(case["min_len"], case["max_len"] + 1, size=case["batch"]).astype(np.int32)
    n[0] = case["max_len"]
    return np.random.default_rng([seed, 1]).permutation(n)


def _mean_lengths(case):
    """Expected sums of the lengths and of their squares over the batch."""
    lo, hi, b = case["min_len"], case["max_len"], case["batch"]
    n = np.arange(lo, hi + 1, dtype=np.float64)
    return hi + (b - 1) * float(n.mean()), hi * hi + (b - 1) * float((n * n).mean())


def _encoder_flops(case, tokens, squares):
    layers, e, _, f = MODELS[case["model"]]
    return layers * (tokens * 2.0 * (4 * e * e + 2 * e * f) + 4.0 * squares * e)


class _Rng:
    """Seeded random tensors on the device."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed))

    def normal(self, *shape, dtype=torch.float32, std=1.0, mean=0.0):
        return (torch.randn(shape, device=DEV, generator=self.g) * std + mean).to(dtype)

    def bytes(self, *shape, amax=4.5):
        """Values ~N(0, 1) quantised with the step amax / 127, and that step."""
        x = torch.randn(shape, device=DEV, generator=self.g)
        return torch.clamp(torch.round(x * (127.0 / amax)), -127, 127).to(torch.int8), amax / 127.0

    def ids(self, *shape, below):
        return torch.randint(0, below, shape, device=DEV, generator=self.g, dtype=torch.int32)


def _cu(lengths):
    return torch.from_numpy(np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)).to(DEV)


def _segments(lengths, seed):
    """Segment id 0 before a random split point of each sequence, 1 after it."""
    g = np.random.default_rng([seed, 2])
    return np.concatenate([(np.arange(n) >= g.integers(1, max(2, n))).astype(np.int32) for n in lengths])


def _prepare_encoder(case, seed):
    layers, e, heads, f = MODELS[case["model"]]
    params = synthetic.make_params(layers, e, heads, f, VOCAB, POSITIONS, SEGMENTS, seed=seed, device=DEV)
    lengths = _lengths(case, seed)
    cu, total, longest = _cu(lengths), int(lengths.sum()), int(lengths.max())
    ids = _Rng(seed + 1).ids(total, below=VOCAB)
    seg = torch.from_numpy(_segments(lengths, seed)).to(DEV)
    if case["dtype"] == "int8":
        # scales from one calibration batch of the same distribution
        calib = T.BertEncoder(params, T.FP16, DEV)
        n = np.full(8, 128, np.int32)
        synthetic.assign_int8_scales(params, calib.calibrate(_Rng(seed + 2).ids(1024, below=VOCAB), torch.from_numpy(_segments(n, seed + 2)).to(DEV), _cu(n), 128))
        calib.close()
    enc = T.BertEncoder(params, T.INT8 if case["dtype"] == "int8" else T.FP16, DEV)
    s = {"enc": enc, "longest": longest, "ids": ids, "seg": seg, "cu": cu}
    if case["host"]:
        for k in ("ids", "seg", "cu"):
            s[k] = s[k].cpu().pin_memory()
        s["out_dev"] = torch.empty((total, e), dtype=torch.float16, device=DEV)
        s["out_host"] = torch.empty((total, e), dtype=torch.float16).pin_memory()
    return s


def _prepare_attention(case, seed):
    r, lengths = _Rng(seed), _lengths(case, seed)
    n, d, b, smax = case["heads"], case["head_size"], case["batch"], int(lengths.max())
    s = {"b": b, "smax": smax, "scales": {}}
    if case["layout"] == "separate":
        shapes = [(b, n, smax, d)] * 3
    elif case["layout"] == "fixed":
        shapes = [(smax, b, 3 * n * d)]
    elif case["layout"] == "packed":
        shapes = [(int(lengths.sum()), 3 * n * d)]
    else:
        shapes = [(3 * n * d // 32, int(lengths.sum()), 32)]
    if case["dtype"] == "int8":
        made = [r.bytes(*shape) for shape in shapes]
        s["x"], step = [t for t, _ in made], made[0][1]
        # the context of a softmax over many keys is narrower than its inputs: output step a quarter of theirs
        s["scales"] = {"scale_bmm1": step * step * d ** -0.5, "scale_softmax": 127.0, "scale_bmm2": 4.0 / 127.0}
    else:
        s["x"] = [r.normal(*shape, dtype=torch.float16) for shape in shapes]
    s["cu"], s["lengths"] = _cu(lengths), torch.from_numpy(lengths).to(DEV)
    return s


def _norm_params(r, hidden, dtype):
    return r.normal(hidden, dtype=dtype, std=0.02, mean=1.0), r.normal(hidden, dtype=dtype, std=0.02)


def _prepare_skip(case, seed):
    r, hidden, tokens = _Rng(seed), case["hidden"], case["tokens"]
    kind = torch.float16 if case["dtype"] == "int8" else TYPES[case["dtype"]]
    s = {"bias": r.normal(hidden, dtype=kind, std=0.02) if case["bias"] else None}
    s["gamma"], s["beta"] = _norm_params(r, hidden, kind)
    if case["dtype"] == "int8":
        (s["x"], s["dq_x"]), (s["skip"], s["dq_skip"]) = r.bytes(tokens, hidden), r.bytes(tokens, hidden)
    else:
        s["x"], s["skip"] = r.normal(tokens, hidden, dtype=kind), r.normal(tokens, hidden, dtype=kind)
    return s


def _prepare_embedding(case, seed):
    r, e, lengths = _Rng(seed), case["hidden"], _lengths(case, seed)
    kind = TYPES[case["dtype"]]
    s = {"tables": [r.normal(rows, e, dtype=kind, std=0.02) for rows in (VOCAB, POSITIONS, SEGMENTS)], "q": 127.0 / 4.5 if case["quantised"] else None}
    s["gamma"], s["beta"] = _norm_params(r, e, torch.float32)
    if case["layout"] == "packed":
        s["cu"], s["smax"] = _cu(lengths), int(lengths.max())
        s["ids"], s["seg"] = r.ids(int(lengths.sum()), below=VOCAB), torch.from_numpy(_segments(lengths, seed)).to(DEV)
    else:
        smax, b = int(lengths.max()), case["batch"]
        s["ids"], s["seg"] = r.ids(smax, b, below=VOCAB), r.ids(smax, b, below=SEGMENTS)
        s["mask"] = (torch.arange(smax, device=DEV)[:, None] < torch.from_numpy(lengths).to(DEV)[None, :]).to(torch.int32)
    return s


def _prepare_fc(case, seed):
    r, m, n, k = _Rng(seed), case["m"], case["n"], case["k"]
    s = {"bias": r.normal(n, std=0.02), "more": {}}
    if case["dtype"] == "int8":
        (s["a"], sa), (w, sw) = r.bytes(m, k), r.bytes(n, k)
        s["w"] = w
        # weights ~N(0, 1 / k): the result is ~N(0, 1)
        s["more"] = {"alpha": sa * sw * k ** -0.5, "out_dtype": TYPES[case["out"]], "out_scale": 127.0 / 4.5 if case["out"] == "int8" else 1.0}
    else:
        s["a"], s["w"] = r.normal(m, k, dtype=torch.float16), r.normal(n, k, dtype=torch.float16, std=k ** -0.5)
    s["act"] = T.ACT_GELU_ERF if case["gelu"] else T.ACT_NONE
    return s


def _prepare_layer(case, seed):
    r, e, f = _Rng(seed), case["hidden"], case["ffn"]
    s = {"x": r.normal(case["seqlen"], case["batch"], e)}
    for name, out, inn in (("qkv", 3 * e, e), ("out", e, e), ("up", f, e), ("down", e, f)):
        s["w_" + name], s["b_" + name] = r.normal(out, inn, std=0.02), r.normal(out, std=0.02)
    for name in ("1", "2"):
        s["gamma" + name], s["beta" + name] = _norm_params(r, e, torch.float32)
    return s


def prepare(case, seed):
    kind = case["kind"]
    if kind == "encoder":
        s = _prepare_encoder(case, seed)
    elif kind == "attention":
        s = _prepare_attention(case, seed)
    elif kind == "interleaved":
        s = _prepare_attention({**case, "dtype": "int8", "layout": "interleaved"}, seed)
        r, hidden = _Rng(seed + 1), case["heads"] * case["head_size"]
        (s["skip"], s["dq_skip"]), (s["gamma"], s["beta"]) = r.bytes(hidden // 32, s["x"][0].shape[1], 32), _norm_params(r, hidden, torch.float16)
    elif kind == "layer_fp32":
        s = _prepare_layer(case, seed)
    else:
        s = {"skip_ln": _prepare_skip, "embedding": _prepare_embedding, "fc": _prepare_fc}[kind](case, seed)
    s["case"] = case
    return s


def _run_layer(s):
    c, x = s["case"], s["x"]
    e, rows = c["hidden"], c["seqlen"] * c["batch"]
    qkv = T.fc(x.view(rows, e), s["w_qkv"], s["b_qkv"])
    ctx = T.mha(qkv.view(c["seqlen"], c["batch"], 3 * e), c["batch"], c["seqlen"], c["heads"], e // c["heads"])
    h = T.skip_layer_norm(T.fc(ctx.view(rows, e), s["w_out"]), x.view(rows, e), s["gamma1"], s["beta1"], bias=s["b_out"])
    up = T.fc(h, s["w_up"], s["b_up"], T.ACT_GELU_ERF)
    return T.skip_layer_norm(T.fc(up, s["w_down"]), h, s["gamma2"], s["beta2"], bias=s["b_down"])


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "encoder":
        if c["host"]:
            return s["enc"].forward_host(s["ids"], s["seg"], s["cu"], s["longest"], s["out_dev"], s["out_host"])
        return s["enc"].forward(s["ids"], s["seg"], s["cu"], s["longest"])
    if kind == "attention":
        if c["layout"] == "separate":
            return T.attention_bnsd(*s["x"], kv_lengths=s["lengths"], **s["scales"])
        where = {"cu_seqlens": s["cu"]} if c["layout"] == "packed" else {"mask_idx": s["lengths"]}
        return T.mha(s["x"][0], s["b"], s["smax"], c["heads"], c["head_size"], **where, **s["scales"])
    if kind == "interleaved":
        ctx = T.mha(s["x"][0], s["b"], s["smax"], c["heads"], c["head_size"], cu_seqlens=s["cu"], interleaved=True, **s["scales"])
        out, preln = T.skip_layer_norm_interleaved(ctx, s["skip"], s["gamma"], s["beta"], s["dq_skip"] / 4, s["dq_skip"], 127.0 / 4.5, 127.0 / 5.0)
        return ctx, out, preln
    if kind == "skip_ln":
        if c["dtype"] == "int8":
            return T.skip_layer_norm_dqq(s["x"], s["skip"], s["gamma"], s["beta"], s["bias"], s["dq_x"], s["dq_skip"], 127.0 / 4.5)
        return T.skip_layer_norm(s["x"], s["skip"], s["gamma"], s["beta"], bias=s["bias"])
    if kind == "embedding":
        if c["layout"] == "packed":
            return T.emb_layer_norm_var_seqlen(s["ids"], s["seg"], s["cu"], s["smax"], *s["tables"], s["gamma"], s["beta"], with_skip=True, q_scale=s["q"])
        return T.emb_layer_norm(s["ids"], s["seg"], *s["tables"], s["gamma"], s["beta"], q_scale=s["q"], mask=s["mask"])
    if kind == "fc":
        return T.fc(s["a"], s["w"], s["bias"], s["act"], **s["more"])
    return _run_layer(s)


def work(case):
    kind = case["kind"]
    if kind in ("encoder", "attention", "interleaved", "embedding"):
        tokens, squares = _mean_lengths(case)
    if kind == "encoder":
        layers, e, _, f = MODELS[case["model"]]
        weights = layers * ((4 * e * e + 2 * e * f) * SIZE[case["dtype"]] + 4 * (3 * e + f) + 2 * 6 * e)
        return {"bytes": weights + tokens * (8 + 2 * e + 2 * e), "flops": _encoder_flops(case, tokens, squares)}
    if kind in ("attention", "interleaved"):
        size = SIZE[case.get("dtype", "int8")]
        e, b, hi = case["heads"] * case["head_size"], case["batch"], case["max_len"]
        if case.get("layout") in ("fixed", "separate"):  # every query row is computed, over the valid keys
            return {"bytes": size * e * (2.0 * b * hi + 2.0 * tokens), "flops": 4.0 * e * hi * tokens}
        extra = 4.0 * tokens * e if kind == "interleaved" else 0.0  # the second input of the sum, its two outputs, and the context read back
        return {"bytes": size * e * 4.0 * tokens + extra, "flops": 4.0 * e * squares}
    if kind == "skip_ln":
        size = SIZE[case["dtype"]]
        return {"bytes": 3.0 * case["tokens"] * case["hidden"] * size + 3 * case["hidden"] * max(2, size), "flops": 0}
    if kind == "embedding":
        size, e = SIZE[case["dtype"]], case["hidden"]
        rows = tokens if case["layout"] == "packed" else case["batch"] * case["max_len"]
        per_row = 8 + e * size * (3 if case["layout"] == "packed" else 2) + (e if case["quantised"] else 0) + (4 if case["layout"] == "fixed" else 0)
        return {"bytes": float(rows * per_row), "flops": 0}
    if kind == "fc":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": float((m * k + n * k) * SIZE[case["dtype"]] + m * n * SIZE[case["out"]] + 4 * n), "flops": 2.0 * m * n * k}
    e, f, rows = case["hidden"], case["ffn"], case["batch"] * case["seqlen"]
    return {"bytes": 4.0 * (4 * e * e + 2 * e * f + 2 * rows * e), "flops": rows * (2.0 * (4 * e * e + 2 * e * f) + 4.0 * case["seqlen"] * e)}


def tolerance(case):
    kind = case["kind"]
    if kind == "encoder":
        # FP16: every stored tensor is rounded to 11 bits, seven times a layer. INT8: a value on the edge between two steps
        # (amax / 127, about a 30th of the standard deviation) may fall either way, and the layers after it see that
        return {"rel": 1e-2 if case["dtype"] == "fp16" else 3e-2}
    if kind == "layer_fp32" or case.get("dtype") == "fp32":
        return {"rel": 1e-5, "differ": 1e-3}
    if kind == "attention" and case["dtype"] == "int8":
        return {"rel": 0.0, "differ": 1e-3}  # whole numbers up to ties of the quantised probabilities
    if kind == "interleaved" or case.get("dtype") == "int8":
        return {"rel": 2e-3, "differ": 5e-3}  # ties of the rounded LayerNorm or of the scaled sum
    return {"rel": 2e-3, "differ": 5e-3}  # one rounding to FP16 of the result, sums in FP32
