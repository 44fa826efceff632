"""The benchmark configurations as end-to-end parity cases.

config 1: one BERT-base post-LN encoder layer (batch 8, seq 128, hidden 768, 12 heads x 64, FFN 3072, erf-GELU), FP32
          oracle / FP16 target, all-valid mask - run through the PLUGIN OBJECTS in the fixed [S, B, E] layout, i.e. the
          path a TensorRT engine would take: FC -> QKVToContext(v4, mask from EmbLayerNorm-style mask index) -> FC ->
          SkipLayerNorm(v5, bias) -> FC(+bias+GELU) -> FC -> SkipLayerNorm(v5, bias).
config 2: BERT-base front end: EmbLayerNorm v6 on B=32, S=128 with lengths in [64, 128] + two layers of the encoder.
config 3: BERT-large, 24 layers, S = 384, 64 sequences, explicit INT8 (the benchmark's headline configuration).
config 4: BERT-large packed variable-length path, lengths uniform in [32, 384] (seed 1), sharded by token count.
"""
import numpy as np
import pytest
import torch

from oracle import bert_oracle as O

pytestmark = pytest.mark.gpu

EMB, QKV, SKIP, FC = ("CustomEmbLayerNormPluginDynamic", "CustomQKVToContextPluginDynamic",
                      "CustomSkipLayerNormPluginDynamic", "CustomFCPluginDynamic")


def _t(a, cuda):
    return torch.from_numpy(np.ascontiguousarray(a)).to(cuda)


def _enqueue(p, ins, outs, in_descs, out_descs, ws=None):
    st = p.enqueue(in_descs, out_descs, [t.data_ptr() for t in ins], [t.data_ptr() for t in outs],
                   ws.data_ptr() if ws is not None else None, torch.cuda.current_stream().cuda_stream)
    assert st == 0, st


def test_config1_single_layer_through_plugins(cuda):
    H = pytest.importorskip("tensorrt_b200.plugin_harness", exc_type=ImportError)  # absent without the TensorRT headers

    rng = np.random.default_rng(0)
    B, S, E, N, F = 8, 128, 768, 12, 3072
    n = lambda *s: (0.02 * rng.standard_normal(s)).astype(np.float32)
    hidden = rng.standard_normal((S, B, E)).astype(np.float16)            # hidden states ~N(0, 1), layout [S, B, E]
    lp = O.LayerParams(w_qkv=n(E, 3 * E).astype(np.float16), b_qkv=n(3 * E), w_out=n(E, E).astype(np.float16), b_out=n(E).astype(np.float16),
                       ln1_gamma=(1 + n(E)).astype(np.float16), ln1_beta=n(E).astype(np.float16), w_ffn1=n(E, F).astype(np.float16),
                       b_ffn1=n(F), w_ffn2=n(F, E).astype(np.float16), b_ffn2=n(E).astype(np.float16),
                       ln2_gamma=(1 + n(E)).astype(np.float16), ln2_beta=n(E).astype(np.float16))
    # oracle on the same rows in packed order (sequence b owns rows [b*S, (b+1)*S))
    x_packed = np.ascontiguousarray(hidden.transpose(1, 0, 2)).reshape(B * S, E)
    cu = np.arange(0, (B + 1) * S, S, dtype=np.int32)
    ref, _ = O.encoder_layer_fp(x_packed.astype(np.float64), lp, B, S, N, cu, round_fp16=True)
    ref = ref.reshape(B, S, E).transpose(1, 0, 2)

    fc = lambda W, out, extra=(): H.Plugin(FC, "2", [("out_dims", out), ("type_id", 1), ("W", W.astype(np.float32).ravel())] + list(extra)).attach()
    p_qkv = fc(lp.w_qkv, 3 * E, [("bias", lp.b_qkv)])
    p_att = H.Plugin(QKV, "4", [("type_id", 1), ("hidden_size", E), ("num_heads", N), ("has_mask", 1)]).attach()
    p_out = fc(lp.w_out, E)
    p_ln1 = H.Plugin(SKIP, "5", [("type_id", 1), ("ld", E), ("beta", lp.ln1_beta.astype(np.float32)),
                                 ("gamma", lp.ln1_gamma.astype(np.float32)), ("bias", lp.b_out.astype(np.float32))]).attach()
    p_f1 = fc(lp.w_ffn1, F, [("bias", lp.b_ffn1), ("activation", 1)])
    p_f2 = fc(lp.w_ffn2, E)
    p_ln2 = H.Plugin(SKIP, "5", [("type_id", 1), ("ld", E), ("beta", lp.ln2_beta.astype(np.float32)),
                                 ("gamma", lp.ln2_gamma.astype(np.float32)), ("bias", lp.b_ffn2.astype(np.float32))]).attach()
    assert all(p.ok for p in (p_qkv, p_att, p_out, p_ln1, p_f1, p_f2, p_ln2))

    d = lambda c: H.make_desc((S, B, c, 1, 1), H.HALF)
    buf = lambda c: torch.empty((S, B, c), dtype=torch.float16, device=cuda)
    x = _t(hidden, cuda)
    qkv, ctx, ao, h1, f1, f2, out = buf(3 * E), buf(E), buf(E), buf(E), buf(F), buf(E), buf(E)
    mask_idx = torch.full((B, 1), S, dtype=torch.int32, device=cuda)      # all-valid mask as the embedding plugin emits it
    _enqueue(p_qkv, [x], [qkv], [d(E)], [d(3 * E)])
    ws = torch.empty(256, dtype=torch.uint8, device=cuda)
    _enqueue(p_att, [qkv, mask_idx], [ctx], [d(3 * E), H.make_desc((B, 1), H.INT32)], [d(E)], ws)
    _enqueue(p_out, [ctx], [ao], [d(E)], [d(E)])
    _enqueue(p_ln1, [ao, x], [h1], [d(E), d(E)], [d(E)])
    _enqueue(p_f1, [h1], [f1], [d(E)], [d(F)])
    _enqueue(p_f2, [f1], [f2], [d(F)], [d(E)])
    _enqueue(p_ln2, [f2, h1], [out], [d(E), d(E)], [d(E)])
    torch.cuda.synchronize()
    ok, worst, bad = O.close_abs_or_rel(out.cpu().numpy(), ref, 1e-2, 1e-2)
    assert ok, (worst, bad)
    for p in (p_qkv, p_att, p_out, p_ln1, p_f1, p_f2, p_ln2):
        p.close()


def test_config2_front_end_and_two_layers(cuda):
    """Config 2 shapes (BERT-base, B = 32, S = 128, lengths in [64, 128], segment split) on the first two layers:
    EmbLayerNorm v6 semantics for the mask index, packed encoder for the layers."""
    import tensorrt_b200 as T

    rng = np.random.default_rng(2)
    B, S = 32, 128
    p = O.make_bert_params(rng, 2, 768, 12, 3072, vocab=30522, max_pos=512)
    lengths = rng.integers(64, 129, size=B).astype(np.int32)
    ids_sb = rng.integers(0, 30522, size=(S, B)).astype(np.int32)
    split = rng.integers(1, 128, size=B)
    seg_sb = (np.arange(S)[:, None] >= split[None, :]).astype(np.int32)
    mask_sb = (np.arange(S)[:, None] < lengths[None, :]).astype(np.int32)
    # mask index output of the front end: bit-exact
    assert np.array_equal(T.compute_mask_idx(_t(mask_sb, cuda)).cpu().numpy(), lengths)
    # the valid tokens, packed, through the encoder
    cu = O.cu_seqlens(lengths)
    ids = np.concatenate([ids_sb[:lengths[b], b] for b in range(B)]).astype(np.int32)
    seg = np.concatenate([seg_sb[:lengths[b], b] for b in range(B)]).astype(np.int32)
    enc = T.BertEncoder(p, T.FP16, cuda)
    out = enc.forward(_t(ids, cuda), _t(seg, cuda), _t(cu, cuda), S).cpu().numpy()
    ref = O.encoder_fp(p, ids, seg, cu, S)
    ok, worst, bad = O.close_abs_or_rel(out, ref, 1e-2, 1e-2)
    assert bad <= out.size * 1e-3 and worst < 5e-2, (worst, bad)
    # the fixed-layout embedding plugin kernel agrees with the packed one on the valid tokens (bit for bit)
    emb_fixed = T.emb_layer_norm(_t(ids_sb, cuda), _t(seg_sb, cuda), enc.word_emb, enc.pos_emb, enc.tok_emb, enc.emb_gamma,
                                 enc.emb_beta).cpu().numpy()
    emb_packed = T.emb_layer_norm_var_seqlen(_t(ids, cuda), _t(seg, cuda), _t(cu, cuda), S, enc.word_emb, enc.pos_emb,
                                             enc.tok_emb, enc.emb_gamma, enc.emb_beta).cpu().numpy()
    gathered = np.concatenate([emb_fixed[:lengths[b], b] for b in range(B)])
    assert np.array_equal(gathered, emb_packed)
    enc.close()


def test_config4_packed_var_len_sharded(cuda):
    """Config 4: lengths uniform in [32, 384], seed 1, B = 256 (about 53k tokens), greedy token balancing over 8
    shards; one BERT-large layer on the packed tokens of the heaviest shard, FP16 and INT8, and the property that a
    sequence's output does not depend on which other sequences share its shard."""
    import tensorrt_b200 as T

    rng = np.random.default_rng(1)
    lengths_all = rng.integers(32, 385, size=256).astype(np.int32)
    assert 50000 < int(lengths_all.sum()) < 56000
    shards = T.shard_by_tokens(lengths_all, 8)
    loads = [int(lengths_all[s].sum()) for s in shards]
    assert max(loads) - min(loads) <= 384
    mine = shards[int(np.argmax(loads))]
    lengths = lengths_all[mine]
    p = O.make_bert_params(rng, 1, 1024, 16, 4096, vocab=30522)
    cu = O.cu_seqlens(lengths)
    total = int(cu[-1])
    ids = rng.integers(0, 30522, size=total).astype(np.int32)
    seg = rng.integers(0, 2, size=total).astype(np.int32)
    enc = T.BertEncoder(p, T.FP16, cuda)
    out = enc.forward(_t(ids, cuda), _t(seg, cuda), _t(cu, cuda), 384).cpu().numpy()
    # oracle on the first three sequences only (the layer is per-sequence independent)
    k = 3
    sub = O.encoder_fp(p, ids[:cu[k]], seg[:cu[k]], cu[:k + 1], 384)
    ok, worst, bad = O.close_abs_or_rel(out[:cu[k]], sub, 1e-2, 1e-2)
    assert bad <= sub.size * 1e-3 and worst < 5e-2, (worst, bad)
    # same three sequences alone give bit-identical rows
    alone = enc.forward(_t(ids[:cu[k]], cuda), _t(seg[:cu[k]], cuda), _t(cu[:k + 1], cuda), 384).cpu().numpy()
    assert np.array_equal(alone, out[:cu[k]])
    enc.close()


def test_config3_bert_large_int8_24_layers(cuda):
    """Config 3 at full size: 24 layers, hidden 1024, 16 heads, FFN 4096, S = 384, a batch of 64 sequences, explicit
    INT8 with per-tensor amax / 127 scales from a seeded calibration batch (the oracle's calibration on two sequences),
    dq_probs = 1 / 127. The oracle runs two sequences of the batch - one at the front and one that a persistent CTA
    meets late in its work list. Layer 1 is held to the operator tolerance (+-1 LSB, a rounding tie of an attention
    probability may cost 2). Through 24 quantised layers a one-LSB difference at any operator is amplified like the
    quantisation noise itself (the two INT8 results end about 3 LSB apart, cosine 0.992), so the end-to-end statement
    is about accuracy: measured against the unquantised FP32 forward of the same network, the product's INT8 result
    is as close as the oracle's INT8 result. (With these synthetic N(0, 0.02) weights attention over 384 keys is close
    to uniform, probabilities of 1/384 quantise to 0 at dq_probs = 1/127, and BOTH INT8 results are far from the FP32
    forward - rms error about 1 on unit-variance outputs; the statement is that the product is no further than the
    exact restatement of the reference's arithmetic.)"""
    import tensorrt_b200 as T

    rng = np.random.default_rng(3)
    B, S = 64, 384
    p = O.make_bert_params(rng, 24, 1024, 16, 4096)
    ids2, seg2, _, cu2 = O.make_inputs(rng, 2, S)
    # O.calibrate_int8, keeping the FP32 forward's final hidden states as the accuracy reference
    O.quantize_weights(p)
    x32, _ = O.emb_layer_norm_var_seqlen(ids2, seg2, cu2, p.word_emb, p.pos_emb, p.tok_emb, p.emb_gamma, p.emb_beta)
    for lp in p.layers:
        lp.scales["s_in"] = O.amax_scale(x32)
        x32, t = O.encoder_layer_fp(x32, lp, 2, S, p.heads, cu2, round_fp16=False)
        lp.scales.update(s_qkv=O.amax_scale(t["qkv"]), s_ctx=O.amax_scale(t["ctx"]), s_attn_out=O.amax_scale(t["ao"]),
                         s_ln1=O.amax_scale(t["h1"]), s_ffn1=O.amax_scale(t["f1"]), s_ffn2=O.amax_scale(t["f2"]),
                         s_out=O.amax_scale(x32))
    ref, ref_i8, _ = O.encoder_int8(p, ids2, seg2, cu2, S, return_all=True)
    # the same two sequences at positions 0 and 41 of a batch of 64
    ids, seg, _, cu = O.make_inputs(rng, B, S)
    where = (0, 41)
    for k, b in enumerate(where):
        ids[b * S:(b + 1) * S] = ids2[k * S:(k + 1) * S]
        seg[b * S:(b + 1) * S] = seg2[k * S:(k + 1) * S]
    rows = np.concatenate([np.arange(b * S, (b + 1) * S) for b in where])

    # layer 1 alone: operator-level tolerance
    p1 = O.BertParams(p.hidden, p.heads, p.ffn, p.word_emb, p.pos_emb, p.tok_emb, p.emb_gamma, p.emb_beta, p.layers[:1], p.dq_probs)
    _, ref1_i8, _ = O.encoder_int8(p1, ids2, seg2, cu2, S, return_all=True)
    enc1 = T.BertEncoder(p1, T.INT8, cuda)
    out1 = enc1.forward(_t(ids, cuda), _t(seg, cuda), _t(cu, cuda), S).cpu().numpy().astype(np.float64)[rows]
    assert enc1.status_word() == 0
    got1 = np.rint(out1 / p.layers[0].scales["s_out"]).astype(np.int32)
    d1 = np.abs(got1 - ref1_i8.astype(np.int32))
    print("config3 layer 1: max", int(d1.max()), "frac > 1", float((d1 > 1).mean()), "exact", float((d1 == 0).mean()))
    # seven operators, each within 1 LSB of the oracle on its own inputs (the two LayerNorms normalise in half2 like the
    # reference's kernel and put a few percent of their values on the neighbouring step): at the end of the layer
    assert d1.max() <= 2 and (d1 > 1).mean() < 5e-3 and (d1 == 0).mean() > 0.7, (int(d1.max()), float((d1 > 1).mean()), float((d1 == 0).mean()))
    enc1.close()

    enc = T.BertEncoder(p, T.INT8, cuda)
    out = enc.forward(_t(ids, cuda), _t(seg, cuda), _t(cu, cuda), S).cpu().numpy().astype(np.float64)
    assert enc.status_word() == 0
    assert enc.launches_per_forward == 2 + 7 * 24
    got = out[rows]
    cos = float((got * ref).sum() / np.sqrt((got * got).sum() * (ref * ref).sum()))
    print("config3 end: cosine", cos)
    assert cos > 0.985, cos
    err_product = float(np.sqrt(np.mean((got - x32) ** 2)))
    err_oracle = float(np.sqrt(np.mean((ref - x32) ** 2)))
    print("config3 end: rms error vs FP32 forward: product", err_product, "oracle", err_oracle)
    assert err_product <= 1.1 * err_oracle, (err_product, err_oracle)
    # a sequence's output does not depend on its place in the batch
    alone = enc.forward(_t(ids2, cuda), _t(seg2, cuda), _t(cu2, cuda), S).cpu().numpy()
    assert np.array_equal(alone, out[rows].astype(np.float16))
    enc.close()
