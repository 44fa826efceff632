"""Parity of fused attention (tcgen05 FP16 / INT8, SIMT FP32) with the CPU oracle."""
import numpy as np
import pytest
import torch

from oracle import bert_oracle as O

pytestmark = pytest.mark.gpu


def _t(a, cuda):
    return torch.from_numpy(np.ascontiguousarray(a)).to(cuda)


def _status(cuda):
    return torch.zeros(4, dtype=torch.int32, device=cuda)


@pytest.mark.parametrize("S,B,N", [(128, 8, 12), (64, 2, 12), (96, 3, 4), (384, 2, 16), (512, 1, 2), (256, 2, 3),
                                   (200, 2, 2), (16, 1, 1)])
def test_mha_fixed_fp16(cuda, S, B, N):
    import tensorrt_b200 as T

    rng = np.random.default_rng(S + B + N)
    d = 64
    qkv = rng.standard_normal((S, B, 3 * N * d)).astype(np.float16)
    lengths = rng.integers(1, S + 1, size=B).astype(np.int32)
    lengths[0] = S
    if B > 1:
        lengths[1] = 0 if S == 128 else lengths[1]  # a sequence without valid keys gives zero rows
    ref = O.mha(qkv, B, S, N, d, lengths=lengths)
    st = _status(cuda)
    out = T.mha(_t(qkv, cuda), B, S, N, mask_idx=_t(lengths, cuda), status=st)
    assert int(st[0]) == 0
    ok, worst, bad = O.close_abs_or_rel(out.cpu().numpy(), ref, 1e-2, 1e-2)
    assert ok, (worst, bad)


@pytest.mark.parametrize("lengths,N", [([384, 32, 129, 1, 0, 257, 128], 16), ([17], 12), ([512, 500], 2)])
def test_mha_packed_fp16(cuda, lengths, N):
    import tensorrt_b200 as T

    rng = np.random.default_rng(len(lengths) + N)
    d = 64
    lengths = np.array(lengths, dtype=np.int32)
    cu = O.cu_seqlens(lengths)
    total, B, S = int(cu[-1]), len(lengths), int(max(lengths.max(), 1))
    qkv = rng.standard_normal((total, 3 * N * d)).astype(np.float16)
    ref = O.mha(qkv, B, S, N, d, cu=cu)
    st = _status(cuda)
    out = T.mha(_t(qkv, cuda), B, S, N, cu_seqlens=_t(cu, cuda), status=st)
    assert int(st[0]) == 0
    ok, worst, bad = O.close_abs_or_rel(out.cpu().numpy(), ref, 1e-2, 1e-2)
    assert ok, (worst, bad)


def _assert_int8_attention(out, ref):
    """+-1 LSB, except where a rounding tie of a quantised probability P_q = rni(p * 127) falls the other way: one
    such flip moves the INT32 accumulator by |v| <= 127, i.e. the output by up to scale_bmm2 * 127 = s_qkv / s_ctx
    (= 2 LSB with the scales used here). At most 1e-5 of the values may therefore be off by 2."""
    d = np.abs(out.astype(np.int32) - ref.astype(np.int32))
    assert d.max() <= 2, int(d.max())
    assert (d > 1).sum() <= max(1, int(1e-5 * d.size)), int((d > 1).sum())
    assert (d == 0).mean() > 0.98


def _int8_case(rng, rows, N, d):
    x = rng.standard_normal((rows, 3 * N * d))
    s_qkv = O.amax_scale(x)
    return O.quantize(x, 1.0 / s_qkv), s_qkv


@pytest.mark.parametrize("lengths,N", [([384, 32, 129, 1, 0, 257, 128], 16), ([64], 2), ([512, 300], 2)])
def test_mha_packed_int8(cuda, lengths, N):
    import tensorrt_b200 as T

    rng = np.random.default_rng(len(lengths) + N + 7)
    d = 64
    lengths = np.array(lengths, dtype=np.int32)
    cu = O.cu_seqlens(lengths)
    total, B, S = int(cu[-1]), len(lengths), int(max(lengths.max(), 1))
    q8, s_qkv = _int8_case(rng, total, N, d)
    dq_probs = 1.0 / 127.0
    s_ctx = s_qkv * 0.5
    s1 = float(np.float32(s_qkv) * np.float32(s_qkv) * np.float32(0.125))
    s2 = dq_probs * s_qkv / s_ctx
    ref = O.mha_int8(q8, B, S, N, d, s1, 1.0 / dq_probs, s2, cu=cu)
    st = _status(cuda)
    out = T.mha(_t(q8, cuda), B, S, N, cu_seqlens=_t(cu, cuda), scale_bmm1=s1, scale_softmax=1.0 / dq_probs,
                scale_bmm2=s2, status=st)
    assert int(st[0]) == 0
    _assert_int8_attention(out.cpu().numpy(), ref)


# pieces of 32 keys and their edges, no key, one key, a full block; probabilities that saturate; many pairs per SM
@pytest.mark.parametrize("lengths,N,scale_softmax", [([128, 1, 31, 0, 32, 33, 64, 65, 95, 96, 97, 127], 5, 127.0),
                                                     ([3, 1, 100, 2, 40], 3, 200.0), ([int(7 * i) % 129 for i in range(150)], 16, 127.0)])
@pytest.mark.parametrize("d,interleaved", [(64, False), (64, True), (32, True), (48, False), (16, False)])
def test_mha_int8_one_key_block_is_the_persistent_kernel_to_the_bit(cuda, lengths, N, scale_softmax, d, interleaved):
    """Sequences of at most 128 tokens have a kernel of their own; with a larger S (an upper bound only, in the packed layouts) the
    same sequences go through the persistent one, which the other tests compare with the oracle. Same bytes."""
    import tensorrt_b200 as T

    gen = torch.Generator(device=cuda).manual_seed(len(lengths) + d)
    cu = _t(O.cu_seqlens(np.array(lengths, dtype=np.int32)), cuda)
    total, B = sum(lengths), len(lengths)
    shape = (3 * N * d // 32, total, 32) if interleaved else (total, 3 * N * d)
    q8 = torch.clamp(torch.round(40 * torch.randn(shape, device=cuda, generator=gen)), -128, 127).to(torch.int8)
    st = _status(cuda)
    for s1 in (2e-4, -1e-5):   # nothing keeps a caller from a scale below zero
        out = [T.mha(q8, B, S, N, d, cu_seqlens=cu, scale_bmm1=s1, scale_softmax=scale_softmax, scale_bmm2=0.02, status=st,
                     interleaved=interleaved) for S in (128, 129)]
        assert int(st[0]) == 0 and torch.equal(out[0], out[1])


@pytest.mark.parametrize("S", [1, 37, 128])
def test_mha_int8_one_key_block_fixed_and_separate(cuda, S):
    """The layouts whose rows S itself places: queries beyond a sequence's keys, a sequence without keys."""
    import tensorrt_b200 as T

    rng = np.random.default_rng(S + 5)
    B, N, d = 4, 3, 64
    q8, s_qkv = _int8_case(rng, S * B, N, d)
    q8 = q8.reshape(S, B, -1)
    lengths = np.array([S, 0, (S + 1) // 2, 1], dtype=np.int32)
    s1 = float(np.float32(s_qkv) * np.float32(s_qkv) * np.float32(0.125))
    s2 = 2.0 / 127.0
    ref = O.mha_int8(q8, B, S, N, d, s1, 127.0, s2, lengths=lengths)
    st = _status(cuda)
    scales = dict(scale_bmm1=s1, scale_softmax=127.0, scale_bmm2=s2, status=st)
    out = T.mha(_t(q8, cuda), B, S, N, mask_idx=_t(lengths, cuda), **scales)
    _assert_int8_attention(out.cpu().numpy(), ref)
    q, k, v = _split_bnsd(q8, S, B, N, d)
    out = T.attention_bnsd(_t(q, cuda), _t(k, cuda), _t(v, cuda), kv_lengths=_t(lengths, cuda), **scales)
    _assert_int8_attention(out.cpu().numpy(), ref.reshape(S, B, N, d).transpose(1, 2, 0, 3))
    assert int(st[0]) == 0


def test_mha_int8_saturating_probabilities(cuda):
    """scale_softmax > 127: probabilities near 1 saturate at 127 like the reference's conversion (the kernel leaves the
    clamp out when scale_softmax <= 127)."""
    import tensorrt_b200 as T

    rng = np.random.default_rng(77)
    N, d = 3, 64
    lengths = np.array([200, 3, 1, 130], dtype=np.int32)   # short sequences have probabilities close to 1
    cu = O.cu_seqlens(lengths)
    total, B, S = int(cu[-1]), len(lengths), 200
    q8, s_qkv = _int8_case(rng, total, N, d)
    s1 = float(np.float32(s_qkv) * np.float32(s_qkv) * np.float32(0.125))
    scale_softmax, s2 = 200.0, 0.4 / 200.0
    ref = O.mha_int8(q8, B, S, N, d, s1, scale_softmax, s2, cu=cu)
    st = _status(cuda)
    out = T.mha(_t(q8, cuda), B, S, N, cu_seqlens=_t(cu, cuda), scale_bmm1=s1, scale_softmax=scale_softmax, scale_bmm2=s2,
                status=st)
    assert int(st[0]) == 0
    _assert_int8_attention(out.cpu().numpy(), ref)


# With four key blocks the clamp is part of the kernel's form: on both sides of 127, few pairs and more than SMs, packed and fixed
@pytest.mark.parametrize("scale_softmax", [127.0, 200.0])
@pytest.mark.parametrize("N", [3, 40])
@pytest.mark.parametrize("packed", [True, False])
def test_mha_int8_clamp_at_four_key_blocks(cuda, scale_softmax, N, packed):
    import tensorrt_b200 as T

    rng = np.random.default_rng(N)
    lengths, S, d = np.array([400, 3, 1, 130], dtype=np.int32), 400, 64   # short sequences have probabilities close to 1
    cu = O.cu_seqlens(lengths)
    q8, s_qkv = _int8_case(rng, int(cu[-1]) if packed else S * len(lengths), N, d)
    s1, s2 = float(np.float32(s_qkv) * np.float32(s_qkv) * np.float32(0.125)), 0.4 / scale_softmax
    st = _status(cuda)
    scales = {"scale_bmm1": s1, "scale_softmax": scale_softmax, "scale_bmm2": s2, "status": st}
    if packed:
        ref = O.mha_int8(q8, len(lengths), S, N, d, s1, scale_softmax, s2, cu=cu)
        out = T.mha(_t(q8, cuda), len(lengths), S, N, cu_seqlens=_t(cu, cuda), **scales)
    else:
        q8 = q8.reshape(S, len(lengths), -1)
        ref = O.mha_int8(q8, len(lengths), S, N, d, s1, scale_softmax, s2, lengths=lengths)
        out = T.mha(_t(q8, cuda), len(lengths), S, N, mask_idx=_t(lengths, cuda), **scales)
    assert int(st[0]) == 0
    _assert_int8_attention(out.cpu().numpy(), ref)


@pytest.mark.parametrize("S,B,N", [(128, 4, 12), (384, 2, 16)])
def test_mha_fixed_int8(cuda, S, B, N):
    import tensorrt_b200 as T

    rng = np.random.default_rng(S)
    d = 64
    q8, s_qkv = _int8_case(rng, S * B, N, d)
    q8 = q8.reshape(S, B, -1)
    lengths = rng.integers(1, S + 1, size=B).astype(np.int32)
    dq_probs = 1.0 / 127.0
    s_ctx = s_qkv * 0.5
    s1 = float(np.float32(s_qkv) * np.float32(s_qkv) * np.float32(0.125))
    s2 = dq_probs * s_qkv / s_ctx
    ref = O.mha_int8(q8, B, S, N, d, s1, 1.0 / dq_probs, s2, lengths=lengths)
    st = _status(cuda)
    out = T.mha(_t(q8, cuda), B, S, N, mask_idx=_t(lengths, cuda), scale_bmm1=s1, scale_softmax=1.0 / dq_probs,
                scale_bmm2=s2, status=st)
    assert int(st[0]) == 0
    _assert_int8_attention(out.cpu().numpy(), ref)


@pytest.mark.parametrize("lengths,N", [([384, 32, 129, 1, 0, 257, 128], 16), ([100], 2)])
def test_mha_interleaved_int8(cuda, lengths, N):
    """CHW32-interleaved I/O of plugin version 6: qkv [3][N][d/32][total][32], out [N][d/32][total][32]."""
    import tensorrt_b200 as T

    rng = np.random.default_rng(len(lengths) + N + 11)
    d = 64
    lengths = np.array(lengths, dtype=np.int32)
    cu = O.cu_seqlens(lengths)
    total, B, S = int(cu[-1]), len(lengths), int(max(lengths.max(), 1))
    q8, s_qkv = _int8_case(rng, total, N, d)           # linear [total, N, 3, d]
    dq_probs = 1.0 / 127.0
    s_ctx = s_qkv * 0.5
    s1 = float(np.float32(s_qkv) * np.float32(s_qkv) * np.float32(0.125))
    s2 = dq_probs * s_qkv / s_ctx
    ref = O.mha_int8(q8, B, S, N, d, s1, 1.0 / dq_probs, s2, cu=cu)            # [total, N*d]
    il = np.ascontiguousarray(q8.reshape(total, N, 3, 2, 32).transpose(2, 1, 3, 0, 4)).reshape(3 * N * 2, total, 32)
    st = _status(cuda)
    out = T.mha(_t(il, cuda), B, S, N, cu_seqlens=_t(cu, cuda), scale_bmm1=s1, scale_softmax=1.0 / dq_probs,
                scale_bmm2=s2, status=st, interleaved=True)
    assert int(st[0]) == 0
    lin = out.cpu().numpy().reshape(N, 2, total, 32).transpose(2, 0, 1, 3).reshape(total, N * d)
    _assert_int8_attention(lin, ref)


@pytest.mark.parametrize("d", [16, 32, 48])
@pytest.mark.parametrize("packed", [False, True])
def test_mha_fp16_small_heads(cuda, d, packed):
    """Head sizes below 64 ride the 64-wide tiles: the missing channels are zero-filled by the TMA unit."""
    import tensorrt_b200 as T

    rng = np.random.default_rng(d + packed)
    N = 5
    lengths = np.array([300, 128, 0, 77, 1], dtype=np.int32)
    B, S = len(lengths), 320
    st = _status(cuda)
    if packed:
        cu = O.cu_seqlens(lengths)
        qkv = rng.standard_normal((int(cu[-1]), 3 * N * d)).astype(np.float16)
        ref = O.mha(qkv, B, S, N, d, cu=cu)
        out = T.mha(_t(qkv, cuda), B, S, N, head_size=d, cu_seqlens=_t(cu, cuda), status=st)
    else:
        qkv = rng.standard_normal((S, B, 3 * N * d)).astype(np.float16)
        ref = O.mha(qkv, B, S, N, d, lengths=lengths)
        out = T.mha(_t(qkv, cuda), B, S, N, head_size=d, mask_idx=_t(lengths, cuda), status=st)
    assert int(st[0]) == 0
    assert out.shape == ref.shape
    ok, worst, bad = O.close_abs_or_rel(out.cpu().numpy(), ref, 1e-2, 1e-2)
    assert ok, (worst, bad)


@pytest.mark.parametrize("d,interleaved", [(16, False), (32, False), (48, False), (32, True)])
def test_mha_int8_small_heads(cuda, d, interleaved):
    import tensorrt_b200 as T

    rng = np.random.default_rng(d + 3)
    N = 6
    lengths = np.array([260, 128, 0, 77, 1], dtype=np.int32)
    cu = O.cu_seqlens(lengths)
    total, B, S = int(cu[-1]), len(lengths), 260
    q8, s_qkv = _int8_case(rng, total, N, d)
    dq_probs = 1.0 / 127.0
    s_ctx = s_qkv * 0.5
    s1 = float(np.float32(s_qkv) * np.float32(s_qkv) * np.float32(1.0 / np.sqrt(d)))
    s2 = dq_probs * s_qkv / s_ctx
    ref = O.mha_int8(q8, B, S, N, d, s1, 1.0 / dq_probs, s2, cu=cu)
    st = _status(cuda)
    kw = dict(head_size=d, cu_seqlens=_t(cu, cuda), scale_bmm1=s1, scale_softmax=1.0 / dq_probs, scale_bmm2=s2, status=st)
    if interleaved:
        g = d // 32
        il = np.ascontiguousarray(q8.reshape(total, N, 3, g, 32).transpose(2, 1, 3, 0, 4)).reshape(3 * N * g, total, 32)
        out = T.mha(_t(il, cuda), B, S, N, interleaved=True, **kw)
        out = out.cpu().numpy().reshape(N, g, total, 32).transpose(2, 0, 1, 3).reshape(total, N * d)
    else:
        out = T.mha(_t(q8, cuda), B, S, N, **kw).cpu().numpy()
    assert int(st[0]) == 0
    _assert_int8_attention(out, ref)


@pytest.mark.parametrize("S,d", [(40, 80), (64, 24), (700, 72), (1100, 128)])
def test_mha_fp16_outside_tensor_core_shapes(cuda, S, d):
    """Heads wider than 64 or not a multiple of 16: FP16 I/O through the SIMT kernel (shapes the reference gives to
    its unfused runner); INT8 is refused there, as in the reference."""
    import tensorrt_b200 as T

    rng = np.random.default_rng(S + d)
    B, N = 2, 2
    lengths = np.array([S, S // 3], dtype=np.int32)
    cu = O.cu_seqlens(lengths)
    qkv = rng.standard_normal((int(cu[-1]), 3 * N * d)).astype(np.float16)
    ref = O.mha(qkv, B, S, N, d, cu=cu)
    out = T.mha(_t(qkv, cuda), B, S, N, head_size=d, cu_seqlens=_t(cu, cuda), use_workspace=False)
    ok, worst, bad = O.close_abs_or_rel(out.cpu().numpy(), ref, 1e-2, 1e-2)
    assert ok, (worst, bad)
    with pytest.raises(RuntimeError, match="INT8 takes"):
        T.mha(torch.zeros_like(_t(qkv, cuda), dtype=torch.int8), B, S, N, head_size=d, cu_seqlens=_t(cu, cuda))


@pytest.mark.parametrize("S,d", [(513, 64), (700, 64), (1100, 32), (1536, 64), (2000, 48)])
@pytest.mark.parametrize("packed", [False, True])
def test_mha_fp16_long_sequences_on_tensor_cores(cuda, S, d, packed):
    """S > 512: up to six key blocks (S <= 768) stay resident for all query tiles of a sequence, longer sequences
    stream their key blocks once per pair of query tiles - either way one softmax over all keys, no workspace.
    Sequences shorter than the longest leave key blocks unused; one sequence has no key at all."""
    import tensorrt_b200 as T

    rng = np.random.default_rng(S + d + packed)
    N = 3
    lengths = np.array([S, 0, 385, S // 2, 1, 384], dtype=np.int32)
    B = len(lengths)
    st = _status(cuda)
    if packed:
        cu = O.cu_seqlens(lengths)
        qkv = rng.standard_normal((int(cu[-1]), 3 * N * d)).astype(np.float16)
        ref = O.mha(qkv, B, S, N, d, cu=cu)
        kw = dict(cu_seqlens=_t(cu, cuda))
    else:
        qkv = rng.standard_normal((S, B, 3 * N * d)).astype(np.float16)
        ref = O.mha(qkv, B, S, N, d, lengths=lengths)
        kw = dict(mask_idx=_t(lengths, cuda))
    q = _t(qkv, cuda)
    p = T._lib.MhaParams(1, B, S, N, d, int(lengths.sum()) if packed else 0, None, None, None, None, 0, 1.0, 1.0, 1.0, None, None, 0)
    assert int(T._lib.lib.bert_b200_mha_workspace_size(T._lib.C.byref(p))) == 0
    out = T.mha(q, B, S, N, head_size=d, status=st, **kw)
    assert int(st[0]) == 0
    assert out.shape == ref.shape
    ok, worst, bad = O.close_abs_or_rel(out.cpu().numpy(), ref, 1e-2, 1e-2)
    assert ok, (worst, bad)


@pytest.mark.parametrize("unit", [128, 32, 7])
@pytest.mark.parametrize("step", [40.0, 3.0, -40.0])
def test_mha_fp16_running_maximum_moves(cuda, unit, step):
    """The online softmax keeps one running maximum per row, tracked per chunk of 32 keys, and rescales what the row has
    accumulated (row sum, context of earlier key blocks, probabilities of the current block written so far) whenever a
    chunk exceeds it by more than the lazy threshold. Keys whose scores rise by `step` every `unit` keys - per key
    block, per chunk, or at odd positions inside chunks; by far more than the threshold, by less than it, or falling -
    exercise every one of those paths."""
    import tensorrt_b200 as T

    rng = np.random.default_rng(99 + unit)
    S, B, N, d = 512, 2, 2, 64
    qkv = rng.standard_normal((S, B, N, 3, d)).astype(np.float32)
    # q . k / sqrt(d) gets the offset (key index // unit) * step: one channel carries the ramp
    qkv[:, :, :, 0, 0] = 8.0
    qkv[:, :, :, 1, 0] = ((np.arange(S) // unit) * step * (unit / 128.0))[:, None, None]
    qkv = qkv.reshape(S, B, -1).astype(np.float16)
    lengths = np.array([S, 300], dtype=np.int32)
    ref = O.mha(qkv, B, S, N, d, lengths=lengths)
    st = _status(cuda)
    out = T.mha(_t(qkv, cuda), B, S, N, mask_idx=_t(lengths, cuda), status=st)
    assert int(st[0]) == 0
    ok, worst, bad = O.close_abs_or_rel(out.cpu().numpy(), ref, 1e-2, 1e-2)
    assert ok, (unit, step, worst, bad)


def _split_bnsd(qkv, S, B, N, d):
    """fixed-layout [S, B, N, 3, d] -> three contiguous [B, N, S, d] arrays"""
    t = qkv.reshape(S, B, N, 3, d).transpose(3, 1, 2, 0, 4)
    return (np.ascontiguousarray(t[i]) for i in range(3))


@pytest.mark.parametrize("S,d", [(200, 64), (384, 32), (512, 64), (40, 16)])
def test_attention_bnsd_fp16(cuda, S, d):
    """Separate Q, K, V of shape [B, N, S, d] (the operand layout of TensorRT's attention layer) through the same
    kernel: must equal the fused-tensor path's oracle, output [B, N, S, d]."""
    import tensorrt_b200 as T

    rng = np.random.default_rng(S + d)
    B, N = 3, 4
    qkv = rng.standard_normal((S, B, 3 * N * d)).astype(np.float16)
    lengths = np.array([S, max(1, S // 3), 0], dtype=np.int32)
    ref = O.mha(qkv, B, S, N, d, lengths=lengths).reshape(S, B, N, d).transpose(1, 2, 0, 3)
    q, k, v = _split_bnsd(qkv, S, B, N, d)
    st = _status(cuda)
    out = T.attention_bnsd(_t(q, cuda), _t(k, cuda), _t(v, cuda), kv_lengths=_t(lengths, cuda), status=st)
    assert int(st[0]) == 0
    ok, worst, bad = O.close_abs_or_rel(out.cpu().numpy(), ref, 1e-2, 1e-2)
    assert ok, (worst, bad)
    full = T.attention_bnsd(_t(q, cuda), _t(k, cuda), _t(v, cuda))   # no lengths: every key valid
    ref_full = O.mha(qkv, B, S, N, d, lengths=np.full(B, S, np.int32)).reshape(S, B, N, d).transpose(1, 2, 0, 3)
    assert O.close_abs_or_rel(full.cpu().numpy(), ref_full, 1e-2, 1e-2)[0]


def test_attention_bnsd_int8(cuda):
    import tensorrt_b200 as T

    rng = np.random.default_rng(21)
    S, B, N, d = 260, 2, 3, 64
    q8, s_qkv = _int8_case(rng, S * B, N, d)
    q8 = q8.reshape(S, B, -1)
    lengths = np.array([260, 77], dtype=np.int32)
    dq_probs = 1.0 / 127.0
    s1 = float(np.float32(s_qkv) * np.float32(s_qkv) * np.float32(0.125))
    s2 = dq_probs * s_qkv / (s_qkv * 0.5)
    ref = O.mha_int8(q8, B, S, N, d, s1, 1.0 / dq_probs, s2, lengths=lengths).reshape(S, B, N, d).transpose(1, 2, 0, 3)
    q, k, v = _split_bnsd(q8, S, B, N, d)
    st = _status(cuda)
    out = T.attention_bnsd(_t(q, cuda), _t(k, cuda), _t(v, cuda), kv_lengths=_t(lengths, cuda), scale_bmm1=s1,
                           scale_softmax=1.0 / dq_probs, scale_bmm2=s2, status=st)
    assert int(st[0]) == 0
    _assert_int8_attention(out.cpu().numpy(), ref)
    with pytest.raises(RuntimeError, match="S <= 512"):
        big = torch.zeros((1, 1, 600, 64), dtype=torch.int8, device=cuda)
        T.attention_bnsd(big, big, big)
    # FP16 has no such limit
    bigh = torch.randn((1, 2, 600, 64), device=cuda).half()
    full = T.attention_bnsd(bigh, bigh, bigh).float()
    p = torch.softmax(bigh.float() @ bigh.float().transpose(-1, -2) / 8.0, dim=-1) @ bigh.float()
    assert (full - p).abs().max().item() < 2e-2


@pytest.mark.parametrize("d", [32, 64])
def test_mha_fp32(cuda, d):
    import tensorrt_b200 as T

    rng = np.random.default_rng(d)
    S, B, N = 40, 3, 3   # the reference FP32 configuration uses tiny hidden sizes with has_mask
    qkv = rng.standard_normal((S, B, 3 * N * d)).astype(np.float32)
    lengths = np.array([40, 13, 0], dtype=np.int32)
    ref = O.mha(qkv, B, S, N, d, lengths=lengths)
    out = T.mha(_t(qkv, cuda), B, S, N, head_size=d, mask_idx=_t(lengths, cuda))
    assert O.close_abs_or_rel(out.cpu().numpy(), ref, 1e-5, 1e-5)[0]


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("d", [4, 20, 64, 72, 96, 128, 132])
def test_mha_simt_tile_edges(cuda, d, half):
    """The FP32-arithmetic kernels around their 64-query / 64-key tiles (one key, a full tile, one past it, several), packed
    and fixed with an empty sequence; head sizes on both sides of every channel padding and beyond the tiled kernel's 128."""
    import tensorrt_b200 as T

    rng = np.random.default_rng(d)
    N, lengths = 2, np.array([1, 64, 65, 200, 0, 63], dtype=np.int32)
    if half and d in (64, 96):
        d += 2   # FP16 multiples of 16 up to 64 belong to the tensor-core kernel; these take the row kernel
    kind, tol = (np.float16, 1e-2) if half else (np.float32, 1e-5)
    cu = O.cu_seqlens(lengths)
    qkv = rng.standard_normal((int(cu[-1]), 3 * N * d)).astype(kind)
    ref = O.mha(qkv, len(lengths), 200, N, d, cu=cu)
    out = T.mha(_t(qkv, cuda), len(lengths), 200, N, head_size=d, cu_seqlens=_t(cu, cuda))
    assert O.close_abs_or_rel(out.cpu().numpy(), ref, tol, tol)[0]
    S = 130
    qkv = rng.standard_normal((S, 3, 3 * N * d)).astype(kind)
    lens = np.array([130, 0, 65], dtype=np.int32)
    ref = O.mha(qkv, 3, S, N, d, lengths=lens)
    out = T.mha(_t(qkv, cuda), 3, S, N, head_size=d, mask_idx=_t(lens, cuda))
    assert O.close_abs_or_rel(out.cpu().numpy(), ref, tol, tol)[0]


# FP32, every form of the launch on 148 SMs (csrc/mha_f32_plan.h), lengths at the edges of rows and blocks of keys, keys ending at and beside fours and eights,
# padded and packed
@pytest.mark.parametrize("S,B,N", [
    (31, 1, 1), (33, 3, 2), (64, 2, 2), (128, 74, 1), (64, 148, 1),               # 64 rows, one CTA per SM, asynchronous copies (64 channels)
    (64, 149, 1), (97, 10, 12), (128, 37, 4), (127, 25, 6), (64, 297, 1),         # two and more
    (129, 3, 2), (192, 49, 1), (257, 7, 4), (259, 15, 4), (192, 149, 1),          # 64 rows, copies between barriers: one, two and more
    (31, 40, 5), (65, 75, 1), (200, 40, 1), (17, 150, 2), (65, 149, 1), (9, 500, 2)])  # 32 rows: two, three and more
@pytest.mark.parametrize("d", [64, 20])
def test_mha_fp32_rows_per_cta(cuda, S, B, N, d):
    import tensorrt_b200 as T

    rng = np.random.default_rng(S + d)
    lengths = np.array([S - 7 * i % S for i in range(B)], dtype=np.int32)
    qkv = rng.standard_normal((S, B, 3 * N * d)).astype(np.float32)
    ref = O.mha(qkv, B, S, N, d, lengths=lengths)
    out = T.mha(_t(qkv, cuda), B, S, N, head_size=d, mask_idx=_t(lengths, cuda))
    assert O.close_abs_or_rel(out.cpu().numpy(), ref, 1e-5, 1e-5)[0]
    out = T.mha(_t(qkv, cuda), B, S, N, head_size=d)   # all lengths S: nothing is left out where S is a multiple of 64
    assert O.close_abs_or_rel(out.cpu().numpy(), O.mha(qkv, B, S, N, d), 1e-5, 1e-5)[0]
    cu = O.cu_seqlens(lengths)
    packed = rng.standard_normal((int(cu[-1]), 3 * N * d)).astype(np.float32)
    ref = O.mha(packed, B, S, N, d, cu=cu)
    out = T.mha(_t(packed, cuda), B, S, N, head_size=d, cu_seqlens=_t(cu, cuda))
    assert O.close_abs_or_rel(out.cpu().numpy(), ref, 1e-5, 1e-5)[0]


@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("block", [0, 64])
def test_mha_fp32_scores_that_overflow(cuda, block, d):
    """A block of 64 keys whose scores all overflow to -inf has no weight; the rows are those of the other keys."""
    import tensorrt_b200 as T

    rng = np.random.default_rng(d + block)
    S, B, N = 150, 2, 2
    qkv = rng.standard_normal((S, B, N, 3, d)).astype(np.float32)
    qkv[..., 0, 0] = 1e30
    qkv[..., 1, 0] = 0.0
    qkv[block:block + 64, :, :, 1, 0] = -1e30
    qkv = qkv.reshape(S, B, 3 * N * d)
    out = T.mha(_t(qkv, cuda), B, S, N, d)
    ok, worst, bad = O.close_abs_or_rel(out.cpu().numpy(), O.mha(qkv, B, S, N, d), 1e-5, 1e-5)
    assert ok, (worst, bad)


def test_mha_full_size_properties(cuda):
    """BERT-large S=384, B=64, N=16: with V = const per head the context equals that constant (rows of the
    softmax sum to one), and attention is invariant to a permutation of the keys."""
    import tensorrt_b200 as T

    S, B, N, d = 384, 64, 16, 64
    gen = torch.Generator(device=cuda).manual_seed(0)
    qkv = torch.randn((S * B, N, 3, d), device=cuda, generator=gen).half()
    const = torch.randn((N, d), device=cuda, generator=gen).half()
    qkv[:, :, 2, :] = const[None]
    cu = torch.arange(0, (B + 1) * S, S, dtype=torch.int32, device=cuda)
    out = T.mha(qkv.reshape(S * B, -1), B, S, N, cu_seqlens=cu).reshape(S * B, N, d)
    assert (out.float() - const.float()[None]).abs().max().item() < 5e-3
    qkv2 = torch.randn((S, N, 3, d), device=cuda, generator=gen).half()
    perm = torch.randperm(S, device=cuda, generator=gen)
    shuffled = qkv2.clone()
    shuffled[:, :, 1:, :] = qkv2[perm][:, :, 1:, :]
    cu1 = torch.tensor([0, S], dtype=torch.int32, device=cuda)
    o1 = T.mha(qkv2.reshape(S, -1), 1, S, N, cu_seqlens=cu1).float()
    o2 = T.mha(shuffled.reshape(S, -1), 1, S, N, cu_seqlens=cu1).float()
    assert (o1 - o2).abs().max().item() < 5e-3


# Sequences of a 64-sequence batch whose 16 (sequence, head) work items sit at every position (first ... seventh) of
# a persistent CTA's work list when 1024 items are dealt round-robin to 148 CTAs.
_QUEUE_SAMPLE = [0, 10, 19, 28, 37, 47, 56, 63]


@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("int8", [False, True])
def test_mha_benchmark_size_against_oracle(cuda, packed, int8):
    """BERT-large S = 384, 64 sequences, 16 heads (1024 work items on 148 persistent CTAs), ragged lengths: whole
    sequences compared element-wise with the oracle, chosen so that every position of a CTA's work list is covered
    (a stale Q / K / V tile or a wrong barrier phase on a CTA's later items would show here)."""
    import tensorrt_b200 as T

    S, B, N, d = 384, 64, 16, 64
    rng = np.random.default_rng(384 + packed + 2 * int8)
    lengths = rng.integers(1, S + 1, size=B).astype(np.int32)
    lengths[[0, 19, 63]] = S
    lengths[28] = 129
    lengths[5] = 0
    cu = O.cu_seqlens(lengths)
    rows = int(cu[-1]) if packed else S * B
    x = rng.standard_normal((rows, 3 * N * d)).astype(np.float32)
    st = _status(cuda)
    if int8:
        s_qkv = O.amax_scale(x)
        data = O.quantize(x, 1.0 / s_qkv)
        s1 = float(np.float32(s_qkv) * np.float32(s_qkv) * np.float32(0.125))
        s2 = (1.0 / 127.0) * s_qkv / (0.5 * s_qkv)
        kw = dict(scale_bmm1=s1, scale_softmax=127.0, scale_bmm2=s2)
    else:
        data = x.astype(np.float16)
        kw = {}
    if packed:
        out = T.mha(_t(data, cuda), B, S, N, cu_seqlens=_t(cu, cuda), status=st, **kw).cpu().numpy()
    else:
        out = T.mha(_t(data.reshape(S, B, -1), cuda), B, S, N, mask_idx=_t(lengths, cuda), status=st, **kw).cpu().numpy()
    assert int(st[0]) == 0
    for b in _QUEUE_SAMPLE + [5]:
        if packed:
            seq = data[int(cu[b]):int(cu[b + 1])]
            got = out[int(cu[b]):int(cu[b + 1])]
            one = dict(cu=np.array([0, seq.shape[0]], dtype=np.int32))
        else:
            seq = data.reshape(S, B, -1)[:, b:b + 1]
            got = out[:, b:b + 1]
            one = dict(lengths=lengths[b:b + 1])
        if seq.shape[0] == 0:
            continue
        if int8:
            ref = O.mha_int8(seq, 1, S, N, d, s1, 127.0, s2, **one)
            _assert_int8_attention(got, ref)
        else:
            ref = O.mha(seq, 1, S, N, d, **one)
            ok, worst, bad = O.close_abs_or_rel(got, ref, 1e-2, 1e-2)
            assert ok, (b, worst, bad)


@pytest.mark.parametrize("seed,N,B,smax", [(1, 16, 39, 1500), (2, 16, 31, 1500), (3, 12, 24, 900), (4, 3, 40, 700)])
def test_mha_fp16_many_long_ragged_sequences(cuda, seed, N, B, smax):
    """Many sequences of very different lengths per CTA, most of them longer than the K / V ring holds: work units of
    one or three query tiles, so that the two query streams of a CTA sit on different sequences and each stage of the
    ring is filled several times between two visits of the same stream. The status word must stay 0 (no bounded wait
    may expire) and sampled sequences must match a float32 reference."""
    import tensorrt_b200 as T

    rng = np.random.default_rng(seed)
    d = 64
    lengths = rng.integers(1, smax + 1, size=B).astype(np.int32)
    lengths[0] = smax
    cu = O.cu_seqlens(lengths)
    total = int(cu[-1])
    g = torch.Generator(device="cpu").manual_seed(seed)
    qkv = torch.randn(total, 3 * N * d, generator=g).half().to(cuda)
    st = _status(cuda)
    out = T.mha(qkv, B, int(lengths.max()), N, cu_seqlens=_t(cu, cuda), status=st)
    torch.cuda.synchronize()
    assert int(st[0]) == 0
    x = qkv.float().view(total, N, 3, d)
    o = out.float().view(total, N, d)
    for b in (0, 1, B // 2, B - 1):
        lo, hi = int(cu[b]), int(cu[b + 1])
        q, k, v = (x[lo:hi, :, i].transpose(0, 1) for i in range(3))
        ref = (torch.softmax(q @ k.transpose(-1, -2) * d ** -0.5, -1) @ v).transpose(0, 1)
        err = (o[lo:hi] - ref).abs()
        assert bool(((err <= 1e-2) | (err <= 1e-2 * ref.abs())).all()), float(err.max())


# Batches around the limits of how the query tiles are divided over the CTAs: one sequence per lane of a warp (32), lengths
# kept in shared memory (128), one sequence per thread (384 / 608), fewer tiles than SMs; empty sequences at both ends.
@pytest.mark.parametrize("B,smax", [(2, 512), (32, 150), (33, 300), (128, 140), (129, 260), (700, 130)])
@pytest.mark.parametrize("packed,int8", [(True, False), (False, False), (True, True), (False, True)])
def test_mha_division_of_ragged_batches(cuda, B, smax, packed, int8):
    import tensorrt_b200 as T

    rng = np.random.default_rng(B + smax)
    N, d = 2, 32
    lengths = rng.integers(0, smax + 1, size=B).astype(np.int32)
    lengths[B // 2] = smax
    lengths[[0, B - 1]] = 0 if B > 2 else (1, smax)
    cu = O.cu_seqlens(lengths)
    shape = (int(cu[-1]), 3 * N * d) if packed else (smax, B, 3 * N * d)
    x = rng.standard_normal(shape)
    where = {"cu": cu} if packed else {"lengths": lengths}
    given = {"cu_seqlens": _t(cu, cuda)} if packed else {"mask_idx": _t(lengths, cuda)}
    st = _status(cuda)
    if int8:
        q8 = np.clip(np.rint(x * (127.0 / 4.0)), -128, 127).astype(np.int8)
        s1, s2 = float((4.0 / 127) ** 2 / np.sqrt(d)), 2.0 / 127
        ref = O.mha_int8(q8, B, smax, N, d, s1, 127.0, s2, **where)
        out = T.mha(_t(q8, cuda), B, smax, N, d, scale_bmm1=s1, scale_softmax=127.0, scale_bmm2=s2, status=st, **given)
        _assert_int8_attention(out.cpu().numpy(), ref)
    else:
        qkv = x.astype(np.float16)
        ref = O.mha(qkv, B, smax, N, d, **where)
        out = T.mha(_t(qkv, cuda), B, smax, N, d, status=st, **given)
        ok, worst, bad = O.close_abs_or_rel(out.cpu().numpy(), ref, 1e-2, 1e-2)
        assert ok, (worst, bad)
    assert int(st[0]) == 0


# INT8 pairs dealt longest first: one pair more than SMs, as many sequences as a CTA puts in order and one more (as they come), as
# many rounds as it lists (64 x 148 pairs) and more; equal lengths among them, empty sequences last
@pytest.mark.parametrize("B,N,smax", [(149, 1, 140), (75, 2, 300), (256, 3, 130), (257, 3, 130), (256, 37, 6), (256, 38, 6), (8, 30, 512)])
@pytest.mark.parametrize("layout", ["packed", "interleaved", "fixed", "separate"])
def test_mha_int8_longest_first(cuda, B, N, smax, layout):
    import tensorrt_b200 as T

    rng = np.random.default_rng(B + N)
    d = 32
    lengths = rng.integers(0, smax + 1, size=B).astype(np.int32)
    lengths[rng.integers(0, B, size=B // 4)] = smax // 2
    lengths[[0, B // 2, B - 1]] = 0, smax, 0
    cu = O.cu_seqlens(lengths)
    packed = layout in ("packed", "interleaved")
    x = rng.integers(-127, 128, size=(int(cu[-1]) if packed else smax * B, 3 * N * d)).astype(np.int8)
    s1, s2 = float((4.0 / 127) ** 2 / np.sqrt(d)), 2.0 / 127
    scales = {"scale_bmm1": s1, "scale_softmax": 127.0, "scale_bmm2": s2}
    st = _status(cuda)
    if packed:
        ref = O.mha_int8(x, B, smax, N, d, s1, 127.0, s2, cu=cu)
    else:
        x = x.reshape(smax, B, 3 * N * d)
        ref = O.mha_int8(x, B, smax, N, d, s1, 127.0, s2, lengths=lengths)
    if layout == "packed":
        out = T.mha(_t(x, cuda), B, smax, N, d, cu_seqlens=_t(cu, cuda), status=st, **scales).cpu().numpy()
    elif layout == "fixed":
        out = T.mha(_t(x, cuda), B, smax, N, d, mask_idx=_t(lengths, cuda), status=st, **scales).cpu().numpy()
    elif layout == "separate":
        q, k, v = (_t(a, cuda) for a in x.reshape(smax, B, N, 3, d).transpose(3, 1, 2, 0, 4))
        out = T.attention_bnsd(q, k, v, kv_lengths=_t(lengths, cuda), status=st, **scales)
        out = out.cpu().numpy().transpose(2, 0, 1, 3).reshape(smax, B, N * d)
    else:
        il = x.reshape(-1, N, 3, d).transpose(0, 2, 1, 3).reshape(-1, 3 * N * d)   # [3][N][d / 32][total][32]
        out = O.from_chw32(T.mha(_t(O.to_chw32(il), cuda), B, smax, N, d, cu_seqlens=_t(cu, cuda), interleaved=True, status=st, **scales).cpu().numpy())
    assert int(st[0]) == 0
    _assert_int8_attention(out, ref)


# One, two or three CTAs of the short kernel per SM: pairs at the edges of the rounds that decide it (148 SMs), against the persistent
# kernel, which an S of more than 128 (an upper bound only, in the packed layout) selects. Same bits.
@pytest.mark.parametrize("B", [148, 149, 296, 297, 444, 445, 592, 593, 889])
def test_mha_fp16_short_kernel_residency(cuda, B):
    import tensorrt_b200 as T

    lengths = np.array([(37 * i) % 129 for i in range(B)], dtype=np.int32)
    lengths[B // 2] = 128
    cu = _t(O.cu_seqlens(lengths), cuda)
    x = torch.randn((int(lengths.sum()), 3 * 64), device=cuda, generator=torch.Generator(device=cuda).manual_seed(B)).half()
    st = _status(cuda)
    short, persistent = (T.mha(x, B, S, 1, 64, cu_seqlens=cu, status=st) for S in (128, 129))
    assert int(st[0]) == 0 and torch.equal(short, persistent)


# Four key blocks in the order in which the sequences come: a CTA's tiles go from one key block to four and back, so that scores of blocks 1 to 3 are formed
# beside a tile that has none of them. 9 x 12 pairs of four tiles (432 items), and more sequences than a CTA puts in order; some without keys between
@pytest.mark.parametrize("B,N,S,layout", [(9, 12, 512, "fixed"), (9, 12, 512, "separate"), (9, 12, 400, "fixed"), (260, 1, 512, "packed"), (260, 1, 400, "interleaved")])
@pytest.mark.parametrize("scale_softmax", [127.0, 200.0])
def test_mha_int8_four_key_blocks_as_they_come(cuda, B, N, S, layout, scale_softmax):
    import tensorrt_b200 as T

    rng = np.random.default_rng(B + S)
    d = 32
    lengths = np.array([(20, S, 1, S - 3, 130, 0, 128, 385)[(i + i // 8) % 8] for i in range(B)], dtype=np.int32)
    lengths[1] = S
    cu = O.cu_seqlens(lengths)
    packed = layout in ("packed", "interleaved")
    x = rng.integers(-127, 128, size=(int(cu[-1]) if packed else S * B, 3 * N * d)).astype(np.int8)
    s1, s2 = float((4.0 / 127) ** 2 / np.sqrt(d)), 2.0 / 127
    st = _status(cuda)
    scales = {"scale_bmm1": s1, "scale_softmax": scale_softmax, "scale_bmm2": s2, "status": st}
    if packed:
        ref = O.mha_int8(x, B, S, N, d, s1, scale_softmax, s2, cu=cu)
    else:
        x = x.reshape(S, B, 3 * N * d)
        ref = O.mha_int8(x, B, S, N, d, s1, scale_softmax, s2, lengths=lengths)
    if layout == "packed":
        out = T.mha(_t(x, cuda), B, S, N, d, cu_seqlens=_t(cu, cuda), **scales).cpu().numpy()
    elif layout == "fixed":
        out = T.mha(_t(x, cuda), B, S, N, d, mask_idx=_t(lengths, cuda), **scales).cpu().numpy()
    elif layout == "separate":
        q, k, v = (_t(a, cuda) for a in x.reshape(S, B, N, 3, d).transpose(3, 1, 2, 0, 4))
        out = T.attention_bnsd(q, k, v, kv_lengths=_t(lengths, cuda), **scales).cpu().numpy().transpose(2, 0, 1, 3).reshape(S, B, N * d)
    else:
        il = x.reshape(-1, N, 3, d).transpose(0, 2, 1, 3).reshape(-1, 3 * N * d)   # [3][N][d / 32][total][32]
        out = O.from_chw32(T.mha(_t(O.to_chw32(il), cuda), B, S, N, d, cu_seqlens=_t(cu, cuda), interleaved=True, **scales).cpu().numpy())
    assert int(st[0]) == 0
    _assert_int8_attention(out, ref)


# Few ragged sequences, whose tiles are dealt one by one: as many pairs as SMs, empty sequences, lengths at the edges of tiles, one long one. Then such as
# the host takes for shorter when cut, but the CTAs, counting tiles, keep whole: lengths just beyond a tile, S far above the lengths
@pytest.mark.parametrize("lengths,N,S", [([384, 97, 279, 90, 195, 241, 267, 119], 16, 384), ([1, 0, 512, 129, 128, 127, 257, 0, 385], 16, 512), ([300, 1, 1], 37, 300),
                                         ([0, 500, 3], 49, 500), ([511, 384, 256, 255, 40], 12, 511), ([260] + [16] * 147, 1, 260),
                                         ([160, 153, 160, 133, 160], 16, 160), ([130] + [129] * 6, 12, 130), ([256] + [129] * 91, 1, 256),
                                         ([128] + [100] * 11, 12, 512), ([0, 0, 1, 0], 12, 400), ([300, 5, 260, 129], 37, 512)])
@pytest.mark.parametrize("interleaved", [False, True])
def test_mha_int8_few_ragged_pairs(cuda, lengths, N, S, interleaved):
    import tensorrt_b200 as T

    d, B, smax = 32, len(lengths), S
    cu = O.cu_seqlens(np.array(lengths, dtype=np.int32))
    x = np.random.default_rng(N).integers(-127, 128, size=(int(cu[-1]), 3 * N * d)).astype(np.int8)
    s1, s2 = float((4.0 / 127) ** 2 / np.sqrt(d)), 2.0 / 127
    ref = O.mha_int8(x, B, smax, N, d, s1, 127.0, s2, cu=cu)
    st = _status(cuda)
    scales = {"scale_bmm1": s1, "scale_softmax": 127.0, "scale_bmm2": s2, "cu_seqlens": _t(cu, cuda), "status": st}
    if interleaved:
        il = x.reshape(-1, N, 3, d).transpose(0, 2, 1, 3).reshape(-1, 3 * N * d)   # [3][N][d / 32][total][32]
        out = O.from_chw32(T.mha(_t(O.to_chw32(il), cuda), B, smax, N, d, interleaved=True, **scales).cpu().numpy())
    else:
        out = T.mha(_t(x, cuda), B, smax, N, d, **scales).cpu().numpy()
    assert int(st[0]) == 0
    _assert_int8_attention(out, ref)


@pytest.mark.parametrize("d", [16, 48, 64])
@pytest.mark.parametrize("lengths", [[37], [1, 16, 17, 32, 33, 0, 64, 65, 96, 97, 127, 128], [5] * 150])
def test_mha_fp16_single_key_block(cuda, d, lengths):
    """Launches of sequences up to 128 tokens have a kernel of their own: edges of its 16- and 32-key steps against the oracle,
    and the same bits as the general kernel, which takes over when longer sequences are announced."""
    import tensorrt_b200 as T

    rng = np.random.default_rng(d + len(lengths))
    N, lengths = 3, np.array(lengths, np.int32)
    cu = O.cu_seqlens(lengths)
    B, S = len(lengths), int(lengths.max())
    qkv = rng.standard_normal((int(cu[-1]), 3 * N * d)).astype(np.float16)
    st = _status(cuda)
    out = T.mha(_t(qkv, cuda), B, S, N, d, cu_seqlens=_t(cu, cuda), status=st)
    general = T.mha(_t(qkv, cuda), B, 129, N, d, cu_seqlens=_t(cu, cuda), status=st)
    assert int(st[0]) == 0
    ok, worst, bad = O.close_abs_or_rel(out.cpu().numpy(), O.mha(qkv, B, S, N, d, cu=cu), 1e-2, 1e-2)
    assert ok, (worst, bad)
    assert torch.equal(out, general)
