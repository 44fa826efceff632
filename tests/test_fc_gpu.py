"""Parity of the fully connected kernels (tcgen05 FP16 / INT8 / FP32, SIMT FP32) with the CPU oracle."""
import numpy as np
import pytest
import torch

from oracle import bert_oracle as O

pytestmark = pytest.mark.gpu


def _t(a, cuda):
    return torch.from_numpy(np.ascontiguousarray(a)).to(cuda)


def _status(cuda):
    return torch.zeros(4, dtype=torch.int32, device=cuda)


# (m, k, n): BERT-base / BERT-large projections, ragged m, k not a multiple of the 64-wide k block
SHAPES = [(1024, 768, 2304), (1024, 768, 768), (300, 768, 3072), (129, 3072, 768), (1, 64, 16), (257, 1024, 1024),
          (130, 80, 48), (640, 4096, 1024)]


@pytest.mark.parametrize("m,k,n", SHAPES)
@pytest.mark.parametrize("epi", ["none", "bias", "bias_gelu"])
def test_fc_fp16(cuda, m, k, n, epi):
    import tensorrt_b200 as T

    rng = np.random.default_rng(m + k + n)
    a = rng.standard_normal((m, k)).astype(np.float16)
    w = (0.02 * rng.standard_normal((k, n))).astype(np.float16)   # reference layout [K, out]
    bias = (0.02 * rng.standard_normal(n)).astype(np.float32) if epi != "none" else None
    ref = O.fc(a, w, bias, "gelu" if epi == "bias_gelu" else None)
    st = _status(cuda)
    out = T.fc(_t(a, cuda), _t(np.ascontiguousarray(w.T), cuda), None if bias is None else _t(bias, cuda),
               T.ACT_GELU_ERF if epi == "bias_gelu" else T.ACT_NONE, status=st)
    assert int(st[0]) == 0
    # the reference plugin states 1e-3 for its FP16 GEMM (CustomFCPluginDynamic_PluginConfig.yaml:72-77);
    # outputs here are O(0.5), FP16 rounding alone is 2.4e-4 relative
    ok, worst, bad = O.close_abs_or_rel(out.cpu().numpy(), ref, 2e-3, 2e-3)
    assert ok, (worst, bad)


@pytest.mark.parametrize("m,k,n", SHAPES)
@pytest.mark.parametrize("epi", ["none", "bias_gelu"])
@pytest.mark.parametrize("out_i8", [True, False])
def test_fc_int8(cuda, m, k, n, epi, out_i8):
    import tensorrt_b200 as T

    rng = np.random.default_rng(m + k + n + 1)
    a = rng.integers(-127, 128, size=(m, k)).astype(np.int8)
    w = rng.integers(-127, 128, size=(k, n)).astype(np.int8)
    bias = (0.5 * rng.standard_normal(n)).astype(np.float32) if epi != "none" else None
    alpha = 2.0 / (127 * 127 * np.sqrt(k))
    inv = 1.0 / 0.02
    ref = O.fc_int8(a, w, alpha, bias, "gelu" if epi == "bias_gelu" else None, inv if out_i8 else None)
    st = _status(cuda)
    out = T.fc(_t(a, cuda), _t(np.ascontiguousarray(w.T), cuda), None if bias is None else _t(bias, cuda),
               T.ACT_GELU_ERF if epi == "bias_gelu" else T.ACT_NONE, alpha=alpha,
               out_dtype=torch.int8 if out_i8 else torch.float16, out_scale=inv, status=st)
    assert int(st[0]) == 0
    if out_i8:
        ok, worst, bad = O.int8_within_lsb(out.cpu().numpy(), ref)
        assert ok, (worst, bad)
        # Without activation only rounding ties can differ. With GELU the kernel evaluates a fitted tanh form with
        # the hardware's packed FP16 tanh (absolute error up to ~1e-3 * |x| / 2, a few percent of one INT8 step here),
        # so a few percent of the values land on the neighbouring step - never further.
        assert (out.cpu().numpy() == ref).mean() > (0.93 if epi == "bias_gelu" else 0.99)
    else:
        ok, worst, bad = O.close_abs_or_rel(out.cpu().numpy(), ref, 2e-3, 2e-3)
        assert ok, (worst, bad)


def test_fc_int8_exact_accumulation(cuda):
    """alpha = 1, no rounding anywhere: the INT32 accumulators themselves must be exact (FP16 output of small sums)."""
    import tensorrt_b200 as T

    rng = np.random.default_rng(5)
    m, k, n = 256, 128, 256
    a = rng.integers(-3, 4, size=(m, k)).astype(np.int8)
    w = rng.integers(-3, 4, size=(k, n)).astype(np.int8)
    out = T.fc(_t(a, cuda), _t(np.ascontiguousarray(w.T), cuda), out_dtype=torch.float16)
    ref = a.astype(np.int32) @ w.astype(np.int32)
    assert np.abs(ref).max() < 2048  # exactly representable in FP16
    assert np.array_equal(out.cpu().numpy().astype(np.int32), ref)


@pytest.mark.parametrize("m,k,n", [(100, 96, 72), (64, 768, 768)])
def test_fc_fp32(cuda, m, k, n):
    import tensorrt_b200 as T

    rng = np.random.default_rng(m)
    a = rng.standard_normal((m, k)).astype(np.float32)
    w = (0.02 * rng.standard_normal((k, n))).astype(np.float32)
    bias = (0.02 * rng.standard_normal(n)).astype(np.float32)
    ref = O.fc(a, w, bias, "gelu")
    out = T.fc(_t(a, cuda), _t(np.ascontiguousarray(w.T), cuda), _t(bias, cuda), T.ACT_GELU_ERF)
    assert O.close_abs_or_rel(out.cpu().numpy(), ref, 1e-5, 1e-5)[0]


# one row of a tile, one past a row box / a tile, n on both sides of each tile width and of the switch to two CTAs per SM and
# to pair tiles (148 SMs), K below a ring stage, not a multiple of one, and longer than the ring
@pytest.mark.parametrize("m,k,n", [(1, 16, 16), (7, 80, 48), (9, 1040, 144), (127, 768, 2368), (128, 4096, 2384), (129, 64, 4736), (130, 3088, 1200),
                                   (129, 272, 9488), (257, 768, 12624), (300, 96, 12640), (37, 12288, 768)])
@pytest.mark.parametrize("int8", [False, True])
def test_fc_tile_edges(cuda, m, k, n, int8):
    """Every tile width and both kernels against products summed in float64; the tolerance is that of the shapes above."""
    import tensorrt_b200 as T

    gen = torch.Generator(device=cuda).manual_seed(m + k + n)
    bias = 0.5 * torch.randn(n, device=cuda, generator=gen)
    st = _status(cuda)
    if int8:
        a, w = (torch.randint(-127, 128, s, device=cuda, generator=gen, dtype=torch.int32).to(torch.int8) for s in ((m, k), (n, k)))
        alpha, q = 2.0 / (127 * 127 * k ** 0.5), 50.0
        ref = (a.double() @ w.double().T).float() * alpha + bias
        for kind in (torch.int8, torch.float16):
            out = torch.full((m + 1, n), 77, device=cuda, dtype=kind)
            T.fc(a, w, bias, alpha=alpha, out_dtype=kind, out_scale=q, status=st, out=out[:m])
            want = torch.clamp(torch.round(ref * q), -128, 127) if kind == torch.int8 else ref
            diff = (out[:m].float() - want).abs()
            if kind == torch.int8:
                assert float(diff.max()) <= 1 and float((diff > 0).float().mean()) < 1e-2
            else:
                assert bool((diff <= 2e-3 * torch.clamp(want.abs(), min=1.0)).all())
            assert bool((out[m] == 77).all())
    else:
        a = torch.randn(m, k, device=cuda, generator=gen).half()
        w = (torch.randn(n, k, device=cuda, generator=gen) * k ** -0.5).half()
        ref = (a.double() @ w.double().T).float() + bias
        out = torch.full((m + 1, n), 77, device=cuda, dtype=torch.float16)
        T.fc(a, w, bias, status=st, out=out[:m])
        assert bool(((out[:m].float() - ref).abs() <= 2e-3 * torch.clamp(ref.abs(), min=1.0)).all())
        assert bool((out[m] == 77).all())
        # a row does not depend on how many rows are multiplied with it
        more = T.fc(torch.cat([a, torch.randn(3000, k, device=cuda, generator=gen).half()]), w, bias)
        assert torch.equal(out[:m], more[:m])
    assert int(st[0]) == 0


# up to 64 rows the narrow tiles have 64: edges of the 16 rows a warp stores, of the tile, and n at the widest such tile
@pytest.mark.parametrize("m,k,n", [(15, 80, 16), (17, 1040, 144), (48, 3088, 2368), (63, 768, 4736), (64, 4096, 1024), (65, 768, 48)])
@pytest.mark.parametrize("int8", [False, True])
def test_fc_64_row_tiles(cuda, m, k, n, int8):
    test_fc_tile_edges(cuda, m, k, n, int8)


# pair tiles of 160, 192 and 224 columns (an uneven number of column chunks per epilogue warp): last tiles with few columns, an
# odd number of row blocks, one and several tiles per pair of CTAs
@pytest.mark.parametrize("m,k,n", [(2600, 3088, 2000), (2600, 3088, 1040), (3100, 3088, 1072), (2305, 208, 3072)])
@pytest.mark.parametrize("int8", [False, True])
def test_fc_pair_tile_widths(cuda, m, k, n, int8):
    test_fc_tile_edges(cuda, m, k, n, int8)


# tile and k-block edges of the FP32 kernel: one row, single column past a 64-wide tile, K below and above a k-block, K and
# strides that are no multiple of four (element copies), shapes that divide K over a cluster (uneven segments included)
@pytest.mark.parametrize("m,k,n", [(1, 4, 1), (65, 20, 67), (64, 7, 64), (33, 1001, 130), (38, 3072, 768), (200, 784, 96), (1024, 768, 768)])
@pytest.mark.parametrize("epi", ["none", "bias_gelu"])
def test_fc_fp32_tile_edges(cuda, m, k, n, epi):
    """Tolerance: a random walk of k roundings to 2^-24 of sums of size 0.02 sqrt(k) stays below 0.02 k 2^-24 < 4e-6."""
    import tensorrt_b200 as T

    rng = np.random.default_rng(m + k + n)
    a = rng.standard_normal((m, k)).astype(np.float32)
    w = (0.02 * rng.standard_normal((k, n))).astype(np.float32)
    bias = (0.02 * rng.standard_normal(n)).astype(np.float32) if epi != "none" else None
    ref = O.fc(a, w, bias, "gelu" if epi == "bias_gelu" else None)
    out = torch.full((m + 1, n), 7.0, device=cuda)
    T.fc(_t(a, cuda), _t(np.ascontiguousarray(w.T), cuda), None if bias is None else _t(bias, cuda),
         T.ACT_GELU_ERF if epi == "bias_gelu" else T.ACT_NONE, out=out[:m])
    assert O.close_abs_or_rel(out[:m].cpu().numpy(), ref, 1e-5, 1e-5)[0]
    assert bool((out[m] == 7.0).all())   # nothing written past the last row


# K in one, two, four and eight segments. K below 384 or no multiple of four: multiply-adds, rows for which a tile's segments go to one CTA each
# and to one CTA (`one_wave`, of 64 x 64 tiles on 148 SMs); K = 400, 768 and 3072: tensor cores, with these rows 32 to 128 columns, clusters and single CTAs
@pytest.mark.parametrize("k,n", [(80, 96), (192, 200), (400, 768), (768, 768), (3072, 768), (1001, 130)])
def test_fc_fp32_rows_do_not_depend_on_m(cuda, k, n):
    """The same bits for a row whatever it is multiplied with."""
    import tensorrt_b200 as T

    gen = torch.Generator(device=cuda).manual_seed(k + n)
    one_wave = 64 * (4 * 148 // ((n + 63) // 64)) - 5
    a = torch.randn(one_wave + 1000, k, device=cuda, generator=gen)
    w, bias = 0.02 * torch.randn(n, k, device=cuda, generator=gen), 0.02 * torch.randn(n, device=cuda, generator=gen)
    a[3] = -0.0   # the sign of a zero, too
    every = T.fc(a, w, None)
    assert bool(((every.double() - a.double() @ w.double().T).abs() <= 1e-5 * torch.clamp(every.abs(), min=1.0)).all())
    for m in (1, 37, 130, 520, 1024, 2100, one_wave):
        assert torch.equal(T.fc(a[:m], w, None).view(torch.int32), every[:m].view(torch.int32)), m
    assert torch.equal(T.fc(a[:37], w, bias, T.ACT_GELU_ERF), T.fc(a[:one_wave], w, bias, T.ACT_GELU_ERF)[:37])


# K on either side of where the FP32 product goes to the tensor cores; one row and column, edges of their tiles, a tail of K
@pytest.mark.parametrize("m,k,n", [(1, 384, 1), (70, 380, 130), (129, 388, 97), (70, 1000, 130), (300, 768, 96), (129, 4096, 257)])
def test_fc_fp32_values_without_exact_parts(cuda, m, k, n):
    """Infinities, NaN and numbers with bits below 2^-133 have no three exact BF16 parts: the outputs that they meet come out as FP32 multiply-adds
    give them (infinities and NaN where float64 has them, others within k 2^-24 of the sum of the products' magnitudes)."""
    import tensorrt_b200 as T

    gen = torch.Generator(device=cuda).manual_seed(m + k + n)
    a, w = torch.randn(m, k, device=cuda, generator=gen), torch.randn(n, k, device=cuda, generator=gen)
    plain = T.fc(a, w)
    bound = k * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    assert bool(((plain.double() - a.double() @ w.double().T).abs() <= bound).all())
    a[0, 3] = float("inf")
    w[n - 1, 5] = float("nan")
    if m > 2:
        a[2] *= 1e-36
        a[m - 1, k - 1] = -float("inf")
        a[1] = 0
        w[1] *= 1e-34
        w[2] = 0
    ref, out = a.double() @ w.double().T, T.fc(a, w)
    finite = torch.isfinite(ref)
    assert torch.equal(torch.isnan(ref), torch.isnan(out))
    assert torch.equal(ref[torch.isinf(ref)].float(), out[torch.isinf(ref)])
    size = torch.nan_to_num(a.double().abs(), 0, 0, 0) @ torch.nan_to_num(w.double().abs(), 0, 0, 0).T
    assert bool(((out.double() - ref).abs() <= k * 2.0 ** -24 * size + 1e-42)[finite].all())
    # rows and columns that meet none of these are untouched by them
    rows = [i for i in range(m) if i not in (0, 1, 2, m - 1)]
    if rows:
        assert torch.equal(out[rows][:, 3:n - 1], plain[rows][:, 3:n - 1])


# a group that is cut together (32 numbers of a row of A, 8 of a row of Wt) and its edges; a small number on either side of the limit
@pytest.mark.parametrize("m,k,n", [(130, 384, 140), (3, 772, 33), (200, 4096, 70)])
@pytest.mark.parametrize("size", [1e-41, 1e-38, 2.0 ** -109, 2.0 ** -103, 1e-30])
@pytest.mark.parametrize("small_wt", [False, True])
def test_fc_fp32_small_numbers_beside_large_ones(cuda, m, k, n, size, small_wt):
    """Numbers too small for three BF16 parts, or nearly so, that share a row with ordinary ones, which meet zeros: the outputs consist of the small ones alone.
    k roundings to 2^-24 in a row, as a random walk."""
    import tensorrt_b200 as T

    gen = torch.Generator(device=cuda).manual_seed(m + k + n)
    a, w = torch.randn(m, k, device=cuda, generator=gen), torch.randn(n, k, device=cuda, generator=gen)
    small, large = (w, a) if small_wt else (a, w)
    small *= size
    large *= 1e35
    small[:, ::8] = 1.0
    large[:, ::8] = 0.0
    ref = a.double() @ w.double().T
    assert float((T.fc(a, w).double() - ref).norm() / ref.norm()) <= k ** 0.5 * 2.0 ** -24


def _off_by_four_bytes(x):
    """The same numbers where the TMA unit cannot read them: the product is then formed by the FP32 multiply-add kernel."""
    moved = torch.empty(x.numel() + 1, device=x.device)[1:].view(x.shape)
    return moved.copy_(x)


# one CTA per segment of K and one for all; a row's, a column's and a whole tile's outputs; edges of the 4 x 4 outputs that a warp computes
@pytest.mark.parametrize("m,k,n", [(130, 384, 142), (129, 772, 97), (70, 4096, 130), (1030, 768, 770), (1030, 3072, 770)])
def test_fc_fp32_outputs_computed_again(cuda, m, k, n):
    """Outputs that meet numbers without exact parts: no further from float64 than the multiply-add kernel on the same numbers, and
    the same bits whatever they are multiplied with."""
    import tensorrt_b200 as T

    gen = torch.Generator(device=cuda).manual_seed(m + k + n)
    a, w = torch.randn(m, k, device=cuda, generator=gen), torch.randn(n, k, device=cuda, generator=gen)
    a[2] *= 2.0 ** -120
    a[m - 1] *= 2.0 ** -115
    w[1] *= 2.0 ** -112
    every = T.fc(a, w)
    for rows, cols in ((slice(2, 3), slice(2, n)), (slice(m - 1, m), slice(2, n)), (slice(3, m - 1), slice(1, 2))):
        ref = a[rows].double() @ w[cols].double().T
        plain = T.fc(_off_by_four_bytes(a[rows]), w[cols].contiguous())
        assert float((every[rows, cols].double() - ref).norm()) <= float((plain.double() - ref).norm())
    assert torch.equal(T.fc(a[:33], w).view(torch.int32), every[:33].view(torch.int32))
    a = torch.randn(m, k, device=cuda, generator=gen) * 2.0 ** -112
    ref = a.double() @ w.double().T
    assert float((T.fc(a, w).double() - ref).norm()) <= float((T.fc(_off_by_four_bytes(a), w).double() - ref).norm())


# K from where the tensor cores take it on (a tail included), tiles of few and many columns
@pytest.mark.parametrize("m,k,n", [(200, 384, 130), (200, 772, 130), (1030, 768, 2304), (300, 1024, 770), (200, 3072, 768), (520, 4096, 1024)])
@pytest.mark.parametrize("values", ["normal", "rectified", "one sign", "around one"])
def test_fc_fp32_error_against_float64(cuda, values, m, k, n):
    """No further from float64 (2-norm over m n outputs) than the multiply-add kernel on the same numbers, whatever their signs; on numbers of
    one sign the mean error is below half a unit of the last place too (2^-24)."""
    import tensorrt_b200 as T

    gen = torch.Generator(device=cuda).manual_seed(m + k + n)
    a, w = torch.randn(m, k, device=cuda, generator=gen), torch.randn(n, k, device=cuda, generator=gen)
    if values == "rectified":
        a = torch.clamp(a, min=0.0)
    elif values == "one sign":
        a, w = torch.rand(m, k, device=cuda, generator=gen), torch.rand(n, k, device=cuda, generator=gen)
    elif values == "around one":
        a, w = 1 + 0.2 * a, 1 + 0.2 * w
    st = _status(cuda)
    ref, out, plain = a.double() @ w.double().T, T.fc(a, w, status=st).double(), T.fc(_off_by_four_bytes(a), w).double()
    assert int(st[0]) == 0
    assert float((out - ref).norm()) <= float((plain - ref).norm())
    if values in ("one sign", "around one"):
        assert abs(float(((out - ref) / ref).mean())) <= 2.0 ** -24


@pytest.mark.parametrize("m,k,n", [(130, 384, 142), (1030, 768, 770)])
def test_fc_fp32_sums_near_the_largest_numbers(cuda, m, k, n):
    """Sums of 2^127 on the way to a small result, and the largest number itself, whose BF16 rounding is infinity: exact in any order."""
    import tensorrt_b200 as T

    a, w = torch.full((m, k), 2.0 ** 122, device=cuda), torch.ones(n, k, device=cuda)
    a.view(m, k // 64, 64)[:, :, 32:] = -2.0 ** 122
    a[:, k - 1] = 0.0
    w[:, 0] = 0.5
    a[5] = 0.0
    a[5, 7] = torch.finfo(torch.float32).max
    w[3] = 0.5
    ref, out = a.double() @ w.double().T, T.fc(a, w)
    assert torch.equal(out.double(), ref)


# A tile's place in the ring must not be filled again before all of its numbers have been read: when it was, one launch in some 1500 of 2296 x 3072 x 768 had rows
# that were off. 128, 96, 64 and 32 columns, launch after launch with another shape between, so that the loads find the memory system in all states
@pytest.mark.parametrize("m,k,n", [(2296, 768, 3072), (1024, 768, 3072), (2296, 768, 768), (512, 4096, 1024)])
def test_fc_fp32_same_bits_every_time(cuda, m, k, n):
    import tensorrt_b200 as T

    gen = torch.Generator(device=cuda).manual_seed(m + n)
    a, w = torch.randn(m, k, device=cuda, generator=gen), torch.randn(n, k, device=cuda, generator=gen)
    x, y = torch.randn(700, 1536, device=cuda, generator=gen), torch.randn(768, 1536, device=cuda, generator=gen)
    first = T.fc(a, w)
    ref = a.double() @ w.double().T
    assert float((first.double() - ref).norm()) <= 2.0 ** -22 * float(ref.norm())
    out = torch.empty_like(first)
    wrong = torch.zeros((), dtype=torch.int64, device=cuda)
    for i in range(2500):
        if i % 2:
            T.fc(x, y)
        T.fc(a, w, out=out)
        wrong += (out.view(torch.int32) != first.view(torch.int32)).sum()
    assert int(wrong) == 0


# 96 and 128 columns: the products of a chunk are waited for in two halves, the second by warps that have read the sums of the first. Another stream keeps the
# SMs busy beside them, so that the barriers are asked early and late
@pytest.mark.parametrize("m,k,n", [(6339, 1540, 129), (2115, 3072, 97), (1024, 768, 2304)])
def test_fc_fp32_halves_of_a_tile_beside_other_work(cuda, m, k, n):
    import tensorrt_b200 as T

    gen = torch.Generator(device=cuda).manual_seed(m + n)
    a, w = torch.randn(m, k, device=cuda, generator=gen), torch.randn(n, k, device=cuda, generator=gen)
    x, y = torch.randn(512, 1024, device=cuda, generator=gen).half(), torch.randn(1024, 1024, device=cuda, generator=gen).half()
    st = _status(cuda)
    first = T.fc(a, w, status=st)
    ref = a.double() @ w.double().T
    assert float((first.double() - ref).norm()) <= 2.0 ** -22 * float(ref.norm())   # two units of the last place on average
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for _ in range(20):
        with torch.cuda.stream(side):
            T.fc(x, y)
        assert torch.equal(T.fc(a, w, status=st), first)
    torch.cuda.synchronize()
    assert int(st[0]) == 0


# each width of the tiles, with all segments of K (two, four, eight) in a CTA and with one each, as fcF32 chooses them on 148 SMs; rows, columns and K that
# fill neither a tile nor a chunk
@pytest.mark.parametrize("m,k,n", [
    (4547, 388, 65), (4163, 708, 33), (67, 1540, 1793), (67, 388, 33), (67, 708, 33), (67, 1540, 33),              # 32 columns: 2, 4, 8 held; 2, 4, 8 CTAs
    (6339, 388, 65), (6339, 708, 65), (6339, 1540, 65), (4547, 388, 33), (67, 708, 1025), (67, 1540, 449),         # 64
    (6339, 388, 129), (6339, 708, 129), (6339, 1540, 129), (6339, 452, 65), (67, 708, 2049), (67, 1540, 897),      # 96
    (6339, 388, 193), (6339, 708, 193), (6339, 1540, 193), (2115, 708, 97), (67, 1540, 1345), (1024, 768, 2304)])  # 128 (no two CTAs)
def test_fc_fp32_every_width_and_division_of_k(cuda, m, k, n):
    """No further from float64 than the multiply-add kernel, the bits of fewer rows, outputs computed again, the epilogue, and nothing written beyond."""
    import tensorrt_b200 as T

    gen = torch.Generator(device=cuda).manual_seed(m + k + n)
    a, w, bias = (torch.randn(*s, device=cuda, generator=gen) for s in ((m, k), (n, k), (n,)))
    st = _status(cuda)
    out = torch.full((m + 1, n), 7.0, device=cuda)
    T.fc(a, w, status=st, out=out[:m])
    ref = a.double() @ w.double().T
    assert float((out[:m].double() - ref).norm()) <= float((T.fc(_off_by_four_bytes(a), w).double() - ref).norm())
    assert torch.equal(T.fc(a[-38:], w), out[m - 38:m])
    # erff is good to 2 units of the last place, the sum to half of one of its terms' magnitudes
    want = torch.nn.functional.gelu(out[:m].double() * 0.5 + bias.double())
    assert bool(((T.fc(a, w, bias, T.ACT_GELU_ERF, alpha=0.5).double() - want).abs() <= 2.0 ** -21 * torch.clamp(out[:m].abs() + bias.abs(), min=1.0)).all())
    a[m - 2] *= 2.0 ** -120
    w[n - 1] *= 2.0 ** -120
    a[1, k - 1] = float("nan")
    w[1, 0] = -float("inf")
    again = T.fc(a, w, status=st, out=out[:m])
    ref = a.double() @ w.double().T
    assert int(st[0]) == 0 and bool((out[m] == 7.0).all())
    assert torch.equal(torch.isnan(ref), torch.isnan(again)) and torch.equal(torch.isinf(ref), torch.isinf(again))
    finite = torch.isfinite(ref)
    # the 2-norm of the error is below 2^-23 of the result's for normal values, a result |a| |w| k^-0.5 on average: eight times that for the largest of
    # a million; 2^-140 for what lies below the smallest numbers
    size = torch.nan_to_num(a.double() ** 2, 0, 0, 0).sum(1, keepdim=True).sqrt() * torch.nan_to_num(w.double() ** 2, 0, 0, 0).sum(1).sqrt()
    assert bool(((again.double() - ref).abs()[finite] <= (2.0 ** -20 * k ** -0.5 * size + 2.0 ** -140)[finite]).all())


# products around the smallest normal number, a row of zeros among them
@pytest.mark.parametrize("exponent", [-50, -56, -63, -66, -70])
@pytest.mark.parametrize("m,k,n", [(130, 384, 142), (1030, 768, 770), (70, 4096, 130)])
def test_fc_fp32_sums_near_the_smallest_numbers(cuda, exponent, m, k, n):
    """No further from float64 than the multiply-add kernel (which rounds to 2^-149 there, where the tensor core cuts off). At the smallest
    exponents both round every product to 2^-149: errors of one size, whose norm over m n outputs scatters by (2 m n)^-0.5 on each side."""
    import tensorrt_b200 as T

    gen = torch.Generator(device=cuda).manual_seed(m + k + n)
    a, w = (torch.randn(s, k, device=cuda, generator=gen) * 2.0 ** exponent for s in (m, n))
    a[5] = 0.0
    ref, out, plain = a.double() @ w.double().T, T.fc(a, w), T.fc(_off_by_four_bytes(a), w)
    assert float((out.double() - ref).norm()) <= (1 + 4 / (m * n) ** 0.5) * float((plain.double() - ref).norm())
    assert bool((out[5] == 0.0).all())
    assert torch.equal(T.fc(a[:33], w), out[:33])


def test_fc_linearity_full_size(cuda):
    """BERT-large sizes (24576 x 1024 -> 4096): fc(a1 + a2) == fc(a1) + fc(a2) within FP16 rounding, and a
    checksum of the INT8 product equals the checksum computed from row/column sums."""
    import tensorrt_b200 as T

    gen = torch.Generator(device=cuda).manual_seed(0)
    m, k, n = 24576, 1024, 4096
    a8 = torch.randint(-127, 128, (m, k), device=cuda, generator=gen, dtype=torch.int32).to(torch.int8)
    w8 = torch.randint(-127, 128, (n, k), device=cuda, generator=gen, dtype=torch.int32).to(torch.int8)
    out = T.fc(a8, w8, alpha=1.0 / 65536, out_dtype=torch.float16).double() * 65536
    # sum over all outputs = sum_k (sum_m a[m,k]) * (sum_n w[n,k])
    expect = (a8.double().sum(0) * w8.double().sum(0)).sum().item()
    got = out.sum().item()
    scale = (a8.double().abs().sum(0) * w8.double().abs().sum(0)).sum().item()
    assert abs(got - expect) / scale < 1e-4
    a1 = torch.randn((2048, k), device=cuda, generator=gen).half()
    a2 = torch.randn((2048, k), device=cuda, generator=gen).half()
    wt = (0.02 * torch.randn((n, k), device=cuda, generator=gen)).half()
    lhs = T.fc((a1.float() + a2.float()).half(), wt).float()
    rhs = T.fc(a1, wt).float() + T.fc(a2, wt).float()
    assert (lhs - rhs).abs().max().item() < 2e-2


def _sampled_rows(m, rng):
    """Rows spread over the whole range: two of every 256-row block (the unit a pair of CTAs owns), the last 32 rows
    and some at random - so that every tile a persistent cluster takes, not only its first, is compared."""
    rows = [blk * 256 + int(o) for blk in range(m // 256) for o in rng.integers(0, 256, size=2)]
    rows += list(range(m - 32, m)) + list(rng.integers(0, m, size=128))
    return np.unique(np.array(rows, dtype=np.int64))


# the four projections of a BERT-large layer at the benchmark's row count (64 sequences x 384 tokens)
LARGE = [(24576, 1024, 3072, "bias"), (24576, 1024, 1024, "none"), (24576, 1024, 4096, "bias_gelu"), (24576, 4096, 1024, "none")]


@pytest.mark.parametrize("m,k,n,epi", LARGE)
def test_fc_fp16_benchmark_shapes(cuda, m, k, n, epi):
    """Element-wise against the oracle at the benchmarked size: 312-1248 tiles on 74 CTA pairs, i.e. the second and
    later tiles of every persistent cluster (accumulator double-buffering, stage parities) are checked too."""
    import tensorrt_b200 as T

    rng = np.random.default_rng(m + k + n)
    gen = torch.Generator(device=cuda).manual_seed(k + n)
    a = torch.randn((m, k), device=cuda, generator=gen).half()
    wt = (0.02 * torch.randn((n, k), device=cuda, generator=gen)).half()
    bias = (0.02 * torch.randn((n,), device=cuda, generator=gen)).float() if epi != "none" else None
    st = _status(cuda)
    out = T.fc(a, wt, bias, T.ACT_GELU_ERF if epi == "bias_gelu" else T.ACT_NONE, status=st)
    assert int(st[0]) == 0
    rows = _sampled_rows(m, rng)
    idx = torch.from_numpy(rows).to(cuda)
    ref = O.fc(a[idx].cpu().numpy(), wt.cpu().numpy().T, None if bias is None else bias.cpu().numpy(),
               "gelu" if epi == "bias_gelu" else None)
    ok, worst, bad = O.close_abs_or_rel(out[idx].cpu().numpy(), ref, 2e-3, 2e-3)
    assert ok, (worst, bad)


@pytest.mark.parametrize("m,k,n,epi", LARGE)
def test_fc_int8_benchmark_shapes(cuda, m, k, n, epi):
    import tensorrt_b200 as T

    rng = np.random.default_rng(m + k + n + 1)
    gen = torch.Generator(device=cuda).manual_seed(k + n + 1)
    a = torch.randint(-127, 128, (m, k), device=cuda, generator=gen, dtype=torch.int32).to(torch.int8)
    wt = torch.randint(-127, 128, (n, k), device=cuda, generator=gen, dtype=torch.int32).to(torch.int8)
    bias = (0.5 * torch.randn((n,), device=cuda, generator=gen)).float() if epi != "none" else None
    alpha = 2.0 / (127 * 127 * np.sqrt(k))
    inv = 1.0 / 0.02
    st = _status(cuda)
    out = T.fc(a, wt, bias, T.ACT_GELU_ERF if epi == "bias_gelu" else T.ACT_NONE, alpha=alpha, out_dtype=torch.int8,
               out_scale=inv, status=st)
    assert int(st[0]) == 0
    rows = _sampled_rows(m, rng)
    idx = torch.from_numpy(rows).to(cuda)
    ref = O.fc_int8(a[idx].cpu().numpy(), wt.cpu().numpy().T, alpha, None if bias is None else bias.cpu().numpy(),
                    "gelu" if epi == "bias_gelu" else None, inv)
    got = out[idx].cpu().numpy()
    ok, worst, bad = O.int8_within_lsb(got, ref)
    assert ok, (worst, bad)
    assert (got == ref).mean() > (0.93 if epi == "bias_gelu" else 0.99)
