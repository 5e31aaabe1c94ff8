"""Linears of one or two tokens (csrc/gemv.cu) through the C ABI, against float64 products of the dequantized weights.

Sizes: fewer rows than SMs, row counts that are no multiple of the granule of four, more warps than work units, an
odd number of 256-weight segments, segments that go round the sixteen warps more than once, long K.

Bounds (2-norm, relative).  Result: rounded once to p significant bits, at most 2^-p of each value: 2^-8 (bf16, p = 8)
and 2^-11 (fp16, p = 11).  Q4_K and Q4_0 hold the
activations as 16-bit fixed point per segment: an error of at most amax / 64000 per element, uniform, that is
3.6e-5 of the root mean square for N(0, 1) (amax about 4).  Q4_K's reference is the shader's half arithmetic, two
roundings of at most 2^-11 per weight that this kernel does not make: 2^-10.  Q8_0 is exact up to float32 sums."""
import numpy as np
import pytest
import torch

from conftest import make_acts, make_weights

pytestmark = pytest.mark.gpu
DT = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
RESULT = {"f16": 2.0 ** -11, "bf16": 2.0 ** -8, "f32": 2e-6}
WEIGHT = {0: 5e-5, 2: 1e-6, 3: 2.0 ** -10}


def _status():
    import mlxr_b200 as mx
    st = torch.zeros(1, dtype=torch.int32)
    mx._capi.check(mx._capi.lib.mlxr_stream_status(torch.cuda.current_stream().cuda_stream, st.data_ptr()))
    return int(st[0])


def _dense(oracle, packed, N, K, qt):
    f, h = oracle.dequantize(packed, N, K, qt)
    return torch.from_numpy((h.view(np.float16) if qt == 3 else f).astype(np.float64).reshape(N, K)).cuda()


@pytest.mark.parametrize("qt,dt", [(3, "bf16"), (3, "f16"), (3, "f32"), (0, "bf16"), (0, "f16"), (0, "f32"), (2, "bf16"), (2, "f16")])
@pytest.mark.parametrize("M,N,K", [(1, 4, 256), (2, 5, 256), (1, 67, 768), (2, 593, 512), (1, 1000, 1280), (2, 2369, 4352), (1, 130, 16640), (2, 70, 20992), (1, 33, 32768), (2, 33, 32768)])
def test_linear(oracle, qt, dt, M, N, K):
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    packed = quantize(make_weights(N, K, 7 + N), qt)
    x = make_acts(M, K, 8 + N, DT[dt])[0].cuda()
    b = make_acts(1, N, 9, DT[dt])[0][0].contiguous().cuda() if N % 2 else None
    args = (x, torch.from_numpy(packed).cuda(), M, N, K, mx.QuantType(qt), mx._capi.lib.mlxr_default_group_size(qt), b)
    y = mx.q_gemm_dequant(*args)
    assert torch.equal(y, mx.q_gemm_dequant(*args))
    assert _status() == 0
    want = x.double() @ _dense(oracle, packed, N, K, qt).T + (b.double() if b is not None else 0)
    assert float((y.double() - want).norm() / want.norm()) <= RESULT[dt] + WEIGHT[qt]


@pytest.mark.parametrize("qt,M,N,K", [(3, 1, 80003, 256), (3, 2, 40961, 1024), (0, 1, 76001, 512), (2, 2, 90001, 256), (2, 1, 5, 16384)])
def test_warps_meet_more_than_once(oracle, qt, M, N, K):
    """More rows per CTA than the places for the warps' sums hold (32 tiles of 16 rows, fewer for two tokens), and one tile
    whose stages go round the warps four times.  Rows are drawn from 4096 quantized ones; every result is compared."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    block = quantize(make_weights(4096, K, 3), qt).reshape(4096, -1)
    which = np.random.Generator(np.random.PCG64(5)).integers(0, 4096, N)
    packed = np.ascontiguousarray(block[which]).reshape(-1)
    x = make_acts(M, K, 4, torch.bfloat16)[0].cuda()
    y = mx.q_gemm_dequant(x, torch.from_numpy(packed).cuda(), M, N, K, mx.QuantType(qt), mx._capi.lib.mlxr_default_group_size(qt))
    assert _status() == 0
    want = (x.double() @ _dense(oracle, block.reshape(-1), 4096, K, qt).T)[:, torch.from_numpy(which).cuda()]
    assert float((y.double() - want).norm() / want.norm()) <= RESULT["bf16"] + WEIGHT[qt]
    # no row may be wrong by itself: the largest results are below 6 rms, their rounding below 6 * 2^-8
    assert float((y.double() - want).abs().max() / want.square().mean().sqrt()) <= 6 * (RESULT["bf16"] + WEIGHT[qt])


@pytest.mark.parametrize("qt", [0, 2, 3])
@pytest.mark.parametrize("scale", [1e-30, 1.0, 1e30])
def test_range_of_bf16(oracle, qt, scale):
    """Activations of any magnitude: the segments' scales carry it, nothing over- or underflows inside."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    N, K = 64, 1024
    packed = quantize(make_weights(N, K, 1), qt)
    x = (make_acts(1, K, 2, torch.float32)[0] * scale).to(torch.bfloat16).cuda()
    x[0, 512:] *= 2.0 ** -12
    y = mx.q_gemm_dequant(x, torch.from_numpy(packed).cuda(), 1, N, K, mx.QuantType(qt), mx._capi.lib.mlxr_default_group_size(qt))
    want = x.double() @ _dense(oracle, packed, N, K, qt).T
    assert float((y.double() - want).norm() / want.norm()) <= RESULT["bf16"] + WEIGHT[qt]


@pytest.mark.parametrize("qt", [0, 2, 3])
@pytest.mark.parametrize("M,H,I", [(1, 512, 1280), (2, 768, 2304), (2, 256, 24320)])
def test_block(oracle, qt, M, H, I):
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    g, u, d = (quantize(make_weights(n, k, s), qt) for n, k, s in ((I, H, 1), (I, H, 2), (H, I, 3)))
    xt, xf = make_acts(M, H, 4, torch.bfloat16)
    nt, nf = make_acts(1, H, 5, torch.bfloat16)
    y = mx.mlp_block(xt.cuda(), nt[0].contiguous().cuda(), *(torch.from_numpy(w).cuda() for w in (g, u, d)), I, mx.QuantType(qt), 1e-5)
    assert _status() == 0
    assert oracle.rel_l2(y.float().cpu().numpy(), oracle.mlp_block(xf, nf[0], g, u, d, I, qt, 1e-5, oracle.BF16)) <= 1e-2


@pytest.mark.parametrize("qt,M", [(33, 1), (33, 2), (16, 1)])
def test_formats_of_the_small_batch_kernel(oracle, qt, M):
    """Canonical Q4_K, and NF4 with an odd number of segments, at one and two tokens: the weights keep 16 bits."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    N, K = 300, 1280
    if qt == 33:
        import gguf
        import gguf.quants as gq
        rng = np.random.Generator(np.random.PCG64(3))
        raw = rng.integers(0, 256, size=(N * (K // 256), 144), dtype=np.uint8)
        raw[:, 0:4] = (rng.random((raw.shape[0], 2)) * 0.002 + 0.0005).astype(np.float16).view(np.uint8)
        packed = raw.reshape(-1)
        w = torch.from_numpy(gq.dequantize(packed.reshape(N, -1), gguf.GGMLQuantizationType.Q4_K).astype(np.float64)).cuda()
    else:
        packed = quantize(make_weights(N, K, 1), qt)
        w = _dense(oracle, packed, N, K, qt)
    x = make_acts(M, K, 2, torch.bfloat16)[0].cuda()
    y = mx.q_gemm_dequant(x, torch.from_numpy(packed).cuda(), M, N, K, mx.QuantType(qt), mx._capi.lib.mlxr_default_group_size(qt))
    assert _status() == 0
    want = x.double() @ w.T
    assert float((y.double() - want).norm() / want.norm()) <= RESULT["bf16"] + 2.0 ** -16


@pytest.mark.parametrize("qt", [0, 3])
@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("M,H,I", [(1, 1024, 2816), (2, 1280, 768), (1, 17408, 512), (2, 17408, 512)])
def test_block_rounds_the_normalised_input(qt, dt, M, H, I):
    """n = rmsnorm(x) enters the products rounded to the activation type, as RMSNorm called by itself returns it (rows of
    more than 16384 elements are read a second time for that).  Against the block made of this package's own operators: g,
    u, h and y are rounded on both sides.  Before that the two sides differ by the step of the fixed point at most, where a
    segment's largest value fell to another neighbour and with it the scale: d = sqrt(2) 3.6e-5 of the result.  A rounding
    to p bits turns a difference d into sqrt(d 2^(1 - p)) in the 2-norm (a share d 2^(p - 1) of the values moves by an
    ulp): 6.3e-4 for bf16, 2.2e-4 for fp16, and d itself.  An unrounded n comes out at 4.6e-3 and 6e-4."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    g, u, d = (torch.from_numpy(quantize(make_weights(n, k, s), qt)).cuda() for n, k, s in ((I, H, 1), (I, H, 2), (H, I, 3)))
    x, nw = make_acts(M, H, 4, DT[dt])[0].cuda(), make_acts(1, H, 5, DT[dt])[0][0].contiguous().cuda()
    q, gs = mx.QuantType(qt), mx._capi.lib.mlxr_default_group_size(qt)
    y = mx.mlp_block(x, nw, g, u, d, I, q, 1e-5)
    assert _status() == 0
    n = mx.rmsnorm_fused(x, nw, 1e-5)
    h = mx.swiglu(mx.q_gemm_dequant(n, g, M, I, H, q, gs), mx.q_gemm_dequant(n, u, M, I, H, q, gs))
    want = mx.q_gemm_dequant(h, d, M, H, I, q, gs).double()
    assert float((y.double() - want).norm() / want.norm()) <= {"bf16": 7e-4, "f16": 2.8e-4}[dt]


@pytest.mark.parametrize("qt", [0, 2, 3])
@pytest.mark.parametrize("scale", [2.0 ** -120, 2.0 ** -102, 2.0 ** 126])
def test_ends_of_the_range_of_bf16(oracle, qt, scale):
    """Segments whose largest value lies near either end of the type's range, up to 2.9e38.  The scale of a 4-bit segment
    is 1 / 32000 of its largest value: at 2^-120 a float32 of 13 bits or more (denormal), 2^-13 of the result."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    N, K = 64, 1024
    packed = quantize(make_weights(N, K, 1, std=0.005), qt)
    x = (make_acts(1, K, 2, torch.float32)[0] * scale).clamp(-2.9e38, 2.9e38).to(torch.bfloat16).cuda()
    y = mx.q_gemm_dequant(x, torch.from_numpy(packed).cuda(), 1, N, K, mx.QuantType(qt), mx._capi.lib.mlxr_default_group_size(qt))
    want = x.double() @ _dense(oracle, packed, N, K, qt).T
    assert float((y.double() - want).norm() / want.norm()) <= RESULT["bf16"] + WEIGHT[qt] + 2.0 ** -13


@pytest.mark.parametrize("qt", [0, 2, 3])
@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("norm", [False, True])
def test_nan_reaches_its_row_only(qt, dt, norm):
    """A NaN among finite values makes all of its token's outputs NaN and leaves the other token's alone; one that the
    conversion to fixed point lost came out as finite numbers."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    N, K, M = 96, 768, 2
    w = torch.from_numpy(quantize(make_weights(N, K, 3), qt)).cuda()
    x = make_acts(M, K, 4, DT[dt])[0].cuda()
    x[1, 300] = float("nan")
    q, gs = mx.QuantType(qt), mx._capi.lib.mlxr_default_group_size(qt)
    if norm:
        d = torch.from_numpy(quantize(make_weights(K, 768, 5), qt)).cuda()
        g = torch.from_numpy(quantize(make_weights(768, K, 6), qt)).cuda()
        y = mx.mlp_block(x, torch.ones(K, device="cuda", dtype=DT[dt]), g, g, d, 768, q, 1e-5)
    else:
        y = mx.q_gemm_dequant(x, w, M, N, K, q, gs)
    assert torch.isnan(y[1]).all() and torch.isfinite(y[0]).all()


def test_infinity_beside_large_values_q8_0():
    """bf16, one infinity per token and, in the same segment, a value outside fp16's range: the outputs are infinities with
    the sign of their weight, as the float32 products give them, not NaN."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    N, K, M = 64, 512, 2
    wf = make_weights(N, K, 3)
    wf[:, 40] = np.where(np.arange(N) % 2 == 0, 0.05, -0.05)
    wf[:, 41] = -wf[:, 40]
    x = make_acts(M, K, 4, torch.bfloat16)[0].cuda()
    x[:, 40] = float("inf")
    x[:, 41] = 1e6
    y = mx.q_gemm_dequant(x, torch.from_numpy(quantize(wf, 2)).cuda(), M, N, K, mx.QuantType.Q8_0, 32).float().cpu().numpy()
    assert np.array_equal(y, np.tile(np.where(np.arange(N) % 2 == 0, np.inf, -np.inf).astype(np.float32), (M, 1)))


@pytest.mark.parametrize("M", [1, 2])
def test_float32_activations_of_one_segment(oracle, M):
    """Q4_0 rows of 256 weights: float32 products and sums, no fixed point (2.6e-5)."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    N, K = 500, 256
    packed = quantize(make_weights(N, K, 1), 0)
    x = make_acts(M, K, 2, torch.float32)[0].cuda()
    y = mx.q_gemm_dequant(x, torch.from_numpy(packed).cuda(), M, N, K, mx.QuantType.Q4_0, 32)
    want = x.double() @ _dense(oracle, packed, N, K, 0).T
    assert float((y.double() - want).norm() / want.norm()) <= RESULT["f32"]


@pytest.mark.parametrize("qt,dt,M,N,K", [(3, "bf16", 1, 4096, 2048), (3, "f16", 1, 4097, 2048), (3, "bf16", 1, 300, 2304), (3, "f16", 2, 8192, 1024), (3, "bf16", 2, 8193, 1024), (3, "f32", 2, 4097, 2048),
                                         (3, "bf16", 1, 4096, 4096), (3, "bf16", 1, 4097, 4096), (3, "f16", 1, 8192, 256), (3, "f16", 1, 8193, 256),
                                         (3, "bf16", 2, 2048, 4096), (3, "bf16", 2, 2049, 4096), (3, "f32", 2, 77, 4096), (3, "f32", 1, 77, 4352),
                                         (2, "f16", 1, 1000, 256), (2, "bf16", 2, 1024, 1024), (2, "f16", 2, 1025, 1024), (2, "bf16", 1, 3072, 2048), (2, "bf16", 1, 3073, 2048), (2, "f16", 2, 2048, 2048), (2, "f16", 2, 2049, 2048),
                                         (2, "bf16", 6, 1024, 1024), (2, "bf16", 6, 1025, 1024), (16, "bf16", 4, 2730, 1536), (16, "bf16", 4, 2731, 1536),
                                         (16, "f16", 8, 1536, 512), (16, "f16", 8, 1537, 512), (33, "bf16", 1, 1280, 1024), (33, "bf16", 1, 1281, 1024)])
def test_borders_of_the_small_matrices(oracle, qt, dt, M, N, K):
    """On both sides of the sizes where a linear of a few tokens changes kernels, with bias.  Bounds as above; NF4 and canonical
    Q4_K keep 16 significant bits of the weights or all."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    if qt == 33:
        import gguf
        import gguf.quants as gq
        raw = np.random.Generator(np.random.PCG64(3)).integers(0, 256, size=(N * (K // 256), 144), dtype=np.uint8)
        raw[:, 0:4] = (np.random.Generator(np.random.PCG64(4)).random((raw.shape[0], 2)) * 0.002 + 0.0005).astype(np.float16).view(np.uint8)
        packed = raw.reshape(-1)
        w = torch.from_numpy(gq.dequantize(packed.reshape(N, -1), gguf.GGMLQuantizationType.Q4_K).astype(np.float64)).cuda()
    else:
        packed = quantize(make_weights(N, K, 7), qt)
        w = _dense(oracle, packed, N, K, qt)
    x, b = make_acts(M, K, 8, DT[dt])[0].cuda(), make_acts(1, N, 9, DT[dt])[0][0].contiguous().cuda()
    args = (x, torch.from_numpy(packed).cuda(), M, N, K, mx.QuantType(qt), mx._capi.lib.mlxr_default_group_size(qt), b)
    y = mx.q_gemm_dequant(*args)
    assert torch.equal(y, mx.q_gemm_dequant(*args))
    assert _status() == 0
    want = x.double() @ w.T + b.double()
    assert float((y.double() - want).norm() / want.norm()) <= RESULT[dt] + WEIGHT.get(qt, 2.0 ** -16)


@pytest.mark.parametrize("H,I", [(1024, 1536), (4096, 4096), (4096, 4608)])
def test_one_token_block_of_nf4_at_the_border(oracle, H, I):
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    g, u, d = (quantize(make_weights(n, k, s), 16) for n, k, s in ((I, H, 1), (I, H, 2), (H, I, 3)))
    xt, xf = make_acts(1, H, 4, torch.bfloat16)
    nt, nf = make_acts(1, H, 5, torch.bfloat16)
    y = mx.mlp_block(xt.cuda(), nt[0].contiguous().cuda(), *(torch.from_numpy(w).cuda() for w in (g, u, d)), I, mx.QuantType.NF4, 1e-5)
    assert oracle.rel_l2(y.float().cpu().numpy(), oracle.mlp_block(xf, nf[0], g, u, d, I, 16, 1e-5, oracle.BF16)) <= 1e-2


@pytest.mark.parametrize("M,H,QH,KH", [(1, 512, 5, 1), (2, 512, 5, 1), (1, 2048, 48, 8), (1, 2048, 50, 8)])
def test_stacked_projections_of_a_small_hidden_size(M, H, QH, KH):
    """q / k / v of Q4_K at one and two tokens, on both sides of the border of the kernel for small matrices, against the
    package's own linears and RoPE on the normalised input.  The kernels multiply the unrounded n: x is a row of equal
    magnitudes and the norm weight 1, so n is x either way."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    D = 64
    ws = [torch.from_numpy(quantize(make_weights(n * D, H, 9 + i), 3)).cuda() for i, n in enumerate((QH, KH, KH))]
    cos, sin = mx.compute_rope_tables(16, D, 10000.0, device=torch.device("cuda"))
    x = torch.sign(make_acts(M, H, 4, torch.float32)[0]).half().cuda()
    pos = torch.arange(3, 3 + M, dtype=torch.int32, device="cuda")
    out = mx.qkv_rope(x, torch.ones(H, device="cuda", dtype=torch.float16), *ws, cos, sin, pos, QH, KH, D, mx.QuantType.Q4_K, 0.0)
    assert _status() == 0
    for i, (got, heads) in enumerate(zip(out, (QH, KH, KH))):
        y = mx.q_gemm_dequant(x, ws[i], M, heads * D, H, mx.QuantType.Q4_K, 256).reshape(M, heads, D)
        want = mx.rope_apply(y, cos, sin, pos) if i < 2 else y
        # one ulp of the linear's result at most, 2^-10, where the two sums round to different sides
        assert float((got.double() - want.double()).norm() / want.double().norm()) <= 2.0 ** -11


@pytest.mark.parametrize("M,N,K", [(1, 5120, 512), (1, 5121, 512), (1, 2048, 1280), (1, 2049, 1280), (1, 256, 1536), (1, 257, 1536), (2, 4096, 512), (2, 4097, 512), (2, 2560, 1024), (2, 2561, 1024), (2, 256, 1536), (2, 64, 8192)])
def test_borders_of_small_q8_0(oracle, M, N, K):
    for dt in ("bf16", "f16"):
        test_borders_of_the_small_matrices(oracle, 2, dt, M, N, K)


@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("N,K", [(200, 512), (1000, 1024)])
def test_small_q8_0_multiplies_float32(oracle, M, N, K):
    """One and two tokens of small Q8_0 matrices: float32 products with the bf16 activations as they are, of any range.  Each segment of 256 has
    one of 2^20 on weights of zero, the others are 2^-30: to 16 bits of one scale they are lost."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    wf = make_weights(N, K, 3)
    wf[:, 5::256] = 0.0
    packed = quantize(wf, 2)
    x = make_acts(M, K, 4, torch.float32)[0] * 2.0 ** -30
    x[:, 5::256] = 2.0 ** 20
    x = x.to(torch.bfloat16).cuda()
    y = mx.q_gemm_dequant(x, torch.from_numpy(packed).cuda(), M, N, K, mx.QuantType.Q8_0, 32)
    want = x.double() @ _dense(oracle, packed, N, K, 2).T
    assert float((y.double() - want).norm() / want.norm()) <= RESULT["bf16"] + WEIGHT[2]
