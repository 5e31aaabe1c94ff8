"""Small-batch tensor-core linear (Q4_K and Q4_0, 3 <= M <= 64; csrc/smallm.cu) through the C ABI vs the oracle.

Gate 2e-2 relative L2.  The tests use 2e-3 for fp16 activations (the weights are converted with
the shader's own fp16 arithmetic, q_gemm_dequant.metal:244-256) and 1e-2 for bf16 (scale, min and
weight are rounded to bf16: about 3e-3 relative).  Shapes cover every padded batch width (16, 32,
64), N that is not a multiple of the 128-row tile, a single super-block of K, tiles shared by
several CTAs (more work units than one CTA's share) and tiles owned by one CTA."""
import numpy as np
import pytest
import torch

from conftest import make_acts, make_weights

pytestmark = pytest.mark.gpu
DT = {"f16": torch.float16, "bf16": torch.bfloat16}
TIGHT = {"f16": 2e-3, "bf16": 1e-2}


def _status():
    import mlxr_b200 as mx
    st = torch.zeros(1, dtype=torch.int32)
    mx._capi.check(mx._capi.lib.mlxr_stream_status(torch.cuda.current_stream().cuda_stream, st.data_ptr()))
    return int(st[0])


def _run(oracle, M, N, K, dt, bias=False, seed=0, rows=None, twice=False, qt=3):
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    packed = quantize(make_weights(N, K, 100 + seed), qt)
    xt, xf = make_acts(M, K, 200 + seed, DT[dt])
    bt = bf = None
    if bias:
        bt, bf = make_acts(1, N, 300 + seed, DT[dt])
        bt, bf = bt[0].contiguous(), bf[0]
    xd, wd, bd = xt.cuda(), torch.from_numpy(packed).cuda(), (bt.cuda() if bias else None)
    gs = mx._capi.lib.mlxr_default_group_size(qt)
    y = mx.q_gemm_dequant(xd, wd, M, N, K, mx.QuantType(qt), gs, bd)
    if twice:   # the tile counters must have cleared themselves, and the result must not depend on arrival order
        y2 = mx.q_gemm_dequant(xd, wd, M, N, K, mx.QuantType(qt), gs, bd)
        assert torch.equal(y, y2)
    torch.cuda.synchronize()
    assert _status() == 0
    yn = y.float().cpu().numpy()
    if rows is not None:
        return oracle.rel_l2(yn[rows], oracle.linear(xf[rows], packed, N, qt, bf))
    return oracle.rel_l2(yn, oracle.linear(xf, packed, N, qt, bf))


@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("M,N,K", [(3, 128, 256), (4, 130, 512), (8, 1000, 768), (9, 256, 256), (16, 512, 1024),
                                   (17, 384, 1280), (32, 640, 2048), (33, 200, 512), (64, 1024, 1024)])
def test_shapes(oracle, dt, M, N, K):
    assert _run(oracle, M, N, K, dt, seed=M, twice=True) <= TIGHT[dt]


@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("M,N,K", [(3, 128, 256), (9, 200, 512), (16, 512, 1024), (33, 384, 1280), (64, 1000, 768)])
def test_q4_0_shapes(oracle, dt, M, N, K):
    """Q4_0: the same 144 bytes per 256 weights of a row, read as eight 18-byte blocks."""
    assert _run(oracle, M, N, K, dt, seed=M + 50, twice=True, qt=0, bias=(N == 200)) <= TIGHT[dt]


def test_q4_0_decode_shape_sampled_rows(oracle):
    assert _run(oracle, 32, 5632, 2048, "f16", rows=np.array([0, 17, 31]), seed=8, twice=True, qt=0) <= TIGHT["f16"]


@pytest.mark.parametrize("dt", ["bf16", "f16"])
def test_bias_and_ragged_rows(oracle, dt):
    assert _run(oracle, 5, 8, 256, dt, bias=True, seed=1) <= TIGHT[dt]
    assert _run(oracle, 48, 257, 768, dt, bias=True, seed=2, twice=True) <= TIGHT[dt]


@pytest.mark.parametrize("M,N,K", [(16, 14336, 4096), (32, 4096, 14336), (64, 28672, 4096)])
def test_decode_shapes_sampled_rows(oracle, M, N, K):
    """Llama-3-8B-shaped linears at small batch: a sample of batch rows against the oracle."""
    rows = np.array([0, M // 2, M - 1])
    assert _run(oracle, M, N, K, "bf16", rows=rows, seed=7, twice=True) <= TIGHT["bf16"]


def test_many_units_per_cta_and_shared_tiles(oracle):
    """N = 148 * 128 + 64 rows and K = 3 super-blocks: every CTA's range of work units crosses a
    tile boundary, so most tiles are summed from two CTAs' partial sums."""
    assert _run(oracle, 12, 148 * 128 + 64, 768, "f16", rows=np.array([0, 5, 11]), seed=9, twice=True) <= TIGHT["f16"]


def test_non_finite_input_propagates():
    """A NaN in one batch row reaches that row's outputs only."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    N, K, M = 256, 512, 6
    packed = torch.from_numpy(quantize(make_weights(N, K, 3), 3)).cuda()
    x = torch.randn(M, K).to(torch.bfloat16)
    x[2, 17] = float("nan")
    y = mx.q_gemm_dequant(x.cuda(), packed, M, N, K, mx.QuantType(3), 256, None).float().cpu()
    assert torch.isnan(y[2]).all()
    assert torch.isfinite(y[[0, 1, 3, 4, 5]]).all()


def test_bit_identical_over_many_launches():
    """Launches of different geometry back to back, many times: every result of a shape equals the
    first one bit for bit (tiles shared between CTAs are summed in CTA order, whatever the arrival
    order; a stale barrier phase or a counter left over from another shape would show here)."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    shapes = [(64, 1536, 2048), (32, 640, 3584), (9, 1024, 1024)]
    data = []
    for i, (M, N, K) in enumerate(shapes):
        w = torch.from_numpy(quantize(make_weights(N, K, 40 + i), 3)).cuda()
        x = torch.randn(M, K, generator=torch.Generator().manual_seed(i)).to(torch.bfloat16).cuda()
        data.append((x, w, M, N, K, mx.q_gemm_dequant(x, w, M, N, K, mx.QuantType(3), 256, None).clone()))
    for _ in range(60):
        for x, w, M, N, K, first in data:
            assert torch.equal(mx.q_gemm_dequant(x, w, M, N, K, mx.QuantType(3), 256, None), first)
    torch.cuda.synchronize()
    assert _status() == 0


@pytest.mark.parametrize("qt", [2, 16, 33])
@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("M,N,K", [(3, 2, 256), (8, 129, 768), (9, 131, 1280), (17, 200, 512), (64, 385, 768)])
def test_other_formats(oracle, qt, dt, M, N, K):
    """Q8_0, NF4 and canonical ggml Q4_K: odd row counts and odd numbers of super-blocks (NF4 rows are
    then only 8-byte aligned).  Against float32 products of the dequantized weights.  Up to batch 8,
    and for canonical Q4_K at any, the weights keep 16 (bf16) or 22 (fp16) significant bits, so the
    result's own rounding is what is left: at most 2^-9 (2^-12) of each value, about 0.6 of that in the
    2-norm; 2^-9 and 2^-11 leave room for sums that cancel.  Wider batches round the weight once more:
    twice that."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    if qt == 33:
        rng = np.random.Generator(np.random.PCG64(M + N))
        raw = rng.integers(0, 256, size=(N * (K // 256), 144), dtype=np.uint8)
        raw[:, 0:2] = (rng.random(raw.shape[0]) * 0.002 + 0.0005).astype(np.float16).view(np.uint8).reshape(-1, 2)
        raw[:, 2:4] = (rng.random(raw.shape[0]) * 0.004 + 0.0005).astype(np.float16).view(np.uint8).reshape(-1, 2)
        packed = raw.reshape(-1)
        import gguf
        import gguf.quants as gq
        w = gq.dequantize(packed.reshape(N, -1), gguf.GGMLQuantizationType.Q4_K).astype(np.float64)
    else:
        packed = quantize(make_weights(N, K, 100 + M), qt)
        w = oracle.dequantize(packed, N, K, qt)[0].astype(np.float64).reshape(N, K)
    xt, xf = make_acts(M, K, 200 + M, DT[dt])
    bt, bf = make_acts(1, N, 300, DT[dt])
    want = xf.astype(np.float64) @ w.T + bf[0]
    args = (xt.cuda(), torch.from_numpy(packed).cuda(), M, N, K, mx.QuantType(qt), mx._capi.lib.mlxr_default_group_size(qt), bt[0].contiguous().cuda())
    y = mx.q_gemm_dequant(*args)
    assert torch.equal(y, mx.q_gemm_dequant(*args))
    assert _status() == 0
    bound = {"bf16": 2.0 ** -9, "f16": 2.0 ** -11}[dt] * (1 if M <= 8 or qt == 33 else 2)
    assert oracle.rel_l2(y.float().cpu().numpy(), want) <= bound


@pytest.mark.parametrize("qt", [2, 16])
@pytest.mark.parametrize("M,H,I", [(5, 256, 768), (33, 768, 1280)])
def test_gate_up_other_formats(oracle, qt, M, H, I):
    """The SiLU(gate) * up form of Q8_0 and NF4, with odd numbers of super-blocks, inside the block."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    g, u, d = (quantize(make_weights(n, k, s), qt) for n, k, s in ((I, H, 1), (I, H, 2), (H, I, 3)))
    xt, xf = make_acts(M, H, 4, torch.bfloat16)
    nt, nf = make_acts(1, H, 5, torch.bfloat16)
    y = mx.mlp_block(xt.cuda(), nt[0].contiguous().cuda(), *(torch.from_numpy(w).cuda() for w in (g, u, d)), I, mx.QuantType(qt), 1e-5)
    assert _status() == 0
    assert oracle.rel_l2(y.float().cpu().numpy(), oracle.mlp_block(xf, nf[0], g, u, d, I, qt, 1e-5, oracle.BF16)) <= TIGHT["bf16"]


@pytest.mark.parametrize("qt", [0, 2, 3, 16])
@pytest.mark.parametrize("M,H,QH,KH,D", [(3, 768, 5, 1, 64), (20, 512, 4, 2, 128), (64, 1280, 3, 3, 32)])
def test_stacked_projections_with_rope(oracle, qt, M, H, QH, KH, D):
    """q, k and v as one launch (row counts that do not fill their last tile, odd numbers of super-blocks), then
    q and k rotated in one: against this package's own linear (bit-equal is not required: the tiles are
    shared by other CTAs, which adds the float32 sums in another order) and rope_apply on its result."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    ws = [torch.from_numpy(quantize(make_weights(n * D, H, 9 + i), qt)).cuda() for i, n in enumerate((QH, KH, KH))]
    x = make_acts(M, H, 4, torch.float16)[0].cuda()
    nw = make_acts(1, H, 5, torch.float16)[0][0].contiguous().cuda()
    cos, sin = mx.compute_rope_tables(512, D, 10000.0, device=torch.device("cuda"))
    pos = torch.from_numpy(np.random.Generator(np.random.PCG64(1)).integers(0, 512, M).astype(np.int32)).cuda()
    out = mx.qkv_rope(x, nw, *ws, cos, sin, pos, QH, KH, D, mx.QuantType(qt), 1e-5)
    assert _status() == 0
    n = mx.rmsnorm_fused(x, nw, 1e-5)
    gs = mx._capi.lib.mlxr_default_group_size(qt)
    for i, (got, heads) in enumerate(zip(out, (QH, KH, KH))):
        y = mx.q_gemm_dequant(n, ws[i], M, heads * D, H, mx.QuantType(qt), gs).reshape(M, heads, D)
        want = mx.rope_apply(y, cos, sin, pos) if i < 2 else y
        # one ulp of the linear's result at most, 2^-10, where the two sums round to different sides
        assert float((got.double() - want.double()).norm() / want.double().norm()) <= 2.0 ** -11


@pytest.mark.parametrize("N", [4095, 4096, 4097])
def test_two_tokens_nf4_at_the_border(oracle, N):
    """Two tokens change kernels at 2^24 weights; bias, and a last tile of one row above it.  Bound as for
    three tokens in test_other_formats: 2^-9 of the bf16 result."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    K, M = 4096, 2
    packed = quantize(make_weights(N, K, 5), 16)
    xt, xf = make_acts(M, K, 6, torch.bfloat16)
    bt, bf = make_acts(1, N, 7, torch.bfloat16)
    want = xf.astype(np.float64) @ oracle.dequantize(packed, N, K, 16)[0].astype(np.float64).reshape(N, K).T + bf[0]
    y = mx.q_gemm_dequant(xt.cuda(), torch.from_numpy(packed).cuda(), M, N, K, mx.QuantType(16), 64, bt[0].contiguous().cuda())
    assert _status() == 0
    assert oracle.rel_l2(y.float().cpu().numpy(), want) <= 2.0 ** -9


@pytest.mark.parametrize("qt", [0, 3])
@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("M,H,QH,KH,D", [(3, 768, 5, 1, 64), (8, 1280, 3, 3, 32), (8, 4096, 32, 8, 128)])
def test_few_tokens_of_stacked_4_bit_weights_are_not_rounded(oracle, qt, dt, M, H, QH, KH, D):
    """v of q / k / v up to 8 tokens: products with the float32 weights, as for the formats above, so 2^-9 (bf16) and 2^-11
    (fp16) for the result's rounding.  Q4_K's reference is the shader's half arithmetic, two roundings of at most 2^-11
    per weight that the kernel does not make.  Weights with scale and min rounded to bf16 come out at 3.4e-3."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    packed = [quantize(make_weights(n * D, H, 9 + i), qt) for i, n in enumerate((QH, KH, KH))]
    x = make_acts(M, H, 4, DT[dt])[0].cuda()
    cos, sin = mx.compute_rope_tables(16, D, 10000.0, device=torch.device("cuda"))
    pos = torch.arange(M, dtype=torch.int32, device="cuda")
    v = mx.qkv_rope(x, None, *(torch.from_numpy(w).cuda() for w in packed), cos, sin, pos, QH, KH, D, mx.QuantType(qt), 1e-5)[2]
    assert _status() == 0
    f, h = oracle.dequantize(packed[2], KH * D, H, qt)
    w = torch.from_numpy((h.view(np.float16) if qt == 3 else f).astype(np.float64).reshape(KH * D, H)).cuda()
    want = (x.double() @ w.T).reshape(M, KH, D)
    assert float((v.double() - want).norm() / want.norm()) <= {"bf16": 2.0 ** -9, "f16": 2.0 ** -11}[dt] + (2.0 ** -11 if qt == 3 else 0)


def _with_large_blocks(packed, rows, block, d):
    """Every third row's first block gets the scale d."""
    p = packed.reshape(rows, -1).copy()
    p[::3, 0:2] = np.frombuffer(np.float16(d).tobytes(), np.uint8)
    return p.reshape(-1)


@pytest.mark.parametrize("qt,M", [(2, 3), (2, 8), (33, 5), (33, 40)])
@pytest.mark.parametrize("N,K", [(200, 768), (385, 4096)])
def test_weights_beyond_the_range_of_fp16(oracle, qt, M, N, K):
    """fp16 activations and weights up to 2.5e5: the float32 products are finite and so is the result.  Bound as in
    test_other_formats (22 significant bits of the weights): the result's rounding, 2^-11."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    if qt == 33:
        import gguf
        import gguf.quants as gq
        rng = np.random.Generator(np.random.PCG64(1))
        raw = rng.integers(0, 256, size=(N * (K // 256), 144), dtype=np.uint8)
        raw[:, 0:4] = (rng.random((raw.shape[0], 2)) * 0.002 + 0.0005).astype(np.float16).view(np.uint8)
        packed = _with_large_blocks(raw.reshape(-1), N, 256, 200.0)
        w = gq.dequantize(packed.reshape(N, -1), gguf.GGMLQuantizationType.Q4_K).astype(np.float64)
    else:
        packed = _with_large_blocks(quantize(make_weights(N, K, 3), qt), N, 32, 2000.0)
        w = oracle.dequantize(packed, N, K, qt)[0].astype(np.float64).reshape(N, K)
    assert np.abs(w).max() > 65504
    x = (make_acts(M, K, 4, torch.float32)[0] * 1e-3).half()
    want = x.double().numpy() @ w.T
    y = mx.q_gemm_dequant(x.cuda(), torch.from_numpy(packed).cuda(), M, N, K, mx.QuantType(qt), mx._capi.lib.mlxr_default_group_size(qt))
    assert _status() == 0
    assert oracle.rel_l2(y.float().cpu().numpy(), want) <= 2.0 ** -11


def test_weights_beyond_the_range_of_fp16_in_the_other_forms(oracle):
    """The same in the gate / up form (Q8_0) and in the stacked one (Q4_0).  Block: g, u, h and y are rounded to fp16 on both
    sides, 2e-3 as everywhere for fp16."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    M, H, I = 5, 512, 768
    g, u, d = (quantize(make_weights(n, k, s), 2) for n, k, s in ((I, H, 1), (I, H, 2), (H, I, 3)))
    g, u = _with_large_blocks(g, I, 32, 2000.0), _with_large_blocks(u, I, 32, 1500.0)
    xt = (make_acts(M, H, 4, torch.float32)[0] * 1e-4).half()
    deq = lambda w, n, k: torch.from_numpy(oracle.dequantize(w, n, k, 2)[0].astype(np.float64).reshape(n, k))
    half = lambda t: t.half().double()
    h = half(torch.nn.functional.silu(half(xt.double() @ deq(g, I, H).T)) * half(xt.double() @ deq(u, I, H).T))
    y = mx.mlp_block(xt.cuda(), None, *(torch.from_numpy(w).cuda() for w in (g, u, d)), I, mx.QuantType.Q8_0)
    assert oracle.rel_l2(y.float().cpu().numpy(), (h @ deq(d, H, I).T).numpy()) <= 2e-3
    QH, KH, D = 3, 1, 64
    packed = [_with_large_blocks(quantize(make_weights(n * D, H, 9 + i), 0), n * D, 32, 20000.0) for i, n in enumerate((QH, KH, KH))]
    cos, sin = mx.compute_rope_tables(16, D, 10000.0, device=torch.device("cuda"))
    v = mx.qkv_rope(xt.cuda(), None, *(torch.from_numpy(w).cuda() for w in packed), cos, sin, torch.arange(M, dtype=torch.int32, device="cuda"), QH, KH, D, mx.QuantType.Q4_0)[2]
    want = xt.double() @ torch.from_numpy(oracle.dequantize(packed[2], KH * D, H, 0)[0].astype(np.float64).reshape(KH * D, H)).T
    assert oracle.rel_l2(v.float().cpu().numpy().reshape(M, -1), want.numpy()) <= 2.0 ** -11
    assert _status() == 0


@pytest.mark.parametrize("qt", [2, 16])
@pytest.mark.parametrize("dt", ["bf16", "f16"])
def test_infinite_activation_in_two_parts(qt, dt):
    """One infinity in a token: infinities with the sign of its weights, as float32 products give them, in that token only."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    N, K, M = 300, 512, 4
    wf = make_weights(N, K, 3)
    wf[:, 40] = np.where(np.arange(N) % 2 == 0, 0.047, -0.047)
    x = make_acts(M, K, 4, DT[dt])[0].cuda()
    x[2, 40] = float("inf")
    y = mx.q_gemm_dequant(x, torch.from_numpy(quantize(wf, qt)).cuda(), M, N, K, mx.QuantType(qt), mx._capi.lib.mlxr_default_group_size(qt)).float().cpu()
    assert np.array_equal(y[2].numpy(), np.where(np.arange(N) % 2 == 0, np.inf, -np.inf).astype(np.float32))
    assert torch.isfinite(y[[0, 1, 3]]).all()


# The two-part weights of this kernel at few tokens: more activations than the kernel of whole rows takes, or more tokens
@pytest.mark.parametrize("qt,M,N,K", [(2, 8, 200, 8192), (2, 3, 385, 16640), (33, 9, 200, 768), (33, 12, 385, 4096)])
def test_weights_beyond_the_range_of_fp16_here(oracle, qt, M, N, K):
    import mlxr_b200 as mx
    assert M > 8 or M * K > 49152
    test_weights_beyond_the_range_of_fp16(oracle, qt, M, N, K)


def test_weights_beyond_the_range_of_fp16_in_the_other_forms_here(oracle):
    """As in ..._in_the_other_forms: gate / up of Q8_0 and v of stacked Q4_0, 8 tokens of hidden size 8192."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    M, H, I = 8, 8192, 512
    g, u, d = (quantize(make_weights(n, k, s), 2) for n, k, s in ((I, H, 1), (I, H, 2), (H, I, 3)))
    g, u = _with_large_blocks(g, I, 32, 2000.0), _with_large_blocks(u, I, 32, 1500.0)
    xt = (make_acts(M, H, 4, torch.float32)[0] * 1e-4).half()
    deq = lambda w, n, k, qt: torch.from_numpy(oracle.dequantize(w, n, k, qt)[0].astype(np.float64).reshape(n, k))
    half = lambda t: t.half().double()
    h = half(torch.nn.functional.silu(half(xt.double() @ deq(g, I, H, 2).T)) * half(xt.double() @ deq(u, I, H, 2).T))
    y = mx.mlp_block(xt.cuda(), None, *(torch.from_numpy(w).cuda() for w in (g, u, d)), I, mx.QuantType.Q8_0)
    assert oracle.rel_l2(y.float().cpu().numpy(), (h @ deq(d, H, I, 2).T).numpy()) <= 2e-3
    QH, KH, D = 3, 1, 64
    packed = [_with_large_blocks(quantize(make_weights(n * D, H, 9 + i), 0), n * D, 32, 20000.0) for i, n in enumerate((QH, KH, KH))]
    cos, sin = mx.compute_rope_tables(16, D, 10000.0, device=torch.device("cuda"))
    v = mx.qkv_rope(xt.cuda(), None, *(torch.from_numpy(w).cuda() for w in packed), cos, sin, torch.arange(M, dtype=torch.int32, device="cuda"), QH, KH, D, mx.QuantType.Q4_0)[2]
    assert oracle.rel_l2(v.float().cpu().numpy().reshape(M, -1), (xt.double() @ deq(packed[2], KH * D, H, 0).T).numpy()) <= 2.0 ** -11
    assert _status() == 0


@pytest.mark.parametrize("qt,dt,M,K", [(2, "bf16", 8, 8192), (2, "f16", 4, 12544), (16, "bf16", 12, 512), (2, "f16", 40, 512)])
def test_infinite_activation_here(qt, dt, M, K):
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    N = 300
    wf = make_weights(N, K, 3)
    wf[:, 40] = np.where(np.arange(N) % 2 == 0, 0.047, -0.047)
    x = make_acts(M, K, 4, DT[dt])[0].cuda()
    x[2, 40] = float("inf")
    y = mx.q_gemm_dequant(x, torch.from_numpy(quantize(wf, qt)).cuda(), M, N, K, mx.QuantType(qt), mx._capi.lib.mlxr_default_group_size(qt)).float().cpu()
    assert np.array_equal(y[2].numpy(), np.where(np.arange(N) % 2 == 0, np.inf, -np.inf).astype(np.float32))
    assert torch.isfinite(y[[m for m in range(M) if m != 2]]).all()


@pytest.mark.parametrize("dt,M", [("bf16", 12), ("f16", 40)])
def test_infinite_activation_canonical(dt, M):
    """Canonical Q4_K weights of code 0 are their offset, of either sign or zero: what float32 products give."""
    import mlxr_b200 as mx
    N, K = 300, 512
    rng = np.random.Generator(np.random.PCG64(1))
    b = rng.integers(0, 256, (N * K // 256, 144), dtype=np.uint8)
    b[:, :4] = rng.uniform(1e-4, 3e-4, (N * K // 256, 2)).astype(np.float16).view(np.uint8)
    w = torch.from_numpy(b.reshape(-1)).cuda()
    x = make_acts(M, K, 4, DT[dt])[0].cuda()
    x[2, 77] = float("inf")
    y = mx.q_gemm_dequant(x, w, M, N, K, mx.QuantType(33), 256).float()
    want = x.float()[2, 77] * mx.dequantize(w, N, K, mx.QuantType(33), torch.float32)[:, 77]
    nan = torch.isnan(want)
    assert torch.equal(torch.isnan(y[2]), nan) and torch.equal(y[2][~nan], want[~nan])
    assert torch.isfinite(y[[m for m in range(M) if m != 2]]).all()
