"""Linears of up to eight tokens (csrc/gemv_tokens.cu) through the C ABI, against float64 products of the dequantized weights.

Sizes: fewer rows than SMs, row counts that are no multiple of the granule of four, more warps than work units, an odd number
of 256-weight segments, every token count, rows that make the warps meet more than once, one ring stage.

Bounds (2-norm, relative).  Result: rounded once to p significant bits, at most 2^-8 (bf16) and 2^-11 (fp16).  Products and sums
are float32: 1e-6.  Q4_K's reference is the shader's half arithmetic, two roundings of at most 2^-11 per weight that the kernel does
not make: 2^-10."""
import numpy as np
import pytest
import torch

from conftest import make_acts, make_weights

pytestmark = pytest.mark.gpu
DT = {"f16": torch.float16, "bf16": torch.bfloat16}
RESULT = {"f16": 2.0 ** -11, "bf16": 2.0 ** -8}
WEIGHT = {0: 1e-6, 2: 1e-6, 3: 2.0 ** -10, 33: 1e-6}


def _status():
    import mlxr_b200 as mx
    st = torch.zeros(1, dtype=torch.int32)
    mx._capi.check(mx._capi.lib.mlxr_stream_status(torch.cuda.current_stream().cuda_stream, st.data_ptr()))
    return int(st[0])


def _weights(N, K, qt, seed):
    """Packed weights on the device: quantized, or for canonical Q4_K random blocks with scales of ordinary size."""
    from mlxr_b200.quantize import quantize
    if qt != 33:
        return torch.from_numpy(quantize(make_weights(N, K, seed), qt)).cuda()
    rng = np.random.Generator(np.random.PCG64(seed))
    b = rng.integers(0, 256, (N * K // 256, 144), dtype=np.uint8)
    b[:, :4] = rng.uniform(1e-4, 3e-4, (N * K // 256, 2)).astype(np.float16).view(np.uint8)
    return torch.from_numpy(b.reshape(-1)).cuda()


def _dense(w, N, K, qt):
    import mlxr_b200 as mx
    return mx.dequantize(w, N, K, mx.QuantType(qt), torch.float32).double()


def _linear(x, w, N, K, qt, b=None):
    import mlxr_b200 as mx
    return mx.q_gemm_dequant(x, w, x.shape[0], N, K, mx.QuantType(qt), mx._capi.lib.mlxr_default_group_size(qt), b)


def _check(y, want, dt, qt):
    assert float((y.double() - want).norm() / want.norm()) <= RESULT[dt] + WEIGHT[qt]
    # no result may be wrong by itself: the largest are below 6 rms
    assert float((y.double() - want).abs().max() / want.square().mean().sqrt()) <= 6 * (RESULT[dt] + WEIGHT[qt]) + 1e-3


@pytest.mark.parametrize("qt,dt", [(33, "f16"), (33, "bf16"), (2, "f16"), (2, "bf16"), (0, "bf16"), (3, "bf16")])
@pytest.mark.parametrize("M,N,K", [(3, 4, 256), (4, 67, 768), (5, 593, 512), (6, 1000, 1280), (7, 2369, 256), (8, 130, 2048), (3, 40, 16384)])
def test_linear(qt, dt, M, N, K):
    w = _weights(N, K, qt, 7 + N)
    x = make_acts(M, K, 8 + N, DT[dt])[0].cuda()
    b = make_acts(1, N, 9, DT[dt])[0][0].contiguous().cuda() if N % 2 else None
    y = _linear(x, w, N, K, qt, b)
    assert torch.equal(y, _linear(x, w, N, K, qt, b)) and _status() == 0
    _check(y, x.double() @ _dense(w, N, K, qt).T + (b.double() if b is not None else 0), dt, qt)


@pytest.mark.parametrize("qt,M,N,K", [(33, 1, 5, 256), (33, 2, 4097, 1792), (33, 1, 300, 32768), (33, 8, 41001, 256), (2, 3, 45003, 256), (0, 3, 33001, 256), (33, 8, 700, 6144)])
def test_few_and_many_rows(qt, M, N, K):
    w = _weights(N, K, qt, 3)
    x = make_acts(M, K, 4, torch.bfloat16)[0].cuda()
    y = _linear(x, w, N, K, qt)
    assert _status() == 0
    _check(y, x.double() @ _dense(w, N, K, qt).T, "bf16", qt)


@pytest.mark.parametrize("qt,dt", [(0, "f16"), (0, "bf16"), (2, "f16"), (2, "bf16"), (3, "f16"), (3, "bf16")])
@pytest.mark.parametrize("M,H,QH,KH,D", [(3, 512, 3, 1, 64), (8, 1280, 10, 2, 128)])
def test_stacked_is_the_three_linears(qt, dt, M, H, QH, KH, D):
    """q, k and v of one launch, without RMSNorm and with positions at zero (a rotation by nothing)."""
    import mlxr_b200 as mx
    w = [_weights(n * D, H, qt, i) for i, n in enumerate((QH, KH, KH))]
    x = make_acts(M, H, 5, DT[dt])[0].cuda()
    cos, sin = mx.compute_rope_tables(4, D, 10000.0, device=torch.device("cuda"))
    out = mx.qkv_rope(x, None, *w, cos, sin, torch.zeros(M, dtype=torch.int32, device="cuda"), QH, KH, D, mx.QuantType(qt), 1e-5)
    assert _status() == 0
    for y, p, n in zip(out, w, (QH, KH, KH)):
        _check(y.reshape(M, -1), x.double() @ _dense(p, n * D, H, qt).T, dt, qt)


@pytest.mark.parametrize("qt", [0, 2, 3])
@pytest.mark.parametrize("M,H,I", [(3, 256, 1280), (8, 512, 1024), (5, 768, 2304)])
def test_gate_up(qt, M, H, I):
    """The block without a norm weight: h and y are rounded to bf16, h from rounded gate and up."""
    import mlxr_b200 as mx
    wg, wu, wd = _weights(I, H, qt, 1), _weights(I, H, qt, 2), _weights(H, I, qt, 3)
    x = make_acts(M, H, 4, torch.bfloat16)[0].cuda()
    y = mx.mlp_block(x, None, wg, wu, wd, I, mx.QuantType(qt), 1e-5)
    assert _status() == 0
    g, u = (x.double() @ _dense(w, I, H, qt).T for w in (wg, wu))
    h = torch.nn.functional.silu(g.bfloat16().double()) * u.bfloat16().double()
    want = h.bfloat16().double() @ _dense(wd, H, I, qt).T
    # rounding of g, u, h and y: each at most 2^-8, independent
    assert float((y.double() - want).norm() / want.norm()) <= 2 * RESULT["bf16"] + WEIGHT[qt]


@pytest.mark.parametrize("qt", [2, 33])
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_values_that_are_not_finite(qt, dt):
    """An infinite activation: every result of its token is what the float32 weights give (a canonical weight of code 0 is its
    offset), the other tokens' are what they are without it.  A NaN reaches its token only."""
    M, N, K = 4, 300, 512
    w = _weights(N, K, qt, 1)
    x = make_acts(M, K, 2, DT[dt])[0].cuda()
    clean = _linear(x, w, N, K, qt)
    x[1, 77], x[2, 300] = float("inf"), float("nan")
    y = _linear(x, w, N, K, qt)
    d = _dense(w, N, K, qt).float()
    want = x.float()[1, 77] * d[:, 77]
    assert torch.equal(torch.isnan(y[1]), torch.isnan(want))
    assert torch.equal(y[1].float()[~torch.isnan(want)], want[~torch.isnan(want)])
    assert torch.isnan(y[2]).all() and torch.equal(y[0], clean[0]) and torch.equal(y[3], clean[3])


@pytest.mark.parametrize("scale", [2.0 ** -100, 2.0 ** 100])
def test_range_of_bf16(scale):
    """Activations of any magnitude, segments of one row apart by 2^12."""
    N, K = 200, 1024
    w = _weights(N, K, 33, 1)
    x = (make_acts(3, K, 2, torch.float32)[0] * scale).to(torch.bfloat16).cuda()
    x[:, 512:] *= 2.0 ** -12
    _check(_linear(x, w, N, K, 33), x.double() @ _dense(w, N, K, 33).T, "bf16", 33)


@pytest.mark.parametrize("qt,dt,M", [(33, "f16", 1), (33, "bf16", 3), (33, "f16", 8), (2, "f16", 3), (2, "bf16", 8), (0, "bf16", 3), (3, "bf16", 5)])
def test_large_activations_that_cancel(qt, dt, M):
    """Every block of 32 has activations 256 and -256 on equal weights; the others are at most 2^-5, in steps of 2^-9.  A block's sums of
    code * x stay below 2^13, so float32 holds them exactly in any order and the large ones leave nothing behind: the
    bounds are those of the small ones alone.  (Sums of 17 bits leave 1 to 3 % of the results.)"""
    N, K = 130, 512 if qt in (2, 33) else 1536
    p = _weights(N, K, qt, 3).cpu().numpy().reshape(-1, {0: 18, 2: 34, 3: 144, 33: 144}[qt])
    if qt == 33:
        p[:, 16:].reshape(-1, 4, 32)[..., 20] = p[:, 16:].reshape(-1, 4, 32)[..., 2]      # byte i: element i of two blocks
    elif qt == 3:
        p[:, 16:].reshape(-1, 8, 16)[..., 10] = p[:, 16:].reshape(-1, 8, 16)[..., 1]      # byte i: elements 2 i and 2 i + 1
    else:
        p[:, 2 + (20 if qt == 2 else 10)] = p[:, 2 + (2 if qt == 2 else 1)]
    w = torch.from_numpy(p.reshape(-1)).cuda()
    d = _dense(w, N, K, qt)
    assert torch.equal(d[:, 2::32], d[:, 20::32])
    x = torch.randint(-16, 17, (M, K), generator=torch.Generator().manual_seed(5)).double() / 512
    x[:, 2::32], x[:, 20::32] = 256.0, -256.0
    x = x.to(DT[dt]).cuda()
    _check(_linear(x, w, N, K, qt), x.double() @ d.T, dt, qt)


# The rule of sizes sends these here: remainders of rows, warps without work, an odd number of segments, one ring stage, meetings
# of the warps in the middle of a CTA's tiles
HERE = [(0, "bf16", 3, 1000, 1280), (3, "bf16", 4, 67, 1536), (0, "bf16", 5, 593, 1792), (3, "bf16", 6, 2369, 1536), (0, "bf16", 8, 130, 2048), (3, "bf16", 8, 2, 2048), (0, "bf16", 3, 41, 4352),
        (3, "bf16", 3, 3001, 3328), (33, "bf16", 8, 4102, 6144), (33, "f16", 1, 4097, 32768), (33, "bf16", 1, 3501, 24576), (2, "bf16", 3, 4099, 16384), (2, "f16", 8, 4097, 5632),
        (33, "bf16", 1, 1025, 512), (33, "f16", 2, 5, 768)]


@pytest.mark.parametrize("qt,dt,M,N,K", HERE)
def test_sizes_that_the_rule_sends_here(qt, dt, M, N, K):
    import mlxr_b200 as mx
    assert mx._capi.lib.mlxr_debug_few_tokens_rule(qt, M, K, N, 0, {"f16": 0, "bf16": 1}[dt]) == 1
    w = _weights(N, K, qt, 7 + N)
    x = make_acts(M, K, 8 + N, DT[dt])[0].cuda()
    b = make_acts(1, N, 9, DT[dt])[0][0].contiguous().cuda() if N % 2 else None
    y = _linear(x, w, N, K, qt, b)
    assert torch.equal(y, _linear(x, w, N, K, qt, b)) and _status() == 0
    _check(y, x.double() @ _dense(w, N, K, qt).T + (b.double() if b is not None else 0), dt, qt)


@pytest.mark.parametrize("qt,M,N,K", [(33, 1, 1024, 512), (33, 3, 700, 14336), (2, 8, 1000, 5632), (3, 3, 6145, 1792), (3, 8, 1000, 4096), (0, 4, 4097, 1280)])
def test_sizes_beyond_the_rule(qt, M, N, K):
    """The other kernels' sizes next to these.  Q4_K and Q4_0: weights rounded to bf16, 2^-9 each, and the result."""
    import mlxr_b200 as mx
    assert mx._capi.lib.mlxr_debug_few_tokens_rule(qt, M, K, N, 0, 1) == 0
    w = _weights(N, K, qt, 7)
    x = make_acts(M, K, 8, torch.bfloat16)[0].cuda()
    y = _linear(x, w, N, K, qt)
    want = x.double() @ _dense(w, N, K, qt).T
    assert _status() == 0 and float((y.double() - want).norm() / want.norm()) <= RESULT["bf16"] + (2.0 ** -9 if qt in (0, 3) else 2.0 ** -15)


@pytest.mark.parametrize("qt", [0, 3])
@pytest.mark.parametrize("M,H,I", [(3, 1536, 1280), (8, 2048, 1536)])
def test_gate_up_of_the_rule(qt, M, H, I):
    import mlxr_b200 as mx
    assert mx._capi.lib.mlxr_debug_few_tokens_rule(qt, M, H, 2 * I, 1, 1) == 1
    test_gate_up(qt, M, H, I)


def _canonical(codes, d, dmin, sc=1, mn=8):
    """Canonical Q4_K blocks of codes [rows, K] with one scale and minimum: w = d sc code - dmin mn."""
    c = codes.astype(np.uint8).reshape(-1, 4, 2, 32)
    head = np.concatenate([np.array([d, dmin], np.float16).view(np.uint8), np.array([sc] * 4 + [mn] * 4 + [sc | (mn << 4)] * 4, np.uint8)])
    return np.concatenate([np.broadcast_to(head, (c.shape[0], 16)), (c[:, :, 0] | (c[:, :, 1] << 4)).reshape(-1, 128)], 1).reshape(-1)


@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_infinite_activation_in_gate_up(dt):
    """Gate weights that are small multiples of a positive scale, without a minimum: their codes below 8 make infinity minus infinity of an
    infinite activation in the kernel's arithmetic, infinity in float32.  Up weights of either sign, down weights of up's sign times the
    output row's: every output is an infinity with the sign of its row."""
    import mlxr_b200 as mx
    M, H, I = 4, 512, 1024
    rng = np.random.Generator(np.random.PCG64(7))
    gate = rng.integers(1, 16, (I, H))
    up = rng.choice([3, 5, 11, 14], (I, H))
    s, t = np.where(up[:, 77] > 8, 1, -1), rng.choice([-1, 1], H)
    down = np.where(t[:, None] * s[None, :] > 0, 13, 2)
    wg, wu, wd = (torch.from_numpy(p).cuda() for p in (_canonical(gate, 1e-3, 0.0), _canonical(up, 1e-3, 1e-3), _canonical(down, 1e-3, 1e-3)))
    assert torch.equal(torch.sign(_dense(wu, I, H, 33)[:, 77]).cpu(), torch.from_numpy(s).double()) and bool((_dense(wg, I, H, 33)[:, 77] > 0).all())
    x = make_acts(M, H, 2, DT[dt])[0].cuda()
    run = lambda: mx.mlp_block(x, None, wg, wu, wd, I, mx.QuantType(33), 1e-5)
    clean = run()
    x[1, 77] = float("inf")
    y = run()
    assert _status() == 0
    assert np.array_equal(y[1].float().cpu().numpy(), t * np.float32(np.inf))
    assert torch.equal(y[[0, 2, 3]], clean[[0, 2, 3]])


@pytest.mark.parametrize("qt,dt", [(33, "f16"), (33, "bf16"), (0, "f16"), (3, "bf16"), (2, "bf16")])
def test_infinite_activation_in_stacked_matrices(qt, dt):
    """v of q / k / v (q and k are rotated: infinity times a sine of zero): the third matrix, whose rows begin inside a CTA's."""
    import mlxr_b200 as mx
    M, H, QH, KH, D = 5, 512, 3, 1, 44
    w = [_weights(n * D, H, qt, i) for i, n in enumerate((QH, KH, KH))]
    x = make_acts(M, H, 5, DT[dt])[0].cuda()
    cos, sin = mx.compute_rope_tables(4, D, 10000.0, device=torch.device("cuda"))
    run = lambda: mx.qkv_rope(x, None, *w, cos, sin, torch.zeros(M, dtype=torch.int32, device="cuda"), QH, KH, D, mx.QuantType(qt), 1e-5)
    clean = run()
    x[1, 77] = float("inf")
    out = run()
    assert _status() == 0
    want = float("inf") * _dense(w[2], KH * D, H, qt)[:, 77].float()
    nan = torch.isnan(want)
    v = out[2].reshape(M, -1).float()
    assert torch.equal(torch.isnan(v[1]), nan) and torch.equal(v[1][~nan], want[~nan])
    for a, b in zip(out, clean):
        assert torch.equal(a[[0, 2, 3, 4]], b[[0, 2, 3, 4]])
    assert not torch.isfinite(out[1][1]).any()


@pytest.mark.parametrize("qt", [2, 33])
@pytest.mark.parametrize("scale", [2.0 ** -100, 1.0, 2.0 ** 100])
def test_small_segments_decide(qt, scale):
    """Segments of one row 2^12 apart where the large ones are not there (one token has zeros in them) or meet weights of zero (some
    rows): norms per token and, for those rows, by themselves."""
    N, K = 200, 1024
    w = _weights(N, K, qt, 1)
    if qt == 2:
        w.view(N, K // 32, 34)[::3, :16, 2:] = 0
    x = (make_acts(3, K, 2, torch.float32)[0] * scale).to(torch.bfloat16).cuda()
    x[:, 512:] *= 2.0 ** -12
    x[1, :512] = 0.0
    y, want = _linear(x, w, N, K, qt), x.double() @ _dense(w, N, K, qt).T
    for m in range(3):
        _check(y[m:m + 1], want[m:m + 1], "bf16", qt)
    if qt == 2:
        _check(y[:, ::3].contiguous(), want[:, ::3], "bf16", qt)


@pytest.mark.parametrize("M", [1, 2, 3, 8])
def test_neighbours_of_a_large_activation(M):
    """bf16 activations are fp16 numbers times a power of two per 256 from the large Q8_0 matrices of one token on: exact down to 2^-31 of the segment's
    largest.  A large one on weights of zero, the others 2^-30 to 2^-29 of it."""
    from mlxr_b200.quantize import quantize
    N, K = 600, 2304
    wf = make_weights(N, K, 3)
    wf[:, 9::256] = 0.0
    w = torch.from_numpy(quantize(wf, 2)).cuda()
    x = make_acts(M, K, 4, torch.float32)[0]
    x = torch.sign(x) * (1.0 + x.abs().clamp(max=0.99)) * 2.0 ** -20
    x[:, 9::256] = 2.0 ** 10
    x = x.to(torch.bfloat16).cuda()
    _check(_linear(x, w, N, K, 2), x.double() @ _dense(w, N, K, 2).T, "bf16", 2)
