"""RMSNorm, SwiGLU and RoPE through the C ABI vs the oracle.  RMSNorm uses the reference
test's own closeness rule |a-b| <= atol + rtol*|b| with its tolerances
(tests/unit/rmsnorm_primitive_test.cpp:36-52, :76, :141, :198)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def arrays_close(a, b, rtol, atol):
    a = np.asarray(a, dtype=np.float64)
    b = np.asarray(b, dtype=np.float64)
    return bool(np.all(np.abs(a - b) <= atol + rtol * np.abs(b)))


def _rms(oracle, shape, dtype, eps, seed, scale=1.0, residual=False):
    import mlxr_b200 as mx
    g = torch.Generator().manual_seed(seed)
    x = (torch.randn(shape, generator=g) * scale).to(dtype)
    w = (1 + 0.1 * torch.randn(shape[-1], generator=g)).to(dtype)
    r = torch.randn(shape, generator=g).to(dtype) if residual else None
    y = mx.rmsnorm_fused(x.cuda(), w.cuda(), eps, r.cuda() if residual else None).float().cpu().numpy()
    ref = oracle.rmsnorm(x.float().numpy(), w.float().numpy(), eps)
    if residual:
        ref = ref + r.float().numpy()
    return y, ref


@pytest.mark.parametrize("hidden", [32, 64, 128, 256, 512, 1024, 2048, 4096, 8192, 100, 5000, 12288])
def test_rmsnorm_fp32_hidden_sizes(oracle, hidden):
    y, ref = _rms(oracle, (4, hidden), torch.float32, 1e-6, hidden)
    assert arrays_close(y, ref, 1e-4, 1e-5)


@pytest.mark.parametrize("batch", [1, 2, 4, 8, 16, 32])
def test_rmsnorm_batch_sizes(oracle, batch):
    y, ref = _rms(oracle, (batch, 16, 128), torch.float32, 1e-6, batch)
    assert arrays_close(y, ref, 1e-4, 1e-5)


@pytest.mark.parametrize("eps", [1e-8, 1e-6, 1e-5, 1e-4, 1e-2])
def test_rmsnorm_eps(oracle, eps):
    y, ref = _rms(oracle, (2, 8, 128), torch.float32, eps, 3)
    assert arrays_close(y, ref, 1e-4, 1e-5)


def test_rmsnorm_fp16_bf16(oracle):
    y, ref = _rms(oracle, (2, 8, 4096), torch.float16, 1e-5, 4)
    assert arrays_close(y, ref, 1e-2, 1e-3)
    y, ref = _rms(oracle, (2, 8, 4096), torch.bfloat16, 1e-5, 4)
    assert arrays_close(y, ref, 2e-2, 1e-2)


def test_rmsnorm_large_values_and_residual(oracle):
    y, ref = _rms(oracle, (2, 8, 128), torch.float32, 1e-6, 5, scale=100.0)
    assert arrays_close(y, ref, 1e-3, 1e-4)
    y, ref = _rms(oracle, (3, 2048), torch.float32, 1e-6, 6, residual=True)
    assert arrays_close(y, ref, 1e-4, 1e-5)


def test_rmsnorm_non_contiguous_and_errors(oracle):
    import mlxr_b200 as mx
    x = torch.randn(8, 4, 128, device="cuda").transpose(0, 1)  # non-contiguous
    w = torch.ones(128, device="cuda")
    y = mx.rmsnorm_fused(x, w, 1e-6)
    ref = oracle.rmsnorm(x.contiguous().cpu().numpy(), w.cpu().numpy(), 1e-6)
    assert arrays_close(y.cpu().numpy(), ref, 1e-4, 1e-5)
    with pytest.raises(ValueError):
        mx.rmsnorm_fused(x, torch.ones(64, device="cuda"))
    with pytest.raises(ValueError):
        mx.rmsnorm_fused(x, torch.ones(2, 64, device="cuda"))
    # [16, 512, 4096] sanity: finite, unit RMS before the weight
    big = torch.randn(16, 512, 4096, device="cuda", dtype=torch.float16)
    out = mx.rmsnorm_fused(big, torch.ones(4096, device="cuda", dtype=torch.float16), 1e-5)
    assert torch.isfinite(out).all()
    assert abs(out.float().pow(2).mean().sqrt().item() - 1.0) < 1e-2


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
def test_swiglu(oracle, dtype):
    import mlxr_b200 as mx
    g = (torch.randn(3, 5632) * 3).to(dtype)
    u = torch.randn(3, 5632).to(dtype)
    g[0, :4] = torch.tensor([-100.0, 100.0, 0.0, -20.0]).to(dtype)  # saturating sigmoid
    h = mx.swiglu(g.cuda(), u.cuda()).float().cpu().numpy()
    ref = oracle.swiglu(g.float().numpy(), u.float().numpy())
    ref = oracle.round_to(ref, {torch.float16: 0, torch.bfloat16: 1, torch.float32: 2}[dtype])
    assert arrays_close(h, ref, 1e-2 if dtype != torch.float32 else 1e-5, 1e-6)
    s = mx.swish(g.cuda()).float().cpu().numpy()
    ref_s = oracle.swiglu(g.float().numpy(), np.ones_like(g.float().numpy()))
    assert arrays_close(s, ref_s, 1e-2 if dtype != torch.float32 else 1e-5, 1e-6)


def test_rope_tables_bit_exact(oracle):
    """compute_rope_tables vs the oracle (same libm, same rounding): identical bits."""
    import mlxr_b200 as mx
    for base, d in ((10000.0, 64), (500000.0, 128)):
        c, s = mx.compute_rope_tables(512, d, base)
        co, so = oracle.rope_tables(512, d, base)
        assert np.array_equal(c.numpy().view(np.uint16), co)
        assert np.array_equal(s.numpy().view(np.uint16), so)
    c, s = mx.compute_rope_tables(64, 32, 10000.0, mx.RoPEScalingMode.LINEAR, 4.0)
    co, so = oracle.rope_tables(64, 32, 10000.0, 3, 4.0)
    assert np.array_equal(c.numpy().view(np.uint16), co) and np.array_equal(s.numpy().view(np.uint16), so)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("layout", ["3d", "4d"])
def test_rope_apply(oracle, dtype, layout):
    import mlxr_b200 as mx
    code = {torch.float16: 0, torch.bfloat16: 1, torch.float32: 2}[dtype]
    heads, d, max_seq = 8, 128, 8192
    cos, sin = mx.compute_rope_tables(max_seq, d, 500000.0)
    g = torch.Generator().manual_seed(1)
    if layout == "3d":
        x = torch.randn(13, heads, d, generator=g).to(dtype)
        pos = torch.randint(0, max_seq, (13,), generator=g, dtype=torch.int32)
        x4 = x.unsqueeze(1)
    else:
        x = torch.randn(3, 5, heads, d, generator=g).to(dtype)
        pos = torch.randint(0, max_seq, (3, 5), generator=g, dtype=torch.int32)
        x4 = x
    y = mx.rope_apply(x.cuda(), cos.cuda(), sin.cuda(), pos.cuda())
    ref = oracle.rope_apply(x4.float().numpy(), cos.numpy().view(np.uint16), sin.numpy().view(np.uint16), pos.numpy())
    ref = oracle.round_to(ref, code).reshape(x.shape)
    # same fp32 operations in the same order, one rounding: identical values
    assert np.array_equal(y.float().cpu().numpy(), ref)
    # in place and LINEAR scaling with an offset
    x2 = x.clone().cuda()
    out = mx.rope_apply(x2, cos.cuda(), sin.cuda(), (pos // 2).cuda(), mx.RoPEScalingMode.LINEAR, 0.5, 3, inplace=True)
    assert out.data_ptr() == x2.data_ptr()
    ref2 = oracle.rope_apply(x4.float().numpy(), cos.numpy().view(np.uint16), sin.numpy().view(np.uint16),
                             (pos // 2).numpy(), 3, 0.5, 3)
    assert np.array_equal(x2.float().cpu().numpy(), oracle.round_to(ref2, code).reshape(x.shape))


def test_rope_errors():
    import mlxr_b200 as mx
    from mlxr_b200._capi import MlxrError
    cos, sin = mx.compute_rope_tables(16, 8)
    cos, sin = cos.cuda(), sin.cuda()
    x = torch.zeros(2, 4, 8, device="cuda", dtype=torch.float16)
    with pytest.raises(MlxrError, match="positions must have shape"):
        mx.rope_apply(x, cos, sin, torch.zeros(3, dtype=torch.int32, device="cuda"))
    with pytest.raises(MlxrError, match="cos_table must have shape"):
        mx.rope_apply(x, cos[:, :2].contiguous(), sin, torch.zeros(2, dtype=torch.int32, device="cuda"))
    with pytest.raises(MlxrError, match="outside"):
        mx.rope_apply(x, cos, sin, torch.tensor([0, 16], dtype=torch.int32, device="cuda"))
    with pytest.raises(MlxrError, match="3D"):
        mx.rope_apply(x[0], cos, sin, torch.zeros(2, dtype=torch.int32, device="cuda"))


def test_swiglu_mlp_dense_matches_composition():
    """swiglu_mlp() with dense weights and biases (swiglu_mlp_primitive.mm:47-82) against the
    same chain in float64."""
    import mlxr_b200 as mx
    g = torch.Generator().manual_seed(5)
    M, H, I = 3, 96, 224
    x = torch.randn(M, H, generator=g)
    wg, wu, wd = (torch.randn(I, H, generator=g) * 0.1, torch.randn(I, H, generator=g) * 0.1,
                  torch.randn(H, I, generator=g) * 0.1)
    bg, bu, bd = torch.randn(I, generator=g) * 0.1, torch.randn(I, generator=g) * 0.1, torch.randn(H, generator=g) * 0.1
    y = mx.swiglu_mlp(x.cuda(), wg.cuda(), wu.cuda(), wd.cuda(), bg.cuda(), bu.cuda(), bd.cuda()).cpu().double()
    xd = x.double()
    gt = xd @ wg.double().T + bg.double()
    ut = xd @ wu.double().T + bu.double()
    want = (gt * torch.sigmoid(gt) * ut) @ wd.double().T + bd.double()
    assert float((y - want).norm() / want.norm()) < 1e-5
    with pytest.raises(ValueError):
        mx.swiglu_mlp(x.cuda(), wg.cuda(), wu.cuda()[:, :8].contiguous(), wd.cuda())


def test_swiglu_is_rounded_from_float32():
    """16-bit swiglu is a float32 result rounded once, also where the exponential is small: an error of k float32 ulp
    before the rounding moves 2 k / 2^16 of all bf16 results to the other neighbour.  expf (1 ulp by its
    documented bound), 1 + e, the division and two products (half an ulp each) make k at most 3.5 and the share at most
    1.1e-4; an exponential whose error grows with the argument (2 + 1.17 |x| ulp, 58 on average here) moves 1.8e-3."""
    import mlxr_b200 as mx
    g = torch.Generator().manual_seed(1)
    gate = (-80 + 60 * torch.rand(1 << 21, generator=g)).to(torch.bfloat16).cuda()
    up = (1e20 * (1 + torch.rand(1 << 21, generator=g))).to(torch.bfloat16).cuda()
    want = (torch.nn.functional.silu(gate.double()) * up.double()).to(torch.bfloat16)
    assert float((mx.swiglu(gate, up) != want).float().mean()) <= 2e-4


def test_position_check_of_two_threads_on_one_stream():
    """The call that has the bad position gets the error, and only that one: the calls of both threads go to the same
    stream and overlap, since a call releases the interpreter lock while it waits."""
    import threading
    import mlxr_b200 as mx
    cos, sin = mx.compute_rope_tables(64, 64, 10000.0, device=torch.device("cuda"))
    x = torch.randn(64, 8, 64, device="cuda").half()
    good = torch.arange(64, dtype=torch.int32, device="cuda")
    bad = good + 1
    seen = {"good": 0, "bad": 0}

    def run(name, pos):
        for _ in range(400):
            try:
                mx.rope_apply(x, cos, sin, pos)
            except mx._capi.MlxrError:
                seen[name] += 1

    threads = [threading.Thread(target=run, args=a) for a in (("good", good), ("bad", bad), ("good", good))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert seen == {"good": 0, "bad": 400}


def test_in_place_and_behind_a_kernel_that_still_runs():
    """Every operator may write over what it reads, and may follow the kernel that writes its input without a pause
    between them: the results are those of a call on a copy, alone on the device."""
    import mlxr_b200 as mx
    from mlxr_b200._capi import check, lib
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(3)
    H, N = 4096, 2048
    for M in (1, 64):
        x = torch.randn(M, H, device="cuda", generator=g).half()
        r = torch.randn(M, N, device="cuda", generator=g).half()
        w = torch.randn(N, device="cuda", generator=g).half()
        blocks = torch.randint(0, 256, (N * H // 32, 18), dtype=torch.uint8, device="cuda", generator=g)
        blocks[:, :2] = torch.tensor([0, 0x18], dtype=torch.uint8, device="cuda")       # scale 2^-9
        lin = lambda: mx.q_gemm_dequant(x, blocks, M, N, H, mx.QuantType.Q4_0, 32)
        cos, sin = mx.compute_rope_tables(M, 64, 10000.0, device=torch.device("cuda"))
        pos = torch.arange(M, dtype=torch.int32, device="cuda")
        y = lin()
        torch.cuda.synchronize()
        want = [mx.rmsnorm_fused(y, w, 1e-5, r), mx.swiglu(y, r), mx.rope_apply(y.reshape(M, -1, 64), cos, sin, pos).reshape(M, N)]
        torch.cuda.synchronize()
        for _ in range(50):
            a, b, c, d, e = (lin() for _ in range(5))
            res, gate = r.clone(), r.clone()
            a = lin()
            check(lib.mlxr_rmsnorm(a.data_ptr(), w.data_ptr(), r.data_ptr(), a.data_ptr(), M, N, 1e-5, 0, st))       # over x
            b = lin()
            check(lib.mlxr_rmsnorm(b.data_ptr(), w.data_ptr(), res.data_ptr(), res.data_ptr(), M, N, 1e-5, 0, st))   # over the residual
            c = lin()
            check(lib.mlxr_swiglu(c.data_ptr(), r.data_ptr(), c.data_ptr(), M * N, 0, st))
            d = lin()
            check(lib.mlxr_swiglu(d.data_ptr(), gate.data_ptr(), gate.data_ptr(), M * N, 0, st))
            e = lin().reshape(M, -1, 64)
            mx.rope_apply(e, cos, sin, pos, inplace=True, check_positions=False)
            for got, ref in ((a, want[0]), (res, want[0]), (c, want[1]), (gate, want[1]), (e.reshape(M, N), want[2])):
                assert torch.equal(got, ref)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_swiglu_of_many_elements_is_that_of_few(dtype):
    """The vector kernel's quotient against the other kernel's IEEE division, every 16-bit gate (infinities and NaN among them):
    up to 2^18 elements take the one, more take the other."""
    import mlxr_b200 as mx
    gate = torch.arange(-32768, 32768, dtype=torch.int32, device="cuda").to(torch.int16).view(dtype)
    for scale in (1.0, 0.37, 250.0):
        up = torch.full((65536,), scale, device="cuda").to(dtype)
        few = mx.swiglu(gate, up)
        many = mx.swiglu(gate.repeat(5), up.repeat(5)).reshape(5, -1)
        nan = torch.isnan(few)
        assert torch.equal(torch.isnan(many), nan.expand(5, -1))
        assert torch.equal(many.view(torch.int16)[:, ~nan], few.view(torch.int16)[~nan].expand(5, -1))


@pytest.mark.parametrize("tokens,heads,dim", [(1, 1, 8), (257, 3, 24), (1001, 5, 64), (3000, 2, 136)])
def test_rope_of_odd_shapes_and_its_check(tokens, heads, dim):
    """Quotients of the vector's number by any count of vectors per token and head, bit for bit; the check sees the last of many
    positions, leaves that token alone and says so, and a call that was told so leaves nothing behind for the next."""
    import mlxr_b200 as mx
    cos, sin = mx.compute_rope_tables(512, dim, 10000.0, device=torch.device("cuda"))
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(tokens, heads, dim, device="cuda", generator=g).to(torch.float16)
    pos = torch.randint(0, 512, (tokens,), device="cuda", generator=g, dtype=torch.int32)
    c, s = cos[pos.long()].float()[:, None], sin[pos.long()].float()[:, None]
    e, o = x[..., 0::2].float(), x[..., 1::2].float()
    want = torch.stack([e * c - o * s, o * c + e * s], -1).reshape(x.shape).half()
    assert torch.equal(mx.rope_apply(x, cos, sin, pos), want)
    bad = pos.clone()
    bad[-1] = 512
    y = x.clone()
    with pytest.raises(mx._capi.MlxrError):
        mx.rope_apply(y, cos, sin, bad, inplace=True)
    torch.cuda.synchronize()
    assert torch.equal(y[:-1], want[:-1]) and torch.equal(y[-1], x[-1])
    assert torch.equal(mx.rope_apply(x, cos, sin, pos), want)


def test_checked_rope_behind_a_long_queue():
    """Positions written by a kernel far back in the stream's queue: the call waits for them however long that takes."""
    import mlxr_b200 as mx
    cos, sin = mx.compute_rope_tables(64, 64, 10000.0, device=torch.device("cuda"))
    x = torch.randn(64, 8, 64, device="cuda").half()
    pos = torch.full((64,), 99, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    torch.cuda._sleep(20_000_000)         # about 10 ms
    pos.copy_(torch.arange(64, dtype=torch.int32, device="cuda"))
    good = mx.rope_apply(x, cos, sin, pos)
    assert torch.equal(good, mx.rope_apply(x, cos, sin, torch.arange(64, dtype=torch.int32, device="cuda")))
    torch.cuda._sleep(20_000_000)
    pos.fill_(99)
    with pytest.raises(mx._capi.MlxrError):
        mx.rope_apply(x, cos, sin, pos)


@pytest.mark.parametrize("route", ["native", "interpreted", "abi"])
@pytest.mark.parametrize("bad", [False, True])
def test_checked_rope_has_ended_when_it_returns(route, bad):
    """A checked call returns, or raises, with the rotation done, whatever the path: its result may be used from another stream and its
    inputs released or overwritten at once.  In place, on a side stream, 256 MB (0.1 ms of rotation after the last
    position is known); the bad position is the last token's."""
    import mlxr_b200 as mx

    class Tagged(torch.Tensor):
        pass

    tokens, heads, dim = 32768, 32, 128
    cos, sin = mx.compute_rope_tables(512, dim, 10000.0, device=torch.device("cuda"))
    x = torch.ones(tokens, heads, dim, device="cuda", dtype=torch.float16)
    pos = torch.zeros(tokens, device="cuda", dtype=torch.int32)
    pos[-1] = 512 if bad else 0
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        raised = False
        if route == "abi":      # any non-zero value of the check argument
            raised = mx._capi.lib.mlxr_rope_apply(x.data_ptr(), cos.data_ptr(), sin.data_ptr(), pos.data_ptr(), x.data_ptr(), tokens, 1, heads, dim,
                                                  512, 0, 1.0, 0, 0, 2, st.cuda_stream) != 0
        else:
            try:
                mx.rope_apply(x if route == "native" else x.as_subclass(Tagged), cos, sin, pos, inplace=True)
            except mx._capi.MlxrError:
                raised = True
        assert st.query()
    assert raised == bad and torch.equal(x, torch.ones_like(x))      # a rotation by position 0 changes nothing


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_swiglu_quotients_by_many_products(dtype):
    """Every 16-bit gate times 64 values of up of all magnitudes: the vector kernel's results are those of the IEEE division."""
    import mlxr_b200 as mx
    gate = torch.arange(-32768, 32768, dtype=torch.int32, device="cuda").to(torch.int16).view(dtype)
    g = torch.Generator(device="cuda").manual_seed(5)
    ups = (torch.randn(64, device="cuda", generator=g) * 2.0 ** torch.randint(-12, 12, (64,), device="cuda", generator=g)).to(dtype)
    many = mx.swiglu(gate.repeat(64), ups.repeat_interleave(65536)).reshape(64, -1)
    for i in range(64):
        few = mx.swiglu(gate, ups[i].expand(65536).contiguous())
        nan = torch.isnan(few)
        assert torch.equal(torch.isnan(many[i]), nan)
        assert torch.equal(many[i].view(torch.int16)[~nan], few.view(torch.int16)[~nan])
