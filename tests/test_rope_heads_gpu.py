"""rope_apply where a thread rotates several heads of a token (csrc/elementwise.cu: four or two from about 450,000 or 230,000 vectors of eight on) and
where the kernel answers a checked call itself."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _want(x, cos, sin, pos):
    c, s = cos[pos.long()].float()[:, None], sin[pos.long()].float()[:, None]
    e, o = x[..., 0::2].float(), x[..., 1::2].float()
    return torch.stack((e * c - o * s, o * c + e * s), -1).flatten(-2).to(x.dtype)


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("tokens,heads,d", [(3, 5, 64), (6000, 5, 64), (11500, 5, 64), (4100, 7, 128), (2100, 7, 128), (120, 1, 8)])
def test_heads_of_a_thread(dt, tokens, heads, d):
    """Head counts that four and two do not divide.  float32 products and one rounding on both sides: the same values."""
    import mlxr_b200 as mx
    g = torch.Generator(device="cuda").manual_seed(tokens)
    cos, sin = mx.compute_rope_tables(512, d, 10000.0, device=torch.device("cuda"))
    x = torch.randn(tokens, heads, d, device="cuda", generator=g).to(dt)
    pos = torch.randint(0, 512, (tokens,), device="cuda", generator=g, dtype=torch.int32)
    want = _want(x, cos, sin, pos)
    for check in (True, False):
        assert torch.equal(mx.rope_apply(x, cos, sin, pos, check_positions=check), want)
    # a position outside the table: reported, the other tokens rotated; the next call finds clean words
    pos[tokens // 2] = 512
    y = x.clone()
    with pytest.raises(mx._capi.MlxrError):
        mx.rope_apply(y, cos, sin, pos, inplace=True)
    want[tokens // 2] = x[tokens // 2]
    assert torch.equal(y, want)
    pos[tokens // 2] = 0
    assert torch.equal(mx.rope_apply(x, cos, sin, pos), _want(x, cos, sin, pos))


def test_answer_behind_longer_work():
    """A checked call behind work that takes longer than the host looks for the answer itself."""
    import mlxr_b200 as mx
    cos, sin = mx.compute_rope_tables(64, 64, 10000.0, device=torch.device("cuda"))
    x = torch.randn(100, 4, 64, device="cuda").half()
    pos = torch.randint(0, 64, (100,), device="cuda", dtype=torch.int32)
    a = torch.randn(4096, 4096, device="cuda")
    for _ in range(10):
        a = torch.nn.functional.normalize(a @ a)
    assert torch.equal(mx.rope_apply(x, cos, sin, pos), _want(x, cos, sin, pos))


def test_threads_that_share_a_stream_handle():
    """Two threads that both pass cudaStreamPerThread share the handle, not the stream: each call's answer and rotation are its own, whatever
    the other's number of CTAs (4 and 1200), and the rotation is done when the call returns."""
    import threading
    import mlxr_b200 as mx
    from mlxr_b200._capi import ERR_SHAPE, OK, lib
    per_thread, D, P = 2, 64, 512
    cos, sin = mx.compute_rope_tables(P, D, 10000.0, device=torch.device("cuda"))
    wrong = []

    def run(tokens, heads):
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            x = torch.randn(tokens, heads, D, device="cuda").half()
            good = torch.randint(0, P, (tokens,), device="cuda", dtype=torch.int32)
            bad = good.clone()
            bad[-1] = P
            want, y = _want(x, cos, sin, good), torch.empty_like(x)
            for i in range(300):
                pos, code = (bad, ERR_SHAPE) if i % 3 == 1 else (good, OK)
                y.zero_()
                side.synchronize()
                r = lib.mlxr_rope_apply(x.data_ptr(), cos.data_ptr(), sin.data_ptr(), pos.data_ptr(), y.data_ptr(), 1, tokens, heads, D, P, 0, 1.0, 0, 0, 1, per_thread)
                n = tokens - 1 if pos is bad else tokens
                if r != code or not torch.equal(y[:n], want[:n]):
                    wrong.append((tokens, i, r))

    torch.cuda.synchronize()
    threads = [threading.Thread(target=run, args=a) for a in ((16, 8), (9600, 16), (16, 8))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("tokens,q_heads,kv_heads,d", [(512, 61, 3, 64), (512, 125, 1, 64), (512, 123, 3, 64), (2100, 7, 1, 128), (4100, 7, 2, 128)])
def test_q_and_k_in_one_launch(tokens, q_heads, kv_heads, d):
    """Two (the first and fourth sizes) and four heads a thread, of both tensors, with head counts that they do not divide: what the
    rotation of each by itself gives."""
    import mlxr_b200 as mx
    H, qt = 256, mx.QuantType.Q8_0
    g = torch.Generator(device="cuda").manual_seed(tokens)
    x = torch.randn(tokens, H, device="cuda", generator=g).half()
    cos, sin = mx.compute_rope_tables(512, d, 10000.0, device=torch.device("cuda"))
    pos = torch.randint(0, 512, (tokens,), device="cuda", generator=g, dtype=torch.int32)

    def weights(heads):
        b = torch.randint(0, 256, (heads * d * H // 32, 34), dtype=torch.uint8, device="cuda", generator=g)
        b[:, :2] = torch.tensor([0, 0x18], dtype=torch.uint8, device="cuda")       # scale 2^-9
        return b.reshape(-1)

    ws = [weights(h) for h in (q_heads, kv_heads, kv_heads)]
    got = mx.qkv_rope(x, None, *ws, cos, sin, pos, q_heads, kv_heads, d, qt)
    lin = [mx.q_gemm_dequant(x, w, tokens, h * d, H, qt, 32).reshape(tokens, h, d) for w, h in zip(ws, (q_heads, kv_heads, kv_heads))]
    assert torch.equal(got[0], _want(lin[0], cos, sin, pos)) and torch.equal(got[1], _want(lin[1], cos, sin, pos)) and torch.equal(got[2], lin[2])


def test_more_work_than_ctas():
    """80,000 tokens of four heads of 128: 5000 CTAs' worth of units for 4736 CTAs; the position outside the table is among the last ones."""
    import mlxr_b200 as mx
    tokens, d = 80000, 128
    cos, sin = mx.compute_rope_tables(64, d, 10000.0, device=torch.device("cuda"))
    x = torch.randn(tokens, 4, d, device="cuda").half()
    pos = torch.randint(0, 64, (tokens,), device="cuda", dtype=torch.int32)
    want = _want(x, cos, sin, pos)
    assert torch.equal(mx.rope_apply(x, cos, sin, pos), want)
    pos[-2] = 64
    want[-2] = x[-2]          # left as it was
    with pytest.raises(mx._capi.MlxrError):
        mx.rope_apply(x, cos, sin, pos, inplace=True)
    assert torch.equal(x, want)


def test_a_checked_call_readies_its_stream():
    """A stream whose first call was a checked one can be captured: what calls in it need is there."""
    import mlxr_b200 as mx
    cos, sin = mx.compute_rope_tables(64, 64, 10000.0, device=torch.device("cuda"))
    x = torch.randn(100, 4, 64, device="cuda").half()
    pos = torch.randint(0, 64, (100,), device="cuda", dtype=torch.int32)
    y = torch.empty_like(x)
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        mx.rope_apply(x, cos, sin, pos)
    st.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        y.copy_(mx.rope_apply(x, cos, sin, pos, check_positions=False))
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, _want(x, cos, sin, pos))
