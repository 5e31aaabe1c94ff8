"""The native call path from torch tensors (cpp/torch_ops.cpp): what it leaves to the interpreted wrapper, which errors
come out, and that the interpreter survives them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _qkv(**over):
    import mlxr_b200 as mx
    H, QH, KH, D, M = 256, 2, 1, 64, 3
    x = torch.randn(M, H, device="cuda", dtype=torch.float16)
    cos, sin = mx.compute_rope_tables(16, D, 10000.0, device=torch.device("cuda"))
    a = dict(x=x, norm=torch.ones(H, device="cuda", dtype=torch.float16), cos=cos, sin=sin, pos=torch.arange(M, device="cuda", dtype=torch.int32),
             **{n: torch.zeros(h * D * 144, device="cuda", dtype=torch.uint8) for n, h in (("wq", QH), ("wk", KH), ("wv", KH))})
    a.update(over)
    return mx.qkv_rope(a["x"], a["norm"], a["wq"], a["wk"], a["wv"], a["cos"], a["sin"], a["pos"], QH, KH, D, mx.QuantType.Q4_K)


def test_tensors_without_memory():
    """vmap's and torch.func.grad's wrappers and fake tensors have no memory to point at: an error, raised with the
    interpreter lock held."""
    import mlxr_b200 as mx
    from torch._subclasses.fake_tensor import FakeTensorMode
    x = torch.randn(4, 64, device="cuda", dtype=torch.float16)
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda t: mx.swiglu(t, t))(x)
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: mx.rmsnorm_fused(t, t[0]).sum())(x.float())
    with FakeTensorMode() as mode:
        f = mode.from_tensor(x)
        with pytest.raises(RuntimeError):
            mx.swiglu(f, f)
    assert torch.isfinite(mx.swiglu(x, x)).all()


def test_subclass_is_kept():
    import mlxr_b200 as mx

    class Tagged(torch.Tensor):
        pass

    x = torch.randn(4, 64, device="cuda", dtype=torch.float16)
    w = torch.ones(64, device="cuda", dtype=torch.float16)
    y = mx.rmsnorm_fused(x.as_subclass(Tagged), w)
    assert type(y) is Tagged and torch.equal(y.as_subclass(torch.Tensor), mx.rmsnorm_fused(x, w))
    assert type(mx.swiglu(x.as_subclass(Tagged), x.as_subclass(Tagged))) is Tagged
    assert torch.equal(mx.rmsnorm_fused(x, torch.nn.Parameter(w)), mx.rmsnorm_fused(x, w))


def test_out_of_memory_keeps_its_type():
    import mlxr_b200 as mx
    n = 1 << 20                                     # 2 TB of result
    x, w = torch.zeros(n, 32, device="cuda", dtype=torch.float16), torch.zeros(n * 18, device="cuda", dtype=torch.uint8)
    with pytest.raises(torch.OutOfMemoryError):
        mx.q_gemm_dequant(x, w, n, n, 32, mx.QuantType.Q4_0, 32)


@pytest.mark.parametrize("over", [dict(wq=128 * 144 - 1), dict(wk=64 * 144 - 16), dict(wv=0), dict(cos=(16, 16)), dict(sin=(15, 32)), dict(norm=255)])
def test_qkv_rope_refuses_short_buffers(over):
    import mlxr_b200 as mx
    (name, size), = over.items()
    dt = torch.uint8 if name[0] == "w" else torch.float16
    with pytest.raises(mx._capi.MlxrError):
        _qkv(**{name: torch.zeros(size, device="cuda", dtype=dt)})
    assert len(_qkv()) == 3


def test_other_operators_refuse_short_buffers():
    import mlxr_b200 as mx
    x, w = torch.randn(4, 64, device="cuda", dtype=torch.float16), torch.ones(64, device="cuda", dtype=torch.float16)
    for r in (x[:3], x.float()):
        with pytest.raises(mx._capi.MlxrInvalidArgument):
            mx.rmsnorm_fused(x, w, 1e-5, r)
    cos, sin = mx.compute_rope_tables(16, 64, 10000.0, device=torch.device("cuda"))
    with pytest.raises(mx._capi.MlxrError):
        mx.rope_apply(x.reshape(4, 1, 64), cos, sin[:8], torch.arange(4, device="cuda", dtype=torch.int32))
