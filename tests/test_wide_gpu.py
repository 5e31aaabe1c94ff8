"""Linears of more than 64 tokens (csrc/widem.cu: weights converted beside the MMAs; csrc/dense.cu: converted to
16 bits in a pass of their own) through the C ABI.

Sizes are the edges of the kernels' tiles: one token more and less than a token tile, weight rows that end inside a
tile of 128 or 256 and, odd, inside a 16-byte store, an odd number of super-blocks (NF4 rows then start 8 bytes
off), few and many units per CTA, tiles shared by CTAs, and K that is no multiple of 256 or of 64.

Bound: the products are exact and accumulate in float32; the weight is rounded once to the activation dtype and the
result once more, each by at most 2^-8 (bf16, eight significant bits) or 2^-11 (fp16) of itself and about 0.4 of
that in the root mean square (Q4_K's scale and min round in half precision in both sides), so the 2-norm of the
two together is below 2^-8 and 2^-11."""
import numpy as np
import pytest
import torch

from conftest import make_acts, make_weights

pytestmark = pytest.mark.gpu
DT = {"f16": torch.float16, "bf16": torch.bfloat16}
BOUND = {"f16": 2.0 ** -11, "bf16": 2.0 ** -8}


def _status():
    import mlxr_b200 as mx
    st = torch.zeros(1, dtype=torch.int32)
    mx._capi.check(mx._capi.lib.mlxr_stream_status(torch.cuda.current_stream().cuda_stream, st.data_ptr()))
    return int(st[0])


def _dense(oracle, packed, N, K, qt):
    """The weights as float64: the shader's half values for Q4_K, the float32 products otherwise."""
    f, h = oracle.dequantize(packed, N, K, qt)
    w = h.view(np.float16) if qt == 3 else f
    return torch.from_numpy(w.astype(np.float64).reshape(N, K)).cuda()


def _check(oracle, qt, dt, M, N, K, bias=True, offset=0):
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    packed = quantize(make_weights(N, K, 7 + M), qt)
    xt, _ = make_acts(M, K, 8 + M, DT[dt])
    b = make_acts(1, N, 9, DT[dt])[0][0].contiguous().cuda() if bias else None
    x = xt.cuda()
    buf = torch.empty(packed.size + offset, dtype=torch.uint8, device="cuda")
    w = buf[offset:]
    w.copy_(torch.from_numpy(packed))
    args = (x, w, M, N, K, mx.QuantType(qt), mx._capi.lib.mlxr_default_group_size(qt), b)
    y = mx.q_gemm_dequant(*args)
    assert torch.equal(y, mx.q_gemm_dequant(*args))     # nothing depends on the order of arrival
    assert _status() == 0
    want = x.double() @ _dense(oracle, packed, N, K, qt).T + (b.double() if bias else 0)
    assert float((y.double() - want).norm() / want.norm()) <= BOUND[dt]


@pytest.mark.parametrize("qt", [0, 2, 3, 16])
@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("M,N,K", [(65, 2, 256), (128, 257, 768), (129, 1000, 1280), (257, 385, 512), (333, 2304, 2816)])
def test_beside_the_mmas(oracle, qt, dt, M, N, K):
    _check(oracle, qt, dt, M, N, K)


@pytest.mark.parametrize("qt", [0, 2, 3, 16])
@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("M,N,K", [(2048, 255, 512), (2049, 520, 256), (4095, 1001, 768)])
def test_in_a_pass_of_its_own(oracle, qt, dt, M, N, K):
    _check(oracle, qt, dt, M, N, K, bias=(N == 520))


@pytest.mark.parametrize("qt,M,N,K,offset", [(0, 9, 33, 96, 0), (2, 130, 300, 320, 0), (16, 70, 129, 448, 0), (0, 100, 256, 512, 2), (2, 20, 64, 256, 2)])
def test_ragged_k_and_rows_off_16_bytes(oracle, qt, M, N, K, offset):
    _check(oracle, qt, "f16", M, N, K, offset=offset)


@pytest.mark.parametrize("qt", [0, 2, 3, 16])
@pytest.mark.parametrize("M,H,I", [(100, 768, 1280), (2100, 256, 768)])
def test_gate_up(oracle, qt, M, H, I):
    """The SiLU(gate) * up forms of both kernels inside the block, against the block built from this package's own
    single operators in float64: n and h are rounded to bf16 on both sides (2^-9 each where they differ by an ulp),
    weights and result once: 1e-2 covers the four."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    g, u, d = (quantize(make_weights(n, k, s), qt) for n, k, s in ((I, H, 1), (I, H, 2), (H, I, 3)))
    x = make_acts(M, H, 4, torch.bfloat16)[0].cuda()
    nw = make_acts(1, H, 5, torch.bfloat16)[0][0].contiguous().cuda()
    y = mx.mlp_block(x, nw, *(torch.from_numpy(w).cuda() for w in (g, u, d)), I, mx.QuantType(qt), 1e-5)
    assert _status() == 0
    n = mx.rmsnorm_fused(x, nw, 1e-5).double()
    gate, up = (n @ _dense(oracle, w, I, H, qt).T for w in (g, u))
    h = (torch.nn.functional.silu(gate.bfloat16().double()) * up.bfloat16().double()).bfloat16().double()
    want = h @ _dense(oracle, d, H, I, qt).T
    assert float((y.double() - want).norm() / want.norm()) <= 1e-2


@pytest.mark.parametrize("qt", [0, 2])
@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("M,K", [(9, 96), (70, 1056)])
def test_weights_are_not_rounded_at_32_mod_64(oracle, qt, dt, M, K):
    """Rows of an odd number of 32-weight blocks multiply the float32 weights: the result's own rounding is left, at most 2^-8
    (2^-11) of each value and about 0.42 of that in the 2-norm; with rounded weights it is 0.6 of it."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    N = 300
    packed = quantize(make_weights(N, K, 7), qt)
    x = make_acts(M, K, 8, DT[dt])[0].cuda()
    y = mx.q_gemm_dequant(x, torch.from_numpy(packed).cuda(), M, N, K, mx.QuantType(qt), 32)
    want = x.double() @ _dense(oracle, packed, N, K, qt).T
    assert float((y.double() - want).norm() / want.norm()) <= BOUND[dt] / 2


def _launches(fn):
    from mlxr_b200._capi import lib
    before = lib.mlxr_launch_count()
    y = fn()
    return y, lib.mlxr_launch_count() - before


@pytest.mark.parametrize("qt", [0, 2, 3, 16])
@pytest.mark.parametrize("M,N,K,launches", [(65, 2, 2816, 1), (128, 257, 2816, 1), (129, 1000, 4096, 1), (257, 385, 2816, 1), (333, 2304, 2816, 1), (65, 4097, 768, 1),
                                            (512, 8001, 1280, 1), (65, 2, 256, 2), (1100, 2304, 4096, 2), (2048, 255, 512, 2), (2049, 520, 256, 2), (4095, 1001, 768, 2)])
def test_either_kernel_for_certain(oracle, qt, M, N, K, launches):
    """Which of the two kernels runs follows from their estimated times: small matrices take the pass and the GEMM (two
    launches) from 65 tokens on.  The edges of the wide kernel's tiles at sizes that it takes, and both of them told apart."""
    import mlxr_b200 as mx
    x = torch.zeros(M, K, device="cuda", dtype=torch.bfloat16)
    w = torch.zeros(mx.compute_quantized_weight_size(N, K, mx.QuantType(qt)), device="cuda", dtype=torch.uint8)
    assert _launches(lambda: mx.q_gemm_dequant(x, w, M, N, K, mx.QuantType(qt), mx._capi.lib.mlxr_default_group_size(qt)))[1] == launches
    _check(oracle, qt, "bf16" if M % 2 else "f16", M, N, K)


@pytest.mark.parametrize("qt", [0, 2, 3, 16])
@pytest.mark.parametrize("M,H,I", [(100, 2816, 1280), (200, 2816, 3008)])
def test_gate_up_beside_the_mmas(oracle, qt, M, H, I):
    """As test_gate_up, at a hidden size for which gate / up is one launch of the wide kernel (odd numbers of super-blocks, tiles
    shared by CTAs; 3008 rows do not fill their last tile): 1e-2 as there, for down's K only formats of 32- and 64-blocks."""
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    if qt == 3 and I % 256:
        I = 3072
    g, u, d = (quantize(make_weights(n, k, s), qt) for n, k, s in ((I, H, 1), (I, H, 2), (H, I, 3)))
    x = make_acts(M, H, 4, torch.bfloat16)[0].cuda()
    args = [torch.from_numpy(w).cuda() for w in (g, u, d)]
    down = _launches(lambda: mx.q_gemm_dequant(torch.zeros(M, I, device="cuda", dtype=torch.bfloat16), args[2], M, H, I, mx.QuantType(qt), mx._capi.lib.mlxr_default_group_size(qt)))[1]
    y, launches = _launches(lambda: mx.mlp_block(x, None, *args, I, mx.QuantType(qt)))
    assert launches == 1 + down and _status() == 0
    gate, up = (x.double() @ _dense(oracle, w, I, H, qt).T for w in (g, u))
    h = (torch.nn.functional.silu(gate.bfloat16().double()) * up.bfloat16().double()).bfloat16().double()
    want = h @ _dense(oracle, d, H, I, qt).T
    assert float((y.double() - want).norm() / want.norm()) <= 1e-2


def _device_blocks(N, K, seed):
    """Q4_0 blocks with scales around 2^-8, made on the device (large matrices)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randint(0, 256, (N * K // 32, 18), dtype=torch.uint8, device="cuda", generator=g)
    w[:, 1] = 0x1C
    return w.reshape(-1)


def test_slices_of_the_16_bit_weights():
    """More than 256 MB of 16-bit weights go through the buffer in slices: three of 6912 rows, which the tile of 160 rows does
    not divide, the last one ragged and the row count odd (K = 64 mod 256 has no other kernel)."""
    import mlxr_b200 as mx
    M, N, K = 700, 20001, 16448
    w = _device_blocks(N, K, 1)
    x = torch.randn(M, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2)).half()
    b = torch.randn(N, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3)).half()
    y, launches = _launches(lambda: mx.q_gemm_dequant(x, w, M, N, K, mx.QuantType.Q4_0, 32, b))
    assert launches == 2 * 3 and _status() == 0
    want = x.double() @ mx.dequantize(w, N, K, mx.QuantType.Q4_0, torch.float32).double().T + b.double()
    assert float((y.double() - want).norm() / want.norm()) <= BOUND["f16"]
    assert float((y.double() - want).norm(dim=0).max() / want.norm(dim=0).mean()) <= 4 * BOUND["f16"]      # no column is someone else's


def test_slices_of_gate_and_up():
    """The same for gate / up (the slices' rows alternate between the two matrices) and, in two slices, for down."""
    import mlxr_b200 as mx
    M, H, I = 700, 16448, 10048
    g, u, d = _device_blocks(I, H, 1), _device_blocks(I, H, 2), _device_blocks(H, I, 3)
    x = torch.randn(M, H, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2)).half()
    y, launches = _launches(lambda: mx.mlp_block(x, None, g, u, d, I, mx.QuantType.Q4_0))
    assert launches == 2 * 3 + 2 * 2 and _status() == 0
    deq = lambda w, n, k: mx.dequantize(w, n, k, mx.QuantType.Q4_0, torch.float32).double()
    gate, up = (x.double() @ deq(w, I, H).T for w in (g, u))
    h = (torch.nn.functional.silu(gate.half().double()) * up.half().double()).half().double()
    want = h @ deq(d, H, I).T
    # g, u, h and the result are rounded to fp16 on both sides from sums over weights rounded on one: 2e-3 as everywhere
    assert float((y.double() - want).norm() / want.norm()) <= 2e-3
    assert float((y.double() - want).norm(dim=0).max() / want.norm(dim=0).mean()) <= 8e-3
