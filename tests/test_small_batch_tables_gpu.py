"""Up to 32 tokens of Q4_K and Q4_0 look their codes up in a table, 33 to 64 tokens compute them (csrc/smallm.cu): the weights are
the same 16-bit numbers.

Sizes: the edges of the padded batches 16 and 32 (the latter with three stages of X between two issuers), row counts for
16-byte stores, for a tile's ragged end and odd ones, more units than stages.

Bound: the two sides differ by the order of float32 sums, about 2e-7 of the result.  A rounding to p bits turns a difference d into
sqrt(d 2^(1 - p)) in the 2-norm: 4e-5 for bf16 (p = 8), 1.4e-5 for fp16 (11).  One wrong code in a thousand gives 1e-2."""
import pytest
import torch

from conftest import make_acts, make_weights

pytestmark = pytest.mark.gpu
DT = {"f16": torch.float16, "bf16": torch.bfloat16}


@pytest.mark.parametrize("qt", [0, 3])
@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("N,K", [(264, 2560), (2048, 1792), (1001, 4352), (20480, 512)])
def test_table_and_arithmetic_agree(qt, dt, N, K):
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    w = torch.from_numpy(quantize(make_weights(N, K, 1), qt)).cuda()
    x = make_acts(33, K, 2, DT[dt])[0].cuda()
    q, gs = mx.QuantType(qt), mx._capi.lib.mlxr_default_group_size(qt)
    want = mx.q_gemm_dequant(x, w, 33, N, K, q, gs).double()
    for M in (9, 16, 17, 32):
        y = mx.q_gemm_dequant(x[:M].contiguous(), w, M, N, K, q, gs).double()
        assert float((y - want[:M]).norm() / want[:M].norm()) <= {"bf16": 1.5e-4, "f16": 5e-5}[dt], M


@pytest.mark.parametrize("qt", [0, 3])
@pytest.mark.parametrize("M,H,I", [(16, 1024, 2816), (31, 2816, 1280)])
def test_gate_up(oracle, qt, M, H, I):
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    g, u, d = (quantize(make_weights(n, k, s), qt) for n, k, s in ((I, H, 1), (I, H, 2), (H, I, 3)))
    xt, xf = make_acts(M, H, 4, torch.bfloat16)
    y = mx.mlp_block(xt.cuda(), None, *(torch.from_numpy(w).cuda() for w in (g, u, d)), I, mx.QuantType(qt), 1e-5)
    assert oracle.rel_l2(y.float().cpu().numpy(), oracle.mlp_block(xf, None, g, u, d, I, qt, 1e-5, oracle.BF16)) <= 1e-2
