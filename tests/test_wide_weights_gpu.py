"""The weights that the wide kernel multiplies (csrc/widem.cu), one by one: with rows of the identity as activations every result is one
converted weight.  To 128 tokens a tile the codes go through a table, above that through arithmetic; both round a weight
once, and in fp16 both give the reference shader's half values to the bit.

Sizes: 128 tokens (table) and 256 (either, by the plan) of a matrix whose last tile is ragged, an odd number of super-blocks.
Bound for bf16: half an ulp of the weight, 2^-8 of it at most (eight significant bits), and for Q4_K, whose oracle holds products and sums rounded to half, the half ulp of
each of them, 2^-11 of magnitudes up to max |w| or a few ulp; a wrong code is off by a step of its block, max |w| / 16 or so."""
import numpy as np
import pytest
import torch

from conftest import make_weights
from test_wide_gpu import _dense, _launches

pytestmark = pytest.mark.gpu
DT = {"f16": torch.float16, "bf16": torch.bfloat16}


@pytest.mark.parametrize("qt", [0, 2, 3, 16])
@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("M", [128, 256])
def test_every_weight(oracle, qt, dt, M):
    import mlxr_b200 as mx
    from mlxr_b200.quantize import quantize
    N, K = 1000, 2816
    packed = quantize(make_weights(N, K, 7), qt)
    w, want = torch.from_numpy(packed).cuda(), _dense(oracle, packed, N, K, qt)
    eye = torch.eye(K, device="cuda", dtype=DT[dt])
    got = torch.empty(N, K, device="cuda", dtype=DT[dt])
    for k in range(0, K, M):
        y, launches = _launches(lambda: mx.q_gemm_dequant(eye[k:k + M].contiguous(), w, M, N, K, mx.QuantType(qt), mx._capi.lib.mlxr_default_group_size(qt)))
        assert launches == 1
        got[:, k:k + M] = y.T
    if dt == "f16":
        assert torch.equal(got, want.half())
    else:
        assert bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + (2.0 ** -10 * want.abs().max() if qt == 3 else 0)).all())
