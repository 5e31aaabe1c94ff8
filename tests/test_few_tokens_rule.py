"""Which of the two kernels of up to eight tokens a call goes to (host arithmetic, no GPU): sizes at which each of them was measured to be
the faster one by 5 % and more (Q4_K and Q4_0, more exact in the kernel of whole rows: the other one by an eighth)."""
import pytest

Q4_0, Q8_0, Q4_K, CANONICAL = 0, 2, 3, 33
F16, BF16 = 0, 1
PLAIN, GATE_UP, STACKED = 0, 1, 2


@pytest.mark.parametrize("qt,M,N,K,dtype", [
    (CANONICAL, 3, 256, 16384, BF16), (CANONICAL, 5, 600, 8192, BF16), (CANONICAL, 7, 1000, 5632, BF16), (CANONICAL, 7, 2560, 6656, BF16), (CANONICAL, 1, 600, 49152, BF16), (CANONICAL, 5, 2560, 8192, BF16),
    (CANONICAL, 1, 256, 49152, F16), (CANONICAL, 1, 256, 512, BF16), (CANONICAL, 1, 1000, 256, F16),
    (Q8_0, 3, 1000, 16384, BF16), (Q8_0, 3, 3000, 16384, BF16), (Q8_0, 5, 256, 9728, BF16), (Q8_0, 8, 1000, 5632, BF16), (Q8_0, 3, 600, 16384, F16),
    (Q4_K, 3, 1000, 8192, BF16), (Q4_K, 3, 1000, 16384, BF16), (Q4_K, 4, 6144, 1024, BF16), (Q4_K, 5, 5120, 1280, BF16), (Q4_K, 6, 1000, 4096, BF16),
    (Q4_K, 8, 2048, 3072, BF16), (Q4_K, 3, 8192, 1536, BF16), (Q4_0, 3, 256, 16384, BF16), (Q4_0, 8, 1000, 4096, BF16)])
def test_sizes_of_the_kernel_that_splits_k(qt, M, N, K, dtype):
    from mlxr_b200._capi import lib
    assert lib.mlxr_debug_few_tokens_rule(qt, M, K, N, PLAIN, dtype) == 0


@pytest.mark.parametrize("qt,M,N,K,dtype", [
    (CANONICAL, 1, 1000, 1024, BF16), (CANONICAL, 1, 14336, 4096, BF16), (CANONICAL, 1, 4096, 49152, BF16), (CANONICAL, 5, 4096, 4096, F16), (CANONICAL, 5, 1000, 4096, BF16),
    (CANONICAL, 8, 1000, 5632, F16), (CANONICAL, 3, 4096, 16384, BF16), (CANONICAL, 1, 2048, 32768, BF16), (CANONICAL, 1, 1536, 32768, F16), (Q8_0, 3, 4096, 14336, BF16), (Q8_0, 8, 14336, 4096, BF16), (Q8_0, 8, 1000, 3072, BF16), (Q8_0, 4, 2048, 8192, BF16),
    (Q4_K, 3, 1000, 2048, BF16), (Q4_K, 3, 4096, 3072, BF16), (Q4_K, 8, 1000, 1536, BF16), (Q4_K, 5, 6144, 1536, BF16), (Q4_K, 6, 2048, 2048, BF16), (Q4_0, 5, 1000, 3072, BF16), (Q4_0, 8, 256, 2048, BF16), (Q4_K, 8, 4096, 1024, BF16), (Q4_K, 6, 1000, 3072, BF16), (Q4_K, 3, 1000, 768, BF16)])
def test_sizes_of_the_kernel_of_whole_rows(qt, M, N, K, dtype):
    from mlxr_b200._capi import lib
    assert lib.mlxr_debug_few_tokens_rule(qt, M, K, N, PLAIN, dtype) == 1


@pytest.mark.parametrize("qt,M,H,rows,dtype,want", [
    (Q4_K, 8, 2560, 3584, BF16, 0), (Q8_0, 8, 2560, 3584, BF16, 0), (Q4_K, 8, 3072, 4096, BF16, 0), (CANONICAL, 7, 5120, 6144, BF16, 1), (Q4_K, 8, 4096, 6144, BF16, 1), (Q8_0, 7, 4096, 6144, BF16, 1), (Q4_K, 8, 6144, 6400, BF16, 1),
    (Q4_K, 8, 1024, 1280, BF16, 1), (Q8_0, 8, 2560, 3584, F16, 1), (Q4_0, 5, 2560, 3584, BF16, 1)])
def test_stacked(qt, M, H, rows, dtype, want):
    from mlxr_b200._capi import lib
    assert lib.mlxr_debug_few_tokens_rule(qt, M, H, rows, STACKED, dtype) == want


@pytest.mark.parametrize("qt,M,H,I,want", [(Q4_K, 3, 1024, 2048, 1), (Q4_0, 8, 1024, 2048, 1), (Q4_K, 3, 1024, 3584, 1), (Q4_K, 5, 1024, 3584, 1), (Q4_K, 8, 1024, 2816, 1), (Q4_K, 6, 1024, 3584, 0), (Q8_0, 8, 4096, 14336, 1), (CANONICAL, 8, 4096, 14336, 1)])
def test_gate_up(qt, M, H, I, want):
    from mlxr_b200._capi import lib
    assert lib.mlxr_debug_few_tokens_rule(qt, M, H, 2 * I, GATE_UP, BF16) == want
