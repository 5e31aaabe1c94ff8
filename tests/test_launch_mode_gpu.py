"""mlxr_set_decode_launch_mode reaches every kernel that can start under the previous one of its stream: the launches are
captured into a CUDA graph, where programmatic stream serialization shows as edges of programmatic type."""
import pytest
import torch

pytestmark = pytest.mark.gpu
COOPERATIVE, OVERLAPPED = 0, 2


def _programmatic_edges(fn):
    from cuda.bindings import driver
    s = torch.cuda.Stream()
    fn(s.cuda_stream)                      # workspaces and attributes
    s.synchronize()
    st = driver.CUstream(s.cuda_stream)
    err, = driver.cuStreamBeginCapture(st, driver.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_RELAXED)
    assert err == driver.CUresult.CUDA_SUCCESS
    fn(s.cuda_stream)
    err, graph = driver.cuStreamEndCapture(st)
    assert err == driver.CUresult.CUDA_SUCCESS
    # edges of a type other than the default one cannot be returned by this form of the query
    err = driver.cuGraphGetEdges(graph, 256)[0]
    driver.cuGraphDestroy(graph)
    assert err in (driver.CUresult.CUDA_SUCCESS, driver.CUresult.CUDA_ERROR_LOSSY_QUERY)
    return err == driver.CUresult.CUDA_ERROR_LOSSY_QUERY


def _calls():
    from mlxr_b200._capi import check, lib
    dev, bf16 = torch.device("cuda"), torch.bfloat16
    p = lambda t: t.data_ptr()
    for M, H, qt, gs, per in ((1, 512, 3, 256, 144 / 256), (1, 8192, 3, 256, 144 / 256), (1, 4096, 2, 32, 34 / 32), (8, 2048, 16, 64, 34 / 64), (100, 512, 3, 256, 144 / 256), (2048, 512, 0, 32, 18 / 32)):
        D, heads = 64, H // 64
        x, y = torch.zeros(M, H, device=dev, dtype=bf16), torch.zeros(M, H, device=dev, dtype=bf16)
        w = torch.zeros(int(H * H * per), device=dev, dtype=torch.uint8)
        nw, k, v = torch.ones(H, device=dev, dtype=bf16), torch.zeros_like(x), torch.zeros_like(x)
        cos = torch.zeros(M, D // 2, device=dev, dtype=torch.float16)
        pos = torch.arange(M, device=dev, dtype=torch.int32)

        def linear(st):
            for _ in range(2):
                check(lib.mlxr_q_gemm_dequant(p(x), p(w), None, p(y), M, H, H, qt, gs, 1, st))

        def block(st):
            for _ in range(2):
                check(lib.mlxr_mlp_block(p(x), p(nw), p(w), p(w), p(w), p(y), M, H, H, qt, 1e-5, 1, st))

        def qkv(st):
            for _ in range(2):
                check(lib.mlxr_qkv_rope(p(x), p(nw), p(w), p(w), p(w), p(cos), p(cos), p(pos), p(y), p(k), p(v), M, H, heads, heads, D, M, qt, 1e-5, 0, 1, st))

        def pieces(st):
            for _ in range(2):
                check(lib.mlxr_rmsnorm(p(x), p(nw), None, p(y), M, H, 1e-5, 1, st))
            check(lib.mlxr_rope_apply(p(x), p(cos), p(cos), p(pos), p(y), M, 1, heads, D, M, 0, 1.0, 0, 1, 0, st))

        yield from ((f"{f.__name__} {M} {H} {qt}", f) for f in (linear, block, qkv, pieces))


def test_mode_reaches_every_launch():
    from mlxr_b200._capi import check, lib
    try:
        for name, fn in _calls():
            check(lib.mlxr_set_decode_launch_mode(OVERLAPPED))
            assert _programmatic_edges(fn), name
            check(lib.mlxr_set_decode_launch_mode(COOPERATIVE))
            assert not _programmatic_edges(fn), name
    finally:
        check(lib.mlxr_set_decode_launch_mode(OVERLAPPED))
