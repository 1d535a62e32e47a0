"""Scratch of the ordered INT4 GEMV over the number of rows: one workspace for the largest batch serves every smaller one, its size
does not grow with a long prompt, and any number of rows is accepted."""
import pytest

SHAPES = [(9728, 2560), (4096, 24576), (2560, 6144), (128, 32), (2048, 2048), (12288, 4096), (1152, 1056)]


@pytest.mark.parametrize("K,N", SHAPES)
def test_size_grows_with_the_rows_and_then_stays(K, N):
    from mykuiperllama_b200._lib import kernels
    size = [kernels().kuiper_awq_gemv_workspace_bytes(m, K, N) for m in list(range(1, 200)) + [2048, 65536, 1 << 20]]
    assert all(a <= b for a, b in zip(size, size[1:]))
    assert size[127] == size[-1]


@pytest.mark.gpu
@pytest.mark.parametrize("M,K,N", [(33, 640, 288), (40, 128, 32), (73, 1152, 1056), (128, 640, 544), (129, 256, 288), (300, 1152, 1056), (65536 + 40, 128, 32)])
def test_blocks_of_rows_share_a_workspace(cuda, M, K, N):
    import torch
    from test_gemm_rows_gpu import TOL, _case, _err
    x, w, ref = _case(M, K, N, M + K)
    workspace = cuda.awq_gemv_workspace(128, K, N)
    res = torch.randn((M, N), device="cuda")
    guard = torch.full((M + 1, N), 7.0, device="cuda")
    cuda.awq_gemv(x, *w, workspace=workspace, out=guard[:M])
    added = cuda.awq_gemv(x, *w, workspace=workspace, residual=res, out=res.clone())
    assert torch.equal(guard[:M], cuda.awq_gemv(x, *w, workspace=workspace))  # fixed order, slots reused
    one = cuda.awq_gemv(x[-1:].contiguous(), *w, workspace=workspace)  # the counters were left alone
    torch.cuda.synchronize()
    cuda.awq_gemv_status()
    assert bool((guard[M:] == 7.0).all())
    assert _err(guard[:M], ref) <= TOL and _err(added, ref + res.double()) <= TOL and _err(one, ref[-1:]) <= TOL
    aliased = res.clone()
    assert torch.equal(cuda.awq_gemv(x, *w, workspace=workspace, residual=aliased, out=aliased), added)
