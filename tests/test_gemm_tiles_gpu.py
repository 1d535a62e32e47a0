"""The 256 x 256 tiles of the tensor-core INT4 GEMM (calls of many rows): ragged rows and columns, tile rows of at most 128
and of more rows, runs that start and end inside a tile, every output mode."""
import pytest
import torch

from test_gemm_rows_gpu import _case, _err, cuda  # noqa: F401

pytestmark = pytest.mark.gpu

# The weight (q - z) * s is rounded to fp16 (2^-11 relative, at most half of it per product); over K products of random
# sign the largest deviation stays below 2^-12 * 4 of the largest output.  Only fp32 sums come on top.
TOL = 1e-3


@pytest.mark.parametrize("M,K,N", [(129, 128, 8), (200, 256, 264), (256, 2560, 2560), (257, 1152, 1000), (333, 4096, 1536), (384, 128, 520),
                                   (512, 640, 6144), (700, 384, 256), (1025, 1024, 2080), (1153, 256, 12320)])
def test_many_rows(cuda, M, K, N):  # noqa: F811
    x, w, ref = _case(M, K, N, M + K + N)
    res = torch.randn((M, N), device="cuda")
    guard = torch.full((M + 3, N), 7.0, device="cuda")
    cuda.awq_gemm(x, *w, y=guard[:M])
    outs = [(guard[:M], ref), (cuda.awq_gemm_f16in(x.half(), *w), ref), (cuda.awq_gemm(x, *w, residual=res), ref + res.double()),
            (cuda.awq_gemm(x, *w, y=res.clone(), accumulate=True), ref + res.double())]
    cuda.set_tuning("gemm_split_k", 0)  # the 128 x 256 tiles: same rounding of the weight, another order of the sums
    try:
        other = cuda.awq_gemm(x, *w)
    finally:
        cuda.set_tuning("gemm_split_k", 1)
    torch.cuda.synchronize()
    cuda.awq_gemm_status()
    assert bool((guard[M:] == 7.0).all())
    for i, (y, r) in enumerate(outs):
        assert _err(y, r) <= TOL, (i, _err(y, r))
    if -(-M // 128) * -(-N // 256) >= 400:  # the fixed order of a launch with many tiles
        assert torch.equal(outs[0][0], cuda.awq_gemm(x, *w)) and torch.equal(outs[2][0], outs[3][0])
    assert _err(outs[0][0], other.double()) <= 1e-5  # fp32 sums of up to 4096 products in two orders
