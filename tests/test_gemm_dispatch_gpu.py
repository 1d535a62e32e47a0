"""Which kernel an INT4 GEMM of 33 rows and more takes is a matter of time only: outputs of few tiles, where either may be chosen, come out the
same from the 256 x 256 tiles and from the chosen kernel."""
import pytest
import torch

from test_gemm_rows_gpu import _case, _err

pytestmark = pytest.mark.gpu


# what the tiles' own tests use, and outputs of few tiles on both sides of the choice (narrow, one group, one wave of split sums)
@pytest.mark.parametrize("M,K,N", [(33, 384, 40), (64, 1024, 232), (129, 128, 8), (200, 256, 264), (256, 2560, 2560), (257, 1152, 1000), (333, 4096, 1536),
                                   (384, 128, 520), (450, 4096, 744), (512, 640, 6144), (700, 384, 256), (700, 2560, 744), (860, 1024, 512),
                                   (1025, 1024, 2080), (200, 128, 40), (256, 128, 64), (256, 128, 72)])
def test_chosen_kernel_and_tiles_agree(cuda, M, K, N):
    x, w, ref = _case(M, K, N, M + K + N)
    res = torch.randn((M, N), device="cuda")
    outs = []
    for always in (0, 1):
        cuda.set_tuning("gemm_tile_always", always)
        try:
            y = torch.full((M + 1, N), float("nan"), device="cuda")
            cuda.awq_gemm(x, *w, y=y[:M])
            assert bool(torch.isnan(y[M:]).all())
            outs.append([y[:M], cuda.awq_gemm_f16in(x.half(), *w, y=res.clone(), accumulate=True), cuda.awq_gemm_any_order(x, *w, residual=res)])
        finally:
            cuda.set_tuning("gemm_tile_always", 0)
    torch.cuda.synchronize()
    cuda.awq_gemm_status()
    for i, r in enumerate((ref, ref + res.double(), ref + res.double())):
        assert _err(outs[0][i], outs[1][i].double()) <= 1e-5  # fp32 sums of up to 4096 products in two orders (see test_gemm_tiles_gpu.py)
        assert _err(outs[0][i], r) <= 1e-3                    # the weight rounded to fp16
