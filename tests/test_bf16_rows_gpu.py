"""The bf16 product of several row blocks in one launch (bf16_gemv.cu): edges of the eight-row blocks and of the four blocks of a
launch, and ragged weight rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,N", [(8, 64, 40), (9, 1024, 4099), (16, 2560, 1000), (25, 96, 17), (32, 4096, 2048), (33, 1024, 151)])
def test_row_blocks(M, K, N):
    from mykuiperllama_b200 import capi
    g = torch.Generator(device="cuda")
    g.manual_seed(M + N)
    x = torch.randn((M, K), generator=g, device="cuda")
    w = torch.randn((N, K), generator=g, device="cuda").bfloat16()
    guard = torch.full((M + 1, N), 7.0, device="cuda")
    capi.bf16_gemv(x, w, out=guard[:M])
    ref = x.double() @ w.double().T
    # exact 24-bit operands, fp32 sums of K / 32 partial results: sqrt(K / 32) * 2^-24 of the row's norm, times a few
    assert float((guard[:M].double() - ref).abs().max() / ref.abs().max()) <= 2e-6
    assert bool((guard[M:] == 7.0).all())
