"""Branches that only calls of many rows take: the four-element SwiGLU, the 256-thread RMSNorm, GEMM launches that hand out whole tiles
and share the rest, and the 128-row tiles with their K split where they are still the default."""
import pytest
import torch

from test_gemm_rows_gpu import _case, _err

pytestmark = pytest.mark.gpu

HALF = 2.0 ** -11  # relative rounding to fp16


# 148 SMs x 8192 elements is where the four-element kernel starts (148 x 8192, one row less below it); widths that are not a
# multiple of four and rows that are not 16-byte aligned stay with the other one
@pytest.mark.parametrize("M,I,shift", [(148, 8192, 0), (147, 8192, 0), (2048, 3072, 0), (333, 9728, 0), (1000, 1501, 0), (300, 4100, 1)])
@pytest.mark.parametrize("clear", [False, True])
def test_swiglu_of_a_chunk(cuda, M, I, shift, clear):
    g = torch.Generator(device="cuda")
    g.manual_seed(M + I)
    rows = (torch.randn(M * 2 * I + shift, generator=g, device="cuda") * 4)[shift:].view(M, 2 * I)
    ref = torch.nn.functional.silu(rows[:, :I].double()) * rows[:, I:].double()
    for call, rounding in ((cuda.swiglu, 2.0 ** -20), (cuda.swiglu_f16, HALF + 2.0 ** -20)):  # expf, a division, two products in fp32
        held = rows.clone() if shift == 0 else rows
        if shift and clear:
            held = torch.cat((torch.zeros(shift, device="cuda"), rows.flatten()))[shift:].view(M, 2 * I)
        before = held.clone()
        out = call(held, clear_input=clear)
        torch.cuda.synchronize()
        assert out.shape == (M, I)
        assert bool(((out.double() - ref).abs() <= rounding * ref.abs() + 2.0 ** -25).all())  # 2^-25: half the smallest fp16
        assert torch.equal(held, torch.zeros_like(held) if clear else before)


# from two rows per SM on, up to 4096 wide, a row has 256 threads; 1023 and the shifted rows take its scalar passes
@pytest.mark.parametrize("M,H,shift", [(296, 4096, 0), (295, 4096, 0), (2048, 2560, 0), (300, 4100, 0), (777, 100, 0), (300, 1023, 0), (300, 4096, 1)])
def test_rmsnorm_of_a_chunk(cuda, M, H, shift):
    g = torch.Generator(device="cuda")
    g.manual_seed(M + H)
    x = torch.randn(M * H + shift, generator=g, device="cuda")[shift:].view(M, H)
    x *= torch.logspace(-3, 3, M, device="cuda").unsqueeze(1)  # every row has its own scale
    x[1] = 0
    w = (1 + 0.1 * torch.randn(H, generator=g, device="cuda")).bfloat16()
    ref = x.double() / (x.double().square().mean(-1, keepdim=True) + 1e-6).sqrt() * w.double()
    # fp32 sum of H squares over a tree of threads, a square root, a division, two products: a few 2^-24 of each value
    for out, rounding in ((cuda.rmsnorm(x, w, 1e-6), 2.0 ** -20), (cuda.rmsnorm_f16(x, w, 1e-6), HALF + 2.0 ** -20)):
        assert bool(((out.double() - ref).abs() <= rounding * ref.abs() + 2.0 ** -25).all())
    in_place = x.clone()
    assert torch.equal(cuda.rmsnorm(in_place, w, 1e-6, out=in_place), cuda.rmsnorm(x.clone(), w, 1e-6))


TILES = 1e-3  # the weight rounded to fp16, see test_gemm_tiles_gpu.py


def _all_modes(cuda, calls, M, N, ref):
    res = torch.randn((M, N), device="cuda")
    for call, x in calls:
        y = torch.full((M + 3, N), float("nan"), device="cuda")  # what is overwritten may hold anything
        call(x, y=y[:M])
        guard = torch.isnan(y[M:]).all()
        added = call(x, y=res.clone(), accumulate=True)
        with_residual = call(x, residual=res)
        aliased = res.clone()
        call(x, y=aliased, residual=aliased)
        torch.cuda.synchronize()
        cuda.awq_gemm_status()
        assert bool(guard)
        for out, r in ((y[:M], ref), (added, ref + res.double()), (with_residual, ref + res.double()), (aliased, ref + res.double())):
            assert _err(out, r) <= TILES


# whole tiles for every CTA and a remainder that several share: 512 x 19456 is 152 tiles, 1280 x 8192 160 of which column tile 29 is
# whole in part, 1153 x 12320 has a short last tile row and a short last column tile, 257 x 512 no whole tile at all
@pytest.mark.parametrize("M,K,N", [(512, 640, 19456), (1280, 256, 8192), (1153, 256, 12320), (2048, 1024, 6400), (257, 1152, 512)])
def test_whole_and_shared_tiles_of_one_launch(cuda, M, K, N):
    x, w, ref = _case(M, K, N, M + N)
    call = lambda rows, **kw: cuda.awq_gemm_any_order(rows, *w, **kw)
    cuda.set_tuning("gemm_tile_always", 1)
    try:
        _all_modes(cuda, [(call, x), (call, x.half())], M, N, ref)
    finally:
        cuda.set_tuning("gemm_tile_always", 0)


# N % 32 != 0 below 33 rows; 257 to 511 rows whose K split fills one wave of two CTAs per SM (3 x 24 tiles, four splits)
@pytest.mark.parametrize("M,K,N", [(16, 1024, 136), (32, 4096, 1000), (9, 128, 8), (2, 640, 264), (300, 1024, 6144), (384, 512, 6144)])
def test_rows_tiles_with_a_split_sum(cuda, M, K, N):
    x, w, ref = _case(M, K, N, M + N)
    half = lambda rows, **kw: cuda.awq_gemm_f16in(rows, *w, **kw)
    _all_modes(cuda, [(lambda rows, **kw: cuda.awq_gemm(rows, *w, **kw), x), (half, x.half())], M, N, ref)
