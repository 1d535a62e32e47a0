"""Values that are not ordinary numbers in prefill attention: both kernels behind kuiper_flash_prefill treat them alike."""
import pytest
import torch

from test_prefill_tc_gpu import _reference

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[1, 0], ids=["tcgen05", "tiled"])
def attend(request, cuda):
    cuda.set_tuning("prefill_tc_vectors", request.param)
    yield cuda.flash_prefill
    cuda.set_tuning("prefill_tc_vectors", 1024)


@pytest.mark.parametrize("hidden", [1, 64, 128, 200])
def test_scores_below_the_fp32_range(attend, hidden):
    # the first `hidden` cache rows score -1e40, which is -inf in fp32: their probability is 0 for every later row, and rows that
    # see nothing else come out as zeros
    M = 300
    g = torch.Generator(device="cuda")
    g.manual_seed(hidden)
    q = torch.randn((M, 32, 128), generator=g, device="cuda")
    k, v = (torch.randn((1, 8, M, 128), generator=g, device="cuda").bfloat16() for _ in range(2))
    q[..., 0] = 1e20
    k[..., 0] = 0
    k[:, :, :hidden, 0] = -1e21
    out = attend(q, k, v, 0, 0)
    q[..., 0] = 0
    s = q.double().transpose(0, 1) @ k[0].double().repeat_interleave(4, 0).transpose(1, 2) / 128 ** 0.5
    late = torch.arange(M, device="cuda") > torch.arange(M, device="cuda").unsqueeze(1)
    s = s.masked_fill(late, float("-inf"))[:, hidden:, hidden:]
    ref = (s.softmax(-1) @ v[0, :, hidden:].double().repeat_interleave(4, 0)).transpose(0, 1)
    assert bool((out[:hidden] == 0).all())
    # 16 significant bits of q and of the probabilities (see test_prefill_tc_gpu.py)
    assert float((out[hidden:].double() - ref).abs().max() / ref.abs().max()) <= 5e-5


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("M,pos0,Nq,Nkv,bad", [(300, 0, 32, 8, 100), (300, 0, 16, 8, 100), (300, 0, 64, 8, 191), (300, 128, 32, 8, 228),
                                               (513, 64, 32, 8, 64 + 127), (256, 0, 32, 8, 255)])
def test_a_value_row_that_is_not_finite_stays_out_of_earlier_tiles(attend, M, pos0, Nq, Nkv, bad, value):
    g = torch.Generator(device="cuda")
    g.manual_seed(M + bad)
    q = torch.randn((M, Nq, 128), generator=g, device="cuda")
    k, v = (torch.randn((1, Nkv, pos0 + M, 128), generator=g, device="cuda").bfloat16() for _ in range(2))
    clean = attend(q, k, v, pos0, 0)
    v[:, :, bad] = value
    out = attend(q, k, v, pos0, 0)
    first = bad // 64 * 64 - pos0  # earlier rows share no 64-row cache tile with the bad one
    assert torch.equal(out[:first], clean[:first])
    assert not bool(torch.isfinite(out[bad - pos0:]).any())
    ref = _reference(q, k[0], torch.where(torch.isfinite(v[0]), v[0], 0), pos0)[:first]
    assert float((out[:first].double() - ref).abs().max() / ref.abs().max()) <= 5e-5
