"""Prefill attention on tcgen05 (flash_prefill_tc.cu): edges of its query blocks and cache tiles for every group size, large
scores (the running maximum moves), and nothing read beyond the written rows."""
import pytest
import torch

from mykuiperllama_b200._lib import check, kernels

pytestmark = pytest.mark.gpu


@pytest.fixture
def cuda():
    from mykuiperllama_b200 import capi
    capi.set_tuning("prefill_tc_vectors", 1)
    yield capi
    capi.set_tuning("prefill_tc_vectors", 1024)


def _reference(q, k, v, pos0):
    M, Nq, D = q.shape
    k, v = (t[:, :pos0 + M].double().repeat_interleave(Nq // t.shape[0], 0) for t in (k, v))
    s = q.double().transpose(0, 1) @ k.transpose(1, 2) / D ** 0.5
    late = torch.arange(pos0 + M, device="cuda") > pos0 + torch.arange(M, device="cuda").unsqueeze(1)
    return (s.masked_fill(late, float("-inf")).softmax(-1) @ v).transpose(0, 1)


@pytest.mark.parametrize("M,pos0,Nq,Nkv,std", [(1, 0, 8, 8, 1), (16, 0, 32, 8, 1), (64, 0, 32, 8, 4), (65, 63, 32, 8, 1), (128, 128, 16, 8, 8),
                                               (129, 0, 16, 8, 1), (255, 1, 8, 8, 4), (300, 37, 64, 8, 1), (513, 127, 32, 8, 2)])
def test_matches_64_bit(cuda, M, pos0, Nq, Nkv, std):
    g = torch.Generator(device="cuda")
    g.manual_seed(M + pos0)
    q = torch.randn((M, Nq, 128), generator=g, device="cuda") * std
    k, v = (torch.randn((2, Nkv, pos0 + M + 9, 128), generator=g, device="cuda").bfloat16() for _ in range(2))
    k[:, :, pos0 + M:] = float("nan")  # rows nobody has written yet
    v[:, :, pos0 + M:] = float("nan")
    out = cuda.flash_prefill(q, k, v, pos0, 1)
    assert torch.equal(out, cuda.flash_prefill(q, k, v, pos0, 1))
    check(kernels().kuiper_flash_decode_status())
    ref = _reference(q, k[1], v[1], pos0)
    # q and the probabilities carry 16 significant bits: a score of magnitude |s| is off by 2^-17 |s|, a probability by as much
    # relatively; scores grow with the deviation of q
    assert float((out.double() - ref).abs().max() / ref.abs().max()) <= 5e-5 * max(1, std)
