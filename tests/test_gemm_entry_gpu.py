"""What the entry points of the INT4 GEMM promise beside the numbers: the values of accumulate."""
import pytest
import torch

from mykuiperllama_b200._lib import check, kernels
from test_gemm_rows_gpu import _case, _err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [5, 300])  # the packed-word kernel, the tensor-core tiles
@pytest.mark.parametrize("accumulate", [1, 2, 3, -1, 256])
def test_every_non_zero_accumulate_adds(cuda, M, accumulate):
    K, N = 256, 512
    x, w, ref = _case(M, K, N, M)
    x16 = x.half()
    held = torch.randn((M, N), device="cuda")
    workspace = cuda.awq_gemm_workspace(M, K)
    stream = torch.cuda.current_stream().cuda_stream
    lib = kernels()
    outs = [held.clone() for _ in range(3)]
    ptrs = [t.data_ptr() for t in w]
    check(lib.kuiper_awq_gemm_f32(x.data_ptr(), *ptrs, outs[0].data_ptr(), None, accumulate, M, K, N, 128, workspace.data_ptr(),
                                  workspace.numel(), stream))
    check(lib.kuiper_awq_gemm_f16in_f32(x16.data_ptr(), *ptrs, outs[1].data_ptr(), None, accumulate, M, K, N, 128, stream))
    check(lib.kuiper_awq_gemm_any_order_f32(None, x16.data_ptr(), *ptrs, outs[2].data_ptr(), None, accumulate, M, K, N, 128, None, 0, stream))
    torch.cuda.synchronize()
    for i, y in enumerate(outs):
        assert _err(y, ref + held.double()) <= 1e-3, i  # the weight is rounded to fp16 beyond 32 rows


def test_any_order_takes_one_kind_of_rows(cuda):
    x, w, _ = _case(4, 128, 32, 1)
    x16, y = x.half(), torch.empty((4, 32), device="cuda")
    ptrs = [t.data_ptr() for t in w]
    for a, b in ((None, None), (x.data_ptr(), x16.data_ptr())):
        assert kernels().kuiper_awq_gemm_any_order_f32(a, b, *ptrs, y.data_ptr(), None, 0, 4, 128, 32, 128, None, 0, None) == 7
