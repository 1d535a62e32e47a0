"""Gate|up rows into the accumulating GEMV entry: three to five rows on both sides of the choice between its two kernels."""
import pytest
import torch

from test_gemm_rows_gpu import TOL, _case, _err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [3, 4, 5])
@pytest.mark.parametrize("K,N", [(384, 288), (4096, 544), (3968, 544), (9728, 2560), (9728, 3264)])
def test_few_gate_up_rows(cuda, M, K, N):
    _, w, _ = _case(M, K, N, M + K)
    rows = torch.randn((M, 2 * K), device="cuda")
    held = torch.randn((M, N), device="cuda")
    want = cuda.awq_gemm_f16in(cuda.swiglu_f16(rows), *w, y=held.clone(), accumulate=True)
    got = cuda.swiglu_awq_gemv_accum(rows, *w, held.clone())
    torch.cuda.synchronize()
    cuda.awq_gemv_status()
    # the same fp16 operands and exact products; an operand may round the other way where the two kernels' silu differ in the last bit
    # (2^-11 of one of K values)
    assert _err(got, want.double()) <= TOL + 2.0 ** -11 / K ** 0.5
