"""The packed-word projection of a few token rows (awq_gemm_rows.cu) behind awq_gemm and awq_gemv: edges of its row blocks,
column tiles and runs, every output mode, fixed order where the entry point has one."""
import numpy as np
import pytest
import torch

from helpers import awq_random, rel_err

pytestmark = pytest.mark.gpu

# The operands are exact (fp16 activations, 4-bit weights), so only fp32 additions round: eight tensor-core steps of 16
# products per group, truncating (8 * 2^-23 of the partial sums), then one fp32 addition per group and run.
TOL = 4e-6


@pytest.fixture
def cuda():
    from mykuiperllama_b200 import capi
    capi.set_tuning("gemm_rows_max", 96)  # awq_gemm sends more than 32 rows elsewhere, awq_gemv does not
    yield capi
    capi.set_tuning("gemm_rows_max", 32)


def _case(M, K, N, seed):
    from oracle import cpu_oracle as orc
    rng = np.random.default_rng(seed)
    q, z, s = awq_random(rng, K, N)
    w = tuple(torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (orc.awq_pack(q), orc.awq_pack(z))) + (torch.from_numpy(s.view(np.float16)).cuda(),)
    x = torch.from_numpy(rng.standard_normal((M, K)).astype(np.float32)).cuda()
    qd, zd, sd = (torch.from_numpy(np.ascontiguousarray(a)).cuda().double() for a in (q, z, s.view(np.float16).astype(np.float64)))
    dense = (qd.view(K // 128, 128, N) - zd.view(K // 128, 1, N)) * sd.view(K // 128, 1, N)
    return x, w, x.half().double() @ dense.view(K, N)


def _err(y, ref):
    return rel_err(y.double().cpu().numpy(), ref.cpu().numpy())


@pytest.mark.parametrize("M,K,N", [(2, 128, 32), (3, 256, 288), (7, 1152, 2080), (8, 128, 256), (9, 2048, 544), (15, 9728, 2560), (16, 4096, 256),
                                   (17, 640, 1056), (31, 1024, 6144), (32, 384, 32), (33, 1024, 512), (77, 1024, 4096), (96, 2560, 800)])
def test_few_rows(cuda, M, K, N):
    x, w, ref = _case(M, K, N, M * 7 + K + N)
    res = torch.randn((M, N), device="cuda")
    outs = [(cuda.awq_gemm(x, *w), ref), (cuda.awq_gemm_f16in(x.half(), *w), ref), (cuda.awq_gemm(x, *w, residual=res), ref + res.double()),
            (cuda.awq_gemm(x, *w, y=res.clone(), accumulate=True), ref + res.double())]
    if M < 40:
        ws = cuda.awq_gemv_workspace(M, K, N)
        outs += [(cuda.awq_gemv(x, *w, workspace=ws), ref), (cuda.awq_gemv(x, *w, workspace=ws, residual=res), ref + res.double())]
        assert torch.equal(outs[-2][0], cuda.awq_gemv(x, *w, workspace=ws))  # fixed summation order
        # one-row calls keep their counters at the front of the same workspace
        one = cuda.awq_gemv(x[:1].contiguous(), *w, workspace=ws)
        assert _err(one, ref[:1]) <= TOL
    torch.cuda.synchronize()
    cuda.awq_gemm_status()
    cuda.awq_gemv_status()
    for i, (y, r) in enumerate(outs):
        assert _err(y, r) <= TOL, (i, _err(y, r))


@pytest.mark.parametrize("M,K,N", [(2, 128, 32), (3, 2560, 6144), (5, 12288, 4096), (8, 640, 288)])
def test_fp32_and_gate_up_operands(cuda, M, K, N):
    x, w, ref = _case(M, K, N, M + K + N)
    res = torch.randn((M, N), device="cuda")
    assert _err(cuda.awq_gemv_accum(x, *w, res.clone()), ref + res.double()) <= TOL
    # SwiGLU of gate|up rows, rounded to fp16, is the operand: the same as the separate kernel followed by the product
    gate_up = torch.randn((M, 2 * K), device="cuda")
    operand = cuda.swiglu_f16(gate_up)
    got = cuda.swiglu_awq_gemv_accum(gate_up, *w, res.clone())
    want = cuda.awq_gemm_f16in(operand, *w, y=res.clone(), accumulate=True)
    torch.cuda.synchronize()
    cuda.awq_gemv_status()
    assert _err(got, want.double()) <= TOL


def test_rows_beyond_the_matrix_stay_untouched(cuda):
    x, w, ref = _case(5, 256, 96, 3)
    y = torch.full((9, 96), 7.0, device="cuda")
    cuda.awq_gemm(x, *w, y=y[:5])
    assert _err(y[:5], ref) <= TOL and bool((y[5:] == 7.0).all())


def test_small_workspace_and_unaligned_rows_take_the_general_path(cuda):
    x, w, ref = _case(6, 512, 1024, 4)
    one_row = cuda.awq_gemv_workspace(1, 512, 1024)
    assert _err(cuda.awq_gemv(x, *w, workspace=one_row), ref) <= TOL
    shifted = torch.empty(6 * 512 + 1, device="cuda")[1:].view(6, 512).copy_(x)
    assert _err(cuda.awq_gemv(shifted, *w), ref) <= TOL
