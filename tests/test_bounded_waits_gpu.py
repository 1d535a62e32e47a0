"""Bounded waits of the pipelined kernels: one copy is left out, so that every wait behind it runs out.  The launch has to end with its
copies landed and its tensor memory freed, report a status, and leave the GPU in order for the next launch.  Each case runs in a
process of its own, because the GEMM's error words stay set for the life of the process."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import sys
sys.path.insert(0, {root!r})
sys.path.insert(0, {root!r} + "/tests")
import torch
from mykuiperllama_b200 import capi
from mykuiperllama_b200._lib import kernels
from test_gemm_rows_gpu import _case

def run(call, status, spins_key, drop_key, drop, again=0):
    good = call().clone()
    torch.cuda.synchronize()
    assert status() == 0
    capi.set_tuning(spins_key, 4096)  # about 4 ms a wait
    capi.set_tuning(drop_key, drop)
    call()
    torch.cuda.synchronize()  # the launch ends by itself
    assert status() == 5 and b"bounded" in kernels().kuiper_last_error(), status()
    capi.set_tuning(drop_key, -1)
    capi.set_tuning(spins_key, 0)
    after = [call().clone() for _ in range(3)]
    torch.cuda.synchronize()
    for y in after:
        assert float((y - good).abs().max() / good.abs().max()) <= 1e-5

{body}
"""


def _process(body):
    done = subprocess.run([sys.executable, "-c", PROGRAM.format(root=ROOT, body=body)], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]


# rows, K, N, operand; 4096 x 6144 gives a CTA several units, 512 x 256 one
@pytest.mark.parametrize("M,K,N,call", [(8, 4096, 6144, "gemm"), (32, 4096, 6144, "gemm"), (4, 4096, 6144, "accum"), (16, 512, 256, "gemm"),
                                        (6, 2560, 6144, "ordered")])
@pytest.mark.parametrize("drop", [0, 1])
def test_packed_word_projection(M, K, N, call, drop):
    if K == 512 and drop:
        pytest.skip("every CTA has one unit")
    call = {"gemm": "capi.awq_gemm(x, *w)", "accum": "capi.awq_gemv_accum(x, *w, torch.zeros((%d, %d), device='cuda'))" % (M, N),
            "ordered": "capi.awq_gemv(x, *w)"}[call]
    _process(f"x, w, _ = _case({M}, {K}, {N}, 1)\n"
             f"run(lambda: {call}, kernels().kuiper_awq_gemm_status, 'rows_wait_spins', 'rows_drop_unit', {drop})")


# 300 rows: a full tile row and a short one; 2048 x 6144: several tiles of one CTA.  Stage 0 starts a tile, later ones are in the middle
@pytest.mark.parametrize("M,K,N", [(64, 1024, 2048), (300, 512, 4096), (2048, 512, 6144)])
@pytest.mark.parametrize("drop", [0, 1, 3, 6])
def test_tensor_core_tiles(M, K, N, drop):
    if M < 2048 and drop > 1:
        pytest.skip("a CTA has one group, which is two stages")
    _process(f"capi.set_tuning('gemm_tile_always', 1)\nx, w, _ = _case({M}, {K}, {N}, 1)\n"
             f"run(lambda: capi.awq_gemm(x, *w), kernels().kuiper_awq_gemm_status, 'tile_wait_spins', 'tile_drop_stage', {drop})")


# tiles alternate K0 V0 K1 V1 ...; 300 rows of 32 / 8 heads are five blocks of one to three tiles
@pytest.mark.parametrize("drop", [0, 1, 2, 3, 5])
def test_prefill_attention(drop):
    _process(f"""
g = torch.Generator(device="cuda"); g.manual_seed(1)
q = torch.randn((300, 32, 128), generator=g, device="cuda")
k, v = (torch.randn((1, 8, 300, 128), generator=g, device="cuda").bfloat16() for _ in range(2))
run(lambda: capi.flash_prefill(q, k, v, 0, 0), kernels().kuiper_flash_decode_status, 'prefill_wait_spins', 'prefill_drop_tile', {drop})""")


def test_prefill_attention_reports_a_wait_once():
    _process("""
q = torch.randn((300, 32, 128), device="cuda")
k, v = (torch.randn((1, 8, 300, 128), device="cuda").bfloat16() for _ in range(2))
status = kernels().kuiper_flash_decode_status
run(lambda: capi.flash_prefill(q, k, v, 0, 0), status, 'prefill_wait_spins', 'prefill_drop_tile', 1)
assert status() == 0  # the launches after the one that failed are in order""")
