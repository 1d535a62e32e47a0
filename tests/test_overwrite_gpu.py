"""Passes of many rows write the q|k|v and gate|up projections anew instead of adding into zeroed buffers; what follows them -
a shorter chunk, a longer one, decode steps - has to find those buffers as it needs them."""
import numpy as np
import pytest

from helpers import make_model_weights, rel_err

pytestmark = pytest.mark.gpu

CFG = dict(n_layers=2, hidden=256, n_q_heads=4, n_kv_heads=2, head_dim=128, inter=512, vocab=1000, max_seq=2048, max_batch=2)
STEPS = 6


def _logits(engine, chunks, ids):
    """Logits of every prompt row, fed chunk by chunk, then of the row after STEPS decode steps with given tokens."""
    out, p = [], 0
    for n in chunks:
        out.append(engine.predict(ids[p:p + n], np.arange(p, p + n), np.zeros(n, np.int32), want_logits=True)[0])
        p += n
    engine.decode_begin([int(ids[p])], [p], [0])
    for i in range(STEPS):
        engine.decode_predict([int(ids[p + i])])
    out.append(engine.predict([int(ids[p + STEPS])], [p + STEPS], [0], want_logits=True)[0])
    return np.concatenate(out)


@pytest.mark.parametrize("min_rows,chunks", [(None, (700, 40, 600, 5)), (None, (512, 511)), (1024, (1100, 800)), (600, (650, 550, 20))])
def test_shorter_passes_after_one_that_overwrites(oracle, monkeypatch, min_rows, chunks):
    from mykuiperllama_b200.engine import EngineConfig, Qwen3Engine
    weights = make_model_weights(oracle, oracle.ModelConfig(**CFG, act_round=oracle.ROUND_FP16), seed=5)
    ids = np.random.default_rng(sum(chunks)).integers(0, 1000, sum(chunks) + STEPS + 1).astype(np.int32)
    small = Qwen3Engine(EngineConfig(**CFG, max_rows=64, act_mode=1))
    small.load(weights)
    total = sum(chunks)
    want = _logits(small, [64] * (total // 64) + [total % 64] * (total % 64 > 0), ids)
    small.close()
    if min_rows:
        monkeypatch.setenv("KUIPER_GEMM_MIN_ROWS", str(min_rows))
    engine = Qwen3Engine(EngineConfig(**CFG, max_rows=max(chunks), act_mode=1))
    engine.load(weights)
    got = _logits(engine, chunks, ids)
    engine.synchronize()
    engine.close()
    # passes of 33 rows and more round the weight to fp16 whatever their size; a pass of other rows sums in another order, which now
    # and then rounds an fp16 operand the other way (2^-11 of one value).  Where the rows take the GEMV instead (min_rows) the
    # weight stays exact: 2^-12 per product on average, as between the GEMM and the oracle, which tests/test_model_gpu.py bounds by 5e-3
    assert rel_err(got, want) <= (5e-3 if min_rows else 2e-3)
