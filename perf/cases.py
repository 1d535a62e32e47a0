"""The work this framework is used for, as measurable cases: INT4-AWQ projections and attention called as operators, and
the engine's two directions - reading a prompt (prefill) and writing tokens (decode) - on the three model shapes of
bench.py's workloads.  Sizes run from one 2048 x 2048 projection of one row to a 4096-token prompt of the 8B shape.

    listed()            the cases that are reported
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs, weights and handles on the GPU, made from the seed alone
    run(state)          one pass through the public entry points; returns its outputs
    work(case)          bytes and operations the pass cannot do without
    tolerance(case)     how far another correct implementation may be off
    exact(case, seed)   the outputs of run() as plain 64-bit arithmetic gives them
"""
import numpy as np
import torch

from mykuiperllama_b200 import capi
from mykuiperllama_b200.engine import EngineConfig, Qwen3Engine

GROUP = 128
HEAD = 128
VOCAB = 151936

# layers, hidden, query heads, key/value heads, intermediate (the model shapes of bench.py)
SHAPES = {
    "0.6b": (28, 1024, 16, 8, 3072),
    "4b": (36, 2560, 32, 8, 9728),
    "8b": (36, 4096, 32, 8, 12288),
}
ENGINE_ROWS = 2048  # rows of one prompt chunk
DECODE_STEPS = 24   # tokens generated per sequence in one pass


def listed():
    return [
        # one projection of one token: the smallest call there is, launch latency and host path
        {"name": "proj-1x2048x2048", "kind": "proj", "rows": 1, "K": 2048, "N": 2048},
        # a few sequences (or a few speculated tokens) through the down projection of the 4B shape
        {"name": "proj-6x9728x2560", "kind": "proj", "rows": 6, "K": 9728, "N": 2560},
        # a ragged prompt through the gate|up projection of the 8B shape
        {"name": "proj-333x4096x24576", "kind": "proj", "rows": 333, "K": 4096, "N": 24576},
        # attention of one decoding sequence over a few thousand cached positions
        {"name": "attn-b1-4096", "kind": "attn", "batch": 1, "length": 4096},
        # the widest attention batch over the longest cache
        {"name": "attn-b16-32768", "kind": "attn", "batch": 16, "length": 32768},
        # interactive generation, smallest model: bound by launches
        {"name": "decode-0.6b-b1-64", "kind": "decode", "model": "0.6b", "batch": 1, "prompt": 64},
        # interactive generation, largest model: the headline workload
        {"name": "decode-8b-b1-2048", "kind": "decode", "model": "8b", "batch": 1, "prompt": 2048},
        # a handful of concurrent sequences of different lengths
        {"name": "decode-8b-b5-777", "kind": "decode", "model": "8b", "batch": 5, "prompt": 777},
        # batched serving
        {"name": "decode-4b-b16-512", "kind": "decode", "model": "4b", "batch": 16, "prompt": 512},
        # time to first token: a short question, an ordinary prompt, a long document in two chunks
        {"name": "prefill-0.6b-77", "kind": "prefill", "model": "0.6b", "prompt": 77},
        {"name": "prefill-4b-512", "kind": "prefill", "model": "4b", "prompt": 512},
        {"name": "prefill-8b-4096", "kind": "prefill", "model": "8b", "prompt": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(("proj", "attn", "decode", "prefill"))
    if kind == "proj":
        # widths of any model: inputs in whole quantisation groups, outputs in whole 32-column runs
        return {"kind": kind, "rows": _log_int(rng, 1, 512), "K": GROUP * _log_int(rng, 8, 96), "N": 32 * _log_int(rng, 32, 768)}
    if kind == "attn":
        return {"kind": kind, "batch": rng.randint(1, 16), "length": _log_int(rng, 1000, 32768)}
    model = rng.choice(sorted(SHAPES))
    if kind == "decode":
        return {"kind": kind, "model": model, "batch": _log_int(rng, 1, 16 if model == "8b" else 32), "prompt": _log_int(rng, 64, 2048)}
    return {"kind": kind, "model": model, "prompt": _log_int(rng, 16, 4096)}


# ---- inputs ---------------------------------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _words(g, *shape):
    n = 4
    for d in shape:
        n *= d
    return torch.randint(0, 256, (n,), generator=g, device="cuda", dtype=torch.uint8).view(torch.int32).view(*shape)


def _quantised(g, K, N, std):
    """An INT4-AWQ matrix: uniform nibbles around zero points of 6 to 9, so that (q - z) * s has the given deviation."""
    qweight = _words(g, K, N // 8)
    qzeros = (_words(g, K // GROUP, N // 8) & 0x33333333) + 0x66666666
    scales = (std / 4.7) * (0.75 + 0.5 * torch.rand((K // GROUP, N), generator=g, device="cuda"))
    return qweight, qzeros, scales.half()


def _normal(g, *shape, std=1.0):
    return torch.randn(shape, generator=g, device="cuda") * std


def _lengths(batch, longest):
    """Sequence lengths of a batch: the longest, then ever shorter ones down to about half of it."""
    return [longest - (i * longest) // (2 * batch) for i in range(batch)]


def _weights(case, g):
    """The model's weights one after another: (embedding, final norm, head), then a dict per layer."""
    layers, H, Nq, Nkv, I = SHAPES[case["model"]]

    def norm(n):
        return (1.0 + _normal(g, n, std=0.02)).bfloat16()

    # As in a trained model the layers add small corrections to the residual stream and the output distribution is
    # peaked: the head of token t points along the embedding of token t - 1, so greedy decoding has a clear winner.
    out_std = 0.02 / (2 * layers) ** 0.5
    embed = _normal(g, VOCAB, H, std=0.5).bfloat16()
    yield embed, norm(H), (torch.roll(embed, 1, 0) * 0.04).contiguous()
    del embed
    for _ in range(layers):
        w = {"input_norm": norm(H), "post_norm": norm(H), "q_norm": norm(HEAD), "k_norm": norm(HEAD)}
        for name, K, N, std in (("qkv", H, (Nq + 2 * Nkv) * HEAD, 0.02), ("o", Nq * HEAD, H, out_std), ("gu", H, 2 * I, 0.02),
                                ("down", I, H, out_std)):
            w[name + "_qw"], w[name + "_qz"], w[name + "_s"] = _quantised(g, K, N, std)
        yield w


def _engine(case, g, max_seq, batch, rows):
    layers, H, Nq, Nkv, I = SHAPES[case["model"]]
    engine = Qwen3Engine(EngineConfig(n_layers=layers, hidden=H, n_q_heads=Nq, n_kv_heads=Nkv, head_dim=HEAD, inter=I, vocab=VOCAB,
                                      group=GROUP, max_seq=max_seq, max_batch=batch, max_rows=rows, act_mode=2))
    weights = _weights(case, g)
    engine.load_globals(*next(weights))
    for i, w in enumerate(weights):
        engine.load_layer(i, w)
    return engine


def prepare(case, seed):
    g = _generator(seed)
    ids = np.random.default_rng(seed)
    kind = case["kind"]
    state = dict(case)
    if kind == "proj":
        M, K, N = case["rows"], case["K"], case["N"]
        state["x"] = _normal(g, M, K)
        state["w"] = _quantised(g, K, N, 0.02)
        state["out"] = torch.empty((M, N), device="cuda")
        state["workspace"] = capi.awq_gemv_workspace(M, K, N) if M < 16 else capi.awq_gemm_workspace(M, K)
    elif kind == "attn":
        B, L = case["batch"], case["length"]
        state["q"] = _normal(g, B, 32, HEAD)
        state["k"], state["v"] = (torch.randn((B, 8, L, HEAD), generator=g, device="cuda", dtype=torch.bfloat16) for _ in range(2))
        state["len"] = torch.tensor(_lengths(B, L), dtype=torch.int32, device="cuda")
        state["slot"] = torch.arange(B, dtype=torch.int32, device="cuda")
        state["out"] = torch.empty((B, 32, HEAD), device="cuda")
        state["workspace"] = capi.flash_decode_workspace(B, 32, HEAD, L)
    elif kind == "decode":
        B, n = case["batch"], case["prompt"]
        engine = state["engine"] = _engine(case, g, n + DECODE_STEPS + 8, B, 512)
        state["pos"] = np.array(_lengths(B, n), np.int32)
        state["first"] = np.array([engine.prefill(ids.integers(0, VOCAB, m), slot=b) for b, m in enumerate(state["pos"])], np.int32)
    else:
        n = case["prompt"]
        state["engine"] = _engine(case, g, n + 8, 1, ENGINE_ROWS)
        state["tokens"] = ids.integers(0, VOCAB, n).astype(np.int32)
    return state


# ---- one pass -------------------------------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "proj":
        if state["rows"] < 16:
            return capi.awq_gemv(state["x"], *state["w"], workspace=state["workspace"], out=state["out"])
        return capi.awq_gemm(state["x"], *state["w"], y=state["out"], workspace=state["workspace"])
    if kind == "attn":
        return capi.flash_decode(state["q"], state["k"], state["v"], state["len"], state["slot"], workspace=state["workspace"],
                                 out=state["out"])
    engine = state["engine"]
    if kind == "decode":
        # greedy generation, every token handed to the caller; the last one with its logits
        slots = np.arange(state["batch"], dtype=np.int32)
        token, written = state["first"], []
        engine.decode_begin(token, state["pos"], slots)
        for _ in range(DECODE_STEPS - 1):
            token = engine.decode_predict(token)
            written.append(token)
        logits, token = engine.predict(token, state["pos"] + (DECODE_STEPS - 1), slots, want_logits=True)
        written.append(token)
        return {"tokens": np.stack(written), "logits": logits}
    # the prompt, and the first generated token with its logits
    first = engine.prefill(state["tokens"])
    logits, second = engine.predict([first], [state["prompt"]], want_logits=True)
    return {"tokens": np.array([first, int(second[0])], np.int64), "logits": logits}


# ---- what the pass cannot do without ----------------------------------------------------------------------------------
def _matrix_bytes(K, N):
    return K * N / 2 + (K // GROUP) * N * 2.5


def _kv_bytes(heads, positions):
    return 2 * heads * HEAD * 2 * positions


def _model(case):
    """(bytes of the layers' weights, bytes of the head, operations per row in the layers, operations per row in the head)"""
    layers, H, Nq, Nkv, I = SHAPES[case["model"]]
    matrices = ((H, (Nq + 2 * Nkv) * HEAD), (Nq * HEAD, H), (H, 2 * I), (I, H))
    return (layers * sum(_matrix_bytes(K, N) for K, N in matrices), VOCAB * H * 2.0,
            layers * sum(2.0 * K * N for K, N in matrices), 2.0 * VOCAB * H)


def work(case):
    kind = case["kind"]
    if kind == "proj":
        M, K, N = case["rows"], case["K"], case["N"]
        return {"bytes": _matrix_bytes(K, N) + 4.0 * M * (K + N), "flops": 2.0 * M * K * N}
    if kind == "attn":
        rows = sum(_lengths(case["batch"], case["length"]))
        return {"bytes": _kv_bytes(8, rows) + case["batch"] * 32 * HEAD * 8.0, "flops": 4.0 * 32 * HEAD * rows}
    layers, _, Nq, Nkv, _ = SHAPES[case["model"]]
    weights, head, ops, head_ops = _model(case)
    if kind == "decode":
        B = case["batch"]
        # position p of a sequence reads p + 1 cached rows
        rows = sum(sum(m + s + 1 for s in range(DECODE_STEPS)) for m in _lengths(B, case["prompt"]))
        return {"bytes": DECODE_STEPS * (weights + head) + layers * _kv_bytes(Nkv, rows) + 4.0 * B * VOCAB,
                "flops": DECODE_STEPS * B * (ops + head_ops) + layers * 4.0 * Nq * HEAD * rows}
    n = case["prompt"]
    # every chunk of the prompt needs the weights once; then one generated token
    chunks = -(-n // ENGINE_ROWS)
    return {"bytes": (chunks + 1) * weights + 2 * head + layers * _kv_bytes(Nkv, 2 * n) + 4.0 * VOCAB,
            "flops": (n + 1) * ops + 2 * head_ops + layers * 4.0 * Nq * HEAD * (n + 1.0) * (n + 2.0) / 2}


def tolerance(case):
    """About four times what was measured, per kind (2-norm; largest single value)."""
    kind = case["kind"]
    if kind == "proj":
        # x (and, from 16 rows on, the weight) rounded to fp16: 2.8e-4; 1.5e-3 against 64-bit sums
        return {"rel": 1.2e-3, "max": 6e-3}
    if kind == "attn":
        # fp32 softmax, 16-bit splits of q and the probabilities: 8.0e-6; 3.1e-5 against 64-bit sums
        return {"rel": 3.2e-5, "max": 1.3e-4}
    # all layers: 1.2e-3; 6.3e-3 of the logits against projections with un-rounded fp32 activations, and as much between
    # two passes over the same inputs, because reductions arrive in another order.  The tokens agreed throughout.
    return {"rel": 5e-3, "max": 2.5e-2, "differ": 0.01}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------
def _dense(qweight, qzeros, scales):
    """The matrix of an INT4-AWQ triple: column c of a word lies in nibble c / 2 (even c) or 4 + c / 2 (odd c)."""
    shifts = torch.tensor([4 * (c // 2 + 4 * (c % 2)) for c in range(8)], device="cuda", dtype=torch.int32)
    q, z = (((w.unsqueeze(-1) >> shifts) & 15).flatten(1).to(torch.int8) for w in (qweight, qzeros))
    K, N = q.shape
    return ((q.view(-1, GROUP, N) - z.unsqueeze(1)).double() * scales.double().unsqueeze(1)).view(K, N)


def _attend(q, k, v, start):
    """Causal attention of the rows at positions start, start + 1, ...: q [n, heads, HEAD], k and v [positions, kv heads, HEAD]"""
    n, heads, _ = q.shape
    k, v = (t.repeat_interleave(heads // t.shape[1], 1).transpose(0, 1) for t in (k, v))
    score = q.transpose(0, 1) @ k.transpose(1, 2) / HEAD ** 0.5
    late = torch.arange(k.shape[1], device="cuda") > start + torch.arange(n, device="cuda").unsqueeze(1)
    return (score.masked_fill_(late, float("-inf")).softmax(-1) @ v).transpose(0, 1)


def _norm64(x, w):
    return x / (x.square().mean(-1, keepdim=True) + 1e-6).sqrt() * w.double()


def _rotate(x, pos):
    angle = pos.double().unsqueeze(1) * 1e6 ** (-torch.arange(0, HEAD, 2, device="cuda").double() / HEAD)
    c, s = angle.cos().unsqueeze(1), angle.sin().unsqueeze(1)
    a, b = x[..., :HEAD // 2], x[..., HEAD // 2:]
    return torch.cat((a * c - b * s, b * c + a * s), -1)


class _Model64:
    def __init__(self, case, g):
        _, _, self.Nq, self.Nkv, self.I = SHAPES[case["model"]]
        weights = _weights(case, g)
        self.embed, self.norm, self.head = next(weights)
        self.layers = list(weights)
        self.cache = [{} for _ in self.layers]

    def forward(self, runs):
        """runs: (slot, first position, tokens) per sequence; logits of the last token of each."""
        def product(x, name):
            return x @ _dense(w[name + "_qw"], w[name + "_qz"], w[name + "_s"])

        ids = torch.from_numpy(np.concatenate([np.asarray(t, np.int64) for _, _, t in runs])).cuda()
        pos = torch.cat([p + torch.arange(len(t), device="cuda") for _, p, t in runs])
        sizes = [len(t) for _, _, t in runs]
        h = self.embed[ids].double()
        for w, cache in zip(self.layers, self.cache):
            q, k, v = product(_norm64(h, w["input_norm"]), "qkv").view(len(ids), -1, HEAD).split((self.Nq, self.Nkv, self.Nkv), 1)
            q, k = _rotate(_norm64(q, w["q_norm"]), pos), _rotate(_norm64(k, w["k_norm"]), pos)
            out = []
            for (slot, p, _), qs, ks, vs in zip(runs, q.split(sizes), k.split(sizes), v.split(sizes)):
                if p:
                    ks, vs = torch.cat((cache[slot][0], ks)), torch.cat((cache[slot][1], vs))
                cache[slot] = (ks, vs)
                out.append(_attend(qs, ks, vs, p))
            h = h + product(torch.cat(out).flatten(1), "o")
            gate, up = product(_norm64(h, w["post_norm"]), "gu").split(self.I, 1)
            h = h + product(torch.nn.functional.silu(gate) * up, "down")
        last = h[torch.tensor(sizes, device="cuda").cumsum(0) - 1]
        return _norm64(last, self.norm) @ self.head.double().T


def exact(case, seed):
    kind = case["kind"]
    if kind in ("proj", "attn"):
        state = prepare(case, seed)
        if kind == "proj":
            return state["x"].double() @ _dense(*state["w"])
        return torch.stack([_attend(state["q"][b:b + 1].double(), k[:, :n].double().transpose(0, 1), v[:, :n].double().transpose(0, 1), n)[0]
                            for b, (k, v, n) in enumerate(zip(state["k"], state["v"], state["len"].tolist()))])
    g, ids = _generator(seed), np.random.default_rng(seed)
    model = _Model64(case, g)
    if kind == "prefill":
        prompts, steps = [ids.integers(0, VOCAB, case["prompt"])], 1
    else:
        prompts, steps = [ids.integers(0, VOCAB, m) for m in _lengths(case["batch"], case["prompt"])], DECODE_STEPS
    logits = model.forward([(b, 0, p) for b, p in enumerate(prompts)])
    for s in range(steps):
        token = logits.argmax(1).tolist()
        logits = model.forward([(b, len(p) + s, [t]) for b, (p, t) in enumerate(zip(prompts, token))])
    return {"tokens": None, "logits": logits}
