"""What is timed when this library's speed is judged: the work a user has it do, through its public entry points.

A case is a plain dict.  `listed()` names the fixed ones, `draw(rng)` makes another of the same ranges, `prepare(case, seed)`
builds the state a user's program holds before the call, `run(state)` makes one call, `work(case)` counts the bytes and
operations the call cannot do without, `tolerance(case)` says how far another correct implementation may be off.

Kinds of call:
  gemv      one quantised matrix times 1..8 vectors, operands on the device (LlmContext.matmul_quant_assign)
  token     one decoded token, logits and greedy choice back on the host (Llama2.forward_logits / Gpt2.forward)
  generate  the device-side loop over n tokens, greedy or with the sampler (Llama models: then the last logits)
  batch     one token of each of several sequences (Llama2.decode_batch), logits of all of them back on the host
  prompt    n prompt tokens in one call, the last token's logits back on the host (Llama2.prefill / Gpt2.prefill)
Weights are seeded N(0, 0.02) values quantised on the device, as in bench.py: no checkpoint is at hand offline.
"""
from __future__ import annotations

import numpy as np
import torch

from slai_b200 import _lib, synth
from slai_b200.models import GPT2_XL, LLAMA2_70B, LLAMA2_7B, TINY_LLAMA, Gpt2Params, Llama2Config, synthetic_gpt2_device, synthetic_llama_device
from slai_b200.ops import Backend, GpuQuantMatrix, LlmContext

STD = 0.02


# ---- the cases ---------------------------------------------------------------------------------------------------------
def _llama(cfg: Llama2Config, fmt: str, out_fmt: str, layers: int | None = None) -> dict:
    return dict(arch="llama", dim=cfg.dim, hidden=cfg.hidden_dim, layers=layers or cfg.n_layers, heads=cfg.n_q_heads, kv_heads=cfg.n_kv_heads,
                vocab=cfg.vocab_size, context=cfg.seq_len, fmt=fmt, out_fmt=out_fmt, kv="f16", neox=False)


def _gpt2(p: Gpt2Params, fmt: str) -> dict:
    return dict(arch="gpt2", dim=p.n_embd, hidden=p.ff_len, layers=p.n_layer, heads=p.n_head, kv_heads=p.n_head, vocab=p.n_vocab,
                context=p.n_seq, fmt=fmt, out_fmt=fmt, kv="f16", neox=False)


def listed() -> list[dict]:
    q4 = _llama(LLAMA2_7B, "q4_k", "q6_k")            # the headline model: Q4_K layers, Q6_K logits matrix
    gqa = _llama(LLAMA2_70B, "q4_k", "q6_k", layers=8)  # the large grouped-query shapes, a tenth of the layers
    return [
        # a host engine that calls the operator itself: an attention projection, one vector (the smallest call here)
        dict(name="gemv_q4k_4096x4096", kind="gemv", fmt="q4_k", rows=4096, cols=4096, n_batch=1),
        # the logits product on its own, the tallest matrix of the headline model
        dict(name="gemv_q6k_32000x4096", kind="gemv", fmt="q6_k", rows=32000, cols=4096, n_batch=1),
        # a feed-forward product for a full batch of vectors
        dict(name="gemv_q5k_4096x11008_b8", kind="gemv", fmt="q5_k", rows=4096, cols=11008, n_batch=8),
        # the tiny story model (odd widths, f32 cache, Q8_0): launches and latency are everything
        dict(_llama(TINY_LLAMA, "q8_0", "q8_0"), name="tiny_generate", kind="generate", kv="f32", pos=16, n=64, sampled=False),
        # chat, one token at a time: the host picks the next token from the logits of each call
        dict(q4, name="7b_token", kind="token", pos=515),
        # the answer sampled on the device (temperature, top-p), with the reference's own f32 cache
        dict(q4, name="7b_sampled_generate", kind="generate", kv="f32", pos=515, n=8, sampled=True),
        # serving: eight conversations of different lengths advance together
        dict(q4, name="7b_batch8", kind="batch", pos=150, seqs=8),
        # the prompt of the headline workload
        dict(q4, name="7b_prompt_511", kind="prompt", pos=0, n=511),
        # a short user turn that follows an existing conversation
        dict(q4, name="7b_turn_37", kind="prompt", pos=300, n=37),
        # a long prompt of the grouped-query model, and a token late in a long conversation
        dict(gqa, name="70b_layers_prompt_1023", kind="prompt", pos=0, n=1023),
        dict(gqa, name="70b_layers_long_token", kind="token", pos=3500),
        # GPT-2 XL (Q8_0, width 1600, LayerNorm and biases): completion after a short prompt
        dict(_gpt2(GPT2_XL, "q8_0"), name="gpt2_xl_token", kind="token", pos=127),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(lo * (hi / lo) ** rng.random()))


def _draw_model(rng) -> dict:
    if rng.random() < 0.2:  # a GPT-2 of another size
        head, heads = 64, rng.randint(6, 25)
        dim = head * heads
        return dict(arch="gpt2", dim=dim, hidden=4 * dim, layers=rng.randint(2, 12), heads=heads, kv_heads=heads, vocab=_log_int(rng, 2000, 50257),
                    context=1024, fmt="q8_0", out_fmt="q8_0", kv=rng.choice(["f16", "f16", "f32"]), neox=False)
    head = rng.choice([64, 128, 128])
    unit = 256 // head                       # K-quants: widths are multiples of 256
    heads = unit * max(1, _log_int(rng, 2, 32) * 128 // 256)
    ratios = [r for r in (1, 1, 2, 4, 8) if heads % r == 0]
    dim = head * heads
    hidden = 256 * max(1, round(dim * rng.uniform(2.2, 3.7) / 256))
    fmt = rng.choice(["q4_k", "q4_k", "q5_k", "q6_k", "q8_0"])
    per_layer = dim * (2 * dim + 3 * hidden + dim)
    layers = max(1, min(rng.randint(2, 16), int(1.6e9 / per_layer)))
    return dict(arch="llama", dim=dim, hidden=hidden, layers=layers, heads=heads, kv_heads=heads // rng.choice(ratios), vocab=_log_int(rng, 2000, 50000),
                context=rng.choice([1024, 2048, 4096]), fmt=fmt, out_fmt=rng.choice([fmt, "q6_k"]), kv=rng.choice(["f16", "f16", "f16", "f32"]), neox=rng.random() < 0.2)


def draw(rng) -> dict:
    r = rng.random()
    if r < 0.25:
        fmt = rng.choice(["q4_k", "q4_k", "q5_k", "q6_k", "q8_0"])
        block = 32 if fmt == "q8_0" else 256
        return dict(kind="gemv", fmt=fmt, rows=_log_int(rng, 1000, 40000), cols=block * _log_int(rng, 2048 // block, 11264 // block),
                    n_batch=rng.choice([1, 1, 1, 2, 3, 4, 5, 6, 7, 8]))
    m = _draw_model(rng)
    if r < 0.40:
        return dict(m, kind="token", pos=rng.choice([0, _log_int(rng, 16, 900)]))
    if r < 0.55:
        # f32 cache: see tolerance()
        return dict(m, kind="generate", kv="f32", pos=_log_int(rng, 16, 900), n=rng.randint(4, 12), sampled=m["arch"] == "llama" and rng.random() < 0.5)
    if r < 0.72:
        while m["arch"] != "llama":
            m = _draw_model(rng)
        return dict(m, kind="batch", pos=_log_int(rng, 16, 160), seqs=rng.randint(2, 8))
    return dict(m, kind="prompt", pos=rng.choice([0, 0, rng.randint(1, 150)]), n=_log_int(rng, 20, 850))


# ---- state -------------------------------------------------------------------------------------------------------------
_backend: list[Backend] = []


def _the_backend() -> Backend:
    """A program has one backend (device context and stream), whatever number of models it holds."""
    if not _backend:
        _backend.append(Backend(0))
    return _backend[0]


class _Operand:
    """A torch tensor handed to the operators: they take anything with a device pointer and a length."""

    def __init__(self, t: torch.Tensor):
        self.t, self.ptr, self.n = t, t.data_ptr(), t.numel()

    def __len__(self):
        return self.n


def _model(be: Backend, case: dict, seed: int):
    fmt, out_fmt = synth.FMT_BY_NAME[case["fmt"]], synth.FMT_BY_NAME[case["out_fmt"]]
    kv = _lib.KV_F16 if case["kv"] == "f16" else _lib.KV_F32
    if case["arch"] == "gpt2":
        p = Gpt2Params(n_vocab=case["vocab"], n_seq=case["context"], n_embd=case["dim"], n_head=case["heads"], n_layer=case["layers"],
                       ff_len=case["hidden"], kv_dtype=kv)
        return synthetic_gpt2_device(be, p, fmt, seed=seed, std=STD)
    cfg = Llama2Config(dim=case["dim"], hidden_dim=case["hidden"], n_layers=case["layers"], n_q_heads=case["heads"], n_kv_heads=case["kv_heads"],
                       vocab_size=case["vocab"], seq_len=case["context"], kv_dtype=kv, rope_variant=1 if case["neox"] else 0)
    return synthetic_llama_device(be, cfg, fmt, out_fmt, seed=seed, std=STD)


def prepare(case: dict, seed: int) -> dict:
    be = _the_backend()
    rng = np.random.default_rng([seed, 20])
    if case["kind"] == "gemv":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        m = GpuQuantMatrix.synthetic(be, synth.FMT_BY_NAME[case["fmt"]], case["rows"], case["cols"], 1 + seed * 7919, STD)
        v = torch.randn(case["n_batch"] * case["cols"], generator=gen, device="cuda")
        out = torch.empty(case["n_batch"] * case["rows"], device="cuda")
        torch.cuda.synchronize()
        return dict(case=case, ctx=LlmContext(be), m=m, v=_Operand(v), out=_Operand(out))
    m = _model(be, case, seed)
    s = dict(case=case, model=m)
    ids = lambda n: rng.integers(0, case["vocab"], size=n).astype(np.int32)  # noqa: E731
    if case["kind"] == "batch":
        # conversations of different lengths: sequence b joins later than b - 1, then all advance in lockstep
        n_seq, longest = case["seqs"], case["pos"]
        starts = [longest * b // (2 * n_seq) for b in range(n_seq)]
        m.batch_reserve(n_seq)
        hist = ids((longest, n_seq))
        for t in range(longest):
            m.decode_batch(hist[t], np.array([t - b0 for b0 in starts], dtype=np.int32), want_logits=False)
        s["tokens"], s["positions"] = ids(n_seq), np.array([longest - b0 for b0 in starts], dtype=np.int32)
        return s
    if case["pos"] > 0:
        m.prefill(ids(case["pos"]))
    s["token"] = int(ids(1)[0])
    s["logits"] = np.empty(case["vocab"], dtype=np.float32)
    if case["kind"] == "prompt":
        s["prompt"] = ids(case["n"])
    be.synchronize()
    return s


def run(s: dict):
    case = s["case"]
    kind = case["kind"]
    if kind == "gemv":
        s["ctx"].matmul_quant_assign(s["out"], s["m"], s["v"], n_batch=case["n_batch"])
        return s["out"].t
    m, pos = s["model"], case["pos"]
    if kind == "token":  # (logits, their arg max): the logits say both, and a near tie may go either way
        return (m.forward_logits(pos, s["token"], s["logits"]) if case["arch"] == "llama" else m.forward(s["token"], pos))[0]
    if kind == "batch":
        return m.decode_batch(s["tokens"], s["positions"])[0]
    if kind == "prompt":
        return m.prefill(s["prompt"], pos, want_logits=True)
    if case["sampled"]:
        # random weights give flat logits: the low temperature makes the distribution as peaked as a trained model's
        ids = m.generate_sampled(s["token"], pos, case["n"], 0.1, 0.9, 12345)
    else:
        ids = m.generate(s["token"], pos, case["n"])
    return (ids, m.read_state("logits")) if case["arch"] == "llama" else ids


# ---- what a call cannot do without ---------------------------------------------------------------------------------------
def _layer_params(case: dict) -> int:
    d, h = case["dim"], case["hidden"]
    if case["arch"] == "gpt2":
        return 4 * d * d + 2 * d * h
    return 2 * d * d + 2 * d * (d * case["kv_heads"] // case["heads"]) + 3 * d * h


def work(case: dict) -> dict:
    bpw = synth.BITS_PER_WEIGHT[synth.FMT_BY_NAME[case["fmt"]]] / 8
    if case["kind"] == "gemv":
        M, K, B = case["rows"], case["cols"], case["n_batch"]
        return {"bytes": M * K * bpw + 4 * B * (M + K), "flops": 2.0 * M * K * B}
    bpo = synth.BITS_PER_WEIGHT[synth.FMT_BY_NAME[case["out_fmt"]]] / 8
    L, d, V, pos = case["layers"], case["dim"], case["vocab"], case["pos"]
    layer, head = _layer_params(case) * L, V * d
    kv_row = 2 * L * (d * case["kv_heads"] // case["heads"]) * (2 if case["kv"] == "f16" else 4)  # keys and values of one position
    weights = layer * bpw + head * bpo
    kind = case["kind"]
    if kind == "prompt":
        n = case["n"]
        ctx = sum(pos + i + 1 for i in range(n))
        return {"bytes": weights + kv_row * (pos + n) + 4 * V, "flops": 2.0 * layer * n + 2.0 * head + 4.0 * L * d * ctx}
    if kind == "batch":
        B, longest = case["seqs"], pos
        lens = [longest - longest * b // (2 * B) + 1 for b in range(B)]
        return {"bytes": weights + kv_row * sum(lens) + 4.0 * B * V, "flops": B * 2.0 * (layer + head) + 4.0 * L * d * sum(lens)}
    n = case.get("n", 1) if kind == "generate" else 1
    ctx = [pos + i + 1 for i in range(n)]
    return {"bytes": len(ctx) * weights + kv_row * sum(ctx) + 4.0 * V, "flops": len(ctx) * 2.0 * (layer + head) + 4.0 * L * d * sum(ctx)}


def tolerance(case: dict) -> dict:
    """Measured, times four.  The operator against the same product in 64 bits is off by 1.7e-7, a plain f32 product in
    another order by 4.8e-7.  A prompt token by token against all its tokens at once: 3.3e-4 after 32 layers with an f32
    cache; with an f16 cache, where a key or value that differs in its last bits may round to the other side, 1.5e-3.
    Whole numbers (the ids of a generated sequence) are the same."""
    if case["kind"] == "gemv":
        return {"rel": 2e-6}
    return {"rel": 6e-3 if case["kv"] == "f16" else 1.3e-3}
