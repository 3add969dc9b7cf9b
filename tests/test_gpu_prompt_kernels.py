"""The prompt pass's GEMM variants and its tensor-core attention at the edges of their tiles, and the decode attention whose keys and
values stay in registers: against the sequential pass and against 64-bit arithmetic."""
import ctypes as C

import numpy as np
import pytest

from slai_b200 import synth, _lib
from slai_b200.models import Gpt2Params, Llama2Config, llama_from_host, synthetic_gpt2_device, synthetic_llama_device, synthetic_llama_host
from slai_b200.ops import BatchedMultiqueryAttentionParams
from helpers import rel_l2

pytestmark = pytest.mark.gpu


# Tokens: up to 64 the two planes of the activations are one operand, above two CTAs share a tile or K is split over a cluster; one
# past a tile, ragged last tiles, several tiles per CTA.  768 columns and 192 rows (k, v): a matrix that ends inside a CTA's rows.
@pytest.mark.parametrize("fmt", [synth.FMT_Q4_K, synth.FMT_Q5_K, synth.FMT_Q6_K, synth.FMT_Q8_0])
@pytest.mark.parametrize("T", [16, 17, 64, 65, 129, 300, 1200])
def test_prompt_pass_at_the_edges_of_its_tiles(backend, monkeypatch, fmt, T):
    cfg = Llama2Config(dim=768, hidden_dim=1280, n_layers=1, n_q_heads=12, n_kv_heads=3, vocab_size=300, seq_len=1240, kv_dtype=_lib.KV_F32)
    w = synthetic_llama_host(cfg, fmt, fmt, seed=T, std=0.05, embd_std=1.0)
    batched, seq = llama_from_host(backend, cfg, w, fmt, fmt), llama_from_host(backend, cfg, w, fmt, fmt)
    prompt = np.random.default_rng(T).integers(0, cfg.vocab_size, size=T).astype(np.int32)
    got = batched.prefill(prompt, 0, want_logits=True)
    monkeypatch.setenv("SLAI_PREFILL_SEQUENTIAL", "1")
    want = seq.prefill(prompt, 0, want_logits=True)
    kb, vb = batched.read_kv(0, T)
    ks, vs = seq.read_kv(0, T)
    # operands of 22 bits (2^-22 of each, both planes of both factors at most) and f32 sums of at most 5 blocks of 256: below 1e-5
    assert rel_l2(kb, ks) < 1e-5 and rel_l2(vb, vs) < 1e-5, (rel_l2(kb, ks), rel_l2(vb, vs))
    for t in {0, T // 2, T - 1}:  # every token on its own, the last row of every head included
        assert rel_l2(kb[t], ks[t]) < 2e-5 and rel_l2(vb[t], vs[t]) < 2e-5
    assert rel_l2(got, want) < 1e-4  # one layer and the logits product


# Q8_0 has no scale per super-block: its sums ended with a CTA's share of K, so their error depended on how K was shared out (512 columns, 37 tokens:
# 1.7e-7 over a cluster of four, 5.7e-7 in one CTA; 4096 columns, 400 tokens: 9e-6).
@pytest.mark.parametrize("dim,T", [(512, 16), (512, 37), (512, 300), (2048, 37), (4096, 16), (4096, 400)])
def test_q8_0_sums_do_not_lose_bits_with_k(backend, monkeypatch, dim, T):
    cfg = Llama2Config(dim=dim, hidden_dim=256, n_layers=1, n_q_heads=dim // 64, n_kv_heads=dim // 64, vocab_size=300, seq_len=T, kv_dtype=_lib.KV_F32)
    batched, seq = (synthetic_llama_device(backend, cfg, synth.FMT_Q8_0, synth.FMT_Q8_0, seed=5, std=0.02) for _ in range(2))
    ids = np.random.default_rng(T).integers(0, cfg.vocab_size, size=T).astype(np.int32)
    batched.prefill(ids, 0)
    monkeypatch.setenv("SLAI_PREFILL_SEQUENTIAL", "1")
    seq.prefill(ids, 0)
    # 128 columns are 24 products added up by the tensor core, each truncated by half of 2^-24 of a sum that is half of the last one on average: 3.6e-7;
    # operands of 22 bits, f32 sums over the super-blocks
    for got, want in zip(batched.read_kv(0, T), seq.read_kv(0, T)):
        assert rel_l2(got, want) < 5e-7
    batched.close()
    seq.close()


# The tensor-core attention (f16 cache, heads of 64 and 128): query tiles of 64, position tiles of 64, a first position inside a tile.
@pytest.mark.parametrize("heads,kv_heads", [(8, 8), (16, 4)])  # head size 128, 64
@pytest.mark.parametrize("pos,T", [(0, 16), (0, 63), (0, 65), (48, 17), (64, 64), (5, 200)])
def test_prompt_attention_on_the_tensor_cores(backend, monkeypatch, heads, kv_heads, pos, T):
    cfg = Llama2Config(dim=1024, hidden_dim=1024, n_layers=1, n_q_heads=heads, n_kv_heads=kv_heads, vocab_size=300, seq_len=256, kv_dtype=_lib.KV_F16)
    w = synthetic_llama_host(cfg, synth.FMT_Q8_0, synth.FMT_Q8_0, seed=3, std=0.08, embd_std=1.0)
    batched, seq = (llama_from_host(backend, cfg, w, synth.FMT_Q8_0, synth.FMT_Q8_0) for _ in range(2))
    ids = np.random.default_rng(pos + T).integers(0, cfg.vocab_size, size=pos + T).astype(np.int32)
    monkeypatch.setenv("SLAI_PREFILL_SEQUENTIAL", "1")
    want = seq.prefill(ids, 0, want_logits=True)
    if pos:
        batched.prefill(ids[:pos], 0)
    monkeypatch.delenv("SLAI_PREFILL_SEQUENTIAL")
    got = batched.prefill(ids[pos:], pos, want_logits=True)
    # a cached value may round to the other of two neighbouring halves (2^-11) where the passes differ in the last bits of f32
    assert rel_l2(got, want) < 1e-3


@pytest.mark.parametrize("hs", [64, 128])
@pytest.mark.parametrize("kv_dtype", [_lib.KV_F16, _lib.KV_F32])
@pytest.mark.parametrize("heads,kv_heads", [(4, 4), (4, 2), (6, 2), (8, 1)])
def test_decode_attention_in_registers(backend, ctx, hs, kv_dtype, heads, kv_heads):
    """One query token; positions at the edges of a group's share, of a batch of loads and of a split."""
    n = 2200
    rng = np.random.default_rng(hs + heads)
    dt = np.float16 if kv_dtype == _lib.KV_F16 else np.float32
    k, v = (rng.standard_normal((n, kv_heads, hs)).astype(dt) for _ in range(2))
    q = (2 * rng.standard_normal((heads, hs))).astype(np.float32)
    dk, dv, dq, out = backend.vector(k.ravel(), dt), backend.vector(v.ravel(), dt), backend.vector(q.ravel()), backend.zeros(heads * hs)
    for pos in (0, 1, 7, 8, 15, 16, 31, 32, 33, 64, 515, 2047, 2048, n - 1):
        p = BatchedMultiqueryAttentionParams(seq_len=n, kv_dim=kv_heads * hs, kv_mul=heads // kv_heads, n_heads=heads, head_size=hs, pos=pos)
        ctx.attention(p, dq, dk, dv, out, kv_dtype)
        got = out.to_numpy().reshape(heads, hs)
        # the entry point that allocates nothing serves more query heads per item: the staged path beside the register path
        backend.check(backend.lib.slai_attention_static(backend.h, C.byref(p.to_c()), C.c_void_p(dq.ptr), C.c_void_p(dk.ptr), C.c_void_p(dv.ptr), kv_dtype,
                                                        C.c_void_p(out.ptr)))
        assert rel_l2(out.to_numpy().reshape(heads, hs), got) < 1e-5, pos
        for h in range(heads):
            K, V = k[:pos + 1, h // (heads // kv_heads)].astype(np.float64), v[:pos + 1, h // (heads // kv_heads)].astype(np.float64)
            s = K @ q[h].astype(np.float64) / np.sqrt(hs)
            e = np.exp(s - s.max())
            # f32 scores of up to ~25 are off by a few 2^-24 of that, the exponentials by as much relative: below 1e-5
            assert rel_l2(got[h], e @ V / e.sum()) < 1e-5, (pos, h)


@pytest.mark.parametrize("heads,kv_heads", [(2, 2), (4, 2), (3, 1)])  # one and two query heads an item; three: one each
@pytest.mark.parametrize("kv_dtype", [_lib.KV_F16, _lib.KV_F32])
def test_decode_attention_where_its_splits_change(backend, ctx, kv_dtype, heads, kv_heads):
    """f32 caches of 128-wide heads: 16 positions a split up to 256 positions, 32 beyond; more than 16 splits are merged by groups."""
    hs, n = 128, 1100
    rng = np.random.default_rng(heads)
    dt = np.float16 if kv_dtype == _lib.KV_F16 else np.float32
    k, v = (rng.standard_normal((n, kv_heads, hs)).astype(dt) for _ in range(2))
    q = (2 * rng.standard_normal((heads, hs))).astype(np.float32)
    dk, dv, dq, out = backend.vector(k.ravel(), dt), backend.vector(v.ravel(), dt), backend.vector(q.ravel()), backend.zeros(heads * hs)
    for pos in (239, 240, 254, 255, 256, 287, 511, 512, 543, 544, 1023, 1024, n - 1):
        p = BatchedMultiqueryAttentionParams(seq_len=n, kv_dim=kv_heads * hs, kv_mul=heads // kv_heads, n_heads=heads, head_size=hs, pos=pos)
        ctx.attention(p, dq, dk, dv, out, kv_dtype)
        got = out.to_numpy().reshape(heads, hs)
        for h in range(heads):
            K, V = k[:pos + 1, h // (heads // kv_heads)].astype(np.float64), v[:pos + 1, h // (heads // kv_heads)].astype(np.float64)
            s = K @ q[h].astype(np.float64) / np.sqrt(hs)
            e = np.exp(s - s.max())
            assert rel_l2(got[h], e @ V / e.sum()) < 1e-5, (pos, h)  # f32 scores of up to ~25, as above


def test_longer_prompts_do_not_allocate_anew(backend):
    """Above 256 tokens the buffers of a pass grow in steps of 256 rows (GPT-2: its pass holds nothing that grows with the position)."""
    p = Gpt2Params(n_vocab=300, n_seq=1024, n_embd=1024, n_head=16, n_layer=1, ff_len=4096, kv_dtype=_lib.KV_F16)
    m = synthetic_gpt2_device(backend, p, synth.FMT_Q8_0, seed=1, std=0.02)
    ids = np.random.default_rng(1).integers(0, p.n_vocab, size=1024).astype(np.int32)
    for first, longer in ((257, (300, 400, 512)), (513, (600, 768))):
        m.prefill(ids[:first], 0)
        free = backend.mem_info()[0]
        for n in longer:
            m.prefill(ids[:n], 0)
            assert backend.mem_info()[0] == free, n
