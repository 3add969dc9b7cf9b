"""The prompt pass where its work is dealt out: products whose tiles are shared by neighbouring CTAs (equal shares of the super-blocks), and attention whose
position tiles are shared by a cluster.  Against the sequential pass of the same model."""
import numpy as np
import pytest

from slai_b200 import _lib, synth
from slai_b200.models import Llama2Config, synthetic_llama_device
from helpers import rel_l2

pytestmark = pytest.mark.gpu


# 148 SMs: q/k/v are 96 tiles of 128 rows x 16 super-blocks (10.4 a CTA: a tile lies on up to three), gate and up 172; above 64 tokens pairs of CTAs
# and several token tiles (400: 192 tiles over 74 pairs).
@pytest.mark.parametrize("fmt", [synth.FMT_Q4_K, synth.FMT_Q6_K, synth.FMT_Q8_0])
@pytest.mark.parametrize("T", [16, 40, 64, 400])
def test_products_with_shared_tiles(backend, monkeypatch, fmt, T):
    cfg = Llama2Config(dim=4096, hidden_dim=11008, n_layers=1, n_q_heads=32, n_kv_heads=32, vocab_size=300, seq_len=416, kv_dtype=_lib.KV_F32)
    batched, seq = (synthetic_llama_device(backend, cfg, fmt, fmt, seed=5, std=0.02) for _ in range(2))
    ids = np.random.default_rng(T).integers(0, cfg.vocab_size, size=T).astype(np.int32)
    got = batched.prefill(ids, 0, want_logits=True)
    again = batched.prefill(ids, 0, want_logits=True)
    assert np.array_equal(got, again)  # sums in a fixed order
    k, v = batched.read_kv(0, T)
    monkeypatch.setenv("SLAI_PREFILL_SEQUENTIAL", "1")
    want = seq.prefill(ids, 0, want_logits=True)
    ks, vs = seq.read_kv(0, T)
    # operands of 22 bits, f32 sums of 16 blocks of 256 (Q8_0: 32 of 128): below 2e-5
    assert rel_l2(k, ks) < 2e-5 and rel_l2(v, vs) < 2e-5, (rel_l2(k, ks), rel_l2(v, vs))
    assert rel_l2(got, want) < 2e-4  # one layer and the logits product
    batched.close()
    seq.close()


@pytest.mark.parametrize("heads", [8, 16])  # head size 128, 64
@pytest.mark.parametrize("pos,T", [(64, 16), (110, 40), (200, 17), (448, 16), (500, 70), (0, 128), (575, 64)])  # 2 to 10 tiles for 2 to 8 CTAs
def test_attention_with_shared_tiles(backend, monkeypatch, heads, pos, T):
    cfg = Llama2Config(dim=1024, hidden_dim=1024, n_layers=1, n_q_heads=heads, n_kv_heads=heads // 2, vocab_size=300, seq_len=640, kv_dtype=_lib.KV_F16)
    batched, seq = (synthetic_llama_device(backend, cfg, synth.FMT_Q8_0, synth.FMT_Q8_0, seed=3, std=0.08) for _ in range(2))
    ids = np.random.default_rng(pos + T).integers(0, cfg.vocab_size, size=pos + T).astype(np.int32)
    monkeypatch.setenv("SLAI_PREFILL_SEQUENTIAL", "1")
    want = seq.prefill(ids, 0, want_logits=True)
    if pos:
        batched.prefill(ids[:pos], 0)
    monkeypatch.delenv("SLAI_PREFILL_SEQUENTIAL")
    got = batched.prefill(ids[pos:], pos, want_logits=True)
    assert rel_l2(got, want) < 1e-3  # a cached value may round to the other of two neighbouring halves, as in test_gpu_prompt_kernels.py
    batched.close()
    seq.close()
