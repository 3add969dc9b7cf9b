"""The prompt pass's tensor-core attention (f16 caches, heads of 64 and 128) where halves could run out of range: queries far beyond 65504, an
infinite cached value behind the query.  Layers are made so that the attention can be read off them: the feed-forward adds nothing."""
import numpy as np
import pytest

from oracle import oracle as O
from slai_b200 import _lib, synth
from slai_b200.models import Llama2Config, llama_from_host, synthetic_llama_host
from helpers import rel_l2

pytestmark = pytest.mark.gpu
DIM, FMT = 512, synth.FMT_Q8_0


def one_model(backend, head_size, layers, seq_len, std=0.05):
    cfg = Llama2Config(dim=DIM, hidden_dim=512, n_layers=layers, n_q_heads=DIM // head_size, n_kv_heads=DIM // head_size, vocab_size=64, seq_len=seq_len,
                       kv_dtype=_lib.KV_F16)
    w = synthetic_llama_host(cfg, FMT, FMT, seed=head_size, std=std, embd_std=1.0)
    for l in range(layers):
        w[("w_down", l)] = synth.quantize(FMT, np.zeros(DIM * 512, dtype=np.float32).reshape(DIM, 512))
    return cfg, w


def matrix(w, name, l, shape):
    return O.dequantize(FMT, w[(name, l)]).reshape(shape).astype(np.float64)


def rotated(x, pos, head_size):
    """Adjacent-pair RoPE of [tokens][heads][head_size] at the f32 angles that the library uses."""
    theta = (1.0 / 10000.0 ** (np.arange(0, head_size, 2) / head_size)).astype(np.float32)
    a = (np.asarray(pos, np.float32)[:, None] * theta).astype(np.float64)[:, None, :]
    p = x.reshape(*x.shape[:-1], head_size // 2, 2)
    return np.stack([np.cos(a) * p[..., 0] - np.sin(a) * p[..., 1], np.sin(a) * p[..., 0] + np.cos(a) * p[..., 1]], -1).reshape(x.shape)


@pytest.mark.parametrize("head_size", [64, 128])
@pytest.mark.parametrize("gain", [1.0, 3e3])  # queries of about 1, and of a million (65504 is a half's largest)
@pytest.mark.parametrize("T", [17, 100])
def test_queries_of_any_size(backend, head_size, gain, T):
    cfg, w = one_model(backend, head_size, 1, 128)
    half = DIM // 2  # queries see one half of the channels, times `gain`; keys see the other, divided by it
    rng = np.random.default_rng(T)
    wq, wk = (0.05 * rng.standard_normal((DIM, DIM)).astype(np.float32) for _ in range(2))
    wq[:, half:] = 0
    wk[:, :half] = 0
    big = gain > 1
    w[("wq", 0)], w[("wk", 0)] = synth.quantize(FMT, wq * (150 if big else 1)), synth.quantize(FMT, wk * (0.002 if big else 1))
    norm = np.ones(DIM, dtype=np.float32)
    norm[:half] *= gain
    norm[half:] *= 0.03 if big else 1
    w[("attn_norm", 0)] = norm
    m = llama_from_host(backend, cfg, w, FMT, FMT)
    ids = rng.integers(0, cfg.vocab_size, size=T).astype(np.int32)
    m.prefill(ids, 0)
    H = DIM // head_size
    k, v = (a.astype(np.float64).reshape(T, H, head_size) for a in m.read_kv(0, T))
    emb = np.asarray(w[("token_embd", -1)], np.float64).reshape(cfg.vocab_size, DIM)
    x = emb[ids[-1]]
    h = x / np.sqrt((x * x).mean() + cfg.rms_norm_eps) * norm
    q = rotated((matrix(w, "wq", 0, (DIM, DIM)) @ h).reshape(1, H, head_size), [T - 1], head_size)[0]
    assert not big or np.abs(q).max() / np.sqrt(head_size) > 65504
    s = np.einsum("hd,thd->ht", q, k) / np.sqrt(head_size)
    e = np.exp(s - s.max(axis=1, keepdims=True))
    att = np.einsum("ht,thd->hd", e / e.sum(axis=1, keepdims=True), v).reshape(DIM)
    got = m.read_state("x").astype(np.float64) - x
    # The products' operands carry 22 bits or more: scores are off by a few 2^-22 of |q| |k| / sqrt(head size) <= 4 |s|, weights by as
    # much; x itself is rounded at 2^-24 of its size.
    tol = 1e-5 + 4 * 2.0 ** -22 * 4 * np.abs(s).max()
    assert np.abs(s).max() < 200
    assert rel_l2(got, matrix(w, "wo", 0, (DIM, DIM)) @ att) < tol


@pytest.mark.parametrize("head_size", [64, 128])
def test_an_infinite_value_does_not_reach_the_queries_before_it(backend, head_size):
    """A value too large for the cache's halves becomes infinite there.  Queries of earlier groups of 16 give it the weight zero, and zero
    times infinity must not enter their sums.  Seen in the second layer's keys, which depend on the first one's attention."""
    T, at = 100, 40
    cfg, w = one_model(backend, head_size, 2, 128)
    emb = np.array(w[("token_embd", -1)], np.float32).reshape(cfg.vocab_size, DIM)
    emb[:, 0] = 0
    emb[7] = 0
    emb[7, 0] = 1  # token 7 lives in channel 0 alone
    w[("token_embd", -1)] = emb.reshape(-1)
    w[("attn_norm", 0)] = np.where(np.arange(DIM) == 0, 1e3, 1).astype(np.float32)
    rng = np.random.default_rng(1)
    wv = 0.05 * rng.standard_normal((DIM, DIM)).astype(np.float32)
    wv[:, :32] = 0  # a block of its own, so that its scale leaves the other channels alone
    wv[:, 0] = 10
    w[("wv", 0)] = synth.quantize(FMT, wv)
    for name in ("wq", "wk"):
        z = 0.05 * rng.standard_normal((DIM, DIM)).astype(np.float32)
        z[:, 0] = 0
        w[(name, 0)] = synth.quantize(FMT, z)
    m = llama_from_host(backend, cfg, w, FMT, FMT)
    ids = rng.integers(8, cfg.vocab_size, size=T).astype(np.int32)
    m.prefill(ids, 0)
    want = m.read_kv(1, T)
    ids[at] = 7
    m.prefill(ids, 0)
    assert np.isinf(m.read_kv(0, T)[1][at]).all()
    before = at // 16 * 16
    for got, ref in zip(m.read_kv(1, T), want):
        assert np.array_equal(got[:before], ref[:before])
