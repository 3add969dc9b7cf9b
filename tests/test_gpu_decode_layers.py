"""The layers of a decode step in one launch (decode_layers.cuh) against the oracle, at the edges of its dispatch: one cluster of blocks or the whole chip,
splits of the positions (more positions than a round of lane groups holds), one or two query heads an item, widths that are not multiples of a digit step,
both cache types, every format.  Bars, relative L2 of the logits: 1e-3 with f16 caches, where a key may round to the other of two halves (test_gpu_models.py's bar);
1e-5 with f32 caches, whose steps keep 26 bits: both sides' f32 sums are what is left (measured 2e-7 to 2e-6; the lowest digit of the input alone is 4e-6 of it)."""
import threading

import numpy as np
import pytest

from oracle import oracle as O
from slai_b200 import _lib, synth
from slai_b200._lib import SlaiError
from slai_b200.models import Gpt2Params, Llama2Config, gpt2_from_host, llama_from_host, synthetic_gpt2_host, synthetic_llama_device, synthetic_llama_host
from slai_b200.ops import Backend
from helpers import oracle_gpt2, oracle_llama, rel_l2

pytestmark = pytest.mark.gpu
F16, F32 = _lib.KV_F16, _lib.KV_F32


@pytest.mark.parametrize("dim,hidden,hq,hkv,fmt,kv,n", [
    (256, 512, 4, 4, synth.FMT_Q4_K, F16, 70),      # one cluster
    (288, 768, 6, 6, synth.FMT_Q8_0, F32, 40),      # 48-wide heads, half-empty steps
    (512, 1280, 4, 4, synth.FMT_Q6_K, F32, 200),    # one cluster, up to four splits of 64 positions
    (512, 1280, 8, 2, synth.FMT_Q5_K, F16, 140),    # two query heads an item
    (1024, 2816, 8, 8, synth.FMT_Q4_K, F16, 140),   # the whole chip, 128 positions to a round
    (1024, 2816, 16, 4, synth.FMT_Q8_0, F32, 140),  # two query heads an item, blocks without items
])
def test_decode_against_the_oracle(backend, dim, hidden, hq, hkv, fmt, kv, n):
    cfg = Llama2Config(dim=dim, hidden_dim=hidden, n_layers=2, n_q_heads=hq, n_kv_heads=hkv, vocab_size=400, seq_len=n, kv_dtype=kv)
    w = synthetic_llama_host(cfg, fmt, seed=11, std=0.05, embd_std=1.0)
    m = llama_from_host(backend, cfg, w, fmt)
    ref = oracle_llama(cfg, w, fmt, kv_f16=kv == F16)
    toks = np.random.default_rng(2).integers(0, cfg.vocab_size, size=n)
    for pos, tok in enumerate(toks):
        got = m.forward_logits(pos, int(tok))[0]
        want = ref.forward(int(tok), pos)
        if pos < 3 or pos % 16 < 2 or pos == n - 1:
            bar = 1e-3 if kv == F16 else 1e-5
            assert rel_l2(got, want) < bar, (pos, rel_l2(got, want))
            assert rel_l2(m.read_state("x"), ref.x()) < bar, (pos, rel_l2(m.read_state("x"), ref.x()))
    assert m.launches_per_token() == 4  # embedding, layers, logits, greedy choice
    m.close()


def test_biases_and_a_tall_feed_forward_part(backend):
    """q / k / v biases with adjacent-pair RoPE; few bytes a layer, but more feed-forward rows than one cluster's epilogues take."""
    cfg = Llama2Config(dim=64, hidden_dim=9216, n_layers=2, n_q_heads=2, n_kv_heads=1, vocab_size=200, seq_len=24, kv_dtype=F32)
    fmt = synth.FMT_Q8_0
    w = synthetic_llama_host(cfg, fmt, seed=13, std=0.05, embd_std=1.0)
    rng = np.random.default_rng(1)
    for l in range(cfg.n_layers):
        w[("bq", l)] = (0.1 * rng.standard_normal(64)).astype(np.float32)
        w[("bk", l)], w[("bv", l)] = ((0.1 * rng.standard_normal(32)).astype(np.float32) for _ in range(2))
    m = llama_from_host(backend, cfg, w, fmt)
    ref = oracle_llama(cfg, w, fmt)
    for pos in range(cfg.seq_len):
        tok = int(rng.integers(cfg.vocab_size))
        assert rel_l2(m.forward_logits(pos, tok)[0], ref.forward(tok, pos)) < 1e-5, pos
    assert m.launches_per_token() == 4
    m.close()


@pytest.mark.parametrize("fmt", [synth.FMT_Q4_K, synth.FMT_Q5_K, synth.FMT_Q6_K, synth.FMT_Q8_0])
@pytest.mark.parametrize("dim,hidden,hq,hkv", [(512, 1280, 8, 4), (2048, 5632, 16, 16)])  # one cluster, the whole chip
def test_one_launch_against_the_separate_kernels(backend, monkeypatch, fmt, dim, hidden, hq, hkv):
    """The same model both ways, f32 caches, where the 256-element steps of every norm's output differ by up to 2^12 and the matrices' columns make up for it: each
    step's scale counts, and every digit of it."""
    cfg = Llama2Config(dim=dim, hidden_dim=hidden, n_layers=2, n_q_heads=hq, n_kv_heads=hkv, vocab_size=300, seq_len=24, kv_dtype=F32)
    w = synthetic_llama_host(cfg, fmt, seed=17, std=0.05, embd_std=1.0)
    rng = np.random.default_rng(3)
    for l in range(cfg.n_layers):
        for norm, names in (("attn_norm", ("wq", "wk", "wv")), ("ffn_norm", ("w_gate", "w_up"))):
            p2 = 2.0 ** rng.integers(-6, 7, size=dim // 256).repeat(256)  # (an f16 scale has to hold the inverse)
            w[(norm, l)] = p2.astype(np.float32)
            for name in names:
                r, c = cfg.matrix_shapes()[name]
                w[(name, l)] = synth.quantize(fmt, (synth.normal_matrix([l, r, len(name)], r, c, 0.05) / p2).astype(np.float32))
    one = llama_from_host(backend, cfg, w, fmt)
    many = llama_from_host(backend, cfg, w, fmt)
    toks = rng.integers(0, cfg.vocab_size, size=cfg.seq_len)
    got = [(one.forward_logits(pos, int(t))[0].copy(), one.read_state("x")) for pos, t in enumerate(toks)]
    monkeypatch.setenv("SLAI_SEPARATE_LAYERS", "1")
    for pos, t in enumerate(toks):
        logits = many.forward_logits(pos, int(t))[0]
        # the same digits and integer sums; f32 sums over the steps and warps in another order, a few 2^-24 of the largest terms, over two layers
        assert rel_l2(got[pos][0], logits) < 2e-6 and rel_l2(got[pos][1], many.read_state("x")) < 2e-6, (pos, rel_l2(got[pos][0], logits))
    assert one.launches_per_token() == 4 and many.launches_per_token() == 3 + 5 * cfg.n_layers
    one.close()
    many.close()


def test_gpt2_decode_against_the_oracle(backend):
    p = Gpt2Params(n_vocab=300, n_seq=300, n_embd=960, n_head=15, n_layer=2, ff_len=3840, kv_dtype=F16)
    w = synthetic_gpt2_host(p, synth.FMT_Q8_0, seed=4, std=0.05)
    m = gpt2_from_host(backend, p, w, synth.FMT_Q8_0)
    ref = oracle_gpt2(p, w, kv_f16=True)
    toks = np.random.default_rng(3).integers(0, p.n_vocab, size=p.n_seq)
    for pos, tok in enumerate(toks):  # 256 positions to a round: the last 44 tokens have two splits
        got = m.forward(int(tok), pos)[0]
        want = ref.forward(int(tok), pos)
        if pos < 3 or pos % 32 < 2 or pos == p.n_seq - 1:
            assert rel_l2(got, want) < 1e-3, pos
    m.close()


def test_two_contexts_decode_at_the_same_time():
    """Two threads, two streams: launches whose blocks wait on one another share the chip (one after the other, or side by side where both fit)."""
    shapes = [dict(dim=1024, hidden_dim=2816, n_q_heads=8, n_kv_heads=8), dict(dim=256, hidden_dim=768, n_q_heads=4, n_kv_heads=4)]
    models = []
    for i, sh in enumerate(shapes * 2):
        be = Backend(0)
        cfg = Llama2Config(n_layers=4, vocab_size=500, seq_len=80, kv_dtype=F16, **sh)
        models.append((be, synthetic_llama_device(be, cfg, synth.FMT_Q4_K, synth.FMT_Q4_K, seed=1 + i, std=0.05)))
    alone = [list(m.generate(3, 0, 64)) for _, m in models]
    got = [None] * len(models)

    def work(i):
        for _ in range(3):
            got[i] = list(models[i][1].generate(3, 0, 64))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(models))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert got == alone
    for be, m in models:
        m.close()
        be.close()


def test_short_wait_limit_at_a_long_context():
    """A block's wait for the others takes as long as their phase: the attention over 3900 positions outlasts 64 polls, and is nobody's failure."""
    be = Backend(0)
    cfg = Llama2Config(dim=4096, hidden_dim=4096, n_layers=1, n_q_heads=32, n_kv_heads=32, vocab_size=500, seq_len=4096, kv_dtype=F16)
    m = synthetic_llama_device(be, cfg, synth.FMT_Q4_K, synth.FMT_Q4_K, seed=1, std=0.02)
    want = m.forward_logits(3900, 5)[0].copy()
    be.set_wait_limit(16)
    m2 = synthetic_llama_device(be, cfg, synth.FMT_Q4_K, synth.FMT_Q4_K, seed=1, std=0.02)
    for _ in range(5):
        assert np.array_equal(m2.forward_logits(3900, 5)[0], want)
    m.close()
    m2.close()
    be.close()


def test_what_the_separate_kernels_refuse_is_refused(backend):
    """More than eight query heads to a key head, and a feed-forward part wider than a product takes (28672 fits, its down product's 30720 does not)."""
    for sh in (dict(dim=512, hidden_dim=1024, n_q_heads=16, n_kv_heads=1), dict(dim=256, hidden_dim=30720, n_q_heads=4, n_kv_heads=4)):
        cfg = Llama2Config(n_layers=1, vocab_size=100, seq_len=32, kv_dtype=F16, **sh)
        m = synthetic_llama_device(backend, cfg, synth.FMT_Q4_K, synth.FMT_Q4_K, seed=1, std=0.05)
        for call in (lambda: m.forward_logits(0, 3), lambda: m.generate(3, 0, 4), lambda: m.stats(3, 0)):
            with pytest.raises(SlaiError) as e:
                call()
            assert e.value.code == _lib.ERR_SHAPE
        m.close()


@pytest.mark.parametrize("arch", ["llama", "gpt2"])
def test_small_layers_leave_the_cluster_at_a_long_context(backend, arch):
    """256 wide: one cluster of blocks while the weights of a layer and half of its keys and values are below 3 MB, the whole chip behind that position (for
    these f32 caches 2045 and 1187 positions), in the device loop as in single steps, and back again."""
    n, first = (1300, 1150) if arch == "gpt2" else (2160, 2010)
    if arch == "llama":
        cfg = Llama2Config(dim=256, hidden_dim=768, n_layers=1, n_q_heads=4, n_kv_heads=4, vocab_size=300, seq_len=n, kv_dtype=F32)
        w = synthetic_llama_host(cfg, synth.FMT_Q8_0, seed=21, std=0.05, embd_std=1.0)
        m, ref = llama_from_host(backend, cfg, w, synth.FMT_Q8_0), oracle_llama(cfg, w, synth.FMT_Q8_0)
    else:
        p = Gpt2Params(n_vocab=300, n_seq=n, n_embd=320, n_head=5, n_layer=1, ff_len=1280, kv_dtype=F32)
        w = synthetic_gpt2_host(p, synth.FMT_Q8_0, seed=22, std=0.05)
        m, ref = gpt2_from_host(backend, p, w, synth.FMT_Q8_0), oracle_gpt2(p, w)
    one = (lambda pos, t: m.forward_logits(pos, t)[0]) if arch == "llama" else (lambda pos, t: m.forward(t, pos)[0])
    toks = np.random.default_rng(4).integers(0, 300, size=n)
    m.prefill(toks[:first].astype(np.int32), 0)
    early = one(3, int(toks[3])).copy()
    for pos in range(n):
        want = ref.forward(int(toks[pos]), pos)
        if pos >= first:
            got = one(pos, int(toks[pos]))
            if pos % 8 == 0 or pos == n - 1:
                assert rel_l2(got, want) < 2e-5, pos
    assert np.array_equal(one(3, int(toks[3])), early)
    assert np.array_equal(m.generate(int(toks[first]), first, 100), m.generate(int(toks[first]), first, 100))
    m.close()


@pytest.mark.parametrize("separate", [False, True])
def test_norms_of_tiny_values_keep_their_bits(backend, monkeypatch, separate):
    """x of 1e-32: what comes out of the norms is 1 / sqrt(eps) = 316 times that, still far below one, and has 20 bits of each step's largest element at least."""
    if separate:
        monkeypatch.setenv("SLAI_SEPARATE_LAYERS", "1")
    cfg = Llama2Config(dim=512, hidden_dim=1024, n_layers=2, n_q_heads=4, n_kv_heads=4, vocab_size=300, seq_len=8, kv_dtype=F32)
    w = synthetic_llama_host(cfg, synth.FMT_Q6_K, seed=31, std=0.05, embd_std=1e-32)
    m, ref = llama_from_host(backend, cfg, w, synth.FMT_Q6_K), oracle_llama(cfg, w, synth.FMT_Q6_K)
    for pos, tok in enumerate((5, 17, 200)):
        assert rel_l2(m.forward_logits(pos, tok)[0] * 1e30, ref.forward(tok, pos).astype(np.float64) * 1e30) < 1e-5
    m.close()
