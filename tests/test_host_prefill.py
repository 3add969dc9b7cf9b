"""The prompt GEMM's operand staging (packed quants -> fp16 pairs of columns, row scales, minimum term) executed on the CPU
(tests/host_prefill.cpp) against the oracle's dequantised weights.  Q4_K, Q5_K and Q6_K operands are exact integers times the
block scales: they differ from the oracle's f32 weights by the oracle's own two roundings, 2^-24 each of the two terms
(minimum and product) at most.  Q8_0: pairs of halves carry q * d to 2^-22, plus half a step of the smallest fp16 number."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from oracle import oracle as O
from slai_b200 import synth

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = "/usr/local/cuda/include"


@pytest.fixture(scope="module")
def emul(tmp_path_factory):
    if not os.path.exists(os.path.join(CUDA_INC, "cuda_fp16.h")) or shutil.which("g++") is None:
        pytest.skip("CUDA headers or g++ not available")
    exe = str(tmp_path_factory.mktemp("emul") / "host_prefill")
    subprocess.check_call(["g++", "-std=c++17", "-O1", f"-I{CUDA_INC}", "-o", exe, os.path.join(ROOT, "tests", "host_prefill.cpp"), "-lpthread"])
    return exe


@pytest.mark.parametrize("fmt,K", [(synth.FMT_Q4_K, 256), (synth.FMT_Q4_K, 1024), (synth.FMT_Q5_K, 512), (synth.FMT_Q6_K, 512),
                                   (synth.FMT_Q8_0, 64), (synth.FMT_Q8_0, 320)])
@pytest.mark.parametrize("kind", ["quantized", "random_bits"])
def test_operand_rows_hold_the_weights(emul, tmp_path, fmt, K, kind):
    rng = np.random.default_rng(K + fmt)
    blocks = synth.quantize(fmt, synth.normal_matrix(K, 16, K)) if kind == "quantized" else synth.random_blocks(fmt, 16, K, rng)
    blocks.tofile(tmp_path / "b.bin")
    out = subprocess.run([emul, str(fmt), str(K), str(tmp_path / "b.bin")], capture_output=True, timeout=60)
    assert out.returncode == 0, out.returncode
    got = np.frombuffer(out.stdout, dtype=np.float64).reshape(16, K)
    want = O.dequantize(fmt, blocks).reshape(16, K).astype(np.float64)
    if fmt == synth.FMT_Q8_0:
        assert np.all(np.abs(got - want) <= 2.0 ** -22 * np.abs(want) + 2.0 ** -25)
    else:
        # the largest product or minimum of a row's 256 columns bounds both terms: |w| <= 2 max, each rounded twice
        scale = np.abs(want).reshape(16, -1, 256).max(axis=2).repeat(256, axis=1)
        assert np.all(np.abs(got - want) <= 8 * 2.0 ** -24 * scale)
