"""A process that has some of the SMs only, though the device's properties tell of all of them (a green context): launches whose blocks wait on one another do not
fit as planned, and the layers run kernel by kernel.  In a process of its own: the context stays current there."""
import os
import subprocess
import sys

import numpy as np
import pytest

from slai_b200 import _lib, synth
from slai_b200.models import Llama2Config, synthetic_llama_device
from helpers import rel_l2

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CFG = dict(dim=1024, hidden_dim=2816, n_layers=2, n_q_heads=8, n_kv_heads=8, vocab_size=400, seq_len=64, kv_dtype=_lib.KV_F32)

CHILD = """
import sys
sys.path.insert(0, sys.argv[1])
from cuda.bindings import driver as cu
def ok(r):
    assert r[0] == cu.CUresult.CUDA_SUCCESS, r
    return r[1] if len(r) == 2 else r[1:]
assert cu.cuInit(0)[0] == cu.CUresult.CUDA_SUCCESS
dev = ok(cu.cuDeviceGet(0))
sms = ok(cu.cuDeviceGetDevResource(dev, cu.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
groups = ok(cu.cuDevSmResourceSplitByCount(1, sms, 0, 32))[0]
green = ok(cu.cuGreenCtxCreate(ok(cu.cuDevResourceGenerateDesc([groups[0]], 1)), dev, cu.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
ok_ctx = ok(cu.cuCtxFromGreenCtx(green))
assert cu.cuCtxSetCurrent(ok_ctx)[0] == cu.CUresult.CUDA_SUCCESS
import numpy as np
from slai_b200 import _lib, synth
from slai_b200.models import Llama2Config, synthetic_llama_device
from slai_b200.ops import Backend
be = Backend(0)
m = synthetic_llama_device(be, Llama2Config(**eval(sys.argv[2])), synth.FMT_Q4_K, synth.FMT_Q4_K, seed=9, std=0.05)
logits = np.stack([m.forward_logits(pos, 7 + pos)[0] for pos in range(6)])
print(groups[0].sm.smCount, m.launches_per_token(), list(m.generate(3, 6, 20)))
np.save(sys.argv[3], logits)
"""


def test_layers_run_kernel_by_kernel_where_one_launch_does_not_fit(backend, tmp_path):
    m = synthetic_llama_device(backend, Llama2Config(**CFG), synth.FMT_Q4_K, synth.FMT_Q4_K, seed=9, std=0.05)
    want = np.stack([m.forward_logits(pos, 7 + pos)[0] for pos in range(6)])
    assert m.launches_per_token() == 4
    m.close()
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT, repr(CFG), str(tmp_path / "l.npy")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    sms, launches = r.stdout.split()[:2]
    assert int(sms) < 64 and int(launches) == 3 + 5 * CFG["n_layers"], r.stdout
    assert rel_l2(np.load(tmp_path / "l.npy"), want) < 2e-6
