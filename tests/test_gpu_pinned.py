"""A process that gets next to no page-locked memory: models are made and give the same logits, by copies straight into the caller's memory.
The failure is made on the host: a library loaded ahead of the CUDA runtime answers requests for more than 4 KB of page-locked memory
with an error (the engine's status word is 4 bytes)."""
import os
import subprocess
import sys
import textwrap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHIM = """
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static void* real(const char* name) { return dlsym(dlopen("libcudart.so.12", RTLD_NOLOAD | RTLD_LAZY), name); }
int cudaHostAlloc(void** p, size_t n, unsigned int f) { return n > 4096 ? 2 : ((int (*)(void**, size_t, unsigned int))real("cudaHostAlloc"))(p, n, f); }
int cudaMallocHost(void** p, size_t n) { return n > 4096 ? 2 : ((int (*)(void**, size_t))real("cudaMallocHost"))(p, n); }
"""

RUN = """
import sys
import numpy as np
from alice_llm_b200 import synth
from alice_llm_b200.gpu import GpuEngine, GpuModel
cfg = dict(num_layers=2, hidden_dim=512, intermediate_dim=1024, num_heads=4, num_kv_heads=2, head_dim=128, vocab_size=1000, max_seq_len=64,
           rope_theta=500000.0, eps=1e-5)
eng = GpuEngine(0)
gm = GpuModel.load(eng, synth.make_llama(np.random.default_rng(5), cfg))
one = gm.forward_and_read(3)
gm.forward(4)
rest = gm.forward_rows(list(range(20)), [0, 5, 19])
np.savez(sys.argv[1], one=one, rest=rest, batch=gm.forward_batch_and_read([1, 2, 3]))
eng.close()
"""


def test_without_page_locked_memory(tmp_path):
    (tmp_path / "shim.c").write_text(SHIM)
    shim = tmp_path / "shim.so"
    subprocess.check_call(["gcc", "-shared", "-fPIC", "-o", str(shim), str(tmp_path / "shim.c"), "-ldl"])
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    got = []
    for name, env in (("plain", {}), ("shim", {"LD_PRELOAD": str(shim)})):
        out = tmp_path / (name + ".npz")
        subprocess.check_call([sys.executable, "-c", textwrap.dedent(RUN), str(out)], cwd=root, env={**os.environ, **env}, timeout=300)
        got.append(np.load(out))
    for key in ("one", "rest", "batch"):
        assert np.array_equal(got[0][key], got[1][key]), key
