"""Greedy decoding from the captured step equals stepping and taking the largest logit, for every storage format whose matvec is launched
in clusters (csrc/gemv_planes.cu, csrc/gemv_blocks.cu) and leaves the packed maximum itself. The kernels are the same: equal tokens."""
import numpy as np
import pytest

from alice_llm_b200 import synth
from softmodel import SMOOTH_MIX, soft_model

pytestmark = pytest.mark.gpu
ROLES = ("q", "k", "v", "o", "gate", "up", "down", "output")


@pytest.mark.parametrize("mix", [SMOOTH_MIX, *({n: t for n in ROLES} for t in (synth.Q8_0, synth.Q1_0, synth.Q2_0))], ids=["ternary", "q8_0", "q1_0", "q2_0"])
@pytest.mark.parametrize("hidden", [512, 640])
def test_greedy_equals_stepping(mix, hidden):
    from alice_llm_b200.gpu import GpuEngine, GpuModel
    cfg = dict(num_layers=2, hidden_dim=hidden, intermediate_dim=1280, num_heads=4, num_kv_heads=2, head_dim=128, vocab_size=1003, max_seq_len=64,
               rope_theta=500000.0, eps=1e-5)
    eng = GpuEngine(0)
    gm = GpuModel.load(eng, soft_model(np.random.default_rng(3 + hidden), cfg, mix))
    got = list(gm.decode_greedy(7, 12))
    gm.reset()
    want, tok = [], 7
    for _ in range(12):
        tok = int(np.argmax(gm.forward_and_read(tok)))
        want.append(tok)
    assert [int(t) for t in got] == want
    eng.close()
