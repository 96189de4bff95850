"""Attention of one token (csrc/attn_body.cuh) where its shares and chunks of positions begin and end: shares of 32 positions and more, chunks
of 64 in a ring of three, contexts without a full share, from an empty cache to rings that wrap. Two key / value heads have 64 shares at most.

Against the CPU oracle's forward of a model whose activations stay in f32 (as tests/test_gpu_attention.py, same gate)."""
import numpy as np
import pytest

from softmodel import SMOOTH_MIX, soft_model
from test_gpu_attention import fill, rel_err, rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    from alice_llm_b200.gpu import GpuEngine
    e = GpuEngine(0)
    yield e
    e.close()


@pytest.mark.parametrize("heads", [(4, 2), (10, 2), (16, 2)])       # 8 or 16 lanes a position, even and odd groups
@pytest.mark.parametrize("ctx", [0, 1, 31, 63, 64, 2046, 4095, 20000])
def test_shares_and_chunks(eng, oracle, heads, ctx):
    from alice_llm_b200.gpu import GpuModel
    cfg = dict(num_layers=1, hidden_dim=512, intermediate_dim=512, num_heads=heads[0], num_kv_heads=heads[1], head_dim=128,
               vocab_size=500, max_seq_len=ctx + 8, rope_theta=500000.0, eps=1e-5)
    rng = np.random.default_rng(ctx + heads[0])
    model = soft_model(rng, cfg, SMOOTH_MIX)
    gm, ref = GpuModel.load(eng, model), oracle.LlamaOracle(model)
    if ctx:
        fill(rng, cfg, ctx, gm, [ref])
    for t in (3, 200, 41):                                           # three positions in a row cross the edge
        got, want = gm.forward_and_read(t), ref.forward(t)
        assert rel_err(got, want) <= 1e-3 and rel_l2(got, want) <= 1e-3, (heads, ctx, t)
    k, v = gm.kv_read(0, ctx, 3)
    assert rel_err(k, ref.kcache[0, ctx:ctx + 3]) <= 1e-3 and rel_err(v, ref.vcache[0, ctx:ctx + 3]) <= 1e-3
    gm.free()
