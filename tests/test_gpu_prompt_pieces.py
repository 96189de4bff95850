"""Prompts taken in pieces of up to 256 tokens (csrc/gemm_kq.cu, csrc/attn_tokens.cu) against the same model stepped token by token,
which the other files hold against the oracle. Token counts at the edges of the 8 / 16 / 32 / 64 / 128-token tiles and of a piece,
contexts at the edges of the 32-key steps, every query group, wanted rows in runs of every length. (The widths of a K-quant model are whole row
tiles; parts of tiles are covered product by product in test_gpu_prompt_products.py.)

All-ternary models are smooth: the two paths differ by the order of f32 sums only (terms up to 1000, two layers: 1e-5, held to
1e-4). K-quant models round activations to the Q8_K grid, where a last bit moves single values by a step of 1 / 128: 2e-2, as
far as two orders of the sums end apart."""
import numpy as np
import pytest

from alice_llm_b200 import synth
from softmodel import SMOOTH_MIX, soft_model

pytestmark = pytest.mark.gpu

Q5KM = dict({n: synth.Q5_K for n in ("q", "k", "v", "o", "gate", "up", "output")}, down=synth.Q6_K)


@pytest.fixture(scope="module")
def eng():
    from alice_llm_b200.gpu import GpuEngine
    e = GpuEngine(0)
    yield e
    e.close()


def rel_l2(got, ref):
    got, ref = np.asarray(got, np.float64), np.asarray(ref, np.float64)
    return float(np.linalg.norm(got - ref) / np.linalg.norm(ref))


def compare(eng, mix, heads, hidden, ff, ctx, n, tol, rows=None):
    from alice_llm_b200.gpu import GpuModel
    cfg = dict(num_layers=2, hidden_dim=hidden, intermediate_dim=ff, num_heads=heads[0], num_kv_heads=heads[1], head_dim=128,
               vocab_size=1000, max_seq_len=ctx + n + 8, rope_theta=500000.0, eps=1e-5)
    rng = np.random.default_rng(n * 131 + ctx + heads[0])
    gm = GpuModel.load(eng, soft_model(rng, cfg, mix))
    kv = [(rng.standard_normal((max(ctx, 1), heads[1] * 128), dtype=np.float32), rng.standard_normal((max(ctx, 1), heads[1] * 128), dtype=np.float32)) for _ in range(2)]
    toks = rng.integers(0, 1000, n).tolist()
    rows = sorted({0, n // 2, max(0, n - 2), n - 1}) if rows is None else rows

    def start():
        gm.reset()
        if ctx:
            for l, (k, v) in enumerate(kv):
                gm.kv_write(l, 0, k, v)
            gm.set_position(ctx)

    start()
    ref = [gm.forward_and_read(t) for t in toks]
    ref_kv = [gm.kv_read(l, 0, ctx + n) for l in range(2)]
    start()
    got = gm.forward_rows(toks, rows)
    assert gm.position() == ctx + n
    for i, r in enumerate(rows):
        assert rel_l2(got[i], ref[r]) <= tol, (r, rel_l2(got[i], ref[r]))
    for l in range(2):
        for a, b in zip(gm.kv_read(l, 0, ctx + n), ref_kv[l]):
            assert rel_l2(a, b) <= tol


@pytest.mark.parametrize("heads", [(2, 2), (4, 2), (8, 2), (10, 2), (16, 2)])   # 1, 2, 4, 5, 8 query heads per KV head
@pytest.mark.parametrize("ctx,n", [(0, 2), (31, 8), (33, 5), (500, 40), (0, 67), (1000, 8)])
def test_attention_of_many_tokens(eng, heads, ctx, n):
    compare(eng, SMOOTH_MIX, heads, 512, 1024, ctx, n, 1e-4)


@pytest.mark.parametrize("heads", [(2, 2), (10, 2), (16, 2), (32, 8)])
@pytest.mark.parametrize("ctx,n", [(0, 3), (120, 5), (250, 6), (257, 6), (2048, 8), (5000, 2), (1000, 48)])
def test_shares_of_attention(eng, heads, ctx, n):
    """Tiles of 16, 32, 48 and 64 rows; one share, two to eight in a cluster, more through the scratch, clusters where that is too small"""
    compare(eng, SMOOTH_MIX, heads, 512, 512, ctx, n, 1e-4)


@pytest.mark.parametrize("heads", [(4, 2), (16, 2), (32, 4)])
@pytest.mark.parametrize("ctx,n", [(2040, 8), (2041, 8), (4100, 8), (240, 8), (249, 8), (60, 8), (140, 3), (0, 17), (0, 48)])
def test_shares_and_tiles_at_their_limits(eng, heads, ctx, n):
    """64 steps of 32 positions and 65, where the scratch holds 64 shares for eight tokens; eight steps and nine, where tiles are smaller up to eight;
    three and five, whose clusters have empty shares"""
    compare(eng, SMOOTH_MIX, heads, 512, 512, ctx, n, 1e-4)


@pytest.mark.parametrize("hidden", [256, 1184, 2048, 2304, 8192, 8448])
@pytest.mark.parametrize("n", [8, 9])
def test_prepared_vectors(eng, hidden, n):
    """Up to eight vectors are prepared by CTAs of four warps, more by one of sixteen each: vectors that fit the registers of either and that do not"""
    compare(eng, SMOOTH_MIX, (4, 2), hidden, 512, 20, n, 1e-4)


@pytest.mark.parametrize("n", [2, 9, 16, 17, 33, 64, 65, 129, 256, 300])
@pytest.mark.parametrize("mix", [None, Q5KM], ids=["q4km", "q5km"])
def test_k_quant_prompts(eng, mix, n):
    compare(eng, mix, (4, 2), 512, 256 * 9, 16 if n % 2 else 0, n, 2e-2)


@pytest.mark.parametrize("mix", [SMOOTH_MIX, {n: synth.Q8_0 for n in ("q", "k", "v", "o", "gate", "up", "down", "output")}], ids=["ternary", "q8_0"])
@pytest.mark.parametrize("n,rows", [(20, list(range(20))), (40, [0, 1, 2, 5, 6, *range(9, 27), 30, 39]), (290, [*range(3, 12), *range(250, 262), 280, 289]), (30, [])])
def test_wanted_rows(eng, mix, n, rows):
    """Runs of up to eight rows share a launch of the head; more than eight rows leave without the pinned buffer."""
    compare(eng, mix, (4, 2), 512, 1024, 5, n, 1e-4, rows)
