"""Several tokens at once, one of them or a part of the context not finite: what a token does not see stays out of its result, what it sees
is not lost. Against the same model stepped token by token."""
import numpy as np
import pytest

from alice_llm_b200 import synth

pytestmark = pytest.mark.gpu
ROLES = ("q", "k", "v", "o", "gate", "up", "down", "output")
Q8 = {n: synth.Q8_0 for n in ROLES}
H = 512


@pytest.fixture(scope="module")
def eng():
    from alice_llm_b200.gpu import GpuEngine
    e = GpuEngine(0)
    yield e
    e.close()


def config(heads, ctx, n):
    return dict(num_layers=2, hidden_dim=H, intermediate_dim=1024, num_heads=heads[0], num_kv_heads=heads[1], head_dim=128, vocab_size=64,
                max_seq_len=ctx + n + 8, rope_theta=500000.0, eps=1e-5)


@pytest.mark.parametrize("heads", [(2, 2), (8, 2), (16, 2)])
@pytest.mark.parametrize("n,odd", [(2, 1), (4, 3), (8, 5), (40, 33), (70, 69)])
def test_value_row_of_a_later_token(eng, heads, n, odd):
    """Token 9's value rows of layer 0 overflow (a norm weight of 2e38 on column 0, which every other embedding and every query and key row
    has at zero); the tokens ahead of it must not notice."""
    from alice_llm_b200.gpu import GpuModel
    rng = np.random.default_rng(n)
    model = synth.make_llama(rng, config(heads, 0, n), Q8)
    emb = model["embedding"][1].reshape(64, H // 32, 34)
    emb[:, 0, 2] = 0
    emb[9, 0, 2] = 40
    L = model["layers"][0]
    L["attn_norm"][0] = 2e38
    for name in ("q", "k"):
        L[name][1].reshape(-1, H // 32, 34)[:, 0, 2] = 0
    v = L["v"][1].reshape(-1, H // 32, 34)
    v[:, 0, 2] = 127
    v[:, 0, 0:2] = np.array([8.0], np.float16).view(np.uint8)
    gm = GpuModel.load(eng, model)
    toks = rng.integers(10, 64, n).tolist()
    toks[odd] = 9
    ref = [gm.forward_and_read(t) for t in toks]
    assert np.isfinite(ref[odd - 1]).all() and not np.isfinite(ref[odd]).any()
    gm.reset()
    rows = sorted({0, odd - 1, odd, n - 1})
    got = gm.forward_rows(toks, rows)
    for i, r in enumerate(rows):
        if r < odd:
            a, b = got[i].astype(np.float64), ref[r].astype(np.float64)
            assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b), r
        else:
            assert not np.isfinite(got[i]).any(), r
    gm.free()


@pytest.mark.parametrize("heads", [(2, 2), (16, 2)])
@pytest.mark.parametrize("n", [2, 8])
def test_key_rows_that_are_not_numbers(eng, heads, n):
    """Keys that are NaN over a whole share of the context: so is every result."""
    from alice_llm_b200.gpu import GpuModel
    rng, ctx = np.random.default_rng(5), 1500
    gm = GpuModel.load(eng, synth.make_llama(rng, config(heads, ctx, n), Q8))
    for l in range(2):
        k, v = (rng.standard_normal((ctx, heads[1] * 128), dtype=np.float32) for _ in range(2))
        if l == 0:
            k[:640] = np.nan
        gm.kv_write(l, 0, k, v)
    gm.set_position(ctx)
    toks = rng.integers(0, 64, n).tolist()
    assert np.isnan(gm.forward_and_read(toks[0])).all()
    gm.set_position(ctx)
    assert np.isnan(gm.forward_rows(toks, list(range(n)))).all()
    gm.free()
