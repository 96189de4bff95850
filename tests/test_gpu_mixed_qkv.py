"""Query, key and value projections of different storage formats: each reads the normalised hidden state in its own form (Q8_K blocks,
f32 rounded to the Q8_K grid, plain f32), whatever the others want. The rows a layer appends to the cache are these projections
themselves (position 0 is not rotated, values never are): held against the oracle's matvecs of the oracle's norm of layer 0, where no
earlier rounding can move a value on the grid, within the 1e-3 of the other parity tests."""
import numpy as np
import pytest

from alice_llm_b200 import synth

pytestmark = pytest.mark.gpu
Q4_K, Q5_K, Q6_K, Q8_0, Q1_0, Q2_0, TERNARY = synth.Q4_K, synth.Q5_K, synth.Q6_K, synth.Q8_0, synth.Q1_0, synth.Q2_0, synth.TERNARY


def expect(oracle, entry, x, rows, cols):
    t, data = entry
    if t == TERNARY:
        return oracle.ternary_matvec(*data, rows, cols, x)
    if t == Q8_0:
        return oracle.matvec(t, x, data, rows, cols)
    return oracle.matvec_preq(t, data, rows, cols, oracle.quantize_row_q8_k(x))


@pytest.mark.parametrize("tokens", [1, 3, 12])
@pytest.mark.parametrize("q,k,v", [(Q8_0, Q4_K, Q4_K), (Q8_0, Q8_0, Q6_K), (Q1_0, Q8_0, Q4_K), (Q2_0, Q5_K, Q8_0), (TERNARY, Q4_K, Q6_K),
                                   (Q1_0, TERNARY, Q1_0), (Q4_K, Q8_0, Q5_K)])
def test_rows_of_the_cache(oracle, q, k, v, tokens):
    from alice_llm_b200.gpu import GpuEngine, GpuModel
    cfg = dict(num_layers=2, hidden_dim=512, intermediate_dim=1024, num_heads=4, num_kv_heads=2, head_dim=128, vocab_size=300, max_seq_len=64,
               rope_theta=500000.0, eps=1e-5)
    rng = np.random.default_rng(11)
    model = synth.make_llama(rng, cfg, {"q": q, "k": k, "v": v})
    eng = GpuEngine(0)
    gm = GpuModel.load(eng, model)
    toks = rng.integers(0, 300, tokens).tolist()
    gm.forward_and_read(7)       # leaves vectors of its own in every buffer
    gm.reset()
    gm.forward_rows(toks, [tokens - 1])
    got_k, got_v = gm.kv_read(0, 0, tokens)
    L, H = model["layers"][0], cfg["hidden_dim"]
    table = oracle.dequantize(Q8_0, model["embedding"][1]).reshape(-1, H)
    for i, t in enumerate(toks):
        x = oracle.rms_norm(table[t], L["attn_norm"], cfg["eps"])
        for name, entry, got in (("k", L["k"], got_k[i]), ("v", L["v"], got_v[i])):
            if name == "k" and i:
                continue         # rotated
            want = np.asarray(expect(oracle, entry, x, 256, H), np.float64)
            assert np.linalg.norm(got - want) <= 1e-3 * np.linalg.norm(want), (name, i)
    gm.free()
    eng.close()
