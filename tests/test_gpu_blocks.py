"""Q8_0, Q1_0 and Q2_0 over 1..8 vectors (csrc/gemv_blocks.cu) against 64-bit numpy at the edges of its tiles (16 rows), stages
(8 blocks), 16-byte pieces (rows that start anywhere), column splits over a cluster and pairs of vectors.

Bound: for the bits of the one- and two-bit codes an activation is rounded to 2^-23 of a power of two above the largest of its vector
(2^-30, divided by up to 2^7 first); block sums are exact and rounded to f32 once, and a row adds as many terms as it has blocks, in any
order: 2^-23 of the sum of their magnitudes, times at most 8 for the length of the chains. Q8_0 rounds no activation."""
import numpy as np
import pytest

from alice_llm_b200 import synth

pytestmark = pytest.mark.gpu
Q8_0, Q1_0, Q2_0 = synth.Q8_0, synth.Q1_0, synth.Q2_0


@pytest.fixture(scope="module")
def eng():
    from alice_llm_b200.gpu import GpuEngine
    e = GpuEngine(0)
    yield e
    e.close()


def quant(qtype):
    from alice_llm_b200.gpu import GpuQuantType as Q
    return {Q8_0: Q.Q8_0, Q1_0: Q.Q1_0, Q2_0: Q.Q2_0}[qtype]


def exact(qtype, w, x):
    """x [n, cols], dequantized w [rows, cols] -> sums, bounds"""
    x = x.astype(np.float64)
    s, mag = x @ w.T, np.abs(x) @ np.abs(w).T
    fixed = (0.0 if qtype == Q8_0 else 2.0 ** -23) * 2.0 * np.abs(x).max(1, keepdims=True) * np.abs(w).sum(1)
    return s, fixed + 8 * 2.0 ** -23 * mag + 1e-30


@pytest.mark.parametrize("qtype", [Q8_0, Q1_0, Q2_0])
@pytest.mark.parametrize("rows,blocks", [(1, 1), (17, 7), (16, 8), (15, 9), (33, 16), (300, 33), (2500, 2), (40, 224), (4099, 24)])
def test_blocks_every_batch(eng, oracle, qtype, rows, blocks):
    cols = blocks * (32 if qtype == Q8_0 else 128)
    rng = np.random.default_rng(rows * 7 + cols)
    data = synth.make_weights(qtype, rng, rows, cols)
    w = eng.upload_weights_typed(data, rows, cols, quant(qtype))
    dense = eng.dequantize(w).reshape(rows, cols).astype(np.float64)      # bit-exact against the oracle elsewhere
    x = synth.make_x(rng, cols, 8).reshape(8, cols) * (10.0 ** rng.integers(-3, 4, (8, 1))).astype(np.float32)
    s, bound = exact(qtype, dense, x)
    xd, y = eng.upload_f32(x.reshape(-1)), eng.alloc_f32(8 * rows)
    for batch in (1, 2, 3, 5, 8):
        eng.matvec_dev(w, xd, y, batch)
        got = eng.read_f32(y)[:batch * rows].reshape(batch, rows)
        eng.sync()
        err = np.abs(got - s[:batch]) / bound[:batch]
        assert err.max() <= 1.0, (batch, err.max())


@pytest.mark.parametrize("qtype", [Q8_0, Q1_0, Q2_0])
@pytest.mark.parametrize("rows,cols,batch", [(17, 1024 + 128, 1), (1000, 4096, 3), (150, 8192, 8)])
def test_blocks_swiglu(eng, qtype, rows, cols, batch):
    rng = np.random.default_rng(rows + cols)
    g, u = (eng.upload_weights_typed(synth.make_weights(qtype, rng, rows, cols), rows, cols, quant(qtype)) for _ in range(2))
    x = synth.make_x(rng, cols, batch).reshape(batch, cols)
    y = eng.alloc_f32(rows * batch)
    eng.swiglu_dev(g, u, eng.upload_f32(x.reshape(-1)), y, batch)
    got = eng.read_f32(y).reshape(batch, rows)
    eng.sync()
    (a, da), (b, db) = (exact(qtype, eng.dequantize(m).reshape(rows, cols).astype(np.float64), x) for m in (g, u))
    sig = 1.0 / (1.0 + np.exp(-a))
    assert (np.abs(got - a * sig * b) <= 1.1 * da * np.abs(b) + np.abs(a * sig) * db + 2.0 ** -20 * np.abs(a * sig * b) + 1e-30).all()


@pytest.mark.parametrize("qtype", [Q1_0, Q2_0])
def test_vectors_that_are_not_finite(eng, qtype):
    """Such a vector has no fixed-point form: its results are NaN, its neighbours' are what they are."""
    rng = np.random.default_rng(3)
    rows, cols = 40, 512
    w = eng.upload_weights_typed(synth.make_weights(qtype, rng, rows, cols), rows, cols, quant(qtype))
    x = synth.make_x(rng, cols, 4).reshape(4, cols)
    x[1, 77], x[2, 500] = np.inf, np.nan
    y = eng.alloc_f32(rows * 4)
    eng.matvec_dev(w, eng.upload_f32(x.reshape(-1)), y, 4)
    got = eng.read_f32(y).reshape(4, rows)
    eng.sync()
    assert np.isnan(got[1]).all() and np.isnan(got[2]).all()
    s, bound = exact(qtype, eng.dequantize(w).reshape(rows, cols).astype(np.float64), x[[0, 3]])
    assert (np.abs(got[[0, 3]] - s) <= bound).all()


@pytest.mark.parametrize("qtype", [Q1_0, Q2_0])
@pytest.mark.parametrize("size", [1e-28, 1e-33, 1e-40])
def test_small_activations(eng, qtype, size):
    """Units are never below 2^-149, and an element is a multiple of up to 2^7 of them (the place of its bit in a byte)."""
    rng = np.random.default_rng(4)
    rows, cols = 40, 1024
    w = eng.upload_weights_typed(synth.make_weights(qtype, rng, rows, cols), rows, cols, quant(qtype))
    dense = eng.dequantize(w).reshape(rows, cols).astype(np.float64)
    x = (synth.make_x(rng, cols, 3).reshape(3, cols).astype(np.float64) * size).astype(np.float32)
    for batch in (1, 3):
        y = eng.alloc_f32(batch * rows)
        eng.matvec_dev(w, eng.upload_f32(x.reshape(-1)), y, batch)
        got = eng.read_f32(y).reshape(batch, rows)
        eng.sync()
        s, bound = exact(qtype, dense, x[:batch])
        assert (np.abs(got - s) <= bound - 1e-30 + 2.0 ** -143 * np.abs(dense).sum(1) + 2.0 ** -148).all(), batch
