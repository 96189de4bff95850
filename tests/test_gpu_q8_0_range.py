"""Q8_0 keeps f32 activations, whatever lies beside them in a vector and however many vectors there are: one element far above the
others, infinities, magnitudes down to the smallest f32 numbers. Against 64-bit numpy, for the kernel of a single vector of most widths,
the one of several vectors, and a width (5120) at which a single vector takes the latter too.

Bound: a product rounds once and a row adds its terms in some order: 2^-23 of the sum of their magnitudes, at most 8 times for the length of
the chains; where numbers are that small, 2^-149 for every term."""
import numpy as np
import pytest

from alice_llm_b200 import synth

pytestmark = pytest.mark.gpu
ROWS = 200


@pytest.fixture(scope="module")
def eng():
    from alice_llm_b200.gpu import GpuEngine
    e = GpuEngine(0)
    yield e
    e.close()


def run(eng, data, x, rows=ROWS):
    from alice_llm_b200.gpu import GpuQuantType as Q
    batch, cols = x.shape
    w = eng.upload_weights_typed(data, rows, cols, Q.Q8_0)
    y = eng.alloc_f32(batch * rows)
    eng.matvec_dev(w, eng.upload_f32(x.reshape(-1)), y, batch)
    got = eng.read_f32(y).reshape(batch, rows)
    eng.sync()
    return got, eng.dequantize(w).reshape(rows, cols).astype(np.float64)


def check(got, dense, x):
    x = x.astype(np.float64)
    bound = 8 * 2.0 ** -23 * (np.abs(x) @ np.abs(dense).T) + x.shape[1] * 2.0 ** -149
    err = np.abs(got - x @ dense.T)
    assert (err <= bound).all(), f"{(err / bound).max():.3g} of the bound"


@pytest.mark.parametrize("batch", [1, 2, 3, 8])
@pytest.mark.parametrize("cols", [512, 4096, 5120])
@pytest.mark.parametrize("ratio", [1e4, 1e6, 1e9])
def test_one_large_element(eng, cols, batch, ratio):
    """Its column holds zero weights, so nothing of it is in the results."""
    rng = np.random.default_rng(cols + batch)
    data = synth.make_q8_0(rng, ROWS, cols)
    at = cols // 2 + 5
    data.reshape(ROWS, cols // 32, 34)[:, at // 32, 2 + at % 32] = 0
    x = synth.make_x(rng, cols, batch).reshape(batch, cols)
    x[:, at] = ratio
    got, dense = run(eng, data, x)
    check(got, dense, x)


@pytest.mark.parametrize("batch", [1, 2, 4, 8])
@pytest.mark.parametrize("cols", [512, 4096, 5120])
def test_infinities(eng, cols, batch):
    """A row's result has the sign of its weight at the infinite element, or is not a number where that weight is zero; the neighbours'
    results are what they are."""
    rng = np.random.default_rng(3)
    data = synth.make_q8_0(rng, ROWS, cols)
    data.reshape(ROWS, cols // 32, 34)[:7, 1, 2 + 9] = 0
    x = synth.make_x(rng, cols, batch).reshape(batch, cols)
    x[-1, 32 + 9] = -np.inf
    got, dense = run(eng, data, x)
    want = dense[:, 32 + 9]
    assert np.isnan(got[-1][want == 0]).all() and (got[-1][want > 0] == -np.inf).all() and (got[-1][want < 0] == np.inf).all()
    if batch > 1:
        check(got[:-1], dense, x[:-1])


@pytest.mark.parametrize("batch", [1, 3, 8])
@pytest.mark.parametrize("cols", [512, 4096, 5120])
@pytest.mark.parametrize("size", [1e30, 1e-30, 1e-37, 1e-41])
def test_magnitudes(eng, cols, batch, size):
    rng = np.random.default_rng(cols + batch)
    data = synth.make_q8_0(rng, ROWS, cols)
    x = (synth.make_x(rng, cols, batch).reshape(batch, cols).astype(np.float64) * size).astype(np.float32)
    got, dense = run(eng, data, x)
    check(got, dense, x)
