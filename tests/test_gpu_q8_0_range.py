"""Q8_0 keeps f32 activations, whatever lies beside them in a vector and however many vectors there are: one element far above the
others, infinities, magnitudes down to the smallest f32 numbers. Against 64-bit numpy, for the kernel of a single vector, the one of
several, and the single vectors that the latter takes: large matrices (96 MB) of widths that are no power of two.

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


@pytest.mark.parametrize("rows,cols", [(71003, 1280), (80999, 1120), (17701, 5120)])
def test_one_vector_of_a_large_matrix(eng, rows, cols):
    """Some of the rows: the first and the last tiles and every 997th."""
    from alice_llm_b200.gpu import GpuQuantType as Q
    rng = np.random.default_rng(cols)
    data = rng.integers(0, 256, (rows, cols // 32, 34), dtype=np.uint8)
    data[:, :, 0:2] = rng.uniform(0.001, 0.01, (rows, cols // 32)).astype(np.float16).view(np.uint8).reshape(rows, cols // 32, 2)
    at = cols // 2 + 5
    data[:, at // 32, 2 + at % 32] = 0
    data[:rows // 2, 1, 2 + 9] = 0
    w = eng.upload_weights_typed(data.reshape(-1), rows, cols, Q.Q8_0)
    some = np.unique(np.r_[0:40, 40:rows:997, rows - 40:rows])
    dense = eng.dequantize(w).reshape(rows, cols)[some].astype(np.float64)
    y = eng.alloc_f32(rows)
    base = synth.make_x(rng, cols)
    for change, size in ((None, 1.0), (1e6, 1.0), (None, 1e-37), (np.inf, 1.0)):
        x = (base.astype(np.float64) * size).astype(np.float32).reshape(1, cols)
        if change is not None:
            x[0, at if np.isfinite(change) else 32 + 9] = change
        eng.matvec_dev(w, eng.upload_f32(x.reshape(-1)), y, 1)
        got = eng.read_f32(y)[some].reshape(1, -1)
        eng.sync()
        if change is None or np.isfinite(change):
            check(got, dense, x)
        else:
            want = dense[:, 32 + 9]
            assert np.isnan(got[0][want == 0]).all() and (got[0][want > 0] == np.inf).all() and (got[0][want < 0] == -np.inf).all()
    w.free()
