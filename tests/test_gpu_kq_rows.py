"""K-quants over 2..8 vectors (csrc/gemv_kq_rows.cu) against the kernel of a single vector, which other files hold against the oracle:
edges of the 16-row tiles, of the one- or two-block stages, of the column split over a cluster, rows that begin anywhere, more tiles than
the CTAs of a launch have room for (180003 rows of Q5_K).

Both keep the integer block dots; a row adds the scale and the min term of every block in f32, in another order. Either term is up to
a few times what is left of both (4), and a chain of them rounds a few times (8): 32 times 2^-23 of the sum of magnitudes."""
import numpy as np
import pytest

from alice_llm_b200 import synth

pytestmark = pytest.mark.gpu
Q4_K, Q5_K, Q6_K = synth.Q4_K, synth.Q5_K, synth.Q6_K


@pytest.fixture(scope="module")
def eng():
    from alice_llm_b200.gpu import GpuEngine
    e = GpuEngine(0)
    yield e
    e.close()


def quant(qtype):
    from alice_llm_b200.gpu import GpuQuantType as Q
    return {Q4_K: Q.Q4K, Q5_K: Q.Q5K, Q6_K: Q.Q6K}[qtype]


@pytest.mark.parametrize("qtype", [Q4_K, Q5_K, Q6_K])
@pytest.mark.parametrize("rows,blocks", [(1, 1), (15, 2), (16, 3), (17, 7), (300, 16), (2500, 1), (40, 56), (4099, 5), (180003, 1)])
def test_every_batch(eng, qtype, rows, blocks):
    cols = 256 * blocks
    rng = np.random.default_rng(rows + cols)
    w = eng.upload_weights_typed(synth.make_weights(qtype, rng, rows, cols), rows, cols, quant(qtype))
    mag = np.abs(eng.dequantize(w).reshape(rows, cols)).astype(np.float64)
    x = synth.make_x(rng, cols, 8).reshape(8, cols)
    y = eng.alloc_f32(8 * rows)
    one = []
    for k in range(8):
        eng.matvec_dev(w, eng.upload_f32(x[k]), y, 1)
        one.append(eng.read_f32(y)[:rows].copy())
        eng.sync()
    bound = 32 * 2.0 ** -23 * (1.1 * np.abs(x) @ mag.T) + 1e-30
    xd = eng.upload_f32(x.reshape(-1))
    for batch in (2, 3, 5, 8):
        eng.matvec_dev(w, xd, y, batch)
        got = eng.read_f32(y)[:batch * rows].reshape(batch, rows).astype(np.float64)
        eng.sync()
        err = np.abs(got - np.array(one[:batch], np.float64)) / bound[:batch]
        assert err.max() <= 1.0, (batch, err.max())


@pytest.mark.parametrize("qtype", [Q4_K, Q5_K, Q6_K])
@pytest.mark.parametrize("swiglu", [False, True])
@pytest.mark.parametrize("cols,limit", [(256, 28000000), (4096, 28000000), (4352, 8000000), (8192, 8000000), (8448, 0)])
def test_vector_quantized_in_the_product(eng, qtype, swiglu, cols, limit):
    """A small product makes the Q8_K blocks of its vector itself: the same bits as from blocks made ahead, on both sides of the limits"""
    rng = np.random.default_rng(cols)
    most = limit // (synth.row_bytes(qtype, cols) * (2 if swiglu else 1))
    x = eng.upload_f32(synth.make_x(rng, cols))
    q = eng.alloc_q8k(cols, 1)
    eng.quantize_q8k(x, q)
    for rows in (5, most, most + 1) if cols > 256 and limit else (5, 3000):
        w, u = (eng.upload_weights_typed(synth.make_weights(qtype, rng, rows, cols), rows, cols, quant(qtype)) for _ in range(2))
        y = eng.alloc_f32(rows)
        out = []
        for product in (lambda: eng.swiglu_dev(w, u, x, y, 1), lambda: eng.swiglu_preq_dev(w, u, q, y)) if swiglu else (lambda: eng.matvec_dev(w, x, y, 1), lambda: eng.matvec_preq_dev(w, q, y)):
            product()
            out.append(eng.read_f32(y).view(np.uint32).copy())
            eng.sync()
        assert np.array_equal(out[0], out[1]), rows
        w.free(), u.free()


@pytest.mark.parametrize("qtype", [Q4_K, Q5_K, Q6_K])
@pytest.mark.parametrize("rows,cols,swiglu", [(28672, 8192, False), (28672, 8192, True), (8192, 28672, False), (128256, 4096, False)])
def test_one_pass_at_the_largest_sizes(eng, qtype, rows, cols, swiglu):
    w = eng.upload_weights_typed(np.zeros(rows * synth.row_bytes(qtype, cols), np.uint8), rows, cols, quant(qtype))
    for batch in (2, 3, 8):
        assert eng.batch_plan(w, batch, swiglu=swiglu)[1] == 1, batch
    w.free()


def test_plan_follows_the_kernels(eng):
    """alice_batch_plan: (launches, passes over the weights) of what really runs, for one vector too."""
    from alice_llm_b200.gpu import GpuQuantType as Q
    def plan(t, q, rows, cols, batch, swiglu=False):
        w = eng.upload_weights_typed(np.zeros(rows * synth.row_bytes(t, cols), np.uint8), rows, cols, q)
        return eng.batch_plan(w, batch, swiglu=swiglu)
    assert plan(synth.Q1_0, Q.Q1_0, 256, 28672, 1) == (1, 1)          # the ring kernel would take two column chunks
    assert plan(synth.Q2_0, Q.Q2_0, 256, 28672, 1) == (1, 1)
    assert plan(Q5_K, Q.Q5K, 180000, 256, 8) == (2, 1)                # one pass, the rows over two launches
    assert plan(Q5_K, Q.Q5K, 180000, 256, 1) == (1, 1)
    assert plan(synth.Q8_0, Q.Q8_0, 256, 4096, 8) == (1, 1)
    planes = [np.zeros((256, 28672 // 8), np.uint8)] * 2 + [np.ones(256, np.float32)]
    w = eng.upload_ternary(*planes, 256, 28672)
    assert eng.batch_plan(w, 1) == (1, 1) and eng.batch_plan(w, 8) == (1, 1)
