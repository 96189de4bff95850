"""Ternary planes and packed codes over 1..8 vectors (csrc/gemv_planes.cu) against 64-bit numpy at the edges of its tiles (16 rows),
segments (512 / 256 columns), word and vector loads, column splits over a cluster and pairs of vectors.

Bound: an activation is rounded to 2^-20 of the largest of its vector, the integer sum is exact and two f32 roundings follow."""
import numpy as np
import pytest

from alice_llm_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    from alice_llm_b200.gpu import GpuEngine
    e = GpuEngine(0)
    yield e
    e.close()


def dense(m, cols):
    p, n = (np.unpackbits(a, axis=1, bitorder="little")[:, :cols].astype(np.float64) for a in m[:2])
    return p - n


def upload(eng, oracle, m, rows, cols, sparse):
    if not sparse:
        return eng.upload_ternary(*m, rows, cols)
    active, sign = synth.ternary_to_sparse(m[0], m[1], cols)
    return eng.upload_sparse_ternary(oracle.sparse_pack_2bit(active, sign, rows, cols), m[2], rows, cols)


def check(got, x, m, cols):
    t = dense(m, cols)
    s = x.astype(np.float64) @ t.T
    scale = m[2].astype(np.float64)
    bound = scale * (np.abs(t).sum(1) * np.abs(x).max(1, keepdims=True) * 2.0 ** -20 + np.abs(s) * 2.0 ** -22) + 1e-30
    err = np.abs(got - s * scale)
    assert (err <= bound).all(), f"{(err / bound).max():.2f} of the bound"


@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("rows,cols", [(1, 32), (17, 35), (16, 512), (15, 516), (33, 1024), (300, 8192 + 32), (2500, 256), (40, 28672), (4099, 2048 + 160)])
def test_planes_every_batch(eng, oracle, rows, cols, sparse):
    rng = np.random.default_rng(rows * 7 + cols)
    m = synth.make_ternary(rng, rows, cols)
    w = upload(eng, oracle, m, rows, cols, sparse)
    x = synth.make_x(rng, cols, 8).reshape(8, cols) * (10.0 ** rng.integers(-3, 4, (8, 1))).astype(np.float32)
    xd, y = eng.upload_f32(x.reshape(-1)), eng.alloc_f32(8 * rows)
    alone = []
    for batch in (1, 2, 3, 5, 8):
        eng.matvec_dev(w, xd, y, batch)
        got = eng.read_f32(y)[:batch * rows].reshape(batch, rows)
        eng.sync()
        check(got, x[:batch], m, cols)
        alone.append(got)
    for a in alone:         # integer sums: a vector's result does not depend on its company
        assert np.array_equal(a, alone[-1][:len(a)])


@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("value", [0.9, -0.9999])
def test_equal_signs_over_equal_activations(eng, oracle, sparse, value):
    """The largest sums there are: they need more than 32 bits in fixed-point units."""
    rows, cols = 20, 28672
    pos = np.full((rows, cols // 8), 255, np.uint8)
    pos[1::2] = 0
    m = (pos, 255 - pos, np.ones(rows, np.float32))
    x = np.full((3, cols), value, np.float32)
    w, y = upload(eng, oracle, m, rows, cols, sparse), eng.alloc_f32(3 * rows)
    eng.matvec_dev(w, eng.upload_f32(x.reshape(-1)), y, 3)
    got = eng.read_f32(y).reshape(3, rows)
    eng.sync()
    check(got, x, m, cols)


@pytest.mark.parametrize("rows,cols,batch", [(17, 544, 1), (1000, 4096, 3), (150, 8192, 8), (40, 28672, 8)])
def test_planes_swiglu(eng, oracle, rows, cols, batch):
    rng = np.random.default_rng(rows + cols)
    g, u = synth.make_ternary(rng, rows, cols), synth.make_ternary(rng, rows, cols)
    x = synth.make_x(rng, cols, batch).reshape(batch, cols)
    y = eng.alloc_f32(rows * batch)
    eng.swiglu_dev(upload(eng, oracle, g, rows, cols, False), upload(eng, oracle, u, rows, cols, False), eng.upload_f32(x.reshape(-1)), y, batch)
    got = eng.read_f32(y).reshape(batch, rows)
    eng.sync()
    a, b = (x.astype(np.float64) @ (dense(m, cols) * m[2].astype(np.float64)[:, None]).T for m in (g, u))
    off = [m[2].astype(np.float64) * (np.abs(dense(m, cols)).sum(1) * np.abs(x).max(1, keepdims=True) * 2.0 ** -20) for m in (g, u)]
    silu = a / (1.0 + np.exp(-a))
    bound = 1.1 * off[0] * np.abs(b) + np.abs(silu) * off[1] + 2.0 ** -20 * np.abs(silu * b) + 1e-30
    assert (np.abs(got - silu * b) <= bound).all()


@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("size", [1e-30, 1e-35, 1e-38, 1e-42])
def test_small_activations(eng, oracle, sparse, size):
    """Down to the smallest f32 numbers. A unit is never below 2^-149, and an element is a multiple of up to 2^6 of them (the place of its
    bit in a byte): half of that on top of the bound above."""
    rng = np.random.default_rng(9)
    rows, cols = 40, 1024
    m = synth.make_ternary(rng, rows, cols)
    w = upload(eng, oracle, m, rows, cols, sparse)
    x = (synth.make_x(rng, cols, 3).reshape(3, cols).astype(np.float64) * size).astype(np.float32)
    for batch in (1, 3):
        y = eng.alloc_f32(batch * rows)
        eng.matvec_dev(w, eng.upload_f32(x.reshape(-1)), y, batch)
        got = eng.read_f32(y).reshape(batch, rows)
        eng.sync()
        t, scale = dense(m, cols), m[2].astype(np.float64)
        s = x[:batch].astype(np.float64) @ t.T
        unit = np.maximum(np.abs(x[:batch]).max(1, keepdims=True) * 2.0 ** -20, 2.0 ** -144)
        bound = scale * (np.abs(t).sum(1) * unit + np.abs(s) * 2.0 ** -22) + 2.0 ** -148
        assert (np.abs(got - s * scale) <= bound).all(), batch
