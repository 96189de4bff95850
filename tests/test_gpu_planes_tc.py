"""Ternary planes and packed codes of larger matrices over three vectors and more (csrc/gemv_planes_tc.cu): rows dealt unevenly, ragged last tiles, columns
that end inside a segment, fewer segments than a cluster has CTAs, more tiles than accumulators fit (two launches), gate and up, three matrices in one launch.

Sums are integers and activations are rounded alike, so every vector's result equals, to the bit, that of the vector alone, which
tests/test_gpu_planes.py holds against 64-bit numpy."""
import numpy as np
import pytest

from alice_llm_b200 import synth
from graph_kernels import block_sizes
from softmodel import SMOOTH_MIX, soft_model
from test_gpu_planes import upload

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    from alice_llm_b200.gpu import GpuEngine
    e = GpuEngine(0)
    yield e
    e.close()


def run(eng, call, x, rows):
    """x [batch, cols] through `call` at once and one by one."""
    y = eng.alloc_f32(len(x) * rows)
    call(eng.upload_f32(x.reshape(-1)), y, len(x))
    got = eng.read_f32(y)[:len(x) * rows].reshape(len(x), rows).copy()
    for k in range(len(x)):
        call(eng.upload_f32(x[k]), y, 1)
        one = eng.read_f32(y)[:rows]
        eng.sync()
        assert np.array_equal(got[k], one), (k, np.abs(got[k] - one).max())


@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("rows,cols,batch", [(4097, 8192, 5), (16500, 1152, 8), (2300, 7808, 6), (9001, 8192, 3), (70000, 512, 7), (300000, 256, 8), (700, 28672, 8), (18000, 4096, 4)])
def test_as_alone(eng, oracle, rows, cols, batch, sparse):
    rng = np.random.default_rng(rows + cols + batch)
    m = synth.make_ternary(rng, rows, cols)
    w = upload(eng, oracle, m, rows, cols, sparse)
    x = synth.make_x(rng, cols, batch).reshape(batch, cols) * (10.0 ** rng.integers(-3, 4, (batch, 1))).astype(np.float32)
    run(eng, lambda xd, y, n: eng.matvec_dev(w, xd, y, n), x, rows)
    w.free()


@pytest.mark.parametrize("rows,cols,batch", [(3000, 4224, 8), (6001, 8192, 3), (20000, 8192, 8)])
def test_gate_and_up(eng, oracle, rows, cols, batch):
    rng = np.random.default_rng(rows)
    g, u = (upload(eng, oracle, synth.make_ternary(rng, rows, cols), rows, cols, False) for _ in range(2))
    x = synth.make_x(rng, cols, batch).reshape(batch, cols)
    run(eng, lambda xd, y, n: eng.swiglu_dev(g, u, xd, y, n), x, rows)
    g.free(), u.free()


def test_not_finite_stays_with_its_vector(eng, oracle):
    rng = np.random.default_rng(3)
    rows, cols = 2500, 8192
    w = upload(eng, oracle, synth.make_ternary(rng, rows, cols), rows, cols, False)
    x = synth.make_x(rng, cols, 6).reshape(6, cols)
    x[2, 77] = np.inf
    y = eng.alloc_f32(6 * rows)
    eng.matvec_dev(w, eng.upload_f32(x.reshape(-1)), y, 6)
    got = eng.read_f32(y).reshape(6, rows)
    eng.sync()
    assert np.isnan(got[2]).all() and np.isfinite(np.delete(got, 2, 0)).all()
    w.free()


def test_model_with_three_matrices_in_a_launch(eng):
    """Eight drafted tokens against the same tokens stepped: attention adds in another order, everything else is the same to the bit."""
    from alice_llm_b200.gpu import GpuModel
    cfg = dict(num_layers=1, hidden_dim=4096, intermediate_dim=4096, num_heads=32, num_kv_heads=8, head_dim=128, vocab_size=500, max_seq_len=32,
               rope_theta=500000.0, eps=1e-5)
    model = soft_model(np.random.default_rng(11), cfg, SMOOTH_MIX)
    a, b = GpuModel.load(eng, model), GpuModel.load(eng, model)
    toks = [3, 499, 41, 7, 8, 250, 1, 0]
    got = np.asarray(a.forward_batch_and_read(toks), np.float64).reshape(8, 500)
    want = np.asarray([b.forward_and_read(t) for t in toks], np.float64)
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)
    ka, va = a.kv_read(0, 0, 8)
    kb, vb = b.kv_read(0, 0, 8)
    assert np.array_equal(ka, kb) and np.array_equal(va, vb)      # of the one layer: nothing of attention is in them
    a.free(), b.free()


def test_model_of_few_vectors(eng):
    """Three drafted tokens: 16 digit columns, with the residual of a wide output projection"""
    from alice_llm_b200.gpu import GpuModel
    cfg = dict(num_layers=1, hidden_dim=4096, intermediate_dim=512, num_heads=128, num_kv_heads=16, head_dim=128, vocab_size=500, max_seq_len=16,
               rope_theta=500000.0, eps=1e-5)
    model = soft_model(np.random.default_rng(12), cfg, SMOOTH_MIX)
    a = GpuModel.load(eng, model)
    toks = [3, 499, 41]
    got = np.asarray(a.forward_batch_and_read(toks), np.float64).reshape(3, 500)
    a.reset()
    want = np.asarray([a.forward_and_read(t) for t in toks], np.float64)
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)
    a.free()

TC_THREADS = 672      # of a block of csrc/gemv_planes_tc.cu, and of no other kernel


@pytest.mark.parametrize("rows,cols,batch,sparse,launches", [
    (4097, 8192, 5, False, 1), (2300, 7808, 6, False, 1), (8300, 8192, 3, False, 1), (8300, 8192, 4, False, 1), (70000, 512, 7, False, 1), (300000, 256, 8, False, 2), (60000, 6144, 5, False, 2),
    (4097, 8192, 8, True, 1), (70000, 512, 7, True, 1), (300000, 256, 8, True, 2), (700, 28672, 8, False, 0), (700, 28672, 8, True, 0), (8300, 8192, 2, False, 0), (16500, 1152, 8, False, 0),
    (4097, 8200, 8, False, 0), (7000, 8192, 4, False, 0), (1900, 8192, 5, False, 0)])
def test_kernel_by_size(eng, oracle, rows, cols, batch, sparse, launches):
    """Launches of the tcgen05 kernel: by what the plans cost, none for two vectors, planes that begin off 16-byte boundaries and less than 4 or 16 MB"""
    rng = np.random.default_rng(rows)
    m = synth.make_ternary(rng, rows, cols)
    w = upload(eng, oracle, m, rows, cols, sparse)
    x = synth.make_x(rng, cols, batch).reshape(batch, cols)
    call = lambda xd, y, n: eng.matvec_dev(w, xd, y, n)
    run(eng, call, x, rows)
    xd, y = eng.upload_f32(x.reshape(-1)), eng.alloc_f32(batch * rows)
    assert block_sizes(eng, lambda: call(xd, y, batch)).count(TC_THREADS) == launches
    assert eng.batch_plan(w, batch) == (max(launches, 1), 1)
    w.free()


@pytest.mark.parametrize("rows,cols,batch,sparse,launches", [
    (3000, 4224, 8, False, 1), (6001, 8192, 3, False, 1), (20000, 8192, 8, False, 2), (10000, 4096, 4, False, 1), (3000, 4224, 8, True, 1), (10000, 4096, 6, True, 1), (3500, 13312, 4, True, 1)])
def test_gate_and_up_of_either_format(eng, oracle, rows, cols, batch, sparse, launches):
    rng = np.random.default_rng(rows + batch)
    g, u = (upload(eng, oracle, synth.make_ternary(rng, rows, cols), rows, cols, sparse) for _ in range(2))
    x = synth.make_x(rng, cols, batch).reshape(batch, cols)
    call = lambda xd, y, n: eng.swiglu_dev(g, u, xd, y, n)
    run(eng, call, x, rows)
    xd, y = eng.upload_f32(x.reshape(-1)), eng.alloc_f32(batch * rows)
    assert block_sizes(eng, lambda: call(xd, y, batch)).count(TC_THREADS) == launches
    g.free(), u.free()
