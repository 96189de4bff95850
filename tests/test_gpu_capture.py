"""Products inside a stream capture of the caller's: after one call of a matrix its scratch is there for every number of vectors."""
import numpy as np
import pytest

from alice_llm_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("qtype", [synth.Q8_0, synth.Q1_0, synth.Q2_0, synth.TERNARY])
def test_batch_behind_a_single_vector(qtype):
    import torch
    from alice_llm_b200.gpu import GpuEngine, GpuQuantType as Q
    rng = np.random.default_rng(qtype % 100)
    rows, cols, batch = 300, 8192, 8
    eng = GpuEngine(0)
    data = synth.make_weights(qtype, rng, rows, cols)
    w = eng.upload_ternary(*data, rows, cols) if qtype == synth.TERNARY else eng.upload_weights_typed(
        data, rows, cols, {synth.Q8_0: Q.Q8_0, synth.Q1_0: Q.Q1_0, synth.Q2_0: Q.Q2_0}[qtype])
    x = synth.make_x(rng, cols, batch)
    xd, y = eng.upload_f32(x), eng.alloc_f32(batch * rows)
    eng.matvec_dev(w, xd, y, 1)
    eng.sync()
    stream = torch.cuda.Stream()
    eng.set_stream(stream.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        eng.matvec_dev(w, xd, y, batch)
    graph.replay()
    torch.cuda.synchronize()
    got = eng.read_f32(y).copy()
    eng.write_f32(y, np.zeros(batch * rows, np.float32))
    eng.matvec_dev(w, xd, y, batch)
    assert np.array_equal(got, eng.read_f32(y))
    eng.sync()
    eng.close()


TYPES = {synth.Q4_K: "Q4K", synth.Q5_K: "Q5K", synth.Q6_K: "Q6K"}


@pytest.mark.parametrize("qtype", list(TYPES))
@pytest.mark.parametrize("rows,cols,launches", [(3000, 1024, {4: 1, 5: 1, 6: 1}), (700, 4096, {4: 2, 5: 2, 6: 1}), (300, 8192, {4: 2, 5: 2, 6: 2}), (5700, 3072, {4: 2, 5: 1, 6: 1}), (5800, 3072, {4: 1, 5: 1, 6: 1})])
def test_k_quant_vectors(qtype, rows, cols, launches):
    """One vector: captured before there is scratch, then behind a first call by the rule for replays, and replayed after the scratch has grown"""
    import torch
    from alice_llm_b200.gpu import GpuEngine, GpuQuantType as Q
    from graph_kernels import block_sizes
    rng = np.random.default_rng(rows)
    eng = GpuEngine(0)
    upload = lambda r, c: eng.upload_weights_typed(synth.make_weights(qtype, rng, r, c), r, c, getattr(Q, TYPES[qtype]))
    w, wide = upload(rows, cols), upload(64, 16384)
    x, y = eng.upload_f32(synth.make_x(rng, cols)), eng.alloc_f32(rows)
    assert len(block_sizes(eng, lambda: eng.matvec_dev(w, x, y, 1))) == 1
    eng.matvec_dev(w, x, y, 1)
    want = eng.read_f32(y).copy()
    eng.sync()
    assert len(block_sizes(eng, lambda: eng.matvec_dev(w, x, y, 1))) == launches[int(TYPES[qtype][1])]
    stream = torch.cuda.Stream()
    eng.set_stream(stream.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        eng.matvec_dev(w, x, y, 1)
    eng.matvec_dev(wide, eng.upload_f32(synth.make_x(rng, 8 * 16384)), eng.alloc_f32(8 * 64), 8)
    eng.write_f32(y, np.zeros(rows, np.float32))
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(eng.read_f32(y), want)
    eng.close()


@pytest.mark.parametrize("qtype", list(TYPES))
def test_large_product_behind_a_small_one(qtype):
    """A first call that quantizes in the product leaves the scratch that a captured product of its width needs"""
    from alice_llm_b200.gpu import GpuEngine, GpuQuantType as Q
    from graph_kernels import block_sizes
    rng = np.random.default_rng(5)
    eng = GpuEngine(0)
    small, large = (eng.upload_weights_typed(synth.make_weights(qtype, rng, r, 4096), r, 4096, getattr(Q, TYPES[qtype])) for r in (256, 14336))
    x, y = eng.upload_f32(synth.make_x(rng, 4096)), eng.alloc_f32(14336)
    eng.matvec_dev(small, x, y, 1)
    eng.sync()
    assert len(block_sizes(eng, lambda: eng.matvec_dev(large, x, y, 1))) == 2
    eng.close()
