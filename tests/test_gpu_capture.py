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
