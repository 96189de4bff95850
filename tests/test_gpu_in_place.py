"""K-quant products whose result takes the place of their vector, or of a part of it: all of x counts as it was before the call. Sizes on both sides
of the rule by which a product quantizes its vector itself; the same bits as with memory of its own."""
import numpy as np
import pytest

from alice_llm_b200 import synth
from alice_llm_b200.gpu import GpuQuantType as Q

pytestmark = pytest.mark.gpu
TYPES = {synth.Q4_K: Q.Q4K, synth.Q5_K: Q.Q5K, synth.Q6_K: Q.Q6K}


@pytest.fixture(scope="module")
def eng():
    from alice_llm_b200.gpu import GpuEngine
    e = GpuEngine(0)
    yield e
    e.close()


@pytest.mark.parametrize("qtype", list(TYPES))
@pytest.mark.parametrize("swiglu", [False, True])
@pytest.mark.parametrize("rows,cols,first", [(4096, 4096, 0), (256, 256, 0), (2048, 4096, 1000), (6000, 4096, 4092), (3000, 4096, 2996), (8192, 8192, 0), (800, 8192, 40)])
def test_result_over_the_vector(eng, qtype, swiglu, rows, cols, first):
    """The result begins at element `first` of the vector, then the vector at that element of the result."""
    import torch
    rng = np.random.default_rng(rows + cols + first)
    w, u = (eng.upload_weights_typed(synth.make_weights(qtype, rng, rows, cols), rows, cols, TYPES[qtype]) for _ in range(2))
    call = (lambda x, y: eng.swiglu_dev(w, u, x, y, 1)) if swiglu else (lambda x, y: eng.matvec_dev(w, x, y, 1))
    v = synth.make_x(rng, cols)
    apart = eng.alloc_f32(rows)
    call(eng.upload_f32(v), apart)
    want = eng.read_f32(apart).copy()
    for xo, yo in ((0, first), (first, 0)):
        mem = torch.zeros(rows + cols + first, device="cuda")
        x, y = (eng.buf_from_device(mem.data_ptr() + 4 * o, n) for o, n in ((xo, cols), (yo, rows)))
        for _ in range(3):
            mem[xo:xo + cols] = torch.from_numpy(v).cuda()
            torch.cuda.synchronize()
            call(x, y)
            eng.sync()
            assert np.array_equal(mem[yo:yo + rows].cpu().numpy().view(np.uint32), want.view(np.uint32)), (xo, yo)
    w.free(), u.free()
