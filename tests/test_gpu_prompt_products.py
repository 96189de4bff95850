"""K-quant products with more than eight vectors (csrc/gemm_kq.cu, csrc/gemm_kq_tc.cu) one by one against 64-bit numpy, from the same
Q8_K blocks: rows and vectors that leave part of every tile (32 to 128 rows, 16 to 128 vectors), one block to 64, the columns of a
tile shared by up to eight CTAs, SwiGLU, a residual, several tiles of each. One to eight vectors (csrc/gemv_stream.cuh, csrc/gemv_kq_rows.cu)
against the same.

The block sums are integers. Up to 64 vectors they are summed in 32 bits and rounded to f32 once; beyond, in f32, exactly up to 2^24. A result
then is a sum of f32 terms: scale times integers (three roundings) and one addition each, nb blocks in any order: 2^-24 of the sum of
their magnitudes, 4 + 2 sqrt(terms) times. A sum that passes 2^24 rounds once more in each of the 16 steps of 16 columns (Q6_K 32), by less
than 2^-23 of what it is by then: test_largest_sums."""
import numpy as np
import pytest

from alice_llm_b200 import synth

pytestmark = pytest.mark.gpu
Q4_K, Q5_K, Q6_K = synth.Q4_K, synth.Q5_K, synth.Q6_K
BYTES = {Q4_K: 144, Q5_K: 176, Q6_K: 210}


@pytest.fixture(scope="module")
def eng():
    from alice_llm_b200.gpu import GpuEngine
    e = GpuEngine(0)
    yield e
    e.close()


def f16(v):
    return np.array([v], np.float16).view(np.uint8)


def upload(eng, qtype, data, rows, cols):
    from alice_llm_b200.gpu import GpuQuantType as Q
    return eng.upload_weights_typed(data, rows, cols, {Q4_K: Q.Q4K, Q5_K: Q.Q5K, Q6_K: Q.Q6K}[qtype])


def integers(eng, qtype, data, rows, cols):
    """-> d, dmin [rows, nb] and scale * quant, min [rows, cols] as integers: the dequantizer with block scales of 1 or 0"""
    blk = data.reshape(-1, BYTES[qtype])
    at = {"d": 208} if qtype == Q6_K else {"d": 0, "dmin": 2}
    field = {k: np.ascontiguousarray(blk[:, o:o + 2]).view(np.float16).astype(np.float64).reshape(rows, -1) for k, o in at.items()}

    def with_scales(d, dmin):
        b = blk.copy()
        b[:, at["d"]:at["d"] + 2] = f16(d)
        if "dmin" in at:
            b[:, at["dmin"]:at["dmin"] + 2] = f16(dmin)
        return eng.dequantize(upload(eng, qtype, b.reshape(-1), rows, cols)).reshape(rows, cols).astype(np.float64)

    main = with_scales(1.0, 0.0)
    mins = -with_scales(0.0, 1.0) if "dmin" in at else np.zeros_like(main)
    return field["d"], field.get("dmin", np.zeros_like(field["d"])), main, mins


def exact(eng, qtype, data, rows, cols, q8):
    """-> sums and bounds [batch, rows]"""
    e, qs, _ = q8
    d, dmin, main, mins = integers(eng, qtype, data, rows, cols)
    batch, nb = e.shape
    s, mag = np.zeros((batch, rows)), np.zeros((batch, rows))
    for b in range(nb):
        c = slice(256 * b, 256 * b + 256)
        x = qs[:, b].astype(np.float64)
        t, m = (x @ main[:, c].T) * d[:, b] * e[:, b:b + 1], (x @ mins[:, c].T) * dmin[:, b] * e[:, b:b + 1]
        s += t - m
        parts = sum(np.abs(x[:, k:k + 64] @ main[:, 256 * b + k:256 * b + k + 64].T) for k in range(0, 256, 64))
        mag += parts * np.abs(d[:, b]) * np.abs(e[:, b:b + 1]) + np.abs(m)
    return s, 2.0 ** -24 * (4 + 2 * np.sqrt(5.0 * nb)) * mag + 1e-30


def run(eng, qtype, data, rows, cols, q8, up=None, resid=None):
    e, qs, bs = q8
    batch = e.shape[0]
    q = eng.upload_q8k(e, qs, bs, cols, batch)
    y = eng.alloc_f32(batch * rows)
    eng.debug_prompt_product(upload(eng, qtype, data, rows, cols), q, y, None if up is None else upload(eng, qtype, up, rows, cols),
                             None if resid is None else eng.upload_f32(resid.reshape(-1)))
    got = eng.read_f32(y).reshape(batch, rows).astype(np.float64)
    eng.sync()
    return got


def vectors(rng, batch, nb):
    qs = rng.integers(-128, 128, (batch, nb, 256)).astype(np.int8)
    e = (rng.uniform(0.5, 1.5, (batch, nb)) * rng.choice([-1.0, 1.0], (batch, nb)) / 100).astype(np.float32)
    return e, qs, qs.reshape(batch, nb, 16, 16).sum(3, dtype=np.int64).astype(np.int16)


BATCHES = [9, 16, 17, 33, 64, 65, 128, 129, 256]


@pytest.mark.parametrize("qtype", [Q4_K, Q5_K, Q6_K])
@pytest.mark.parametrize("rows,nb", [(1, 1), (31, 2), (129, 9), (300, 16), (70, 33), (40, 64), (2500, 3), (9001, 1)])
def test_products(eng, qtype, rows, nb):
    cols, rng = 256 * nb, np.random.default_rng(rows + nb)
    data = synth.make_weights(qtype, rng, rows, cols)
    q8 = vectors(rng, 256, nb)
    s, bound = exact(eng, qtype, data, rows, cols, q8)
    for batch in BATCHES if rows * nb < 4000 else [33, 129]:
        err = np.abs(run(eng, qtype, data, rows, cols, [a[:batch] for a in q8]) - s[:batch]) / bound[:batch]
        assert err.max() <= 1.0, (batch, err.max())


@pytest.mark.parametrize("qtype", [Q4_K, Q5_K, Q6_K])
@pytest.mark.parametrize("rows,nb", [(1, 1), (15, 2), (17, 7), (300, 16), (2500, 1), (40, 56), (4099, 5)])
def test_few_vectors(eng, qtype, rows, nb):
    cols, rng = 256 * nb, np.random.default_rng(rows + nb)
    data = synth.make_weights(qtype, rng, rows, cols)
    q8 = vectors(rng, 8, nb)
    s, bound = exact(eng, qtype, data, rows, cols, q8)
    w, y = upload(eng, qtype, data, rows, cols), eng.alloc_f32(8 * rows)
    for batch in (1, 2, 3, 5, 8):
        e, qs, bs = (a[:batch] for a in q8)
        eng.matvec_preq_dev(w, eng.upload_q8k(e, qs, bs, cols, batch), y)
        got = eng.read_f32(y)[:batch * rows].reshape(batch, rows).astype(np.float64)
        eng.sync()
        err = np.abs(got - s[:batch]) / bound[:batch]
        assert err.max() <= 1.0, (batch, err.max())


@pytest.mark.parametrize("qtype", [Q4_K, Q5_K, Q6_K])
@pytest.mark.parametrize("rows,nb", [(1, 2), (65, 9), (130, 17), (33, 64), (5000, 2)])
@pytest.mark.parametrize("batch", [16, 40, 64, 100, 200])
def test_swiglu(eng, qtype, rows, nb, batch):
    cols, rng = 256 * nb, np.random.default_rng(rows + nb)
    gate, up = synth.make_weights(qtype, rng, rows, cols), synth.make_weights(qtype, rng, rows, cols)
    q8 = vectors(rng, batch, nb)
    q8[0][:] /= np.float32(np.sqrt(cols))
    (g, dg), (u, du) = (exact(eng, qtype, w, rows, cols, q8) for w in (gate, up))
    sig = 1.0 / (1.0 + np.exp(-np.clip(g, -700, 700)))
    got = run(eng, qtype, gate, rows, cols, q8, up)
    bound = 1.1 * dg * (np.abs(u) + du) + np.abs(g * sig) * du + 2.0 ** -20 * np.abs(g * sig * u) + 1e-30
    assert (np.abs(got - g * sig * u) <= bound).all(), (np.abs(got - g * sig * u) / bound).max()


@pytest.mark.parametrize("qtype", [Q4_K, Q5_K, Q6_K])
@pytest.mark.parametrize("rows,nb,batch,swiglu", [(9600, 9, 256, False), (9601, 8, 200, False), (14000, 10, 256, False), (19000, 17, 128, False), (6300, 16, 300, False), (4800, 9, 200, True)])
def test_tiles_over_whole_waves(eng, qtype, rows, nb, batch, swiglu):
    """Up to half a wave of tiles over whole waves of 148: their columns shared by clusters of two to eight, the other tiles whole"""
    cols, rng = 256 * nb, np.random.default_rng(rows + nb)
    gate, up = (synth.make_weights(qtype, rng, rows, cols) for _ in range(2))
    q8 = vectors(rng, batch, nb)
    q8[0][:] /= np.float32(np.sqrt(cols))
    g, dg = exact(eng, qtype, gate, rows, cols, q8)
    got = run(eng, qtype, gate, rows, cols, q8, up if swiglu else None)
    if not swiglu:
        assert (np.abs(got - g) <= dg).all(), (np.abs(got - g) / dg).max()
        return
    u, du = exact(eng, qtype, up, rows, cols, q8)
    sig = 1.0 / (1.0 + np.exp(-np.clip(g, -700, 700)))
    bound = 1.1 * dg * (np.abs(u) + du) + np.abs(g * sig) * du + 2.0 ** -20 * np.abs(g * sig * u) + 1e-30
    assert (np.abs(got - g * sig * u) <= bound).all(), (np.abs(got - g * sig * u) / bound).max()


@pytest.mark.parametrize("qtype", [Q4_K, Q6_K])
@pytest.mark.parametrize("batch", [20, 100])
def test_residual(eng, qtype, batch):
    rows, nb, rng = 200, 18, np.random.default_rng(1)
    data, q8 = synth.make_weights(qtype, rng, rows, 256 * nb), vectors(rng, batch, nb)
    resid = rng.standard_normal((batch, rows)).astype(np.float32) * 100
    s, bound = exact(eng, qtype, data, rows, 256 * nb, q8)
    got = run(eng, qtype, data, rows, 256 * nb, q8, resid=resid)
    assert (np.abs(got - s - resid) <= bound + 2.0 ** -23 * (np.abs(s) + np.abs(resid))).all()


@pytest.mark.parametrize("qtype", [Q4_K, Q5_K, Q6_K])
@pytest.mark.parametrize("nb", [1, 9])
@pytest.mark.parametrize("sign", [1, -1])
def test_largest_sums(eng, qtype, nb, sign):
    """Weights and activations of one sign near their largest values: block sums of up to 2^27, odd ones among them. All terms have the sign of
    the sum, so what every step may lose is a share of the result."""
    rows, batch, rng = 150, 100, np.random.default_rng(nb)
    blk = synth.make_weights(qtype, rng, rows, 256 * nb).reshape(-1, BYTES[qtype])
    high = lambda n, lo, hi: rng.integers(lo, hi, (len(blk), n)).astype(np.uint8)
    if qtype == Q6_K:      # quants of -32 .. -29 (low nibble 0 .. 3, high bits 0) times scales of -128 .. -120
        blk[:, :128] = high(128, 0, 4) | (high(128, 0, 4) << 4)
        blk[:, 128:192] = 0
        blk[:, 192:208] = (256 - high(16, 120, 128).astype(np.int64)).astype(np.uint8)
        blk[:, 208:210] = f16(2.0 ** -10)
    else:                  # scales of 62 or 63, mins of 0 .. 3, nibbles of 12 .. 15, fifth bits set
        sc, mn = high(8, 62, 64), high(8, 0, 4)
        blk[:, 4:8] = (sc[:, :4] & 63) | ((sc[:, 4:] >> 4) << 6)
        blk[:, 8:12] = mn[:, :4]
        blk[:, 12:16] = (sc[:, 4:] & 15) | (mn[:, 4:] << 4)
        blk[:, 16:48] = 255
        blk[:, -128:] = high(128, 12, 16) | (high(128, 12, 16) << 4)
        blk[:, 0:2], blk[:, 2:4] = f16(2.0 ** -10), f16(2.0 ** -9)
    qs = (rng.integers(120, 128, (batch, nb, 256)) * sign).astype(np.int8)
    q8 = (np.full((batch, nb), 2.0 ** -6, np.float32), qs, qs.reshape(batch, nb, 16, 16).sum(3, dtype=np.int64).astype(np.int16))
    data = blk.reshape(-1)
    s, bound = exact(eng, qtype, data, rows, 256 * nb, q8)
    assert np.abs(integers(eng, qtype, data, rows, 256 * nb)[2][0, :256] @ qs[0, 0].astype(np.float64)) > 2.0 ** 24
    got = run(eng, qtype, data, rows, 256 * nb, q8)
    small = np.concatenate([run(eng, qtype, data, rows, 256 * nb, [a[k:k + 50] for a in q8]) for k in (0, 50)])
    worst = [float((np.abs(v - s) / np.abs(s)).max() * 2 ** 24) for v in (got, small)]
    print("largest sums", qtype, nb, "of 2^-24:", worst)
    assert (np.abs(small - s) <= bound).all()
    steps = 32 if qtype == Q6_K else 16
    assert (np.abs(got - s) <= bound + steps * 2.0 ** -23 * np.abs(s)).all()
    if nb == 1:            # one block: integer sums are exact, so what is left are the roundings of the terms
        assert worst[1] <= 3.0, worst
