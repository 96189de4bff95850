"""What users of this framework have it do, as cases that can be timed and compared.

Four kinds of work, each through the public calls of ``alice_llm_b200``:

  matvec  one quantized matrix times 1..8 vectors, device buffers (GpuEngine.matvec_dev) - the call a host program binds for
          single projections
  ffn     the SwiGLU feed-forward block, swiglu_dev then matvec_dev - the largest part of a decoded token
  llama   a whole quantized Llama-style model: "decode" reads the logits of every token (sampling on the host), "verify" runs a
          draft of several tokens in one pass and reads all their logits, "prompt" takes a prompt from an empty context and
          reads the logits of its last token
  stack   a bfloat16 layer-stack model: "request" is a reset, a prompt and some decoded tokens

Weights are drawn in the storage formats themselves with the spread of a trained matrix (zero mean, 1 / sqrt(columns)).
"""
import math

import numpy as np
import torch

from alice_llm_b200 import stack
from alice_llm_b200.gpu import GpuEngine, GpuModel, GpuModelConfig, GpuQuantType as Q

DEV = "cuda"
TYPES = {"q4k": Q.Q4K, "q5k": Q.Q5K, "q6k": Q.Q6K, "q8_0": Q.Q8_0, "q1_0": Q.Q1_0, "q2_0": Q.Q2_0, "ternary": Q.Ternary, "sparse": Q.SparseTernary}
BLOCK = {"q4k": (256, 144), "q5k": (256, 176), "q6k": (256, 210), "q8_0": (32, 34), "q1_0": (128, 18), "q2_0": (128, 34)}   # elements, bytes
K_QUANTS = ("q4k", "q5k", "q6k")
ROLES = ("q", "k", "v", "o", "gate", "up", "down")
# storage type of every projection, of down and of the head
MIXES = {"q4km": ("q4k", "q6k", "q6k"), "q5km": ("q5k", "q6k", "q6k"), "q8_0": ("q8_0", "q8_0", "q8_0"), "q1_0": ("q1_0", "q1_0", "q8_0"),
         "ternary": ("ternary", "ternary", "ternary")}


def matvec(type, rows, cols, batch):
    return dict(kind="matvec", type=type, rows=rows, cols=cols, batch=batch)


def ffn(mix, hidden, ff, batch):
    return dict(kind="ffn", mix=mix, hidden=hidden, ff=ff, batch=batch)


def llama(mode, mix, layers, hidden, ff, heads, kv_heads, vocab, context, tokens):
    return dict(kind="llama", mode=mode, mix=mix, layers=layers, hidden=hidden, ff=ff, heads=heads, kv_heads=kv_heads, vocab=vocab, context=context, tokens=tokens)


def stacked(family, layers, width, ff, heads, kv_heads, vocab, prompt, tokens):
    return dict(kind="stack", family=family, layers=layers, width=width, ff=ff, heads=heads, kv_heads=kv_heads, vocab=vocab, prompt=prompt, tokens=tokens)


def listed():
    named = {
        # one attention projection of an 8B model: the smallest call, launches and latency
        "matvec_q4k_4096": matvec("q4k", 4096, 4096, 1),
        # a projection of a pruned or unusual width, three vectors: no size a power of two, no whole number of tiles
        "matvec_q5k_ragged_b3": matvec("q5k", 5003, 2816, 3),
        # feed-forward block at 8B shapes, one token being decoded
        "ffn_8b_b1": ffn("q4km", 4096, 14336, 1),
        # the same block for a draft of four tokens
        "ffn_8b_b4": ffn("q4km", 4096, 14336, 4),
        # feed-forward block at 70B shapes in ternary bit planes
        "ffn_70b_ternary_b1": ffn("ternary", 8192, 28672, 1),
        # chat with an 8B model, sampling on the host: four tokens behind 2048
        "decode_8b": llama("decode", "q4km", 32, 4096, 14336, 32, 8, 128256, 2048, 4),
        # the prompt of such a chat
        "prompt_8b": llama("prompt", "q4km", 32, 4096, 14336, 32, 8, 128256, 0, 256),
        # a 27B model in one bit per weight, behind a long context
        "decode_27b_q1_0": llama("decode", "q1_0", 64, 5120, 25600, 40, 8, 151936, 4096, 2),
        # speculative decoding: eight drafted tokens through a 70B ternary model
        "verify_70b_ternary": llama("verify", "ternary", 80, 8192, 28672, 64, 8, 32000, 2048, 8),
        # reading a document: a long prompt, few tokens of answer
        "zamitar_document": stacked("Zamitar", 8, 4096, 14336, 32, 32, 32000, 2048, 1),
        "suborax_document": stacked("Suborax", 8, 4096, 14336, 32, 8, 32000, 2048, 1),
        # a short question and its answer on a smaller model: nearly all of it decoding
        "zamitar_answer": stacked("Zamitar", 8, 2048, 8192, 16, 16, 32000, 33, 24),
    }
    return [dict(c, name=n) for n, c in named.items()]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` between lo and hi, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(max(round(v / step), -(-lo // step)), hi // step) * step)


def draw(rng):
    limits = [max(work(c)["bytes"] for c in listed()), max(work(c)["flops"] for c in listed())]
    while True:
        c = _draw(rng)
        w = work(c)
        if w["bytes"] <= limits[0] and w["flops"] <= limits[1]:
            return c


def _draw(rng):
    kind = rng.choice(("matvec", "ffn", "llama", "stack"))
    batch = rng.choice((1, 1, 1, 2, 3, 4, 5, 8))
    if kind == "matvec":
        t = rng.choice(tuple(TYPES))
        step = 256 if t in K_QUANTS else 32 if t in ("q8_0", "ternary", "sparse") else 128
        cols = _log(rng, 512, 16384, step)
        rows = _log(rng, 256, 131072)
        return matvec(t, min(rows, (1 << 29) // cols), cols, batch)
    if kind == "ffn":
        return ffn(rng.choice(tuple(MIXES)), _log(rng, 1024, 8192, 256), _log(rng, 2048, 28672 if rng.random() < 0.5 else 14336, 256) // 256 * 256, batch)
    if kind == "llama":
        mix, mode = rng.choice(tuple(MIXES)), rng.choice(("decode", "verify", "prompt"))
        kv, group = rng.choice(((8, 4), (8, 5), (8, 8), (4, 4), (4, 8), (16, 1), (8, 2)))
        hidden = kv * group * 128
        ff = min(_log(rng, 2 * hidden, 4 * hidden, 256), 16384 if mix == "q8_0" else 28672)
        vocab = rng.choice((32000, 50257, 128256, 151936))
        tokens = {"decode": rng.randint(1, 4), "verify": rng.randint(2, 8), "prompt": _log(rng, 2, 256)}[mode]
        context = 0 if mode == "prompt" else _log(rng, 16, 8192)
        return llama(mode, mix, rng.choice((2, 4, 8, 16, 32)), hidden, ff, kv * group, kv, vocab, context, tokens)
    family, heads = rng.choice(("Zamitar", "Suborax")), rng.choice((8, 16, 24, 32))
    prompt, tokens = (_log(rng, 128, 2048), rng.randint(1, 4)) if rng.random() < 0.5 else (_log(rng, 2, 128), rng.randint(8, 24))
    return stacked(family, rng.choice((2, 4, 6, 8)), heads * 128, _log(rng, 256 * heads, 512 * heads, 64), heads, heads if family == "Zamitar" else heads // 4,
                   rng.choice((8192, 32000, 50257)), prompt, tokens)


# ---- weights in their storage formats ---------------------------------------------------------------------

def _f16(t):
    return t.to(torch.float16).view(torch.uint8).reshape(*t.shape, 2)


def _blocks(gen, t, rows, cols, gain=1.0):
    """Raw rows of a block format, or (planes, scales) of a ternary one, on the device."""
    rand = lambda n, w: torch.randint(0, 256, (n, w), dtype=torch.uint8, device=DEV, generator=gen)
    near = lambda n: 1.0 + 0.2 * torch.rand(n, device=DEV, generator=gen)
    sigma = gain / math.sqrt(cols)
    if t in ("ternary", "sparse"):
        scales = near(rows) * sigma * math.sqrt(2.0)
        if t == "ternary":
            pb = (cols + 31) // 32 * 4
            a, b = rand(rows, pb), rand(rows, pb)
            planes = torch.stack([a & b, ~a & b], dim=1).reshape(rows, 2 * pb)
            if cols % 32:
                raise ValueError("ternary columns come in multiples of 32 here")
            return planes, scales
        a, b = (rand(rows, (cols + 15) // 16 * 4) & 0x55 for _ in range(2))
        return a | ((a & b) << 1), scales       # 00 = 0, 01 = +1, 11 = -1
    elems, size = BLOCK[t]
    n = rows * (cols // elems)
    blk = rand(n, size)
    if t in ("q4k", "q5k"):
        # scale and min of a sub-block alike, dmin the middle code times d: a mean of zero
        sc = torch.randint(24, 64, (n, 8), dtype=torch.uint8, device=DEV, generator=gen)
        blk[:, 4:8] = blk[:, 8:12] = (sc[:, :4] & 63) | ((sc[:, 4:] >> 4) << 6)
        blk[:, 12:16] = (sc[:, 4:] & 15) | ((sc[:, 4:] & 15) << 4)
        d = near(n) * sigma / (44.0 * (4.6 if t == "q4k" else 9.2))
        blk[:, 0:2], blk[:, 2:4] = _f16(d), _f16(d * (7.5 if t == "q4k" else 15.5))
    elif t == "q6k":
        blk[:, 192:208] = torch.randint(-48, 49, (n, 16), dtype=torch.int8, device=DEV, generator=gen).view(torch.uint8)
        blk[:, 208:210] = _f16(near(n) * sigma / (28.0 * 18.5))
    elif t == "q8_0":
        blk[:, 2:] = torch.randint(-127, 128, (n, 32), dtype=torch.int8, device=DEV, generator=gen).view(torch.uint8)
        blk[:, 0:2] = _f16(near(n) * sigma / 73.6)
    elif t == "q1_0":
        blk[:, 0:2] = _f16(near(n) * sigma)
    else:
        s = torch.randint(0, 3, (n, 32, 4), dtype=torch.uint8, device=DEV, generator=gen)
        blk[:, 2:] = s[..., 0] | (s[..., 1] << 2) | (s[..., 2] << 4) | (s[..., 3] << 6)
        blk[:, 0:2] = _f16(near(n) * sigma * 1.22)
    return blk.reshape(rows, -1), None


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


_ENGINE = []


def engine():
    if not _ENGINE:
        _ENGINE.append(GpuEngine(0))
    return _ENGINE[0]


def _handle(t, rows, cols, raw, scales):
    e = engine()
    if t == "ternary":
        return e.ternary_from_device(raw.data_ptr(), scales.data_ptr(), rows, cols)
    if t == "sparse":
        return e.upload_sparse_ternary(raw.cpu().numpy(), scales.cpu().numpy(), rows, cols)
    return e.weights_from_device(raw.data_ptr(), raw.numel(), rows, cols, TYPES[t])


def _matrices(case):
    """[(name, type, rows, cols)] of the quantized matrices, in the order they are drawn."""
    if case["kind"] == "matvec":
        return [("w", case["type"], case["rows"], case["cols"])]
    most, down, head = MIXES[case["mix"]]
    h, f = case["hidden"], case["ff"]
    if case["kind"] == "ffn":
        return [("gate", most, f, h), ("up", most, f, h), ("down", down, h, f)]
    kv = case["kv_heads"] * 128
    per = {"q": (h, h), "k": (kv, h), "v": (kv, h), "o": (h, h), "gate": (f, h), "up": (f, h), "down": (h, f)}
    out = [(f"{i}.{r}", down if r == "down" else most, *per[r]) for i in range(case["layers"]) for r in ROLES]
    return out + [("embedding", "q8_0", case["vocab"], h), ("output", head, case["vocab"], h)]


def _weights(case, seed):
    """name -> (type, rows, cols, raw, scales). In a whole model embeddings have unit spread and the matrices that write into the
    residual stream are smaller, as trained ones are: the stream outweighs what a layer adds."""
    out = {}
    for i, (name, t, rows, cols) in enumerate(_matrices(case)):
        gain = 1.0
        if case["kind"] == "llama":
            gain = math.sqrt(cols) if name == "embedding" else 1.0 / math.sqrt(2 * case["layers"]) if name.endswith((".o", ".down")) else 1.0
        out[name] = (t, rows, cols, *_blocks(_gen(seed * 1000003 + i), t, rows, cols, gain))
    return out


def _vectors(case, seed):
    n = case["cols"] if case["kind"] == "matvec" else case["hidden"]
    return torch.randn(case["batch"], n, device=DEV, generator=_gen(seed * 1000003 + 900001))


def _llama_inputs(case, seed):
    rng = np.random.default_rng(seed)
    norms = [(1.0 + 0.02 * rng.standard_normal(case["hidden"])).astype(np.float32) for _ in range(2 * case["layers"] + 1)]
    tokens = rng.integers(0, case["vocab"], case["tokens"]).astype(np.uint32)
    g = _gen(seed * 1000003 + 900002)
    k, v = (torch.randn(case["context"], case["kv_heads"] * 128, device=DEV, generator=g) for _ in range(2))
    return norms, tokens, k, v


# ---- layer-stack models -----------------------------------------------------------------------------------

def _stack_config(case):
    w, f, h = case["width"], case["ff"], case["heads"]
    mlp, base = {"kind": "dense", "ff": f}, {"vocab": case["vocab"], "width": w, "norm": {"eps": 1e-6}, "embedding": {"scale": 1.0}}
    if case["family"] == "Suborax":
        layer = {"type": "attention", "mlp": mlp,
                 "mixer": dict(heads=h, kv_heads=case["kv_heads"], dim=128, vdim=128, scale=128 ** -0.5, softcap=30.0,
                               rot=dict(base=10000.0, dims=128, scaling=dict(factor=4.0, low=1.0, high=4.0, original=4096)))}
        return dict(base, architecture="Suborax", postln_alpha=2.0, layers=[layer] * case["layers"])
    latent = {"type": "latent_attention", "mlp": mlp,
              "mixer": dict(heads=h, dim=128, rot_dim=64, vdim=128, q_rank=w * 3 // 8 // 64 * 64, kv_rank=512, scale=192 ** -0.5, rot=dict(base=10000.0, dims=64))}
    delta = {"type": "channel_delta", "mlp": mlp, "mixer": dict(heads=h, kv_heads=h, dim=128, vdim=128, conv=4)}
    return dict(base, architecture="Zamitar", loop=None, layers=[delta if i % 2 == 0 else latent for i in range(case["layers"])])


def _stack_weights(case, seed):
    """(StackConfig, [(matrices, vectors)] in the packed layout of alice_stack_create, embedding, head or None, final norm, prompt, tokens)"""
    gen, rng = _gen(seed * 1000003 + 900003), np.random.default_rng(seed)
    cfg = stack.StackConfig(_stack_config(case), case["prompt"] + case["tokens"])

    def mat(rows, cols, spread=None):
        return (torch.randn(rows, cols, device=DEV, generator=gen) * (spread or cols ** -0.5)).to(torch.bfloat16)

    one = lambda n: (1.0 + 0.02 * rng.standard_normal(n)).astype(np.float32)
    small = lambda *n: (0.1 * rng.standard_normal(n)).astype(np.float32)
    packed, w = [], cfg.width
    for L in cfg.layers:
        L.decay_rank = L.gate_rank = 128 if L.kind == stack.MIX_DELTA else 0
        mats = {n: mat(*shape) for n, shape in L.packed_shapes(w).items()}
        if L.kind == stack.MIX_GROUPED:
            packed.append((mats, dict(norm=one(w), norm2=one(w), sink=small(L.heads))))
            continue
        vecs = dict(norm=one(w), ls1=0.5 * one(w), ls2=0.5 * one(w), gate_bias=small(L.ff), up_bias=small(L.ff), down_bias=small(w))
        if L.kind == stack.MIX_LATENT:
            vecs.update(q_norm=one(L.q_rank), kv_norm=one(L.kv_rank), sink=small(L.heads))
        else:
            vecs.update(conv=0.5 + small(L.conv_taps, 3 * L.heads * 128), a_log=small(L.heads), dt_bias=small(L.heads * 128) - 2.0, head_norm=one(L.vdim))
        packed.append((mats, vecs))
    embed = mat(cfg.vocab_size, w, 1.0 if cfg.family.tied is False else w ** -0.5)
    head = None if cfg.family.tied else mat(cfg.vocab_size, w)
    return cfg, packed, embed, head, one(w), rng.integers(0, case["vocab"], case["prompt"]).astype(np.uint32), rng.integers(0, case["vocab"], case["tokens"]).tolist()


# ---- the cases --------------------------------------------------------------------------------------------

def prepare(case, seed):
    e = engine()
    kind = case["kind"]
    if kind == "stack":
        cfg, packed, embed, head, final, prompt, tokens = _stack_weights(case, seed)
        bf16 = lambda t: e.weights_from_device(t.data_ptr(), t.numel() * 2, t.shape[0], t.shape[1], Q.BF16)
        torch.cuda.synchronize()
        h, keep = stack.create(e, cfg, [({n: bf16(t) for n, t in m.items()}, v) for m, v in packed], bf16(embed), final, None, False, None if head is None else bf16(head))
        return dict(kind=kind, model=GpuModel(e, h, cfg, [keep]), prompt=prompt, tokens=tokens, keep=(packed, embed, head))
    weights = _weights(case, seed)
    torch.cuda.synchronize()
    handles = {n: _handle(*w) for n, w in weights.items()}
    if kind != "llama":
        x = _vectors(case, seed)
        rows = case["rows"] if kind == "matvec" else case["hidden"]
        y = torch.empty(case["batch"], rows, device=DEV)
        h = torch.empty(case["batch"], case.get("ff", 1), device=DEV)
        buf = lambda t: e.buf_from_device(t.data_ptr(), t.numel())
        torch.cuda.synchronize()
        return dict(kind=kind, w=handles, batch=case["batch"], x=buf(x), h=buf(h), y=buf(y), out=y, keep=(weights, x, h))
    norms, tokens, k, v = _llama_inputs(case, seed)
    cfg = GpuModelConfig(case["layers"], case["hidden"], case["ff"], case["heads"], case["kv_heads"], 128, 500000.0, 1e-5, case["context"] + case["tokens"], case["vocab"])
    layers = [dict({r: handles[f"{i}.{r}"] for r in ROLES}, attn_norm=norms[2 * i], ffn_norm=norms[2 * i + 1]) for i in range(case["layers"])]
    model = GpuModel.load(e, {"layers": layers, "embedding": handles["embedding"], "output": handles["output"], "output_norm": norms[-1]}, cfg)
    if case["context"]:
        k, v = k.cpu().numpy(), v.cpu().numpy()
        for i in range(case["layers"]):
            model.kv_write(i, 0, k, v)
    model.set_position(case["context"])
    return dict(kind=kind, mode=case["mode"], model=model, context=case["context"], tokens=tokens, keep=weights)


def run(state):
    e, kind = engine(), state["kind"]
    if kind == "matvec":
        e.matvec_dev(state["w"]["w"], state["x"], state["y"], state["batch"])
        return state["out"]
    if kind == "ffn":
        w = state["w"]
        e.swiglu_dev(w["gate"], w["up"], state["x"], state["h"], state["batch"])
        e.matvec_dev(w["down"], state["h"], state["y"], state["batch"])
        return state["out"]
    m = state["model"]
    if kind == "stack":
        m.reset()
        n = len(state["prompt"])
        return [m.forward_rows(state["prompt"], [n - 1])[0]] + [m.forward_and_read(t) for t in state["tokens"]]
    m.rollback_to(state["context"])     # what a sequence that is thrown away costs: nothing is cleared
    if state["mode"] == "decode":
        return [m.forward_and_read(int(t)) for t in state["tokens"]]
    if state["mode"] == "verify":
        return m.forward_batch_and_read(state["tokens"])
    return m.forward_rows(state["tokens"], [len(state["tokens"]) - 1])


def _row_bytes(t, cols):
    return cols // 4 if t in ("ternary", "sparse") else cols // BLOCK[t][0] * BLOCK[t][1]


def work(case):
    if case["kind"] == "stack":
        w, f, h, kv, n = case["width"], case["ff"], case["heads"], case["kv_heads"], case["tokens"]
        total = case["prompt"] + n
        pairs = sum(range(1, total + 1))        # (query, key) pairs of one causal head
        if case["family"] == "Suborax":
            mixers = [(w * (2 * h + 2 * kv) * 128, 4 * h * 128 * pairs, kv * 256 * 2 * total)] * case["layers"]
        else:
            qr = w * 3 // 8 // 64 * 64
            latent = (w * (qr + 576 + 2 * h * 128) + h * (192 * qr + 256 * 512), 2 * h * 320 * pairs, 576 * 2 * total)
            delta = (w * (4 * h * 128 + h + 256) + 2 * 128 * h * 128, 6 * h * 128 * 128 * total, 2 * h * 128 * 128 * 4)
            mixers = [delta if i % 2 == 0 else latent for i in range(case["layers"])]
        body = sum(m[0] for m in mixers) + case["layers"] * 3 * w * f
        head = case["vocab"] * w
        # the prompt reads the weights once, every decoded token once more; the cache is read by every decoded token
        return {"bytes": (1 + n) * 2 * (body + head) + (1 + n) * sum(m[2] for m in mixers), "flops": 2 * body * total + 2 * head * (1 + n) + sum(m[1] for m in mixers)}
    mats = [m for m in _matrices(case) if m[0] != "embedding"]
    weights, elems = sum(r * _row_bytes(t, c) for _, t, r, c in mats), sum(r * c for _, _, r, c in mats)
    if case["kind"] == "matvec":
        return {"bytes": weights + 4 * case["batch"] * (case["rows"] + case["cols"]), "flops": 2 * elems * case["batch"]}
    if case["kind"] == "ffn":
        return {"bytes": weights + 8 * case["batch"] * case["hidden"], "flops": 2 * elems * case["batch"]}
    n, kv = case["tokens"], case["layers"] * case["kv_heads"] * 128 * 8     # bytes a cached position takes
    pairs = sum(case["context"] + i + 1 for i in range(n))
    flops = 2 * elems * n + 4 * case["layers"] * case["heads"] * 128 * pairs
    if case["mode"] == "decode":
        return {"bytes": n * weights + kv * pairs + 4 * n * case["vocab"], "flops": flops}
    if case["mode"] == "verify":
        return {"bytes": weights + kv * (case["context"] + n) + 4 * n * case["vocab"], "flops": flops}
    return {"bytes": weights + kv * n + 4 * case["vocab"], "flops": flops - 2 * case["vocab"] * case["hidden"] * (n - 1)}


def tolerance(case):
    """About four times what these calls are off the same in 64 bits, or what two orders of their sums differ by."""
    if case["kind"] == "matvec":
        return {"rel": {"ternary": 5e-6, "sparse": 5e-6, "q1_0": 3e-5, "q2_0": 3e-5}.get(case["type"], 2e-6)}
    if case["kind"] == "stack":
        return {"rel": 0.03}        # bfloat16 activations
    if case["kind"] == "ffn":       # the hidden vector of the K-quants is rounded to the Q8_K grid: a last bit moves single values by a step
        return {"rel": 3e-3 if MIXES[case["mix"]][1] in K_QUANTS else {"q8_0": 2e-6, "ternary": 2e-5, "q1_0": 8e-5}[case["mix"]]}
    # the same rounding in every layer: two orders of the sums end 1.2e-2 apart, as far as each is off the unrounded model
    return {"rel": 5e-5 if case["mix"] in ("q8_0", "ternary") else 0.03}


# ---- the same in 64 bits ----------------------------------------------------------------------------------

def _dequantize(t, raw, scales, cols):
    """Rows of a storage format in 64 bits."""
    n = raw.shape[0]
    if t in ("ternary", "sparse"):
        if t == "ternary":
            bits = ((raw.reshape(n, 2, -1, 1) >> torch.arange(8, device=DEV, dtype=torch.uint8)) & 1).reshape(n, 2, -1)[..., :cols]
            w = bits[:, 0].double() - bits[:, 1].double()
        else:
            code = ((raw.reshape(n, -1, 1) >> torch.arange(0, 8, 2, device=DEV, dtype=torch.uint8)) & 3).reshape(n, -1)[:, :cols]
            w = (code & 1).double() * (1.0 - (code & 2).double())
        return w * scales.double()[:, None]
    elems, size = BLOCK[t]
    b = raw.reshape(-1, size)
    f16 = lambda o: b[:, o:o + 2].contiguous().view(torch.float16).double()
    if t in ("q4k", "q5k"):
        lo, mn, hi = b[:, 4:8], b[:, 8:12], b[:, 12:16]
        sc = torch.cat([lo & 63, (hi & 15) | ((lo >> 6) << 4)], 1).double()
        m = torch.cat([mn & 63, (hi >> 4) | ((mn >> 6) << 4)], 1).double()
        qs = b[:, size - 128:].reshape(-1, 4, 1, 32)
        q = torch.cat([qs & 15, qs >> 4], 2).reshape(-1, 8, 32)
        if t == "q5k":
            q = q + (((b[:, 16:48].reshape(-1, 1, 32) >> torch.arange(8, device=DEV, dtype=torch.uint8)[:, None]) & 1) << 4)
        w = f16(0)[:, :, None] * sc[:, :, None] * q.double() - f16(2)[:, :, None] * m[:, :, None]
    elif t == "q6k":
        ql, qh = b[:, :128].reshape(-1, 2, 2, 32), b[:, 128:192].reshape(-1, 2, 1, 32)
        q = torch.cat([ql & 15, ql >> 4], 2) | (((qh >> torch.arange(0, 8, 2, device=DEV, dtype=torch.uint8)[:, None]) & 3) << 4)
        sc = b[:, 192:208].contiguous().view(torch.int8).double()
        w = (q.double() - 32.0).reshape(-1, 16, 16) * sc[:, :, None] * f16(208)[:, :, None]
    elif t == "q8_0":
        w = b[:, 2:].contiguous().view(torch.int8).double() * f16(0)
    elif t == "q1_0":
        w = (((b[:, 2:, None] >> torch.arange(8, device=DEV, dtype=torch.uint8)) & 1).reshape(-1, 128).double() * 2.0 - 1.0) * f16(0)
    else:
        w = (((b[:, 2:, None] >> torch.arange(0, 8, 2, device=DEV, dtype=torch.uint8)) & 3).reshape(-1, 128).double() - 1.0) * f16(0)
    return w.reshape(n, cols)


def _times(x, w):
    """x [n, cols] times the matrix, in slices of its rows."""
    t, rows, cols, raw, scales = w
    step = max(1, (1 << 26) // cols)
    return torch.cat([x @ _dequantize(t, raw[i:i + step], None if scales is None else scales[i:i + step], cols).T for i in range(0, rows, step)], 1)


def _q8k(x):
    """Activations on the Q8_K grid: per 256 the element of largest magnitude becomes -128 (quantize_row_q8_k, src/gguf.rs:1323)."""
    b = x.float().reshape(-1, 256)
    top = b.gather(1, b.abs().argmax(1, keepdim=True))
    inv = 128.0 / top
    q = torch.round(inv * b).clamp(-128, 127)
    return (q.double() * (1.0 / inv).double()).reshape(x.shape)


def _silu(x):
    return x * torch.sigmoid(x)


def _causal(q, k, v, scale, cap=None, sink=None):
    """q [n, h, d] behind the first of k, v [m, h, .]: the last query sees every key."""
    n, m = q.shape[0], k.shape[0]
    out = torch.empty(n, q.shape[1], v.shape[2], dtype=q.dtype, device=q.device)
    for h in range(q.shape[1]):
        s = q[:, h] @ k[:, h].T * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill(torch.ones(n, m, dtype=torch.bool, device=q.device).triu(m - n + 1), -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(n, 1)], 1)
        out[:, h] = torch.softmax(s, 1)[:, :m] @ v[:, h]
    return out


def _exact_llama(case, seed):
    """Activations are not rounded here (the K-quant and one-bit models put them on the Q8_K grid): both sides are as far off."""
    w, (norms, tokens, kc, vc) = _weights(case, seed), _llama_inputs(case, seed)
    norms = [torch.from_numpy(n).to(DEV).double() for n in norms]
    n, ctx, group = case["tokens"], case["context"], case["heads"] // case["kv_heads"]
    rms = lambda x, g: x / torch.sqrt((x * x).mean(1, keepdim=True) + 1e-5) * g
    freq = (1.0 / np.float32(500000.0) ** (np.arange(0, 128, 2, dtype=np.float32) / np.float32(128))).astype(np.float32)
    ang = torch.from_numpy(np.arange(ctx, ctx + n, dtype=np.float32)[:, None] * freq).to(DEV).double()
    c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]

    def turn(x):
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * c - v * s, u * s + v * c], -1).reshape(x.shape)

    t, rows, cols, raw, _ = w["embedding"]
    x = _dequantize(t, raw[torch.from_numpy(tokens.astype(np.int64)).to(DEV)], None, cols)
    for i in range(case["layers"]):
        L = lambda r: w[f"{i}.{r}"]
        h = rms(x, norms[2 * i])
        q, k, v = (_times(h, L(r)).reshape(n, -1, 128) for r in "qkv")
        k = torch.cat([kc.double().reshape(ctx, case["kv_heads"], 128), turn(k)])
        v = torch.cat([vc.double().reshape(ctx, case["kv_heads"], 128), v])
        a = _causal(turn(q), k.repeat_interleave(group, 1), v.repeat_interleave(group, 1), 128 ** -0.5)
        x = x + _times(a.reshape(n, -1), L("o"))
        h = rms(x, norms[2 * i + 1])
        x = x + _times(_silu(_times(h, L("gate"))) * _times(h, L("up")), L("down"))
    if case["mode"] == "prompt":
        x = x[-1:]
    logits = _times(rms(x, norms[-1]), w["output"])
    return list(logits) if case["mode"] == "decode" else logits.reshape(-1) if case["mode"] == "verify" else logits


def _exact_stack(case, seed):
    cfg, packed, embed, head, final, prompt, tokens = _stack_weights(case, seed)
    d = lambda a: (torch.from_numpy(np.asarray(a)).to(DEV) if not torch.is_tensor(a) else a).double()
    ids = np.concatenate([prompt.astype(np.int64), np.array(tokens, np.int64)])
    T, eps, offset = len(ids), cfg.eps, case["family"] == "Suborax"
    x = embed[torch.from_numpy(ids).to(DEV)].double()

    def layer_norm(x, g):
        m = x - x.mean(-1, keepdim=True)
        return m / torch.sqrt((m * m).mean(-1, keepdim=True) + eps) * g

    rms = lambda x, g=1.0: x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * g
    norm = rms if offset else layer_norm

    def turn(x, L):
        half = L.rot_dims // 2
        f = L.rot_base ** (-2.0 * np.arange(half) / L.rot_dims)
        if L.rot_factor:
            wave = 2.0 * math.pi / f
            keep = np.clip((L.rot_original / wave - L.rot_low) / (L.rot_high - L.rot_low), 0.0, 1.0)
            f = (1.0 - keep) * f / L.rot_factor + keep * f
        a = (torch.arange(T, device=DEV).double()[:, None] * d(f))[:, None]
        u, v = x[..., :half], x[..., half:2 * half]
        return torch.cat([u * torch.cos(a) - v * torch.sin(a), v * torch.cos(a) + u * torch.sin(a), x[..., 2 * half:]], -1)

    def mlp(h, m, v, L):
        g = d(m["gu"]).reshape(-1, 2, 64, cfg.width)
        a, b = (h @ g[:, i].reshape(-1, cfg.width).T for i in range(2))
        if "gate_bias" in v:
            a, b = a + d(v["gate_bias"]), b + d(v["up_bias"])
        y = (_silu(a) * b) @ d(m["down"]).T
        return y + d(v["down_bias"]) if "down_bias" in v else y

    def grouped(h, m, v, L):
        q, k, val = torch.split(h @ d(m["in"]).T, [L.heads * 128, L.kv_heads * 128, L.kv_heads * 128], 1)
        q, k = (rms(turn(a.reshape(T, -1, 128), L)) for a in (q, k))
        k, val = (a.reshape(T, -1, 128).repeat_interleave(L.heads // L.kv_heads, 1) for a in (k, val))
        return _causal(q, k, val, L.scale, L.softcap, d(v["sink"])).reshape(T, -1) @ d(m["o"]).T

    def latent(h, m, v, L):
        kv, H = L.kv_rank, L.heads
        cq, ckv, _, gate = torch.split(h @ d(m["in"]).T, [L.q_rank, kv + 64, 0, H * 128], 1)
        q = (rms(cq, d(v["q_norm"])) @ d(m["uq"]).T).reshape(T, H, 192)
        c = rms(ckv[:, :kv], d(v["kv_norm"]))
        kr = turn(ckv[:, None, kv:], L).expand(T, H, 64)
        k = torch.cat([(c @ d(m["uk"]).T).reshape(T, H, 128), kr], -1)
        q = torch.cat([q[..., :128], turn(q[..., 128:], L)], -1)
        o = _causal(q, k, (c @ d(m["uv"]).T).reshape(T, H, 128), L.scale, None, d(v["sink"])).reshape(T, -1)
        return (o * torch.sigmoid(gate)) @ d(m["o"]).T

    def delta(h, m, v, L):
        H, n = L.heads, L.heads * 128
        p = h @ d(m["in"]).T
        qkv, step, low, glow = p[:, :3 * n], p[:, 3 * n:3 * n + H], p[:, 3 * n + stack.pad(H):][:, :128], p[:, 3 * n + stack.pad(H) + 128:][:, :128]
        taps = d(v["conv"])
        qkv = torch.cat([torch.zeros(L.conv_taps - 1, 3 * n, dtype=torch.float64, device=DEV), qkv])
        q, k, val = (a.reshape(T, H, 128) for a in torch.split(_silu(sum(qkv[j:j + T] * taps[j] for j in range(L.conv_taps))), n, 1))
        unit = lambda a: a / torch.sqrt((a * a).sum(-1, keepdim=True) + 1e-6)
        q, k, beta = unit(q) * 128 ** -0.5, unit(k), torch.sigmoid(step)[..., None]
        rate = torch.nn.functional.softplus(low @ d(m["a2"]).T + d(v["dt_bias"]).reshape(-1)).reshape(T, H, 128)
        g = torch.exp(-torch.exp(d(v["a_log"]))[:, None] * rate)
        S, out = torch.zeros(H, 128, 128, dtype=torch.float64, device=DEV), torch.empty_like(val)
        for t in range(T):
            S = S * g[t][:, :, None]
            u = beta[t] * (val[t] - torch.bmm(k[t][:, None], S)[:, 0])
            S = torch.baddbmm(S, k[t][:, :, None], u[:, None])
            out[t] = torch.bmm(q[t][:, None], S)[:, 0]
        o = rms(out, d(v["head_norm"])).reshape(T, -1) * torch.sigmoid(glow @ d(m["g2"]).T)
        return o @ d(m["o"]).T

    mixer = {stack.MIX_GROUPED: grouped, stack.MIX_LATENT: latent, stack.MIX_DELTA: delta}
    for L, (m, v) in zip(cfg.layers, packed):
        if offset:
            x = norm(cfg.alpha * x + mixer[L.kind](x, m, v, L), d(v["norm"]))
            x = norm(cfg.alpha * x + mlp(x, m, v, L), d(v["norm2"]))
        else:
            h = norm(x, d(v["norm"]))
            x = x + mixer[L.kind](h, m, v, L) * d(v["ls1"]) + mlp(h, m, v, L) * d(v["ls2"])
    x = norm(x[len(prompt) - 1:], d(final))
    return list(x @ d(embed if head is None else head).T)


def exact(case, seed):
    if case["kind"] == "llama":
        return _exact_llama(case, seed)
    if case["kind"] == "stack":
        return _exact_stack(case, seed)
    w, x = _weights(case, seed), _vectors(case, seed)
    if case["kind"] == "matvec":
        return _times(_q8k(x) if case["type"] in K_QUANTS else x.double(), w["w"])
    x = x.double()      # the hidden vector is not rounded to the Q8_K grid here, nor is x: both sides are as far off
    return _times(_silu(_times(x, w["gate"])) * _times(x, w["up"]), w["down"])
