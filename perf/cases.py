"""Measured cases of the quantized attention path: the calls a user's program makes, through the package's own entry points,
over the range of sizes, data types and options they are used with.

  prefill        attention forward on quantised vectors (ops.att_fwd)
  prefill_block  one layer's forward: int8 projections with rope and quantisation, attention, combiner product
  train          attention forward and backward (ops.att_fwd, ops.att_bwd)
  train_block    one layer's forward and backward: producers, attention, combiner product and the way back through all of them
  decode         two tokens of one layer over int8 KV caches (KVCache.append, KVCache.decode)
  infer          two tokens of the whole int8 model over its KV caches (InferContext.compute_prediction)

A case is a dict of plain values; `listed` gives the fixed ones, `draw` more of the same ranges.
"""
import math
import random

import numpy as np
import torch

from tscale_b200 import abi, infer, ops

DEV = torch.device("cuda:0")
WHOLE = 1 << 20  # decode: a window longer than any context
VEC = 1.0 / 24   # scale of a unit vector's int8 codes
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


def listed():
    return [
        # one short prompt: the call's latency
        dict(name="prefill_short", kind="prefill", rows=77, frags=1, ragged=False, heads=12, d=64, qk="e4m3", v="e4m3", window=0, slope=0.0, out="bf16"),
        # a batch of documents through a sliding-window layer with ALiBi, and through the full-causal layer of the same model
        dict(name="prefill_window", kind="prefill", rows=65536, frags=16, ragged=False, heads=12, d=64, qk="e4m3", v="e4m3", window=64, slope=0.5,
             out="bf16"),
        dict(name="prefill_full", kind="prefill", rows=65536, frags=16, ragged=False, heads=12, d=64, qk="e4m3", v="e4m3", window=0, slope=0.0, out="bf16"),
        # long-context prefill, the largest call
        dict(name="prefill_long", kind="prefill", rows=131072, frags=4, ragged=False, heads=32, d=128, qk="e4m3", v="e4m3", window=0, slope=0.0, out="bf16"),
        # a layer's forward from the normalised int8 state, prompts of unequal length
        dict(name="prefill_block", kind="prefill_block", rows=12345, frags=8, ragged=True, heads=16, d=128, window=0, slope=0.0),
        # fine-tuning on a few short documents: every step of the layer and its back-propagation
        dict(name="train_block_short", kind="train_block", rows=3001, frags=5, ragged=True, heads=12, d=64, window=0, slope=0.0),
        # training batch: window layer and full-causal layer
        dict(name="train_window", kind="train", rows=32768, frags=8, ragged=False, heads=16, d=128, qk="i8", v="e4m3", window=256, slope=0.0, grad="bf16"),
        dict(name="train_full", kind="train", rows=32768, frags=8, ragged=False, heads=16, d=128, qk="i8", v="e4m3", window=0, slope=0.0, grad="bf16"),
        # one user's conversation: the step's latency; a serving batch: the stream of the caches
        dict(name="decode_single", kind="decode", seqs=1, ctx_lo=1000, ctx_hi=1000, heads=12, d=64, scale="f32", out="f32", window=WHOLE, slope=0.0),
        dict(name="decode_batch", kind="decode", seqs=64, ctx_lo=1024, ctx_hi=8192, heads=16, d=128, scale="f16", out="f32", window=WHOLE, slope=0.0),
        # the same two through the whole model (three window-64 layers and a wide one, repeated)
        dict(name="infer_single", kind="infer", seqs=1, ctx_lo=500, ctx_hi=500, layers=12, heads=12, d=64, relu_mult=1, vocab=50304, labels=1),
        dict(name="infer_batch", kind="infer", seqs=64, ctx_lo=1024, ctx_hi=8192, layers=12, heads=12, d=64, relu_mult=1, vocab=50304, labels=1),
    ]


def _log(rng, lo, hi):
    """Log-uniform integer in [lo, hi]."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


# attended pairs x heads x head size: the costliest case of each kind stays below the largest listed ones
MOST_WORK = {"prefill": 4 * 32 * 128 * 32768.0 ** 2 / 2, "prefill_block": 16 * 16 * 128 * 4096.0 ** 2 / 2, "train": 8 * 16 * 128 * 4096.0 ** 2 / 2,
              "train_block": 8 * 16 * 128 * 4096.0 ** 2 / 4}


def draw(rng):
    kind = rng.choice(("prefill", "prefill", "prefill_block", "train", "train_block", "decode", "infer"))
    if kind == "infer":
        seqs = _log(rng, 1, 64)
        lo = _log(rng, 16, 4096)
        heads, d = rng.choice(((8, 64), (12, 64), (16, 64), (4, 128), (8, 128)))
        return dict(kind=kind, seqs=seqs, ctx_lo=lo, ctx_hi=min(8192, lo + rng.randrange(lo + 1)), layers=rng.randrange(2, 9), heads=heads, d=d,
                    relu_mult=rng.choice((1, 2)), vocab=_log(rng, 1000, 60000), labels=rng.randrange(1, 4))
    if kind == "decode":
        lo = _log(rng, 16, 8192)
        heads, d = rng.choice(((8, 64), (12, 64), (16, 64), (5, 128), (16, 128), (32, 128)))
        return dict(kind=kind, seqs=_log(rng, 1, 64), ctx_lo=lo, ctx_hi=min(12000, lo + rng.randrange(lo + 1)), heads=heads, d=d,
                    scale=rng.choice(("f16", "f32")), out=rng.choice(("f32", "bf16", "f16")), window=rng.choice((WHOLE, WHOLE, 64, 256, 1024)),
                    slope=rng.choice((0.0, 0.5)))
    heads, d = rng.choice(((4, 64), (12, 64), (16, 64), (5, 128), (16, 128), (32, 128)))
    c = dict(kind=kind, heads=heads, d=d, window=rng.choice((0, 0, 64, 256)), slope=rng.choice((0.0, 0.0, 0.5)))
    if kind == "prefill":
        c["qk"], c["v"] = rng.choice((("e4m3", "e4m3"), ("e4m3", "e4m3"), ("i8", "e4m3"), ("i8", "i8")))
        c["out"] = rng.choice(("bf16", "bf16", "f16", "f32"))
    elif kind == "train":
        c["qk"], c["v"] = rng.choice((("i8", "e4m3"), ("i8", "e4m3"), ("e4m3", "e4m3")))
        c["grad"] = rng.choice(("bf16", "bf16", "f16"))
    rows = _log(rng, 16, 65536 if kind == "prefill" else 16384)
    c.update(rows=rows, frags=_log(rng, 1, max(1, rows // 64)), ragged=True)
    while _pairs(c) * heads * d > MOST_WORK[kind]:
        c["rows"] = c["rows"] * 3 // 4
        c["frags"] = min(c["frags"], c["rows"])
    return c


# ---------------------------------------------------------------------------------------------------- sizes that follow from a case
def _frag_lens(c):
    rows, frags = c["rows"], c["frags"]
    if not c["ragged"]:
        return [rows // frags] * frags
    cuts = sorted(random.Random(rows * 31 + frags).sample(range(1, rows), frags - 1)) if frags > 1 else []
    return [b - a for a, b in zip([0] + cuts, cuts + [rows])]


def _pairs(c):
    """Attended (query, key) pairs: row i of a fragment sees the min(i, window) rows before it (window 0: all of them)."""
    total = 0
    for n in _frag_lens(c):
        w = c["window"] if 0 < c["window"] < n else n
        total += w * (w - 1) // 2 + (n - w) * w
    return total


def _contexts(c):
    """Tokens in each sequence's cache, spread evenly over [ctx_lo, ctx_hi] in a shuffled order."""
    span = c["ctx_hi"] - c["ctx_lo"]
    return [c["ctx_lo"] + int(span * ((i * 0.6180339887) % 1.0)) for i in range(c["seqs"])]


def _layer_plan(c):
    return [(64, 0.5) if i % 4 != 3 else (WHOLE, 0.0) for i in range(c["layers"])]


# ---------------------------------------------------------------------------------------------------- inputs
def _normal(gen, rows, cols, scale, dtype=torch.float32):
    return (torch.randn((rows, cols), generator=gen, device=DEV) * scale).to(dtype)


def _quantised(gen, rows, hd, dtype, d):
    """N(0, 1/4) vectors through the library's abs-max quantiser: bytes [rows][hd] and scales [H][rows]."""
    b = torch.empty((rows, hd), dtype=torch.uint8, device=DEV)
    s = torch.empty((hd // d, rows), dtype=torch.float32, device=DEV)
    for r in range(0, rows, 32768):
        n = min(32768, rows - r)
        b[r:r + n], s[:, r:r + n] = ops.quant_rows(_normal(gen, n, hd, 0.5), "absmax", dtype, d)
    return b, s


def _codes(gen, shape):
    """int8 codes of normalised vectors (a unit component is 24)."""
    return torch.randn(shape, generator=gen, device=DEV).mul_(24.0).round_().clamp_(-127, 127).to(torch.int8)


def _rope(lens, d):
    """Rope rows of concatenated fragments: per 64-element block 32 cosines and 32 sines of the row's position."""
    pos = torch.cat([torch.arange(n, device=DEV) for n in lens]).to(torch.float32)[:, None]
    freq = torch.exp(torch.arange(d // 2, device=DEV) * (-2.0 * math.log(500000.0) / d))
    table = torch.empty((pos.shape[0], d), device=DEV)
    for blk in range(0, d, 64):
        angle = pos * freq[None, blk // 2:blk // 2 + 32]
        table[:, blk:blk + 32] = angle.cos()
        table[:, blk + 32:blk + 64] = angle.sin()
    return table


def _workspace(nbytes):
    return torch.empty(max(256, nbytes), dtype=torch.uint8, device=DEV)


def prepare(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    return {"prefill": _prepare_prefill, "prefill_block": _prepare_prefill_block, "train": _prepare_train, "train_block": _prepare_train_block,
            "decode": _prepare_decode, "infer": _prepare_infer}[case["kind"]](case, gen, seed)


def _attention_state(c, cfg, heads, rows, lens):
    """What every attention caller keeps: the mask on the device, workspace, status word."""
    L = abi.lib()
    mask = ops.Mask.window(lens, c["window"])
    mask.dev(DEV)
    return dict(case=c, cfg=cfg, mask=mask, ws=_workspace(L.tsa_att_fwd_workspace_bytes(cfg, heads, rows)),
                status=torch.zeros(1, dtype=torch.int32, device=DEV))


def _prepare_prefill(c, gen, seed):
    rows, heads, d = c["rows"], c["heads"], c["d"]
    hd = heads * d
    out = DTYPES[c["out"]]
    st = _attention_state(c, ops.make_cfg(c["qk"], c["v"], d, d, out_dtype=out), heads, rows, _frag_lens(c))
    for nm, dt in (("q", c["qk"]), ("k", c["qk"]), ("v", c["v"])):
        st[nm], st["s" + nm] = _quantised(gen, rows, hd, dt, d)
    # the caller's own result buffers
    st["out"] = torch.empty((rows, hd), dtype=out, device=DEV)
    st["lse"] = torch.empty((heads, rows), dtype=torch.float32, device=DEV)
    return st


def _prepare_train(c, gen, seed):
    rows, heads, d = c["rows"], c["heads"], c["d"]
    hd = heads * d
    grad = DTYPES[c["grad"]]
    cfg = ops.make_cfg(c["qk"], c["v"], d, d, out_dtype=grad, grad_dtype=grad)
    st = _attention_state(c, cfg, heads, rows, _frag_lens(c))
    st["bws"] = _workspace(abi.lib().tsa_att_bwd_workspace_bytes(cfg, heads, rows))
    for nm, dt in (("q", c["qk"]), ("k", c["qk"]), ("v", c["v"])):
        st[nm], st["s" + nm] = _quantised(gen, rows, hd, dt, d)
    st["d_out"] = _normal(gen, rows, hd, 1e-2, grad)
    st["out"] = torch.empty((rows, hd), dtype=grad, device=DEV)
    st["lse"] = torch.empty((heads, rows), dtype=torch.float32, device=DEV)
    return st


def _prepare_prefill_block(c, gen, seed):
    rows, heads, d = c["rows"], c["heads"], c["d"]
    dim = hd = heads * d
    lens = _frag_lens(c)
    st = _attention_state(c, ops.make_cfg("e4m3", "e4m3", d, d, out_dtype=torch.bfloat16), heads, rows, lens)
    st["x"] = _codes(gen, (rows, dim))
    st["w"] = [_codes(gen, (hd, dim)) for _ in range(4)]
    st["rope"] = _rope(lens, d)
    st["scale"] = VEC * VEC / math.sqrt(dim)
    return st


def _prepare_train_block(c, gen, seed):
    rows, heads, d = c["rows"], c["heads"], c["d"]
    hd = heads * d
    lens = _frag_lens(c)
    cfg = ops.make_cfg("i8", "e4m3", d, d, out_dtype=torch.bfloat16, grad_dtype=torch.bfloat16)
    st = _attention_state(c, cfg, heads, rows, lens)
    st["bws"] = _workspace(abi.lib().tsa_att_bwd_workspace_bytes(cfg, heads, rows))
    st["raw"] = [_normal(gen, rows, hd, 1.0, torch.bfloat16) for _ in range(3)]  # q, k, v as the projections left them
    st["comb"] = _normal(gen, rows, hd, 1.0, torch.bfloat16)                     # combiner keys
    st["dkv"] = _normal(gen, rows, 4 * hd, 1e-2, torch.bfloat16)
    st["rope"] = _rope(lens, d)
    return st


def _prepare_decode(c, gen, seed):
    seqs, heads, d = c["seqs"], c["heads"], c["d"]
    ctx = _contexts(c)
    scale_t = DTYPES[c["scale"]]
    cache = ops.KVCache(seqs, max(ctx) + 2, heads, d, DEV, scale_dtype=scale_t, out_dtype=DTYPES[c["out"]], qk_vec_scale=VEC)
    for s in range(seqs):
        cache.k[s] = _codes(gen, cache.k[s].shape)
        cache.v[s] = _codes(gen, cache.v[s].shape)
    cache.k_scale.copy_((torch.rand(cache.k_scale.shape, generator=gen, device=DEV) + 0.5) * VEC)
    cache.v_scale.fill_(VEC)
    tokens = [[_codes(gen, (seqs, heads * d)) for _ in range(3)] for _ in range(2)]
    scales = [((torch.rand((seqs, heads), generator=gen, device=DEV) + 0.5) * VEC).to(scale_t) for _ in range(2)]
    return dict(case=c, cache=cache, lens=torch.tensor(ctx, dtype=torch.int32, device=DEV), longest=max(ctx), tokens=tokens, k_scales=scales,
                v_scale=torch.full((seqs, heads), VEC, dtype=scale_t, device=DEV), status=torch.zeros(1, dtype=torch.int32, device=DEV),
                out=[torch.empty((seqs, heads * d), dtype=DTYPES[c["out"]], device=DEV) for _ in range(2)])


def _prepare_infer(c, gen, seed):
    seqs, heads, d = c["seqs"], c["heads"], c["d"]
    dim = hs = heads * d
    relu = heads * 128 * c["relu_mult"]
    rng = np.random.default_rng(seed)

    def mat(rows, cols):
        return rng.integers(-60, 61, (rows, cols), dtype=np.int8)

    layers = [dict(qk=mat(hs, dim), qv=mat(hs, dim), k=mat(hs, dim), v=mat(hs, dim), combiner=mat(dim, hs * 4), expand=mat(relu, dim),
                   contract=mat(dim, relu), qv_scale=1 / 32.0, combiner_scale=1 / 32.0, contract_scale=1 / 32.0, width=width, slope=slope)
              for width, slope in _layer_plan(c)]
    vocab = c["vocab"]
    ctx = _contexts(c)
    model = infer.InferModel(dict(dim=dim, head_dim=d, heads=heads, relu_mult=c["relu_mult"], vocab=vocab, label_count=vocab + 33, layers=layers,
                                  label_embed=mat(vocab + 33, dim), label_embed_scale=1 / 32.0, final_layer=mat(vocab, dim),
                                  final_layer_scale=1 / 32.0, bias=np.zeros(vocab, dtype=np.float32)), _rope([max(ctx) + 2], d).cpu().numpy(), DEV)
    ic = infer.InferContext(model, seqs, max(ctx) + 2)
    for l in range(c["layers"]):
        ic.k[l].copy_(_codes(gen, ic.k[l].shape))
        ic.v[l].copy_(_codes(gen, ic.v[l].shape))
    ic.k_scale.copy_((torch.rand(ic.k_scale.shape, generator=gen, device=DEV) + 0.5) * VEC)
    ic.v_scale.fill_(VEC)
    ic.set_lengths(ctx)
    return dict(case=c, ic=ic, lens=ic.ctx_lens.clone(), longest=max(ctx),
                labels=[torch.randint(0, vocab, (seqs, c["labels"]), generator=gen, device=DEV, dtype=torch.int32) for _ in range(2)],
                prediction=[torch.empty((seqs, vocab), dtype=torch.float32, device=DEV) for _ in range(2)])


# ---------------------------------------------------------------------------------------------------- one pass
def run(state):
    return {"prefill": _run_prefill, "prefill_block": _run_prefill_block, "train": _run_train, "train_block": _run_train_block,
            "decode": _run_decode, "infer": _run_infer}[state["case"]["kind"]](state)


def _run_prefill(st):
    c = st["case"]
    return ops.att_fwd(st["cfg"], st["q"], st["k"], st["v"], st["sk"], st["mask"], c["slope"], c["heads"], qk_scale=st["sq"], v_scale=st["sv"],
                       out=st["out"], lse=st["lse"], workspace=st["ws"], status=st["status"])


def _run_train(st):
    c = st["case"]
    out, lse = _run_prefill(st)
    grads = ops.att_bwd(st["cfg"], st["q"], st["k"], st["v"], st["sk"], st["d_out"], out, lse, st["mask"], c["slope"], c["heads"],
                        qk_scale=st["sq"], v_scale=st["sv"], workspace=st["bws"], status=st["status"])
    return (out, lse) + grads


def _run_prefill_block(st):
    c, x, (wq, wk, wv, wc), rope = st["case"], st["x"], st["w"], st["rope"]
    heads, d = c["heads"], c["d"]
    args = dict(src_scale=st["scale"], status=st["status"])
    q, sq = ops.matmul_norm_rope_quant(x, wq, rope, "e4m3", heads, d, vec_scale=0.25, **args)
    k, sk = ops.matmul_norm_rope_quant(x, wk, rope, "e4m3", heads, d, vec_scale=0.25, **args)
    v, sv = ops.matmul_norm_rope_quant(x, wv, None, "e4m3", heads, d, vec_scale=0.25, **args)
    comb, sc = ops.matmul_norm_rope_quant(x, wc, None, torch.bfloat16, heads, d, vec_scale=1.0, **args)
    out, lse = ops.att_fwd(st["cfg"], q, k, v, sk, st["mask"], c["slope"], heads, qk_scale=sq, v_scale=sv, workspace=st["ws"], status=st["status"])
    return ops.kv_product(comb, out, heads, d), out, lse, q, sq, k, sk, v, sv, comb, sc


def _run_train_block(st):
    c, (rq, rk, rv), rope = st["case"], st["raw"], st["rope"]
    heads, d = c["heads"], c["d"]
    q, sq = ops.norm_rope_quant(rq, rope, "i8", heads, d, vec_scale=VEC)
    k, sk = ops.norm_rope_quant(rk, rope, "i8", heads, d, vec_scale=VEC)
    v, sv = ops.norm_rope_quant(rv, None, "e4m3", heads, d, vec_scale=0.25)
    out, lse = ops.att_fwd(st["cfg"], q, k, v, sk, st["mask"], c["slope"], heads, qk_scale=sq, v_scale=sv, workspace=st["ws"], status=st["status"])
    kv = ops.kv_product(st["comb"], out, heads, d)
    d_comb, d_out, d_scale = ops.kv_product_bwd(st["comb"], out, st["dkv"], heads, d)
    dq, dk, dv = ops.att_bwd(st["cfg"], q, k, v, sk, d_out, out, lse, st["mask"], c["slope"], heads, qk_scale=sq, v_scale=sv, d_scale=d_scale,
                             workspace=st["bws"], status=st["status"])
    gq = ops.rope_norm_bwd(rq, dq, rope, heads, d)
    gk = ops.rope_norm_bwd(rk, dk, rope, heads, d)
    gv = ops.rope_norm_bwd(rv, dv, None, heads, d)
    return kv, out, lse, d_comb, d_scale, gq, gk, gv


def _run_decode(st):
    """Two tokens of every sequence, so that the second attends to what the first appended; the counts go back first, as when
    a continuation is sampled again."""
    c, cache = st["case"], st["cache"]
    cache.ctx_lens.copy_(st["lens"])
    cache.max_ctx = st["longest"]
    for i in range(2):
        k, v, q = st["tokens"][i]
        cache.append(k, st["k_scales"][i], v, st["v_scale"], status=st["status"])
        cache.decode(q, None, c["window"], c["slope"], out=st["out"][i], status=st["status"])
    return st["out"], cache.ctx_lens


def _run_infer(st):
    """Two tokens of every sequence, counts back first (see _run_decode)."""
    ic = st["ic"]
    ic.ctx_lens.copy_(st["lens"])
    ic.max_ctx = st["longest"]
    for i in range(2):
        ic.compute_prediction(st["labels"][i], prediction=st["prediction"][i])
    return st["prediction"], ic.ctx_lens


# ---------------------------------------------------------------------------------------------------- work and tolerance
def work(case):
    """Bytes (each input read once, each output written once) and operations of one pass."""
    c = case
    kind, heads, d = c["kind"], c["heads"], c["d"]
    hd = heads * d
    if kind == "decode":
        esz, osz = torch.empty(0, dtype=DTYPES[c["scale"]]).element_size(), torch.empty(0, dtype=DTYPES[c["out"]]).element_size()
        keys = sum(min(n + i, c["window"]) for n in _contexts(c) for i in range(2))
        tokens = 2 * c["seqs"]
        return {"bytes": keys * heads * (2 * d + 2 * esz) + tokens * hd * (5 + osz), "flops": 4.0 * keys * hd}
    if kind == "infer":
        relu = heads * 128 * c["relu_mult"]
        weights = c["layers"] * (8 * hd * hd + 2 * relu * hd) + c["vocab"] * hd
        keys = sum(min(n + i, w) for n in _contexts(c) for i in range(2) for w, _ in _layer_plan(c))
        tokens = 2 * c["seqs"]
        # the weights are needed once for each of the two tokens, which depend on one another
        return {"bytes": 2 * weights + keys * heads * (2 * d + 8) + tokens * (hd * c["labels"] + c["layers"] * 2 * hd + 4 * c["vocab"]),
                "flops": 2.0 * weights * tokens + 4.0 * keys * hd}
    rows, pairs = c["rows"], _pairs(c)
    plane = 4 * heads * rows
    forward = 4.0 * pairs * hd
    if kind == "prefill":
        osz = torch.empty(0, dtype=DTYPES[c["out"]]).element_size()
        return {"bytes": rows * hd * (3 + osz) + 4 * plane, "flops": forward}
    if kind == "prefill_block":
        # state, four matrices and rope in; three quantised planes, combiner keys, output and product out
        return {"bytes": rows * hd + 4 * hd * hd + 4 * rows * d + rows * hd * (3 + 2 + 2 + 8) + 5 * plane, "flops": forward + 8.0 * rows * hd * hd}
    if kind == "train":
        return {"bytes": rows * hd * (3 + 2 + 2 + 6) + 4 * plane, "flops": 3.5 * forward}
    # raw projections, combiner keys, dKv and rope in; product, output and four gradients out
    return {"bytes": rows * hd * 2 * (3 + 1 + 4 + 4 + 1 + 4) + 4 * rows * d + 2 * plane, "flops": 3.5 * forward}


def tolerance(case):
    if case["kind"] == "infer":
        # every stage of a token is rounded to int8 codes again: attention sums in another order flip a few of those roundings by
        # one code, and twelve layers pass the flips on
        return {"rel": 2e-2, "max": 0.25}
    if case["kind"] == "decode":
        # weights are 16-bit integers relative to their batch's largest; 16-bit outputs round once more
        return {"rel": 1e-4 if case["out"] == "f32" else 4e-3}
    # weights in e4m3, gradients through bf16 products, 16-bit outputs
    return {"rel": 1e-2}
