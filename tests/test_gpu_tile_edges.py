"""The sizes at which the kernels' tiles, half tiles, rings and work splits end, against the CPU oracle."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests import util
from tests.test_gpu_attention import _run_fwd
from tests.test_gpu_infer import _deviation, _run_gpu
from tests.test_gpu_quant_decode import _decode_case

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _custom(rows):
    spans, ptr = [], [0]
    for r in rows:
        spans.extend(r)
        ptr.append(len(spans))
    return np.array(spans, dtype=np.int32).reshape(-1, 2), np.array(ptr, dtype=np.int32)


def _edge_rows(length):
    """Spans that begin and end on both sides of the 64-key halves and 128-key tiles; a tile of rows without keys."""
    rows = []
    for i in range(length):
        first = (0, 1, 63, 64, 65, 127, 128, 129)[i % 8]
        last = first + (0, 1, 62, 63, 64, 65, 126, 127, 128, 129)[i % 10]
        if 128 <= i < 256 or i == 0:
            rows.append([])
        else:
            rows.append([(min(first, length - 1), min(last, length - 1))])
    return rows


@pytest.mark.parametrize("length", [1, 129, 391])
@pytest.mark.parametrize("d,qk_dtype,v_dtype,slope", [(64, "e4m3", "e4m3", 0.0), (128, "i8", "e4m3", 0.5), (64, "i8", "i8", 0.0)])
def test_fwd_half_tiles(length, d, qk_dtype, v_dtype, slope):
    rows = _edge_rows(length) if length > 1 else [[(0, 0)]]
    out, lse, ref, _ = _run_fwd(50, [length], None, slope, 3, d, qk_dtype, v_dtype, out_dtype=torch.float32, scale=0.5, custom=_custom(rows))
    mx, mean = util.err_stats(out, ref["out"])
    assert mx < util.OUT_MAX_ABS and mean < util.OUT_MEAN_ABS, util.describe(out, ref["out"])
    assert util.err_stats(lse, ref["lse"])[0] < 2e-3, util.describe(lse, ref["lse"])


@pytest.mark.parametrize("step", [-0.05, 0.02, 0.11, 3.0])   # log2 units from key to key: no raise, one now and then, one per group, one per key
@pytest.mark.parametrize("d,qk_dtype,v_dtype,window,slope,form", [
    (64, "e4m3", "e4m3", 0, 0.0, "plain"), (128, "e4m3", "e4m3", 0, 0.0, "plain"), (128, "i8", "e4m3", 0, 0.0, "plain"),
    (64, "i8", "e4m3", 200, 0.0, "plain"), (64, "e4m3", "e4m3", 0, 0.01, "plain"), (64, "i8", "i8", 0, 0.0, "plain"),
    (64, "e4m3", "e4m3", 0, 0.0, "to"), (128, "i8", "e4m3", 0, 0.01, "to"), (64, "i8", "e4m3", 200, 0.0, "to"),
    (64, "e4m3", "e4m3", 0, 0.01, "kv"), (128, "i8", "e4m3", 0, 0.0, "kv"),
])
def test_fwd_rising_logits(step, d, qk_dtype, v_dtype, window, slope, form):
    """Logits that rise along the keys: the reference moves in full halves and in masked blocks, first groups and later ones, and the
    weights formed in front of the vote have to be formed again.  Also with int8 values, with two further destinations and with the
    fused consumer, which are kernels of their own.

    The values are positive, so that an output is bounded by its own size.  P = 128 w sv / svRef is rounded to e4m3: by 2^-4 of itself at
    most, or by 2^-10 where it is subnormal (svRef, the power of two at or above the scales, is 2); with int8 values the residual takes all
    but 2^-4 of that away again, or down to 2^-10.  2^-10 stands for 2^-17 svRef in the sum of w v.  A block that is shrunk again is rounded
    once more, on what the residual left (2^-8).  The sum of the weights is not rounded; a bf16 output by 2^-9."""
    from tscale_b200 import abi, ops
    rows, heads = 420, 2
    c = 0.5 / np.sqrt(d) / 0.693147
    one = 0x38 if qk_dtype == "e4m3" else 1   # the vectors are all ones, their product is d
    q8 = torch.full((rows, heads * d), one, dtype=torch.uint8, device=DEV)
    sk = (torch.arange(rows, dtype=torch.float64) * step / (d * c)).to(torch.float32).expand(heads, rows).contiguous()
    sq = torch.ones(heads, rows)
    gen = torch.Generator().manual_seed(60)
    if v_dtype == "e4m3":
        v8 = (torch.randn(rows, heads * d, generator=gen).abs() + 0.25).to(torch.float8_e4m3fn)
    else:
        v8 = torch.randint(1, 128, (rows, heads * d), generator=gen, dtype=torch.int8)
    sv = torch.rand(heads, rows, generator=gen) + 0.5
    out_dtype = torch.bfloat16 if form == "kv" else torch.float32
    cfg = ops.make_cfg(qk_dtype, v_dtype, d, d, out_dtype=out_dtype)
    ws = torch.empty(max(1, abi.lib().tsa_att_fwd_workspace_bytes(cfg, heads, rows)), dtype=torch.uint8, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    copies = [torch.zeros(rows, heads * d, dtype=out_dtype, device=DEV) for _ in range(2)] if form == "to" else None
    comb = torch.ones(rows, heads * d, dtype=torch.bfloat16, device=DEV) if form == "kv" else None
    out, lse, *kv = ops.att_fwd(cfg, q8, q8, v8.view(torch.uint8).to(DEV), sk.to(DEV), ops.Mask.window([rows], window), slope, heads,
                                qk_scale=sq.to(DEV), v_scale=sv.to(DEV), workspace=ws, status=status, out_copies=copies, combiner_k=comb)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    i = torch.arange(rows)
    seen = (i[None, :] < i[:, None]) & ((i[None, :] >= i[:, None] - window) if window else True)
    z = ((sk[0].double() * d * c).expand(rows, rows) - slope * (i[:, None] - i[None, :])).masked_fill(~seen, -np.inf)
    m = z.amax(1, keepdim=True).clamp_min(0)
    w = torch.exp2(z - m)
    total = w.sum(1, keepdim=True) + torch.exp2(-m)
    v = v8.double().view(rows, heads, d)
    want = torch.einsum("ij,jhd->ihd", w / total, v * sv.t().double()[:, :, None])
    bound = (2.0 ** -4 + 2.0 ** -8 if v_dtype == "e4m3" else 2.0 ** -8 + 2.0 ** -8) * want
    bound += 2.0 ** -17 * 2 * torch.einsum("ij,jhd->ihd", seen.double() / total, v)
    if form == "kv":
        bound += 2.0 ** -9 * want
    err = (out.cpu().double().view(rows, heads, d) - want).abs()
    assert (err <= bound).all(), float((err / bound.clamp_min(1e-30)).max())
    want_lse = (m + torch.log2(total))[:, 0]
    assert ((lse.cpu().double() - want_lse).abs() <= 2e-5 + 1e-6 * want_lse.abs()).all()
    for copy in copies or []:
        assert torch.equal(copy, out)
    if kv:   # keys of one: each of the four blocks is the output
        assert torch.equal(kv[0].view(rows, heads, 4, d), out.view(rows, heads, 1, d).expand(-1, -1, 4, -1))


@pytest.mark.parametrize("length,heads", [(1, 1), (129, 3), (391, 2), (2200, 10)])   # the last: more items than CTAs
@pytest.mark.parametrize("d,grad,pad", [(64, torch.bfloat16, 0), (128, torch.float32, 4), (64, torch.float16, 8), (128, torch.bfloat16, 8)])
def test_bwd_work_items(length, heads, d, grad, pad):
    """Ragged row tiles, row tiles without keys, one and many work items per CTA; `pad` leaves the gradients' rows aligned to 16
    bytes but not to 32."""
    from tscale_b200 import abi, ops
    rows = _edge_rows(length) if length > 1 else [[(0, 0)]]
    out, lse, ref, (g, mask, cfg, spans, ptr, (qd, kd, vd)) = _run_fwd(
        51, [length], None, 0.25, heads, d, "i8", "e4m3", out_dtype=torch.float32, scale=0.5, custom=_custom(rows))
    d_out = (np.random.default_rng(52).standard_normal(out.shape) * 1e-2).astype(np.float32)
    gref = O.att_bwd(qd, kd, vd, d_out, spans, ptr, heads, 0.25, fwd=ref)
    cfg = ops.make_cfg("i8", "e4m3", d, d, out_dtype=torch.float32, grad_dtype=grad)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
    do_t, out_t, lse_t = t(d_out).to(grad), t(ref["out"]), t(ref["lse"])
    whole = [torch.full((length, heads * d + pad), 7.0, dtype=grad, device=DEV) for _ in range(3)]
    dq, dk, dv = (w[:, :heads * d] for w in whole)
    ws = torch.empty(max(1, abi.lib().tsa_att_bwd_workspace_bytes(ctypes.byref(cfg), heads, length)), dtype=torch.uint8, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    p, q = ops.p2d, lambda x: ctypes.c_void_p(x.data_ptr())
    groups, gptr, rgroups, rgptr = mask.dev(DEV)
    abi.check(abi.lib().tsa_att_bwd(ctypes.byref(cfg), None, p(g["q8"]), p(g["k8"]), p(g["sq"]), p(g["sk"]), p(g["v8"]), p(g["sv"]),
                                    p(do_t), p(out_t), p(None), p(lse_t), q(groups), q(gptr), q(rgroups), q(rgptr), 0.25, 1.0,
                                    p(dq), p(dk), p(dv), heads, mask.len_att_tiles, q(ws), ws.numel(), q(status), None))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for name, got, w in (("dq", dq, whole[0]), ("dk", dk, whole[1]), ("dv", dv, whole[2])):
        assert util.rel_l2(util.to_np(got.float()), gref[name]) < util.GRAD_REL_L2, name
        assert pad == 0 or bool((w[:, heads * d:] == 7).all()), name
    empty = [i for i, r in enumerate(rows) if not r]
    assert not empty or float(dq[empty].float().abs().max().item()) == 0


@pytest.mark.parametrize("rows,length,dim,heads,d,with_rope", [
    (1, 1, 128, 1, 64, True), (129, 128, 1152, 5, 64, True), (127, 127, 256, 3, 128, False), (5121, 5000, 256, 17, 64, True),
])
@pytest.mark.parametrize("dst", ["i8", torch.float16])
def test_projection_tiles(dst, rows, length, dim, heads, d, with_rope):
    """Remainders of the 128 x 256 tiles of single CTAs."""
    from tscale_b200 import ops
    rng = np.random.default_rng(rows + dim)
    x = rng.integers(-127, 128, (rows, dim)).astype(np.int8)
    w = rng.integers(-127, 128, (heads * d, dim)).astype(np.int8)
    src_scale = np.float32(1.0 / 4096)
    y = (x[:length].astype(np.float64) @ w.T.astype(np.float64)).astype(np.float32) * src_scale
    table = O.fill_rope(d, rows) if with_rope else None
    want_b, want_s, roped = O.norm_rope_quant("i8", 0.5, y, None if table is None else table[:length], d)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    got, got_s = ops.matmul_norm_rope_quant(torch.from_numpy(x).to(DEV), torch.from_numpy(w).to(DEV),
                                            None if table is None else torch.from_numpy(table).to(DEV), dst, heads, d,
                                            vec_scale=0.5, src_scale=float(src_scale), length=length, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    got, got_s = got.cpu(), got_s.cpu().numpy()
    assert np.array_equal(got_s[:, :length], want_s) and np.abs(got_s[:, length:]).max(initial=0) == 0
    want = torch.from_numpy(want_b.view(np.int8)) if dst == "i8" else torch.from_numpy(roped).to(dst)
    assert torch.equal(got[:length].view(want.dtype), want)
    assert not bool(got[length:].view(want.dtype).float().any())


@pytest.mark.parametrize("dst", ["i8", torch.bfloat16])
@pytest.mark.parametrize("rows,dim,heads,d", [
    (1, 64, 1, 64), (128, 192, 1, 128), (129, 64, 3, 64), (256, 320, 5, 64), (257, 2048, 3, 128), (20000, 192, 5, 128),
])
def test_projection_pairs(dst, rows, dim, heads, d):
    """One to three row tiles, heads that leave part of the columns' weights past the matrix, one chunk to many."""
    test_projection_tiles(dst, rows, rows, dim, heads, d, True)


@pytest.mark.parametrize("dst", ["i8", torch.bfloat16])
@pytest.mark.parametrize("rows,length,dim,heads,d", [
    (1, 1, 1344, 1, 64), (128, 128, 1344, 1, 128), (129, 128, 1280, 3, 64), (256, 200, 1344, 5, 64), (385, 385, 1408, 2, 128),
    # on both sides of the lines between single CTAs and pairs: the inner size, and one tile of 128 x 256 for each of 148 SMs or one more
    (300, 300, 960, 4, 64), (300, 300, 1024, 4, 64), (18944, 18900, 1024, 4, 64), (18945, 18945, 1024, 4, 64), (18945, 18945, 1088, 4, 64),
])
def test_projection_pair_tiles(dst, rows, length, dim, heads, d):
    """Tiles of 256 rows x 256 columns shared by two CTAs, 128 columns of x at a time: a second CTA without rows, half or all of
    its columns' weights past the matrix, an inner size that ends in half a chunk."""
    test_projection_tiles(dst, rows, length, dim, heads, d, True)


@pytest.mark.parametrize("src,dst", [("i8", "i8"), ("i8", torch.float16), ("e4m3", "i8")])
@pytest.mark.parametrize("rows,dim,heads,d,with_rope", [
    (69, 64, 2100, 128, True), (4000, 192, 132, 64, False),      # single CTAs: 1050 and 32 x 33 tiles on 148, at least seven each
    (257, 1344, 520, 128, True), (2048, 1280, 268, 64, False),   # pairs: 2 x 260 and 8 x 67 tiles on 74, at least seven each
])
def test_projection_many_tiles(src, dst, rows, dim, heads, d, with_rope):
    """Several tiles for every CTA or pair: the ring goes round many times, both accumulator sets are waited for in both parities, the
    rope rows change under way.  e4m3 operands: the sums are formed in f32, in steps of 32 products; with a rounding of 2^-22 of a sum
    per step (nothing is known of the order inside) a value is off by dim / 32 * 2^-22 of the largest partial sum, and so is a scale at most.
    A code changes where the value lies that close to a rounding boundary: 2 * 127 * that bound of them."""
    from tscale_b200 import ops
    gen = torch.Generator(device=DEV).manual_seed(rows + dim)
    if src == "i8":
        x, w = (torch.randint(-127, 128, (n, dim), dtype=torch.int8, device=DEV, generator=gen) for n in (rows, heads * d))
        src_scale = float(np.float32(1.0 / 4096))
    else:
        x, w = ((torch.randn(n, dim, device=DEV, generator=gen) * 0.7).to(torch.float8_e4m3fn) for n in (rows, heads * d))
        src_scale = 1.0
    # float64 holds every sum of these products exactly
    y = (x.double() @ w.double().t()).float().cpu().numpy() * np.float32(src_scale)
    table = O.fill_rope(d, rows) if with_rope else None
    vec = 1 / 24.0 if src == "e4m3" else 0.5
    want_b, want_s, roped = O.norm_rope_quant("i8", vec, y, table, d)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    got, got_s = ops.matmul_norm_rope_quant(x.view(torch.int8), w.view(torch.int8), None if table is None else torch.from_numpy(table).to(DEV), dst,
                                            heads, d, vec_scale=vec, src_scale=src_scale, status=status, src=src)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    got, got_s = got.cpu(), got_s.cpu().numpy()
    if src == "e4m3":
        bound = dim / 32 * 2.0 ** -22
        codes, want = got.view(torch.int8).numpy().astype(np.int32), want_b.view(np.int8).astype(np.int32)
        assert np.abs(got_s - want_s).max() <= bound * want_s.max()
        assert np.abs(codes - want).max() <= 1 and np.mean(codes != want) <= 2 * 127 * bound
    else:
        want = torch.from_numpy(want_b.view(np.int8)) if dst == "i8" else torch.from_numpy(roped).to(dst)
        assert np.array_equal(got_s, want_s) and torch.equal(got.view(want.dtype), want)


@pytest.mark.parametrize("ctx,heads,d,window,slope", [
    ([9001], 5, 128, 100000, 0.0), ([4097, 3, 0, 2000], 2, 64, 3000, 0.25), ([1], 7, 64, 100000, 0.0),
])
def test_decode_chunk_merge(ctx, heads, d, window, slope):
    _decode_case(53, ctx, heads, d, window, slope)


@pytest.mark.parametrize("dim,d,heads,relu_mult,n_seq,steps,layers", [
    (256, 128, 5, 1, 3, 70, 2),     # heads that do not fill an attention group
    (384, 64, 12, 1, 2, 70, 2),     # several tokens per load, the last group of heads partly empty
    (256, 64, 1, 3, 64, 3, 2),      # one head, the largest batch
    (256, 64, 1, 1, 1, 2, 33),      # more layers than one launch carries
])
def test_infer_groups(dim, d, heads, relu_mult, n_seq, steps, layers):
    model = O.make_infer_model(54, dim, d, heads, relu_mult, 90, 16, [((100000, 24)[i % 2], (0.0, 0.5)[i % 2]) for i in range(layers)])
    streams = np.random.default_rng(55).integers(0, 16, (min(n_seq, 3), steps, 1)).astype(np.int32)
    labels = streams[np.arange(n_seq) % len(streams)]
    pred, logits = _run_gpu(model, labels, want_logits=True)
    want = np.zeros_like(pred[:len(streams)])
    for s in range(len(streams)):
        orc = O.InferOracle(model, steps, exp_mode="exact")
        for t in range(steps):
            want[s, t], want_logits = orc.step(streams[s, t], want_logits=True)
            if t == 0:
                assert np.array_equal(logits[s, 0], want_logits), s
    dev = _deviation(pred[:len(streams)], want)
    # one int8 rounding that falls the other way stays in the caches and moves every later step by 1e-2
    assert dev.max() < 8e-2 and np.median(dev) < 2e-2 and dev[:, :2].max() < 1e-5, (dev.max(), np.median(dev))
    for s in range(len(streams), n_seq):
        assert np.array_equal(logits[s], logits[s % len(streams)]) and np.array_equal(pred[s], pred[s % len(streams)]), s
