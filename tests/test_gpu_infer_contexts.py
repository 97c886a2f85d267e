"""The token step over caches that already hold unequal contexts: chunks of the keys, the units that take them and the merge of
their partials, against the CPU oracle and between slots of a batch."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

DEV = torch.device("cuda:0")
CONTEXTS = [0, 1, 63, 64, 65, 700, 3000, 8000]
# Logits of one step of one layer, relative 2-norm.  With exact exp2 on both sides only the order of fp32 sums and the 16-bit weights of a
# batch differ (2^-17 of its largest).  That turns a combiner code next to a rounding boundary over now and then, and with it perhaps a
# code or two of the final state, each of which moves the logits by 1 / (24 sqrt(dim)) = 2.6e-3 (the relu block, which would pass on more, is
# scaled to nothing).  32 keys missing from 8000 move them by 3.5e-2 and more.
TOL = 1e-2


def _model(dim, d, heads, layers):
    model = O.make_infer_model(60, dim, d, heads, 1, 256, 16, layers)
    for layer in model["layers"]:
        layer["contract_scale"] = np.float32(0)
    return model


def _caches(rng, layers, tokens, heads, d):
    """Keys that are attended about evenly; every 32 tokens have values of their own, so that no part of a context repeats another."""
    row = heads * d
    keys = rng.integers(-127, 128, (layers, tokens, row)).astype(np.int8)
    signs = rng.integers(0, 2, (layers, (tokens + 31) // 32, row)) * 2 - 1
    vals = (signs.repeat(32, axis=1)[:, :tokens] * rng.integers(64, 128, (layers, tokens, row))).astype(np.int8)
    return keys, (rng.random((layers, tokens, heads)) * 4e-3 + 2e-3).astype(np.float32), vals, \
        (rng.random((layers, tokens, heads)) * 0.1 + 0.1).astype(np.float32)


def _oracle_logits(model, caches, label):
    orc = O.InferOracle(model, caches[0].shape[1] + 1, exp_mode="exact")
    orc.load(*caches)
    return orc.step([label], want_logits=True)[1].astype(np.float64)


def _gpu_context(model, caches):
    from tscale_b200 import infer
    lens = [c[0].shape[1] for c in caches]
    ctx = infer.InferContext(infer.InferModel(model, O.fill_rope(model["head_dim"], max(lens) + 8), DEV), len(caches), max(lens) + 8)
    for s, n in enumerate(lens):
        for dst, src in zip((ctx.k, ctx.k_scale, ctx.v, ctx.v_scale), caches[s]):
            dst[:, s, :n] = torch.from_numpy(src).to(DEV)
    ctx.set_lengths(lens)
    return ctx


def _deviation(got, want):
    return float(np.linalg.norm(got - want) / np.linalg.norm(want))


def test_missing_keys_show():
    """The tolerance of the comparison below tells a context from one with 32 of its keys left out."""
    model = _model(256, 64, 3, [(100000, 0.0)])
    rng = np.random.default_rng(61)
    for tokens in (65, 700, 3000, 8000):
        caches = _caches(rng, 1, tokens, 3, 64)
        want = _oracle_logits(model, caches, 1)
        for first in (0, tokens // 64 * 32, tokens - 32):
            scales = caches[3].copy()
            scales[0, first:first + 32] = 0
            assert _deviation(_oracle_logits(model, caches[:3] + (scales,), 1), want) > 2 * TOL, (tokens, first)


@pytest.mark.gpu
@pytest.mark.parametrize("d,heads,window,slope", [
    (64, 3, 100000, 0.0),     # one head per load, eight streams; chunks of three parts
    (128, 5, 100000, 0.0),    # one head per load, four streams
    (64, 12, 100000, 0.25),   # four heads, two streams
    (64, 12, 64, 0.5),        # rows that fit a unit, all of them apart
    (64, 16, 3000, 0.0),      # eight heads, one stream
    (64, 16, 64, 0.5),        # two units per row
    (64, 17, 100000, 0.0),    # chunks of one part
    (128, 4, 0, 0.0),         # the new token alone
])
def test_contexts_against_oracle(d, heads, window, slope):
    model = _model(256, d, heads, [(window, slope)])
    rng = np.random.default_rng(62)
    caches = [_caches(rng, 1, n, heads, d) for n in CONTEXTS]
    ctx = _gpu_context(model, caches)
    labels = rng.integers(0, 16, (len(CONTEXTS), 1)).astype(np.int32)
    logits = torch.empty((len(CONTEXTS), 256), dtype=torch.float32, device=DEV)
    ctx.compute_prediction(torch.from_numpy(labels).to(DEV), logits=logits)
    got = logits.double().cpu().numpy()
    assert int(ctx.status.item()) == 0
    assert ctx.ctx_lens.cpu().tolist() == [[n + 1 for n in CONTEXTS]]
    dev = [_deviation(got[s], _oracle_logits(model, caches[s], labels[s, 0])) for s in range(len(CONTEXTS))]
    assert max(dev) < TOL, dev


@pytest.mark.gpu
@pytest.mark.parametrize("d,heads", [(64, 12), (128, 4)])
def test_same_bits_in_any_slot(d, heads):
    """A batch of 64 that holds every sequence twice, the second time in another order: equal sequences give equal bits, whatever is
    in front of them.  Four layers and six steps: sums in another order would turn some code over."""
    model = _model(256, d, heads, [(100000, 0.0), (100000, 0.25), (64, 0.5), (900, 0.0)])
    rng = np.random.default_rng(63)
    caches = [_caches(rng, 4, int(n), heads, d) for n in rng.integers(100, 1500, 32)]
    order = np.concatenate([np.arange(32), rng.permutation(32)])
    ctx = _gpu_context(model, [caches[i] for i in order])
    logits = torch.empty((64, 256), dtype=torch.float32, device=DEV)
    for _ in range(6):
        labels = rng.integers(0, 16, (32, 1)).astype(np.int32)[order]
        prediction = ctx.compute_prediction(torch.from_numpy(labels).to(DEV), logits=logits)
        for t in (logits, prediction):
            back = torch.empty_like(t[32:])
            back[torch.from_numpy(order[32:]).to(DEV)] = t[32:]
            assert torch.equal(t[:32], back)
    assert int(ctx.status.item()) == 0
