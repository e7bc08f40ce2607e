"""The latent attention's tensor-memory kernel (csrc/attention_latent_tc.cu) against float64: rows that fill and do not fill a
tile, heads that do and do not divide it, portions after a past, several requests with single tokens among them,
windows, sinks, page sizes; unused cache slots hold NaN."""
import pytest
import torch

from gpu_util import Harness
from vosti_b200 import ops
from vosti_b200.engine.batch import StepEntry
from vosti_b200.parts import PagedCacheSpec

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
RANK, ROT = 512, 64


@pytest.mark.parametrize("heads,lengths,past,page,window,with_sink", [
    (16, (8,), (0,), 16, 0, False), (16, (33,), (0,), 16, 0, True), (16, (40, 1, 9), (100, 77, 0), 16, 0, False),
    (5, (131, 27), (3, 0), 48, 0, True), (128, (3, 2), (0, 61), 32, 0, False), (16, (150,), (13,), 16, 40, False),
    (16, (64, 1, 5), (0, 95, 31), 16, 32, True), (16, (700,), (0,), 16, 0, False)])
def test_against_float64(monkeypatch, heads, lengths, past, page, window, with_sink):
    gen = torch.Generator(device=DEV).manual_seed(sum(lengths) + heads)
    normal = lambda *s, std=1.0: torch.randn(*s, generator=gen, device=DEV) * std
    T = sum(lengths)
    pages = sum(-(-(n + p) // page) for n, p in zip(lengths, past)) + 3
    harness = Harness([PagedCacheSpec(entries=2, heads=1, width=RANK, widths=(RANK, ROT))], [None], torch.bfloat16,
                      num_pages=pages, page_size=page, max_requests=len(lengths))
    if any(past):
        harness.context([StepEntry(i, [0] * p) for i, p in enumerate(past) if p])
    ctx = harness.context([StepEntry(i, [0] * n) for i, n in enumerate(lengths)])
    layer = harness.cache.layer_caches[0]
    for pool in layer.tensors:
        pool.fill_(float("nan"))
    keys = []
    for i, (n, p) in enumerate(zip(lengths, past)):
        at = torch.arange(n + p, device=DEV)
        where = ctx.groups[0].block_table[i, at // page].long()
        rows = (normal(n + p, 1, RANK).bfloat16(), normal(n + p, 1, ROT).bfloat16())
        for pool, row in zip(layer.tensors, rows):
            pool[where, :, at % page] = row
        keys.append((rows[0][:, 0].double(), rows[1][:, 0].double()))
    qk = normal(T, heads, RANK + ROT, std=0.3).bfloat16()
    sink = normal(heads, std=2.0) if with_sink else None
    scale = 0.07
    monkeypatch.setattr(ops, "LATENT_MMA_SPLIT_BELOW", 0)      # no cutting of keys: every portion of enough rows comes here
    calls = []
    monkeypatch.setattr(ops, "_check", lambda code, what, kernels=1, check=ops._check: (calls.append(what), check(code, what, kernels))[1])
    got = ops.latent_attend(ctx, qk, layer.k, layer.v, ctx.groups[0], scale=scale, window=window, sink=sink).double()
    assert calls == ["latent_attend_tc"] and harness.status.item() == 0
    at = 0
    for (n, p), (c, r) in zip(zip(lengths, past), keys):
        q = qk[at:at + n].double()
        scores = (torch.einsum("nhd,kd->nhk", q[..., :RANK], c) + torch.einsum("nhd,kd->nhk", q[..., RANK:], r)) * scale
        pos, key = torch.arange(p, p + n, device=DEV)[:, None], torch.arange(n + p, device=DEV)[None, :]
        seen = (key <= pos) & ((key > pos - window) if window else True)
        scores = scores.masked_fill(~seen[:, None, :], float("-inf"))
        if sink is not None:
            scores = torch.cat([scores, sink.double()[None, :, None].expand(n, heads, 1)], -1)
        weights = torch.softmax(scores, -1)[..., :n + p]
        want = torch.einsum("nhk,kd->nhd", weights, c)
        # the weights carry 16 bits (two bfloat16 terms), the scores are float32 sums of 576 products
        assert torch.allclose(got[at:at + n], want, atol=2e-4, rtol=2e-4), float((got[at:at + n] - want).abs().max())
        at += n


def test_the_cut_does_not_show_in_fixed_order():
    """With one order of arithmetic asked for, no kernel is chosen by how many tokens a portion has: a prompt in one
    portion (640 rows) and in portions of five tokens (80 rows) gives the same bits."""
    heads, T, page = 16, 40, 16
    gen = torch.Generator(device=DEV).manual_seed(9)
    normal = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    qk, rows = (normal(T, heads, RANK + ROT) * 0.3).bfloat16(), (normal(T, RANK).bfloat16(), normal(T, ROT).bfloat16())
    got = []
    ops.set_fixed_order(True)
    try:
        for cut in (T, 5):
            harness = Harness([PagedCacheSpec(entries=2, heads=1, width=RANK, widths=(RANK, ROT))], [None], torch.bfloat16,
                              num_pages=8, page_size=page)
            layer, parts = harness.cache.layer_caches[0], []
            for first in range(0, T, cut):
                ctx = harness.context([StepEntry("r", [0] * cut)])
                at = torch.arange(first, first + cut, device=DEV)
                for pool, row in zip(layer.tensors, rows):
                    pool[ctx.groups[0].block_table[0, at // page].long(), 0, at % page] = row[first:first + cut]
                parts.append(ops.latent_attend(ctx, qk[first:first + cut].contiguous(), layer.k, layer.v, ctx.groups[0], scale=0.07))
            got.append(torch.cat(parts))
    finally:
        ops.set_fixed_order(False)
    assert torch.equal(*got)
