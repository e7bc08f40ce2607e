"""Latent attention over keys and values formed for every head (csrc/attention_latent_heads.cu) against float64: portions that
fill and do not fill a tile, after a past, several requests with single tokens among them, page sizes, sinks and both gates; unused
cache slots hold NaN."""
import pytest
import torch

from gpu_util import Harness
from vosti_b200 import ops
from vosti_b200.engine.batch import StepEntry
from vosti_b200.parts import PagedCacheSpec

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DIM, ROT = 128, 64


@pytest.mark.parametrize("heads,rank,lengths,past,page,with_sink,gate", [
    (16, 512, (8,), (0,), 16, False, "head"), (16, 512, (129,), (0,), 16, True, "none"), (4, 512, (40, 1, 9), (100, 77, 0), 16, False, "element"),
    (8, 256, (131, 27), (3, 0), 48, True, "head"), (40, 512, (300, 2), (0, 61), 32, False, "none"), (16, 512, (700,), (13,), 16, False, "head"),
    (2, 64, (64, 128, 256, 65), (0, 64, 0, 63), 64, True, "element"), (160, 128, (260,), (0,), 16, False, "head")])
def test_against_float64(heads, rank, lengths, past, page, with_sink, gate):
    gen = torch.Generator(device=DEV).manual_seed(sum(lengths) + heads)
    normal = lambda *s, std=1.0: torch.randn(*s, generator=gen, device=DEV) * std
    T = sum(lengths)
    pages = sum(-(-(n + p) // page) for n, p in zip(lengths, past)) + 3
    harness = Harness([PagedCacheSpec(entries=2, heads=1, width=rank, widths=(rank, ROT))], [None], torch.bfloat16,
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
        rows = (normal(n + p, 1, rank).bfloat16(), normal(n + p, 1, ROT).bfloat16())
        for pool, row in zip(layer.tensors, rows):
            pool[where, :, at % page] = row
        keys.append((rows[0][:, 0].double(), rows[1][:, 0].double()))
    q_width = heads * (DIM + ROT)
    width = q_width + (heads * DIM if gate == "element" else 8)
    proj = normal(T, width).bfloat16()
    qr = normal(T, heads, ROT).bfloat16()
    kv_up = normal(2 * heads * DIM, rank, std=rank ** -0.5).bfloat16()
    sink = normal(heads, std=2.0) if with_sink else None
    head_gate = torch.rand(T, heads, generator=gen, device=DEV) if gate == "head" else None
    element = proj[:, q_width: q_width + heads * DIM] if gate == "element" else None
    scale = 0.07
    assert ops.library().vosti_latent_heads_fits(DIM, ROT, DIM, rank, page, width)
    outs = [ops.latent_attend_heads(ctx, proj, qr, kv_up, layer.k, layer.v, ctx.groups[0], heads=heads, dim=DIM, scale=scale, sink=sink,
                                    gate=head_gate, element_gate=element) for _ in range(2)]
    assert torch.equal(*outs) and harness.status.item() == 0
    got = outs[0].double()
    at = 0
    up = kv_up.double().view(2, heads, DIM, rank)
    for (n, p), (c, r) in zip(zip(lengths, past), keys):
        k = torch.einsum("kr,hdr->khd", c, up[0]).float().bfloat16().double()          # keys are rounded, values are not
        v = torch.einsum("kr,hdr->khd", c, up[1])
        q = proj[at:at + n, :q_width].double().view(n, heads, DIM + ROT)[..., :DIM]
        scores = (torch.einsum("nhd,khd->nhk", q, k) + torch.einsum("nhd,kd->nhk", qr[at:at + n].double(), r)) * scale
        seen = torch.arange(n + p, device=DEV)[None, :] <= torch.arange(p, p + n, device=DEV)[:, None]
        scores = scores.masked_fill(~seen[:, None, :], float("-inf"))
        if sink is not None:
            scores = torch.cat([scores, sink.double()[None, :, None].expand(n, heads, 1)], -1)
        want = torch.einsum("nhk,khd->nhd", torch.softmax(scores, -1)[..., :n + p], v)
        if head_gate is not None:
            want = want * head_gate[at:at + n].double()[..., None]
        if element is not None:
            want = want * torch.sigmoid(element[at:at + n].double().view(n, heads, DIM))
        # the result's own rounding (2^-9), and keys whose product lies at a tie of their rounding (2^-9 of one of 128 terms of a
        # score, of size scale: a weight moves by less than 2^-9 of itself)
        assert bool(((got[at:at + n] - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -9 * want.pow(2).mean().sqrt()).all())
        at += n
