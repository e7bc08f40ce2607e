"""The delta rules' long portions in chunks (csrc/delta_chunks.cu) against the recurrences in float64 and against
the token-by-token kernels: lengths around the chunk and the line between the two ways, ragged steps with short
requests between long ones, grouped heads, widths of the value side, decays of every kind (none, total,
mixed), start states, and containment of a token that is not finite."""
import pytest
import torch

from gpu_util import Harness
from vosti_b200 import ops
from vosti_b200.engine.batch import StepEntry
from vosti_b200.parts import StateSpec

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DK = 128


def decays(kind, T, heads, gen):
    u = torch.rand(T, heads, DK, generator=gen, dtype=torch.float64)
    if kind == "near one":
        return 0.98 + 0.02 * u
    if kind == "strong":
        return u ** 8                                  # down to underflow within a chunk
    if kind == "none and total":
        return (u > 0.1).double()
    return torch.where(u > 0.5, 1 - 1e-3 * u, u * 0.3)


def inputs(rule, T, heads, x_heads, dv, kind, gen):
    normal = lambda *s: torch.randn(*s, generator=gen, dtype=torch.float64)
    unit = lambda t: t / t.norm(dim=-1, keepdim=True)
    g, v = decays(kind, T, heads, gen), normal(T, heads, dv)
    if rule == "gated":
        k = unit(normal(T, x_heads, DK))
        k[1::3] = unit(k[1::3] + 4 * k[0:1])           # keys that look alike: the triangular solve matters
        return dict(q=unit(normal(T, x_heads, DK)), k=k, v=v, beta=torch.rand(T, heads, generator=gen, dtype=torch.float64), g=g)
    k = normal(T, heads, DK)
    k[1::3] = k[1::3] + 4 * k[0:1]
    b = unit(k)
    rate = torch.rand(T, heads, DK, generator=gen, dtype=torch.float64)
    return dict(q=normal(T, heads, DK), k=k, v=v, b=b, a=rate * b, g=g)


def recurrence(rule, ins, S, heads):
    """Token by token in float64; S [heads, key, value]."""
    ins = {n: (t.float().double() if t is not None else None) for n, t in ins.items()}
    out = []
    wide = lambda t: t.repeat_interleave(heads // t.shape[0], 0)
    for t in range(ins["v"].shape[0]):
        k, q, v, g = wide(ins["k"][t]), wide(ins["q"][t]), ins["v"][t], ins["g"][t]
        if rule == "gated":
            S = S * g[:, :, None]
            u = ins["beta"][t][:, None] * (v - torch.einsum("hkv,hk->hv", S, k))
            S = S + k[:, :, None] * u[:, None, :]
        else:
            d = torch.einsum("hkv,hk->hv", S, ins["b"][t])
            S = S * g[:, :, None] - ins["a"][t][:, :, None] * d[:, None, :] + k[:, :, None] * v[:, None, :]
        out.append(torch.einsum("hkv,hk->hv", S, q))
    return torch.stack(out), S


def scan(rule, ins, harness, ctx, heads, x_heads, dv):
    flat = {n: t.reshape(t.shape[0], -1).float().contiguous().to(DEV) for n, t in ins.items()}
    state = harness.cache.layer_caches[0].state
    if rule == "gated":
        return ops.delta_scan(flat["q"], flat["k"], flat["v"], flat["beta"], flat["g"], state, ctx, kv_heads=x_heads, heads=heads,
                              dk=DK, dv=dv)
    return ops.general_delta_scan(flat["q"], flat["k"], flat["v"], flat["g"], flat["b"], flat["a"], state, ctx, heads=heads, d=DK)


@pytest.mark.parametrize("kind", ["near one", "strong", "none and total", "mixed"])
@pytest.mark.parametrize("rule,heads,x_heads,dv,lengths", [
    ("gated", 2, 1, 128, (49,)), ("gated", 4, 2, 48, (64, 1, 65)), ("gated", 1, 1, 160, (48, 130, 7)), ("gated", 6, 2, 16, (300, 95)),
    ("general", 2, 2, 128, (49,)), ("general", 1, 1, 128, (96, 48, 1, 97)), ("general", 3, 3, 128, (257, 63))])
def test_chunks(monkeypatch, rule, heads, x_heads, dv, lengths, kind):
    monkeypatch.setattr(ops, "delta_takes_chunks", lambda *a: True)         # also where token by token is faster
    gen = torch.Generator().manual_seed(sum(lengths) + heads)
    T = sum(lengths)
    ins = inputs(rule, T, heads, x_heads, dv, kind, gen)
    starts = torch.randn(len(lengths), heads, dv, DK, generator=gen)
    got = {}
    for way in ("chunks", "tokens"):
        harness = Harness([None], [StateSpec((heads * DK * dv,), torch.float32)], torch.float32, max_requests=len(lengths))
        ctx = harness.context([StepEntry(i, [0] * n) for i, n in enumerate(lengths)])
        assert ctx.layout["delta"]["longs"] == sum(n > ops.DELTA_SHORT for n in lengths)
        if way == "tokens":
            ctx.layout = {k: v for k, v in ctx.layout.items() if k != "delta"}
        state = harness.cache.layer_caches[0].state
        for i, slot in enumerate(ctx.host_state_slots):
            state[slot] = starts[i].reshape(-1).to(DEV)
        out = scan(rule, ins, harness, ctx, heads, x_heads, dv)
        got[way] = out.cpu().double(), state[ctx.host_state_slots].cpu().double()
    at = 0
    for i, n in enumerate(lengths):
        part = {name: t[at:at + n] for name, t in ins.items()}
        want, end = recurrence(rule, part, starts[i].double().transpose(1, 2), heads)
        rel = lambda a, b: float((a - b).norm() / b.norm())
        for which, exact in ((0, want.reshape(n, -1)), (1, end.transpose(1, 2).reshape(-1))):
            error = {way: rel(got[way][which][at:at + n] if which == 0 else got[way][which][i], exact) for way in got}
            # both ways are float32 evaluations of the same sums: of the same order of rounding
            assert error["chunks"] <= 2 * error["tokens"] + 2.0 ** -22, (i, n, which, error)
        at += n


@pytest.mark.parametrize("rule", ["gated", "general"])
def test_a_token_that_is_not_finite_reaches_no_earlier_one(monkeypatch, rule):
    monkeypatch.setattr(ops, "delta_takes_chunks", lambda *a: True)
    gen = torch.Generator().manual_seed(3)
    ins = inputs(rule, 80, 1, 1, 128, "mixed", gen)
    outs = []
    for value in (None, float("inf"), float("nan")):
        case = {n: t.clone() for n, t in ins.items()}
        if value is not None:
            for name in case:
                case[name][45] = value
        harness = Harness([None], [StateSpec((DK * 128,), torch.float32)], torch.float32)
        ctx = harness.context([StepEntry("r", [0] * 80)])
        outs.append(scan(rule, case, harness, ctx, 1, 1, 128).cpu())
    for out in outs[1:]:
        assert torch.equal(out[:45], outs[0][:45]) and not torch.isfinite(out[45:]).any()


@pytest.mark.parametrize("rule", ["gated", "general"])
def test_a_start_state_that_is_not_finite_stays_in_its_value_column(monkeypatch, rule):
    """An infinite entry of a start state (NaN from the first chunk on: its lower terms are inf - inf) spoils that value column's read-outs and
    state, and not a bit of another's."""
    monkeypatch.setattr(ops, "delta_takes_chunks", lambda *a: True)
    gen = torch.Generator().manual_seed(4)
    ins = inputs(rule, 80, 2, 2, 128, "mixed", gen)
    start = torch.randn(2, 128, DK, generator=gen)           # [head, value, key]
    got = []
    for value in (None, float("inf"), float("-inf"), float("nan")):
        case = start.clone()
        if value is not None:
            case[1, 5, 3] = value
        harness = Harness([None], [StateSpec((2 * DK * 128,), torch.float32)], torch.float32)
        ctx = harness.context([StepEntry("r", [0] * 80)])
        state = harness.cache.layer_caches[0].state
        state[ctx.host_state_slots[0]] = case.reshape(-1).to(DEV)
        out = scan(rule, ins, harness, ctx, 2, 2, 128).view(80, 2, 128)
        got.append((out.cpu(), state[ctx.host_state_slots[0]].view(2, 128, DK).cpu()))
    others = torch.ones(2, 128, dtype=torch.bool)
    others[1, 5] = False
    for out, state in got[1:]:
        assert torch.equal(out[:, others], got[0][0][:, others]) and torch.equal(state[others], got[0][1][others])
        assert not torch.isfinite(out[:, 1, 5]).any() and not torch.isfinite(state[1, 5]).any()


@pytest.mark.parametrize("rule,lengths,chunks", [("gated", (49, 3), False), ("gated", (300, 1), True), ("general", (64,), False),
                                                 ("general", (700, 20), True), ("gated", (1000,), True)])
def test_the_rule_itself_chooses(monkeypatch, rule, lengths, chunks):
    """Steps with long portions that the rule leaves token by token, and others: which kernels run, and what comes out."""
    gen = torch.Generator().manual_seed(len(lengths))
    heads, dv = 2, 128
    ins = inputs(rule, sum(lengths), heads, heads, dv, "mixed", gen)
    calls = []
    monkeypatch.setattr(ops, "_check", lambda code, what, kernels=1, check=ops._check: (calls.append(what), check(code, what, kernels))[1])
    got = []
    for laid_out in (True, False):
        harness = Harness([None], [StateSpec((heads * DK * dv,), torch.float32)], torch.float32, max_requests=len(lengths))
        ctx = harness.context([StepEntry(i, [0] * n) for i, n in enumerate(lengths)])
        assert ctx.layout["delta"]["longs"] > 0
        if not laid_out:
            ctx.layout = {}
        del calls[:]
        out = scan(rule, ins, harness, ctx, heads, heads, dv)
        got.append((out, harness.cache.layer_caches[0].state[ctx.host_state_slots].clone()))
        assert ("delta_chunks" in calls) == (chunks and laid_out), calls
        assert len(calls) == (2 if chunks and laid_out and min(lengths) <= ops.DELTA_SHORT else 1)
    for a, b in zip(*got):           # (two float32 evaluations of sums whose terms cancel by a few hundred times at most)
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-4) if chunks else torch.equal(a, b)


@pytest.mark.parametrize("rule", ["gated", "general"])
def test_rounds_of_chunks_give_the_same_bits(monkeypatch, rule):
    """Chunks that don't fit the scratch together run in rounds that may end anywhere in a request."""
    monkeypatch.setattr(ops, "delta_takes_chunks", lambda *a: True)
    gen = torch.Generator().manual_seed(4)
    lengths, heads, dv = (150, 7, 64, 49, 260), 2, 128
    ins = inputs(rule, sum(lengths), heads, heads, dv, "mixed", gen)
    starts = torch.randn(len(lengths), heads * dv * DK, generator=gen)
    got = []
    for chunks in (100, 1, 4, 7):
        monkeypatch.setattr(ops, "DELTA_SCRATCH", chunks * ops.library().vosti_delta_chunk_floats(heads, dv, int(rule == "general")))
        harness = Harness([None], [StateSpec((heads * DK * dv,), torch.float32)], torch.float32, max_requests=len(lengths))
        ctx = harness.context([StepEntry(i, [0] * n) for i, n in enumerate(lengths)])
        state = harness.cache.layer_caches[0].state
        for i, slot in enumerate(ctx.host_state_slots):
            state[slot] = starts[i].to(DEV)
        out = scan(rule, ins, harness, ctx, heads, heads, dv)
        got.append((out, state[ctx.host_state_slots].clone()))
    assert all(torch.equal(a, b) for other in got[1:] for a, b in zip(got[0], other))


def test_scratch_is_bounded(monkeypatch):
    """12,000 tokens of 16 heads would take 396 MB of chunks at once; a layer never takes more than 256."""
    monkeypatch.setattr(ops, "delta_takes_chunks", lambda *a: True)
    T, heads, kv = 12000, 16, 4
    harness = Harness([None], [StateSpec((heads * DK * 128,), torch.float32)], torch.float32)
    ctx = harness.context([StepEntry("r", [0] * T)])
    r = lambda *s: torch.rand(*s, device=DEV)
    q, k, v, beta, g = r(T, kv * DK) / 20, r(T, kv * DK) / 20, r(T, heads * 128), r(T, heads), r(T, heads * DK)
    torch.cuda.synchronize()
    held = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    out = ops.delta_scan(q, k, v, beta, g, harness.cache.layer_caches[0].state, ctx, kv_heads=kv, heads=heads, dk=DK, dv=128)
    peak = torch.cuda.max_memory_allocated() - held
    # (the allocator hands out large blocks in whole 2 MB: up to that much more for each of the two)
    assert peak <= out.numel() * 4 + (256 << 20) + (4 << 20) and torch.isfinite(out).all()


def near(got, want):
    """float32 sums of at most 128 terms and elementary functions against float64: some tens of roundings."""
    return torch.allclose(got.double().cpu(), want, rtol=64 * 2.0 ** -24, atol=64 * 2.0 ** -24)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("taps,per_head,silu", [(1, False, False), (2, True, True), (4, False, True), (4, True, False)])
@pytest.mark.parametrize("kv,heads,lengths", [(1, 2, (1, 2, 3)), (2, 4, (5, 1, 7, 1200)), (2, 4, (5, 1, 7, 5100))])
def test_preparation_of_wide_heads(dtype, taps, per_head, silu, kv, heads, lengths):
    """Heads of 128 (whole words, one or four tokens a warp), portions shorter than the taps and starts from a tail."""
    gen = torch.Generator().manual_seed(taps + heads)
    T, D = sum(lengths), DK
    cq, cv = kv * D, heads * D
    cc, cd = 2 * cq + cv, heads if per_head else heads * D
    normal = lambda *s, std=1.0: (torch.randn(*s, generator=gen) * std).to(dtype)
    proj, rates = normal(T, cc + heads), torch.randn(T, cd + cv, generator=gen)
    conv_w, a_log, dt_bias = normal(cc, taps, std=0.5), normal(heads, std=0.5), normal(cd)
    size = heads * D * D + (taps - 1) * cc
    harness = Harness([None], [StateSpec((size,), torch.float32)], torch.float32, max_requests=len(lengths))
    ctx = harness.context([StepEntry(i, [0] * n) for i, n in enumerate(lengths)])
    state = harness.cache.layer_caches[0].state
    tails = torch.randn(len(lengths), taps - 1, cc, generator=gen)
    for i, slot in enumerate(ctx.host_state_slots):
        state[slot, heads * D * D:] = tails[i].reshape(-1).to(DEV)
    offsets = {"q": 0, "k": cq, "v": 2 * cq, "b": cc}
    got = ops.delta_prep(proj.to(DEV), rates.to(DEV), offsets, kv_heads=kv, heads=heads, dk=D, dv=D, taps=taps, conv_w=conv_w.to(DEV),
                         a_log=a_log.to(DEV), dt_bias=dt_bias.to(DEV), state=state, conv_offset=heads * D * D, ctx=ctx,
                         decay_per_head=per_head, gate_silu=silu)
    x, r = proj.double(), rates.double()
    rows, at = [], 0
    for i, n in enumerate(lengths):
        full = torch.cat([tails[i].double(), x[at:at + n, :cc]])
        y = sum(full[j:j + n] * conv_w.double()[:, j] for j in range(taps))
        rows.append(y * torch.sigmoid(y))
        assert torch.equal(state[ctx.host_state_slots[i], heads * D * D:].cpu().view(taps - 1, cc).double(), full[n:])
        at += n
    y = torch.cat(rows)
    unit = lambda t: (t.view(T, kv, D) / torch.sqrt((t.view(T, kv, D) ** 2).sum(-1, keepdim=True) + 1e-6)).reshape(T, cq)
    decay = torch.exp(-torch.exp(a_log.double())[:, None] * torch.nn.functional.softplus((r[:, :cd] + dt_bias.double()).view(T, heads, -1)))
    z = r[:, cd:]
    want = (unit(y[:, :cq]) * D ** -0.5, unit(y[:, cq:2 * cq]), y[:, 2 * cq:], torch.sigmoid(x[:, cc:]),
            decay.expand(T, heads, D).reshape(T, cv), z * torch.sigmoid(z) if silu else torch.sigmoid(z))
    for name, a, b in zip("q k v beta decay gate".split(), got, want):
        assert near(a, b), (name, float((a.double().cpu() - b).abs().max()))
    assert harness.status.item() == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_general_preparation_of_wide_heads(dtype):
    gen = torch.Generator().manual_seed(8)
    T, heads, D = 37, 5, DK
    W = heads * D
    proj, inner = torch.randn(T, 5 * W + 12, generator=gen).to(dtype), torch.randn(T, W, generator=gen)
    w0, bias = torch.randn(W, generator=gen).to(dtype), torch.randn(W, generator=gen).to(dtype)
    offsets = {name: i * W for i, name in enumerate(("r", "k", "v", "g", "a"))}
    got = ops.general_delta_prep(proj.to(DEV), inner.to(DEV), offsets, heads=heads, d=D, w0=w0.to(DEV), a_bias=bias.to(DEV))
    r, k, v, g, a = (proj.double()[:, i * W:(i + 1) * W] for i in range(5))
    unit = (k.view(T, heads, D) / torch.sqrt((k.view(T, heads, D) ** 2).sum(-1, keepdim=True) + 1e-6)).reshape(T, W)
    decay = torch.exp(-torch.exp(torch.tensor(-0.5, dtype=torch.float64)) * torch.sigmoid(inner.double() + w0.double()))
    for one, want in zip(got, (r, k, v, decay, unit, torch.sigmoid(a + bias.double()) * unit, torch.sigmoid(g))):
        assert near(one, want)
