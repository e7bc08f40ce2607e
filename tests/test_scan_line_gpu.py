"""The selective scan's one pass over long portions (csrc/selective_scan.cu) against float64: lengths around the tile,
single tokens beside them, channels that do not fill a block, start states, both serving types."""
from dataclasses import replace

import pytest
import torch

from gpu_util import Harness
from vosti_b200 import ops
from vosti_b200.engine.batch import StepEntry
from vosti_b200.parts import StateSpec

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
N = 16


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("inner,lengths", [(2048, (65,)), (2049, (64, 1, 129)), (2068, (300, 63, 128, 2))])
def test_against_float64(dtype, inner, lengths):
    gen = torch.Generator().manual_seed(inner)
    normal = lambda *s, std=1.0: torch.randn(*s, generator=gen) * std
    T = sum(lengths)
    x, xz = normal(T, inner).to(dtype), normal(T, 2 * inner).to(dtype)
    dtp, bc = normal(T, inner), normal(T, 2 * N)
    bias, a_log, skip = (torch.rand(inner, generator=gen) * 7 - 6).to(dtype), normal(inner, N, std=0.5).to(dtype), normal(inner).to(dtype)
    starts = normal(len(lengths), inner, N)
    harness = Harness([None], [StateSpec((inner * N + 4,), torch.float32)], torch.float32, max_requests=len(lengths))
    ctx = harness.context([StepEntry(i, [0] * n) for i, n in enumerate(lengths)])
    state = harness.cache.layer_caches[0].state
    for i, slot in enumerate(ctx.host_state_slots):
        state[slot, :inner * N] = starts[i].reshape(-1).to(DEV)
    d = lambda t: t.to(DEV)
    assert ops.library().vosti_scan_one_pass(inner, N)
    got = ops.scan_run(d(x), d(dtp), d(bias), d(bc), d(a_log), d(skip), d(xz), state, ctx, inner=inner, states=N)
    at, A = 0, -torch.exp(a_log.double())
    for i, n in enumerate(lengths):
        S, rows = starts[i].double(), []
        for t in range(at, at + n):
            dt = torch.nn.functional.softplus(dtp[t].double() + bias.double())
            S = torch.exp(dt[:, None] * A) * S + (dt * x[t].double())[:, None] * bc[t, :N].double()
            z = xz[t, inner:].double()
            rows.append((S @ bc[t, N:].double() + skip.double() * x[t].double()) * z * torch.sigmoid(z))
        want, end = torch.stack(rows), S
        have, held = got[at:at + n].double().cpu(), state[ctx.host_state_slots[i], :inner * N].double().cpu().view(inner, N)
        # float32 throughout: n roundings of a state at most, few in the mean; the result rounded once to its type
        rel = lambda a, b: float((a - b).norm() / b.norm())
        assert rel(held, end) <= n ** 0.5 * 2.0 ** -22, rel(held, end)
        assert rel(have, want) <= n ** 0.5 * 2.0 ** -22 + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0), rel(have, want)
        at += n
    assert harness.status.item() == 0


def test_channels_that_forget_at_once_keep_finite_states():
    """A rate beyond float32's range (exp of A_log overflows) means that a state holds its last token alone; the
    places of a tile past the portion's last token must not touch it (70 tokens: two whole groups of four are empty)."""
    gen = torch.Generator().manual_seed(5)
    normal = lambda *s: torch.randn(*s, generator=gen)
    T, inner = 70, 2048
    x, xz, dtp, bc, a_log = normal(T, inner), normal(T, 2 * inner), normal(T, inner), normal(T, 2 * N), normal(inner, N)
    a_log[::3, ::2] = 100.0
    harness = Harness([None], [StateSpec((inner * N,), torch.float32)], torch.float32)
    ctx = harness.context([StepEntry("r", [0] * T)])
    state, d = harness.cache.layer_caches[0].state, lambda t: t.to(DEV)
    y = ops.scan_run(d(x), d(dtp), None, d(bc), d(a_log), None, d(xz), state, ctx, inner=inner, states=N)
    end = state[ctx.host_state_slots[0]].view(inner, N).double().cpu()
    last = (torch.nn.functional.softplus(dtp[-1].double()) * x[-1].double())[:, None] * bc[-1, :N].double()
    assert torch.isfinite(y).all() and torch.isfinite(end).all()
    assert torch.allclose(end[::3, ::2], last[::3, ::2], rtol=2.0 ** -20, atol=1e-30)


def test_a_step_without_host_lengths_gives_the_same_bits():
    """A context made by hand may leave out the host's copies of the lengths; the longest portion is all that is needed."""
    gen = torch.Generator().manual_seed(6)
    d = lambda *s: torch.randn(*s, generator=gen).to(DEV)
    lengths, inner = (100, 3, 70), 2048
    T = sum(lengths)
    x, xz, dtp, bc, a_log = d(T, inner), d(T, 2 * inner), d(T, inner), d(T, 2 * N), d(inner, N)
    got = []
    for known in (True, False):
        harness = Harness([None], [StateSpec((inner * N,), torch.float32)], torch.float32, max_requests=len(lengths))
        ctx = harness.context([StepEntry(i, [0] * n) for i, n in enumerate(lengths)])
        state = harness.cache.layer_caches[0].state
        if not known:
            ctx = replace(ctx, host_q_lens=[], host_kv_lens=[])
        got.append((ops.scan_run(x, dtp, None, bc, a_log, None, xz, state, ctx, inner=inner, states=N), state.clone()))
    assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("with_bias,with_skip", [(False, False), (True, False), (False, True)])
def test_without_step_bias_or_skip(with_bias, with_skip):
    """One pass over 130 tokens against float64, the optional vectors left out."""
    gen = torch.Generator().manual_seed(7)
    normal = lambda *s: torch.randn(*s, generator=gen)
    T, inner = 130, 2048
    x, xz, dtp, bc, a_log = normal(T, inner), normal(T, 2 * inner), normal(T, inner) - 2, normal(T, 2 * N), normal(inner, N) * 0.5
    bias, skip = (normal(inner) if with_bias else None), (normal(inner) if with_skip else None)
    harness = Harness([None], [StateSpec((inner * N,), torch.float32)], torch.float32)
    ctx = harness.context([StepEntry("r", [0] * T)])
    state, d = harness.cache.layer_caches[0].state, lambda t: None if t is None else t.to(DEV)
    y = ops.scan_run(d(x), d(dtp), d(bias), d(bc), d(a_log), d(skip), d(xz), state, ctx, inner=inner, states=N).double().cpu()
    S, A, rows = torch.zeros(inner, N, dtype=torch.float64), -torch.exp(a_log.double()), []
    for t in range(T):
        dt = torch.nn.functional.softplus(dtp[t].double() + (bias.double() if with_bias else 0.0))
        S = torch.exp(dt[:, None] * A) * S + (dt * x[t].double())[:, None] * bc[t, :N].double()
        z = xz[t, inner:].double()
        rows.append((S @ bc[t, N:].double() + (skip.double() * x[t].double() if with_skip else 0.0)) * z * torch.sigmoid(z))
    want = torch.stack(rows)
    assert float((y - want).norm() / want.norm()) <= T ** 0.5 * 2.0 ** -22
