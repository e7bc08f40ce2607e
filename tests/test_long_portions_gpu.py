"""Recurrent mixers at sizes that take the kernels for long portions (heads of 128, 2,048 channels): a prompt in one step
against the same prompt in portions short enough to go token by token, state and convolution tail included."""
import pytest
import torch

from gpu_util import Harness
from vosti_b200 import ops
from vosti_b200.config import PartSpec
from vosti_b200.engine.batch import StepEntry
from vosti_b200.parts import build_mixer

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
WIDTH = 256


def mixer_of(kind, gen):
    spec = {
        "gated_delta": dict(num_heads=4, num_kv_heads=2, head_dim=128, v_head_dim=128, conv_taps=4, eps=1e-6, decay_rank=16, gate_rank=16),
        "general_delta": dict(num_heads=4, head_dim=128, decay_rank=16, eps=1e-6),
        "selective_scan": dict(inner=2048, state=16, conv_taps=4, dt_rank=32),
    }[kind]
    mixer = build_mixer(PartSpec.make(kind, **spec), WIDTH, None)
    weights = {}
    for name, w in mixer.weight_specs().items():
        t = torch.randn(*w.shape, generator=gen) * (0.3 if "conv" in name else 0.5 if len(w.shape) == 1 or name == "A_log" else 0.06)
        # gates around 1, step sizes small enough for channels that keep
        weights[name] = (t + 1.0 if name == "norm" else t - 2.0 if name in ("dt_bias", "dt.b", "w0") else t).to(DEV)
    mixer.load(weights, torch.float32)
    mixer.setup(DEV, torch.float32)
    return mixer


@pytest.mark.parametrize("kind,kernel", [("gated_delta", "delta_chunks"), ("general_delta", "delta_chunks"), ("selective_scan", "scan_run")])
def test_one_step_equals_short_portions(monkeypatch, kind, kernel):
    ops.require_device(DEV)
    gen = torch.Generator().manual_seed(11)
    mixer, lengths = mixer_of(kind, gen), (300, 131)
    rows = [torch.randn(n, WIDTH, generator=gen).to(DEV) for n in lengths]
    calls = []
    monkeypatch.setattr(ops, "_check", lambda code, what, kernels=1, check=ops._check: (calls.append(what), check(code, what, kernels))[1])
    got = []
    for portion in (300, 40):
        harness = Harness([mixer.cache_spec()], [mixer.state_spec()], torch.float32, max_requests=2)
        layer, parts = harness.cache.layer_caches[0], [[], []]
        del calls[:]
        for first in range(0, 300, portion):
            part = {i: rows[i][first:first + portion] for i in range(2) if first < lengths[i]}
            ctx = harness.context([StepEntry(i, [0] * x.shape[0]) for i, x in part.items()])
            y, at = mixer.forward(ctx, torch.cat(list(part.values())), layer), 0
            for i, x in part.items():
                parts[i].append(y[at:at + x.shape[0]])
                at += x.shape[0]
            slots = {**(slots if first else {}), **dict(zip(part, ctx.host_state_slots))}
        assert kernel in calls if portion == 300 else kernel == "scan_run" or kernel not in calls
        got.append([torch.cat(p) for p in parts] + [layer.state[slots[i]].clone() for i in range(2)])
        assert harness.status.item() == 0
    # the products are the same bits; the recurrences are two float32 evaluations of the same sums: tens of roundings
    for a, b in zip(*got):
        assert float((a.double() - b.double()).norm() / b.double().norm()) <= 64 * 2.0 ** -24
