"""The work that is measured: decoder layers, recurrent and latent mixers and a small whole model, through
the package's public entry points, at the sizes of `bench.py`.

Qwen3 layers have the 8B sizes (width 4,096, 32 heads of 128 over 8, feed-forward 12,288, pages of 16);
mixers and the small model have the "s" sizes of the other designs (width 2,048, 16 heads of 128). A step of
one token per request is recorded as a CUDA graph while it is prepared and replayed, as the engine
does with decode steps; every other step is launched call by call, as the engine does with portions.

A case: `kind`, `dtype` ("bfloat16", "float32"), `new` (tokens each request brings, "2048" or "1,1,1") and
`past` (tokens of each request whose keys, or whose traces in the state, are there already).
"""
import math

import torch

PAGE = 16
QWEN_LAYER = dict(width=4096, heads=32, kv=8, ff=12288, layers=1, vocab=8192)
QWEN_SMALL = dict(width=2048, heads=16, kv=4, ff=8192, layers=4, vocab=32768)
LIMIT = 4096                     # positions of the rotation tables
DIM = 128                        # head size everywhere
THETA, EPS = 1000000.0, 1e-6
WIDTH, HEADS, KV = 2048, 16, 4   # the mixers
TAPS, RANK = 4, 64               # convolution taps, ranks of the low-rank pairs
LATENT, ROT, LATENT_THETA = 512, 64, 10000.0
INNER, STATES, DT_RANK = 4096, 16, 128


def _case(kind, dtype, new, past):
    return dict(kind=kind, dtype=dtype, new=",".join(map(str, new)), past=",".join(map(str, past)))


def _ragged(count, low, high):
    """`count` lengths spread over low .. high in a mixed order."""
    return [low + (high - low) * ((i * 37 + 11) % 64) // 63 for i in range(count)]


def listed():
    named = [
        # the smallest call: one user, a short context, the whole of a small model with its logits
        ("model_decode_1", _case("model", "bfloat16", [1], [300])),
        # a layer of the 8B sizes while it generates for one user, for eight (the benchmark's batch), and for a
        # full server whose requests have different lengths
        ("layer_decode_1", _case("layer", "bfloat16", [1], [2047])),
        ("layer_decode_8", _case("layer", "bfloat16", [1] * 8, [2047] * 8)),
        ("layer_decode_64", _case("layer", "bfloat16", [1] * 64, _ragged(64, 600, 3500))),
        # a prompt of the benchmark's length in one step
        ("layer_prefill_2048", _case("layer", "bfloat16", [2048], [0])),
        # a continuous batch: two portions of prompts of odd lengths beside requests that generate
        ("layer_mixed", _case("layer", "bfloat16", [509, 131] + [1] * 13, [1024, 0] + _ragged(13, 70, 2900))),
        # the float32 path of the same layer
        ("layer_prefill_float32", _case("layer", "float32", [384], [0])),
        # recurrent mixers: the gated delta rule over a prompt and while it generates for sixteen, the generalized
        # rule over three prompts of odd lengths, the selective scan over two
        ("delta_prefill_2048", _case("delta", "bfloat16", [2048], [0])),
        ("delta_decode_16", _case("delta", "bfloat16", [1] * 16, [700] * 16)),
        ("general_prefill_ragged", _case("general", "bfloat16", [1031, 700, 317], [0, 512, 0])),
        ("scan_prefill_ragged", _case("scan", "bfloat16", [1499, 549], [0, 600])),
        # latent attention over a prompt
        ("latent_prefill_2048", _case("latent", "bfloat16", [2048], [0])),
    ]
    return [dict(case, name=name) for name, case in named]


def draw(rng):
    spread = lambda low, high: int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    kind = rng.choice(["layer", "layer", "layer", "delta", "general", "scan", "latent"])
    dtype = "float32" if rng.random() < 0.15 else "bfloat16"
    if dtype == "float32":
        # the float32 path is for checking answers: few tokens
        new = [spread(1, 300 if kind == "layer" else 500)]
        return _case(kind, dtype, new, [rng.choice([0, rng.randint(1, 1000)])])
    if rng.random() < 0.45:          # generating
        count = spread(1, 64)
        most = 3500 if kind == "layer" else 2000
        return _case(kind, dtype, [1] * count, [rng.randint(16, most) for _ in range(count)])
    portions = rng.randint(1, 3)     # portions of prompts, perhaps beside requests that generate
    new = [spread(5, 2048 // portions) for _ in range(portions)]
    past = [rng.choice([0, rng.randint(1, 1500)]) if kind != "latent" else rng.choice([0, rng.randint(1, 64)]) for _ in new]
    if rng.random() < 0.4:
        count = rng.randint(1, 12)
        new, past = new + [1] * count, past + [rng.randint(16, 2000) for _ in range(count)]
    return _case(kind, dtype, new, past)


# ---------------------------------------------------------------- inputs, from the seed alone
def _lengths(case):
    return [int(v) for v in case["new"].split(",")], [int(v) for v in case["past"].split(",")]


def _sizes(case):
    return QWEN_LAYER if case["kind"] == "layer" else QWEN_SMALL


def _dtype(case):
    return torch.float32 if case["dtype"] == "float32" else torch.bfloat16


class _Draws:
    def __init__(self, seed, dtype):
        self.gen, self.dtype = torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + 17), dtype

    def normal(self, *shape, std=0.02, mean=0.0, dtype=None):
        out = torch.empty(shape, dtype=dtype or self.dtype, device="cuda")
        return out.normal_(mean, std, generator=self.gen)

    def uniform(self, *shape, low, high):
        out = torch.empty(shape, dtype=self.dtype, device="cuda")
        return out.uniform_(low, high, generator=self.gen)

    def tokens(self, count, vocab):
        return torch.randint(0, vocab, (count,), generator=self.gen, device="cuda")


def _weights(case, d):
    """The tensors of a case by their checkpoint names (a mixer's by its own names)."""
    kind = case["kind"]
    if kind in ("layer", "model"):
        s = _sizes(case)
        W, q, kv, F = s["width"], s["heads"] * DIM, s["kv"] * DIM, s["ff"]
        # rows of the stream have entries of about 1
        out = {"model.embed_tokens.weight": d.normal(s["vocab"], W, std=1.0), "model.norm.weight": d.normal(W, std=0.1, mean=1.0)}
        for i in range(s["layers"]):
            p = f"model.layers.{i}."
            for name in ("input_layernorm", "post_attention_layernorm"):
                out[p + name + ".weight"] = d.normal(W, std=0.1, mean=1.0)
            for name, shape in (("q", (q, W)), ("k", (kv, W)), ("v", (kv, W)), ("o", (W, q))):
                out[p + f"self_attn.{name}_proj.weight"] = d.normal(*shape)
            for name in "qk":
                out[p + f"self_attn.{name}_norm.weight"] = d.normal(DIM, std=0.1, mean=1.0)
            for name, shape in (("gate", (F, W)), ("up", (F, W)), ("down", (W, F))):
                out[p + f"mlp.{name}_proj.weight"] = d.normal(*shape)
        if kind == "model":
            out["lm_head.weight"] = d.normal(s["vocab"], W)
        return out
    q, kv = HEADS * DIM, KV * DIM
    if kind == "delta":
        return {"q": d.normal(kv, WIDTH), "k": d.normal(kv, WIDTH), "v": d.normal(q, WIDTH),
                "q.conv": d.normal(kv, TAPS, std=0.5), "k.conv": d.normal(kv, TAPS, std=0.5), "v.conv": d.normal(q, TAPS, std=0.5),
                "b": d.normal(HEADS, WIDTH), "A_log": d.normal(HEADS, std=0.5), "norm": d.normal(DIM, std=0.1, mean=1.0),
                # step sizes from a few thousandths to about one, so that some channels forget and some keep
                "dt_bias": d.uniform(q, low=-6.0, high=1.0), "o": d.normal(WIDTH, q),
                "a1": d.normal(RANK, WIDTH), "a2": d.normal(q, RANK, std=0.1), "g1": d.normal(RANK, WIDTH), "g2": d.normal(q, RANK, std=0.2)}
    if kind == "general":
        out = {name: d.normal(q, WIDTH) for name in ("r", "k", "v", "g", "a")}
        out.update({"a.b": d.normal(q, std=0.5), "w1": d.normal(RANK, WIDTH), "w2": d.normal(q, RANK, std=0.2),
                    "w0": d.uniform(q, low=-6.0, high=1.0), "norm": d.normal(q, std=0.1, mean=1.0), "o": d.normal(WIDTH, q)})
        return out
    if kind == "scan":
        return {"in": d.normal(2 * INNER, WIDTH), "conv": d.normal(INNER, TAPS, std=0.5), "conv.b": d.normal(INNER, std=0.1),
                "x": d.normal(DT_RANK + 2 * STATES, INNER, std=0.05), "dt": d.normal(INNER, DT_RANK, std=0.2),
                "dt.b": d.uniform(INNER, low=-6.0, high=1.0), "A_log": d.normal(INNER, STATES, std=0.5),
                "D": d.normal(INNER, std=0.1, mean=1.0), "o": d.normal(WIDTH, INNER)}
    return {"q": d.normal(HEADS * (DIM + ROT), WIDTH), "uk": d.normal(q, LATENT, std=0.05), "uv": d.normal(q, LATENT, std=0.05),
            "o": d.normal(WIDTH, q), "dkv": d.normal(LATENT + ROT, WIDTH), "dkv.norm": d.normal(LATENT, std=0.1, mean=1.0),
            "g": d.normal(HEADS, WIDTH)}


def _draw_case(case, seed):
    """(weights, tokens or rows of the step, per layer what every request has cached or its state)."""
    d = _Draws(seed, _dtype(case))
    weights = _weights(case, d)
    new, past = _lengths(case)
    kind = case["kind"]
    if kind in ("layer", "model"):
        s = _sizes(case)
        rows = d.tokens(sum(new), s["vocab"])
        kept = [[(d.normal(p, s["kv"], DIM, std=1.0), d.normal(p, s["kv"], DIM, std=1.0)) for p in past] for _ in range(s["layers"])]
        return weights, rows, kept
    rows = d.normal(sum(new), WIDTH, std=1.0)
    if kind == "latent":
        return weights, rows, [[(d.normal(p, 1, LATENT, std=1.0), d.normal(p, 1, ROT, std=1.0)) for p in past]]
    size = {"delta": HEADS * DIM * DIM + (TAPS - 1) * (2 * KV + HEADS) * DIM, "general": HEADS * DIM * DIM,
            "scan": INNER * STATES + (TAPS - 1) * INNER}[kind]
    return weights, rows, [[d.normal(size, std=0.5, dtype=torch.float32) * (1.0 if p else 0.0) for p in past]]


# ---------------------------------------------------------------- the package's parts
def _qwen_config(s):
    return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", num_hidden_layers=s["layers"], hidden_size=s["width"],
                num_attention_heads=s["heads"], num_key_value_heads=s["kv"], head_dim=DIM, intermediate_size=s["ff"],
                vocab_size=s["vocab"], rope_theta=THETA, rms_norm_eps=EPS, tie_word_embeddings=s["layers"] == 1,
                max_position_embeddings=LIMIT, hidden_act="silu", attention_bias=False, attention_dropout=0.0,
                use_sliding_window=False, sliding_window=None, rope_scaling=None)


def _mixer_spec(kind):
    from vosti_b200.config import PartSpec
    if kind == "delta":
        return PartSpec.make("gated_delta", num_heads=HEADS, num_kv_heads=KV, head_dim=DIM, v_head_dim=DIM, conv_taps=TAPS,
                             eps=EPS, decay_rank=RANK, gate_rank=RANK)
    if kind == "general":
        return PartSpec.make("general_delta", num_heads=HEADS, head_dim=DIM, decay_rank=RANK, eps=EPS)
    if kind == "scan":
        return PartSpec.make("selective_scan", inner=INNER, state=STATES, conv_taps=TAPS, dt_rank=DT_RANK)
    rotation = PartSpec.make("rope", theta=LATENT_THETA, rotary_dim=ROT, scaling=None, max_positions=0)
    return PartSpec.make("latent_attention", num_heads=HEADS, head_dim=DIM, rot_dim=ROT, v_head_dim=DIM, kv_rank=LATENT,
                         scale=(DIM + ROT) ** -0.5, eps=EPS, gate=True, position=rotation)


def _fill_pages(pages, block_table, kept):
    """Put every request's cached rows [past, heads, width] where its block table says."""
    for request, rows in enumerate(kept):
        n = rows.shape[0]
        if n:
            at = torch.arange(n, device=rows.device)
            pages[block_table[request, at // PAGE].long(), :, at % PAGE] = rows


def prepare(case, seed):
    from vosti_b200 import ops
    from vosti_b200.cache import CacheManager
    from vosti_b200.config import model_spec_from_config
    from vosti_b200.engine.batch import StagingBuffer, StepEntry, build_context
    from vosti_b200.engine.graphs import KV_BUCKET, PAGES_BUCKET
    from vosti_b200.engine.runner import ModelRunner
    from vosti_b200.parts import build_mixer

    kind, dtype = case["kind"], _dtype(case)
    new, past = _lengths(case)
    weights, rows, kept = _draw_case(case, seed)
    pages = sum((n + p + PAGE - 1) // PAGE for n, p in zip(new, past)) + 4
    decoding = max(new) == 1
    longest = max(n + p for n, p in zip(new, past))
    bucket = dict(min_pages=-(-longest // PAGE // PAGES_BUCKET) * PAGES_BUCKET + PAGES_BUCKET,
                  kv_bucket=-(-longest // KV_BUCKET) * KV_BUCKET) if decoding else {}
    if kind in ("layer", "model"):
        runner = ModelRunner(spec=model_spec_from_config(_qwen_config(_sizes(case))), tensors=weights, dtype=dtype, device="cuda:0",
                             num_pages=pages, page_size=PAGE, max_requests=len(new), consume_tensors=True)
        cache, step = runner.cache, runner.prepare
        ids = rows.tolist()
    else:
        device = torch.device("cuda:0")
        ops.require_device(device)
        mixer = build_mixer(_mixer_spec(kind), WIDTH, None)
        mixer.load(weights, dtype)
        mixer.setup(device, dtype)
        cache = CacheManager([mixer.cache_spec()], [mixer.state_spec()], num_pages=pages, page_size=PAGE, max_requests=len(new),
                             device=device, dtype=dtype, prefix_reuse=False)
        staging, status = StagingBuffer(device), torch.zeros(1, dtype=torch.int32, device=device)
        step = lambda entries, **more: build_context(staging, cache, entries, status, dtype, **more)
        ids = [0] * sum(new)
    del weights
    for request in range(len(new)):
        cache.begin(request)
    # the past of all requests came in turns of 256 tokens, so their pages lie between one another's
    for start in range(0, max(past), 256):
        turn = [StepEntry(r, [0] * min(256, p - start)) for r, p in enumerate(past) if p > start]
        step(turn)
    entries, at = [], 0
    for request, n in enumerate(new):
        entries.append(StepEntry(request, ids[at:at + n], [n - 1] if kind == "model" else []))
        at += n
    ctx = step(entries, **bucket)
    for layer, layer_kept in zip(cache.layer_caches, kept):
        if layer.state is not None:
            for slot, state in zip(ctx.host_state_slots, layer_kept):
                layer.state[slot, :state.shape[0]] = state
        else:
            for i in range(2):
                _fill_pages(layer.tensors[i], ctx.groups[0].block_table, [k[i] for k in layer_kept])
    del kept
    first = cache.layer_caches[0]

    def forward():
        if kind == "model":
            return (runner.run(ctx),) + first.tensors
        if kind == "layer":
            # the layer, and the norm that adds its last sublayer's output to the stream
            hidden, residual = runner.model.forward(ctx, cache.layer_caches)
            return tuple(runner.model.final_norm.forward_add(ctx, hidden, residual)) + first.tensors
        out = mixer.forward(ctx, rows, first)
        return (out, first.state) if first.state is not None else (out,) + first.tensors

    state = dict(forward=forward, graph=None, keep=(rows, cache, ctx))
    if decoding:
        # recorded once, like the engine's decode steps; what the warm-up changed is put back
        before = None if first.state is None else first.state.clone()

        def record():
            for _ in range(2):
                forward()
            torch.cuda.current_stream().synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                outputs = forward()
            state.update(graph=graph, outputs=outputs, stamp=ops.WORKSPACE_GENERATION)

        record()
        if before is not None:
            first.state.copy_(before)
        state.update(record=record, moved=lambda: state["stamp"] != ops.WORKSPACE_GENERATION)
    return state


def run(state):
    if state["graph"] is None:
        return state["forward"]()
    if state["moved"]():             # a scratch buffer that the recording points to has moved: record again
        state["record"]()
    state["graph"].replay()
    return state["outputs"]


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    new, past = _lengths(case)
    T, kind = sum(new), case["kind"]
    e = 4 if case["dtype"] == "float32" else 2
    pairs = sum(n * p + n * (n + 1) // 2 for n, p in zip(new, past))
    keys = sum(n + p for n, p in zip(new, past))
    if kind in ("layer", "model"):
        s = _sizes(case)
        W, q, kv, F, L = s["width"], s["heads"] * DIM, s["kv"] * DIM, s["ff"], s["layers"]
        per = W * (2 * q + 2 * kv) + 3 * W * F
        flops = L * (2.0 * T * per + 4.0 * q * pairs)
        data = L * (e * per + 2.0 * e * kv * keys) + 3.0 * e * T * W
        if kind == "model":
            flops += 2.0 * len(new) * W * s["vocab"]
            data += e * W * s["vocab"] + 4.0 * len(new) * s["vocab"]
        return {"bytes": data, "flops": flops}
    q, kv = HEADS * DIM, KV * DIM
    ends = T * WIDTH * (e + 4.0)                     # rows in, float32 rows out
    if kind == "delta":
        per = WIDTH * (2 * kv + q + HEADS + 2 * RANK) + 2 * RANK * q + q * WIDTH
        state = 4.0 * (HEADS * DIM * DIM + (TAPS - 1) * (2 * kv + q))
        return {"bytes": e * per + ends + 2 * len(new) * state, "flops": 2.0 * T * per + 6.0 * T * HEADS * DIM * DIM}
    if kind == "general":
        per = WIDTH * (5 * q + RANK) + RANK * q + q * WIDTH
        return {"bytes": e * per + ends + 8.0 * len(new) * HEADS * DIM * DIM, "flops": 2.0 * T * per + 8.0 * T * HEADS * DIM * DIM}
    if kind == "scan":
        per = WIDTH * 2 * INNER + INNER * (DT_RANK + 2 * STATES) + DT_RANK * INNER + INNER * WIDTH
        return {"bytes": e * per + ends + 8.0 * len(new) * INNER * (STATES + TAPS - 1), "flops": 2.0 * T * per + 6.0 * T * INNER * STATES}
    per = WIDTH * (HEADS * (DIM + ROT) + LATENT + ROT + HEADS) + 2 * q * LATENT + q * WIDTH
    return {"bytes": e * per + ends + e * (LATENT + ROT) * keys, "flops": 2.0 * T * per + 2.0 * HEADS * (2 * LATENT + ROT) * pairs}


def tolerance(case):
    # about four times the distance to 64 bits seen over listed and drawn cases (products of bfloat16 operands with
    # float32 sums; float32 throughout in the float32 path)
    if case["dtype"] == "float32":
        return {"rel": 1.5e-5, "max": 5e-4}
    if case["kind"] in ("model", "scan"):
        return {"rel": 0.025, "max": 0.5}
    return {"rel": 0.015, "max": 0.3}


# ---------------------------------------------------------------- the same in 64 bits
def _rms(x, w):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * w


def _rotate(x, positions, theta, dims):
    """Half-split rotation of x [T, heads, dims]; the angles are float32 by definition."""
    inv = 1.0 / (theta ** (torch.arange(0, dims, 2, dtype=torch.int64).float() / dims)).cuda()
    angle = (positions.float()[:, None] * inv[None, :]).double()
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    a, b = x[..., : dims // 2], x[..., dims // 2:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _softmax_rows(scores, past):
    n, keys = scores.shape[-2:]
    seen = torch.arange(keys, device="cuda")[None, :] <= past + torch.arange(n, device="cuda")[:, None]
    return torch.softmax(scores.masked_fill(~seen, float("-inf")), -1)


def _spans(new, past):
    at = 0
    for request, (n, p) in enumerate(zip(new, past)):
        yield request, slice(at, at + n), n, p
        at += n


def _exact_layer(s, w, prefix, x, kept, new, past):
    W, H, G = s["width"], s["heads"], s["kv"]
    g = lambda name: w[prefix + name + ".weight"].double()
    T = x.shape[0]
    positions = torch.cat([torch.arange(p, p + n) for n, p in zip(new, past)]).cuda()
    h = _rms(x, g("input_layernorm"))
    q = _rotate(_rms((h @ g("self_attn.q_proj").T).view(T, H, DIM), g("self_attn.q_norm")), positions, THETA, DIM)
    k = _rotate(_rms((h @ g("self_attn.k_proj").T).view(T, G, DIM), g("self_attn.k_norm")), positions, THETA, DIM)
    v = (h @ g("self_attn.v_proj").T).view(T, G, DIM)
    y = torch.empty(T, H * DIM, dtype=torch.float64, device="cuda")
    for r, span, n, p in _spans(new, past):
        keys = torch.cat([kept[r][0].double(), k[span]]).repeat_interleave(H // G, 1)
        values = torch.cat([kept[r][1].double(), v[span]]).repeat_interleave(H // G, 1)
        a = _softmax_rows(torch.einsum("nhd,khd->hnk", q[span], keys) * DIM ** -0.5, p)
        y[span] = torch.einsum("hnk,khd->nhd", a, values).reshape(n, H * DIM)
    x = x + y @ g("self_attn.o_proj").T
    h = _rms(x, g("post_attention_layernorm"))
    gate = h @ g("mlp.gate_proj").T
    return x + (gate * torch.sigmoid(gate) * (h @ g("mlp.up_proj").T)) @ g("mlp.down_proj").T


def _silu(x):
    return x * torch.sigmoid(x)


def _convolve(x, tail, weight, bias=None):
    """Causal convolution per channel of x [n, C] after the rows `tail` [TAPS - 1, C], and the tail after it."""
    rows = torch.cat([tail, x])
    y = sum(rows[j:j + x.shape[0]] * weight[:, j] for j in range(TAPS))
    return (y if bias is None else y + bias), rows[-(TAPS - 1):]


def _exact_delta(w, x, kept, new, past):
    q, kv, g = HEADS * DIM, KV * DIM, {n: t.double() for n, t in w.items()}
    proj = torch.cat([x @ g[n].T for n in "qkv"], 1)
    beta = torch.sigmoid(x @ g["b"].T)
    speed = torch.exp(g["A_log"])[:, None]
    decay = torch.exp(-speed * torch.nn.functional.softplus(((x @ g["a1"].T) @ g["a2"].T + g["dt_bias"]).view(-1, HEADS, DIM)))
    gate = torch.sigmoid((x @ g["g1"].T) @ g["g2"].T).view(-1, HEADS, DIM)
    conv = torch.cat([g["q.conv"], g["k.conv"], g["v.conv"]])
    out, states = torch.empty(x.shape[0], HEADS, DIM, dtype=torch.float64, device="cuda"), []
    for r, span, n, p in _spans(new, past):
        start = kept[r].double()
        S = start[: HEADS * DIM * DIM].view(HEADS, DIM, DIM).clone()             # [head, value, key]
        y, tail = _convolve(proj[span], start[HEADS * DIM * DIM:].view(TAPS - 1, -1), conv)
        y = _silu(y)
        unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
        qs = (unit(y[:, :kv].reshape(n, KV, DIM)) * DIM ** -0.5).repeat_interleave(HEADS // KV, 1)
        ks = unit(y[:, kv:2 * kv].reshape(n, KV, DIM)).repeat_interleave(HEADS // KV, 1)
        vs, bs, ds, os = y[:, 2 * kv:].reshape(n, HEADS, DIM), beta[span][..., None], decay[span], out[span]
        for t in range(n):
            S = S * ds[t][:, None, :]
            u = bs[t] * (vs[t] - torch.einsum("hvk,hk->hv", S, ks[t]))
            S = S + u[:, :, None] * ks[t][:, None, :]
            os[t] = torch.einsum("hvk,hk->hv", S, qs[t])
        states.append(torch.cat([S.reshape(-1), tail.reshape(-1)]))
    y = _rms(out, g["norm"]) * gate
    return y.reshape(-1, q) @ g["o"].T, torch.stack(states)


def _exact_general(w, x, kept, new, past):
    g = {n: t.double() for n, t in w.items()}
    heads = lambda t: t.reshape(-1, HEADS, DIM)
    r, k, v, gate, a = (heads(x @ g[n].T) for n in ("r", "k", "v", "g", "a"))
    a = torch.sigmoid(a + heads(g["a.b"]))
    decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(heads(torch.tanh(x @ g["w1"].T) @ g["w2"].T) + heads(g["w0"])))
    unit = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    out, states = torch.empty_like(v), []
    for req, span, n, p in _spans(new, past):
        S = kept[req].double().view(HEADS, DIM, DIM).clone()
        us, rs, ks, vs, ws, removal, os = unit[span], r[span], k[span], v[span], decay[span], (a * unit)[span], out[span]
        for t in range(n):
            d = torch.einsum("hvk,hk->hv", S, us[t])
            S = S * ws[t][:, None, :] - d[:, :, None] * removal[t][:, None, :] + vs[t][:, :, None] * ks[t][:, None, :]
            os[t] = torch.einsum("hvk,hk->hv", S, rs[t])
        states.append(S.reshape(-1))
    y = _rms(out, heads(g["norm"])) * torch.sigmoid(gate)
    return y.reshape(x.shape[0], -1) @ g["o"].T, torch.stack(states)


def _exact_scan(w, x, kept, new, past):
    g = {n: t.double() for n, t in w.items()}
    both = x @ g["in"].T
    u, z = both[:, :INNER], both[:, INNER:]
    out, states, A = torch.empty_like(u), [], -torch.exp(g["A_log"])
    for r, span, n, p in _spans(new, past):
        start = kept[r].double()
        S = start[: INNER * STATES].view(INNER, STATES).clone()
        c, tail = _convolve(u[span], start[INNER * STATES:].view(TAPS - 1, INNER), g["conv"], g["conv.b"])
        c = _silu(c)
        small = c @ g["x"].T
        dt = torch.nn.functional.softplus(small[:, :DT_RANK] @ g["dt"].T + g["dt.b"])
        B, C, os = small[:, DT_RANK:DT_RANK + STATES], small[:, DT_RANK + STATES:], out[span]
        for t in range(n):
            S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * c[t])[:, None] * B[t]
            os[t] = S @ C[t]
        os += g["D"] * c
        states.append(torch.cat([S.reshape(-1), tail.reshape(-1)]))
    return (out * _silu(z)) @ g["o"].T, torch.stack(states)


def _exact_latent(w, x, kept, new, past):
    g = {n: t.double() for n, t in w.items()}
    T = x.shape[0]
    positions = torch.cat([torch.arange(p, p + n) for n, p in zip(new, past)]).cuda()
    q = (x @ g["q"].T).view(T, HEADS, DIM + ROT)
    turned = _rotate(q[..., DIM:], positions, LATENT_THETA, ROT)
    down = x @ g["dkv"].T
    c = _rms(down[:, :LATENT], g["dkv.norm"])
    rot = _rotate(down[:, None, LATENT:], positions, LATENT_THETA, ROT)[:, 0]
    gate = torch.sigmoid(x @ g["g"].T)
    plain = torch.einsum("nhd,hdr->nhr", q[..., :DIM], g["uk"].view(HEADS, DIM, LATENT))
    y = torch.empty(T, HEADS, DIM, dtype=torch.float64, device="cuda")
    for r, span, n, p in _spans(new, past):
        cs, rs = torch.cat([kept[r][0][:, 0].double(), c[span]]), torch.cat([kept[r][1][:, 0].double(), rot[span]])
        scores = (torch.einsum("nhr,kr->hnk", plain[span], cs) + torch.einsum("nhd,kd->hnk", turned[span], rs)) * (DIM + ROT) ** -0.5
        mixed = torch.einsum("hnk,kr->nhr", _softmax_rows(scores, p), cs)
        y[span] = torch.einsum("nhr,hdr->nhd", mixed, g["uv"].view(HEADS, DIM, LATENT))
    return (y * gate[..., None]).reshape(T, -1) @ g["o"].T


def exact(case, seed):
    kind = case["kind"]
    new, past = _lengths(case)
    w, rows, kept = _draw_case(case, seed)
    if kind in ("layer", "model"):
        s = _sizes(case)
        x = w["model.embed_tokens.weight"][rows].double()
        for i in range(s["layers"]):
            x = _exact_layer(s, w, f"model.layers.{i}.", x, kept[i], new, past)
        final = _rms(x, w["model.norm.weight"].double())
        # (where the cache keeps its rows is the cache manager's choice)
        if kind == "layer":
            return final, x, None, None
        last = torch.tensor(new).cumsum(0) - 1
        return final[last.cuda()] @ w["lm_head.weight"].double().T, None, None
    x = rows.double()
    if kind == "latent":
        return _exact_latent(w, x, kept[0], new, past), None, None
    # the slots of the requests, in their order
    return {"delta": _exact_delta, "general": _exact_general, "scan": _exact_scan}[kind](w, x, kept[0], new, past)
