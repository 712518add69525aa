"""The serving steps this framework is measured on.

A case is one step of a model runner, the unit of work of everything above it (continuous batching, generation,
replay): ``requests`` decode rows with about ``context`` cached tokens each (ragged), and ``prompts`` prompt chunks of
about ``chunk`` tokens each (ragged) that follow about ``prefix`` cached tokens, in one flat forward.  Decode steps and
steps with few prompt tokens are captured in a CUDA graph and replayed, as a serving loop does; longer prefills run
eagerly.  Designs: Qwen3 with FP8 projections over the bf16 page pool (``qwen3``) or the FP8 one (``qwen3-kv8``),
Tidelorn and Ripesun; widths, head counts and vocabulary are those of ``modelbench.py``.

``run`` returns the step's logits, and what else the step leaves behind: the last cached layer's pages where prompt
tokens were written, the recurrent state where there is one.
"""

from __future__ import annotations

import math
import random

import torch

from mini_inference_engine_b200.engine.model_runner.qwen3_decode import Qwen3DecodeRunner, Qwen3Shape, Qwen3Weights
from mini_inference_engine_b200.engine.model_runner.ripesun import RipesunRunner, RipesunShape, RipesunWeights
from mini_inference_engine_b200.engine.model_runner.tidelorn import TidelornRunner, TidelornShape, TidelornWeights

PAGE, HEAD, VOCAB, WINDOW = 16, 128, 151936, 1024
GRAPH_TOKENS = 1024  # prompt tokens up to which a step is captured
# width: query heads, key/value heads, feed-forward
ATTENTION_SIZES = {2048: (16, 8, 6144), 2560: (32, 8, 9728), 4096: (32, 8, 12288)}
# width: heads, feed-forward, query latent
RIPESUN_SIZES = {2048: (16, 6144, 768), 4096: (32, 12288, 1536)}
ROTATED, KV_RANK, SIDE = 64, 512, 256


def _case(name, design, width, layers, requests=0, context=0, prompts=0, chunk=0, prefix=0):
    case = {"design": design, "width": width, "layers": layers, "requests": requests, "context": context,
            "prompts": prompts, "chunk": chunk, "prefix": prefix}
    return {"name": name, **case} if name else case


def listed():
    return [
        # One user in an interactive session: the whole 36-layer model, bound by latency and the weights.
        _case("qwen3-decode-1", "qwen3", 2560, 36, requests=1, context=611),
        # A small serving batch of the whole model.
        _case("qwen3-decode-24", "qwen3", 2560, 36, requests=24, context=1000),
        # The full batch of the decode benchmark (fewer layers, so that its pages fit more than once).
        _case("qwen3-decode-256", "qwen3", 2560, 8, requests=256, context=2900),
        # A large batch over the FP8 page pool.
        _case("qwen3-kv8-decode-96", "qwen3-kv8", 2560, 12, requests=96, context=1500),
        # Continuous batching: new requests' prompt chunks ride along with running decodes.
        _case("qwen3-mixed-48", "qwen3", 2560, 12, requests=48, context=900, prompts=2, chunk=256, prefix=1024),
        # Requests that arrive together, prefilled whole.
        _case("qwen3-prefill-8", "qwen3", 2560, 4, prompts=8, chunk=1500),
        # One chunk of a long document.
        _case("qwen3-chunk-long", "qwen3", 2560, 4, prompts=1, chunk=4096, prefix=12000),
        # The second design: alternating whole-prefix and windowed layers, bf16 projections.
        _case("tidelorn-decode-40", "tidelorn", 2048, 8, requests=40, context=1800),
        _case("tidelorn-prefill-3", "tidelorn", 4096, 4, prompts=3, chunk=3000),
        # The third design: latent attention and recurrent layers; one user, a batch, and whole prompts.
        _case("ripesun-decode-1", "ripesun", 2048, 8, requests=1, context=777),
        _case("ripesun-decode-64", "ripesun", 4096, 8, requests=64, context=2000),
        _case("ripesun-prefill-5", "ripesun", 2048, 8, prompts=5, chunk=2000),
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    design = rng.choice(["qwen3", "qwen3", "qwen3", "qwen3-kv8", "tidelorn", "tidelorn", "ripesun", "ripesun"])
    width = rng.choice(sorted(RIPESUN_SIZES if design == "ripesun" else ATTENTION_SIZES))
    kind = "decode" if design == "qwen3-kv8" else rng.choice(["decode", "decode", "prefill", "mixed"])
    requests = context = prompts = chunk = prefix = 0
    if kind != "prefill":
        requests = _log_uniform(rng, 1, 256 if kind == "decode" else 64)
        context = _log_uniform(rng, 40, min(6000, 400000 // requests))
    if kind == "prefill":
        prompts = rng.randint(1, 8)
        chunk = _log_uniform(rng, 150, min(4000, 9000 // prompts))
        prefix = 0 if rng.random() < 0.6 else _log_uniform(rng, 100, 8000 // prompts)
    elif kind == "mixed":
        prompts = rng.randint(1, 4)
        chunk = _log_uniform(rng, 16, 512 // prompts)
        prefix = 0 if rng.random() < 0.5 else _log_uniform(rng, 30, 3000)
    return _case(None, design, width, rng.choice([4, 6]), requests, context, prompts, chunk, prefix)


# -- what a case's rows look like (from the case alone) ---------------------------------------------------

def _spread(count, mean, salt, low=1):
    """``count`` ragged sizes around ``mean``."""

    rng = random.Random(f"{salt}/{count}/{mean}")
    sizes = [math.exp(rng.uniform(-1.3, 0.7)) if count > 1 else 1.0 for _ in range(count)]
    total = sum(sizes)
    return [max(low, int(round(s * mean * count / total))) for s in sizes]


def _rows(case):
    """``(first position, tokens)`` of every request: the decode rows, then the prompts."""

    decode = [(n, 1) for n in _spread(case["requests"], case["context"], "context")]
    chunks = _spread(case["prompts"], case["chunk"], "chunk")
    prefixes = _spread(case["prompts"], case["prefix"], "prefix") if case["prefix"] else [0] * case["prompts"]
    return decode, list(zip(prefixes, chunks))


def _outer_decay(heads):
    return [1.0 - 2.0 ** -(5 + i % 8) for i in range(heads)]


def _tidelorn_config(width, layers):
    heads, kv_heads, ff = ATTENTION_SIZES[width]
    entries = []
    for index in range(layers):
        mixer = {"heads": heads, "kv_heads": kv_heads, "dim": HEAD, "vdim": HEAD, "scale": HEAD ** -0.5, "v_mix": True}
        if index % 2 == 0:
            mixer["q_temp"] = {"coef": 0.1, "every": 4096}
        else:
            mixer["mask"] = {"size": WINDOW}
        entries.append({"type": "attention" if index % 2 == 0 else "attention_2", "mixer": mixer,
                        "mlp": {"kind": "dense", "ff": ff, "limit": 7.0}})
    return {"vocab": VOCAB, "width": width, "norm": {"eps": 1e-6}, "postln_alpha": 2.0, "layers": entries,
            "embedding": {"scale": width ** 0.5, "bigram": {"buckets": 65521, "mul_prev": 8191, "mul_cur": 127}}}


def _ripesun_config(width, layers):
    heads, ff, q_rank = RIPESUN_SIZES[width]
    mlp = {"kind": "dense", "ff": ff}
    latent = {"heads": heads, "dim": HEAD, "rot_dim": ROTATED, "vdim": HEAD, "q_rank": q_rank, "kv_rank": KV_RANK,
              "scale": (HEAD + ROTATED) ** -0.5, "mask": {"size": WINDOW}, "rot": {"base": 1e6, "dims": ROTATED}}
    outer = {"heads": heads, "dim": HEAD, "vdim": HEAD, "decay": _outer_decay(heads)}
    entries = []
    for index in range(layers):
        if index % 4 == 0:
            entries.append({"type": "latent_attention", "mixer": {**latent, "kv_from": 0} if index else latent, "mlp": mlp})
        elif index % 4 == 3:
            entries.append({"type": "mingru", "mixer": {"width": width}, "mlp": mlp})
        else:
            entries.append({"type": "lightning", "mixer": outer, "mlp": mlp})
    return {"vocab": VOCAB, "width": width, "norm": {"eps": 1e-6}, "residual_mult": 0.5, "layers": entries,
            "embedding": {"scale": width ** 0.5}, "token_side": {"dim": SIDE}, "logit_softcap": 30.0}


def _qwen3_shape(case):
    heads, kv_heads, ff = ATTENTION_SIZES[case["width"]]
    return Qwen3Shape(layers=case["layers"], hidden=case["width"], q_heads=heads, kv_heads=kv_heads, head_dim=HEAD,
                      intermediate=ff, vocab=VOCAB)


# -- the user's side: runner, inputs, one step ------------------------------------------------------------

class State:
    """A runner and one step's metadata on the device."""


def prepare(case, seed):
    device = torch.device("cuda", torch.cuda.current_device())
    torch.manual_seed(seed)
    decode, chunks = _rows(case)
    spans = decode + chunks
    pages = [-(-(start + count) // PAGE) for start, count in spans]
    live = max(case["requests"], case["prompts"], 1)
    options = dict(num_pages=sum(pages), max_batch=live, max_context=max(start + count for start, count in spans) + 1,
                   decode_buckets=(live,), chunk_buckets=(), kv_init="normal")
    s = State()
    design, width, layers = case["design"], case["width"], case["layers"]
    if design == "tidelorn":
        shape = TidelornShape.from_config(_tidelorn_config(width, layers))
        s.runner = TidelornRunner(TidelornWeights.random(shape, device, seed=seed), **options)
    elif design == "ripesun":
        shape = RipesunShape.from_config(_ripesun_config(width, layers))
        s.runner = RipesunRunner(RipesunWeights.random(shape, device, seed=seed), state_slots=len(spans), **options)
    else:
        weights = Qwen3Weights(_qwen3_shape(case), device, seed=seed)
        # A trained model's residual stream: unit entries, of which every sublayer adds a small part.  (With the
        # layers as drawn the stream is the sum of their outputs, and a rounding difference anywhere grows through
        # the e4m3 activations of the layers after it until it is as large as the quantisation itself.)
        weights.embedding.mul_(50.0)
        for layer in weights.layers:
            layer.o_scale.mul_(0.2 / math.sqrt(2 * layers))
            layer.down_scale.mul_(0.2 / math.sqrt(2 * layers))
        s.runner = Qwen3DecodeRunner(weights, kv_dtype="fp8" if design == "qwen3-kv8" else "bf16", **options)
    # Pages in the order a pool hands them out after a while: any.
    order = torch.randperm(sum(pages), device=device, dtype=torch.int32)
    s.tables = torch.full((len(spans), max(pages)), -1, dtype=torch.int32, device=device)
    cursor = 0
    for row, count in enumerate(pages):
        s.tables[row, :count] = order[cursor:cursor + count]
        cursor += count
    tokens = sum(count for _, count in spans)
    s.ids = torch.randint(0, VOCAB, (tokens,), device=device)
    if design == "tidelorn":  # the cached tokens themselves, which the bigram embedding looks back at
        s.runner.history.random_(0, VOCAB)
    cpu = dict(dtype=torch.int32)
    s.owners = torch.cat([torch.full((n,), r, **cpu) for r, (_, n) in enumerate(spans)]).to(device)
    s.positions = torch.cat([torch.arange(p, p + n, **cpu) for p, n in spans]).to(device)
    s.lengths = torch.tensor([p + 1 for p, _ in decode], **cpu).to(device)
    s.cu = torch.tensor([0, *[n for _, n in chunks]], **cpu).cumsum(0).to(torch.int32).to(device)
    s.kv_lens = torch.tensor([p + n for p, n in chunks], **cpu).to(device)
    s.longest = max([n for _, n in chunks], default=0)
    s.rows = torch.cat([torch.arange(len(decode)), len(decode) + s.cu[1:].cpu().long() - 1]).to(device)
    s.extra, s.starts = {}, {}
    if design == "ripesun":
        s.extra = {"state_slots": torch.randperm(len(spans), dtype=torch.int32, device=device)}
        s.starts = {"chunk_starts": [p for p, _ in chunks]}
    s.decode, s.chunks, s.graph = decode, chunks, None
    if sum(n for _, n in chunks) <= GRAPH_TOKENS:
        s.starts = {}
        side = torch.cuda.Stream(device)
        side.wait_stream(torch.cuda.current_stream(device))
        with torch.cuda.stream(side):
            _step(s)
        torch.cuda.current_stream(device).wait_stream(side)
        torch.cuda.synchronize(device)
        s.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s.graph):
            s.outputs = _step(s)
    if design == "ripesun":  # running requests' states
        s.runner.state.rows.normal_()
    return s


def _step(s):
    runner = s.runner
    if not s.chunks:
        _, logits = runner.decode_forward(s.ids, s.lengths, s.tables, return_logits=True, **s.extra)
        outputs = {"logits": logits}
    else:
        _, logits = runner.mixed_forward(
            s.ids, s.owners, s.positions, s.tables, decode_rows=len(s.decode),
            decode_lengths=s.lengths if s.decode else None, cu_seqlens=s.cu, kv_lens=s.kv_lens,
            max_query_len=s.longest, logit_rows=s.rows, return_logits=True, **s.extra, **s.starts)
        outputs = {"logits": logits, **_pages(runner)}
    if runner.recurrent:
        outputs["state"] = runner.state.rows
    return outputs


def _pages(runner):
    if isinstance(runner, RipesunRunner):
        return {"latents": [pool for pool in runner.latents if pool is not None][-1]}
    return {"keys": runner.key_blocks[-1], "values": runner.value_blocks[-1]}


def run(s):
    if s.graph is None:
        return _step(s)
    s.graph.replay()
    return s.outputs


# -- work and tolerance -----------------------------------------------------------------------------------

def _pairs(start, count, window):
    """Visible (query, key) pairs of tokens [start, start + count)."""

    total = count * start + count * (count + 1) // 2
    if window is None:
        return total
    hidden = [start + i + 1 - window for i in (0, count - 1)]
    if hidden[1] <= 0:
        return total
    first = max(hidden[0], 1)
    return total - (first + hidden[1]) * (hidden[1] - first + 1) // 2


def _seen(start, count, window):
    """Cached or new tokens that any of the tokens [start, start + count) sees."""

    return start + count - (0 if window is None else max(0, start + 1 - window))


def work(case):
    decode, chunks = _rows(case)
    spans, design, width = decode + chunks, case["design"], case["width"]
    tokens = sum(n for _, n in spans)
    size = 1 if design.startswith("qwen3") else 2
    weights = flops = moved = 0
    for index in range(case["layers"]):
        window, pair_flops, row_bytes, per_token = None, 0, 0, 0
        if design == "ripesun":
            heads, ff, q_rank = RIPESUN_SIZES[width]
            weight = 2 * width * ff + 2 * SIDE * width
            if index % 4 == 0:
                window, row_bytes = WINDOW, 2 * (KV_RANK + ROTATED)
                weight += width * q_rank + q_rank * heads * (HEAD + ROTATED) + 2 * heads * HEAD * KV_RANK + width * heads * HEAD
                weight += 0 if index else width * (KV_RANK + ROTATED)
                # A single token attends in the latent space, a chunk over expanded heads.
                flops += sum(2 * heads * (2 * KV_RANK + ROTATED) * _pairs(p, n, window) for p, n in decode)
                flops += sum(2 * heads * (2 * HEAD + ROTATED) * _pairs(p, n, window) for p, n in chunks)
            elif index % 4 == 3:
                weight += 4 * width * width
                moved += len(spans) * 2 * 4 * width
                flops += 6 * width * tokens
            else:
                weight += 5 * width * heads * HEAD
                moved += len(spans) * 2 * 4 * heads * HEAD * HEAD
                flops += 4 * heads * HEAD * HEAD * tokens
        else:
            heads, kv_heads, ff = ATTENTION_SIZES[width]
            weight = width * (2 * heads + 2 * kv_heads) * HEAD + 3 * width * ff
            row_bytes = 2 * kv_heads * (HEAD + 4 if design == "qwen3-kv8" else 2 * HEAD)
            window = WINDOW if design == "tidelorn" and index % 2 else None
            flops += sum(4 * heads * HEAD * _pairs(p, n, window) for p, n in spans)
        weights += weight * size
        flops += 2 * weight * tokens
        moved += row_bytes * (sum(_seen(p, n, window) for p, n in spans) + tokens)
    logits = len(spans) * VOCAB
    weights += 2 * VOCAB * width
    flops += 2 * width * logits
    return {"bytes": weights + moved + logits * (2 if size == 1 else 4) + tokens * 2 * width, "flops": flops}


def tolerance(case):
    # Measured.  Qwen3 and Tidelorn: about four times what other sums make of the step (FP8 GEMMs with their K range cut
    # or not: up to 7e-3 here, the bf16 rounding points against 64 bits: 8e-3).  Ripesun: four times the distance from
    # 64 bits (2.4e-3).
    return {"rel": 1e-2} if case["design"] == "ripesun" else {"rel": 3e-2}


# -- the same step in 64 bits -----------------------------------------------------------------------------

def _rms(x, eps, weight=1.0):
    return x / torch.sqrt(x.square().mean(dim=-1, keepdim=True) + eps) * weight


def _e4m3(x):
    """Groups of 128 along the last dimension as e4m3 values times their group's scale."""

    groups = x.view(*x.shape[:-1], -1, 128)
    scale = groups.abs().amax(dim=-1, keepdim=True) / 448.0
    return ((groups / scale.clamp_min(1e-12)).float().to(torch.float8_e4m3fn).double() * scale).view(x.shape)


def _linear8(x, weight, scales):
    n, k = weight.shape
    full = weight.double().view(n // 128, 128, k // 128, 128) * scales.double()[:, None, :, None]
    return _e4m3(x) @ full.view(n, k).t()


class Cache:
    """A layer's rows per token, [tokens, ...] per request, over a 64-bit copy of its pages."""

    def __init__(self, s, pages):
        self.s, self.pages = s, pages

    def swap(self, new):
        """Write the step's rows; then ``read(request)`` gives that request's rows from position 0."""

        s = self.s
        where = s.tables[s.owners.long(), (s.positions // PAGE).long()].long()
        self.pages[where, :, (s.positions % PAGE).long()] = new
        return self

    def read(self, request, end):
        rows = self.pages[self.s.tables[request, :-(-end // PAGE)].long()]  # [pages, heads, page, dim]
        return rows.transpose(1, 2).reshape(-1, rows.shape[1], rows.shape[3])[:end]


def _attend(s, q, keys, values, scale, window=None, sinks=None):
    """[tokens, heads, value dim]: softmax attention of every token over its request's cached rows."""

    heads, kv_heads = q.shape[1], keys.pages.shape[1]
    out = torch.empty(q.shape[0], heads, values.pages.shape[3], dtype=q.dtype, device=q.device)
    cursor = 0
    for request, (start, count) in enumerate(s.decode + s.chunks):
        k = keys.read(request, start + count).repeat_interleave(heads // kv_heads, dim=1).permute(1, 2, 0)
        v = values.read(request, start + count).repeat_interleave(heads // kv_heads, dim=1).transpose(0, 1)
        for at in range(0, count, 512):
            rows = slice(cursor + at, cursor + min(at + 512, count))
            scores = torch.bmm(q[rows].transpose(0, 1), k) * scale
            distance = s.positions[rows].long()[:, None] - torch.arange(start + count, device=q.device)[None, :]
            hidden = distance < 0 if window is None else (distance < 0) | (distance >= window)
            scores.masked_fill_(hidden, -math.inf)
            if sinks is not None:
                scores = torch.cat([scores, sinks.double()[:, None, None].expand(-1, scores.shape[1], 1)], dim=-1)
            weights = torch.softmax(scores, dim=-1)
            if sinks is not None:
                weights = weights[..., :-1]
            out[rows] = torch.bmm(weights, v).transpose(0, 1)
        cursor += count
    return out


def _exact_qwen3(case, s):
    r = s.runner
    shape, w, tokens = r.shape, r.weights, s.ids.shape[0]
    heads, kv_heads = shape.q_heads, shape.kv_heads
    inv = 1.0 / shape.rope_theta ** (torch.arange(0, HEAD, 2, device=s.ids.device).double() / HEAD)
    angle = torch.cat([s.positions.double()[:, None] * inv] * 2, dim=-1)[:, None]

    def rope(x):
        half = torch.cat([-x[..., HEAD // 2:], x[..., :HEAD // 2]], dim=-1)
        return x * angle.cos() + half * angle.sin()

    x = w.embedding[s.ids].double()
    for index, layer in enumerate(w.layers):
        h = _rms(x, shape.rms_eps, layer.input_norm.double())
        qkv = _linear8(h, layer.qkv, layer.qkv_scale).view(tokens, heads + 2 * kv_heads, HEAD)
        q = rope(_rms(qkv[:, :heads], shape.rms_eps, layer.q_norm.double()))
        k = rope(_rms(qkv[:, heads:heads + kv_heads], shape.rms_eps, layer.k_norm.double()))
        v = qkv[:, heads + kv_heads:]
        if r.kv8 is None:
            pools = [r.key_blocks[index].double(), r.value_blocks[index].double()]
        else:
            data, scales = r.kv8.data[index].view(torch.float8_e4m3fn).double(), r.kv8.scales[index].double()
            pools = list((data * scales[..., None]).unbind(2))
            k, v = _e4m3(k), _e4m3(v)
        keys, values = Cache(s, pools[0]).swap(k), Cache(s, pools[1]).swap(v)
        attended = _attend(s, q, keys, values, HEAD ** -0.5).view(tokens, heads * HEAD)
        x = x + _linear8(attended, layer.o, layer.o_scale)
        h = _rms(x, shape.rms_eps, layer.post_norm.double())
        gate, up = _linear8(h, layer.gate_up, layer.gate_up_scale).chunk(2, dim=-1)
        x = x + _linear8(gate * torch.sigmoid(gate) * up, layer.down, layer.down_scale)
    final = _rms(x[s.rows], shape.rms_eps, w.final_norm.double())
    pages = {"keys": keys.pages, "values": values.pages} if s.chunks else {}
    return {"logits": final @ w.lm_head.double().t(), **pages}


def _exact_tidelorn(case, s):
    r = s.runner
    shape, w, tokens = r.shape, r.weights, s.ids.shape[0]
    # The token before each one: its neighbour in the step, or what the cache holds.
    before = (s.positions - 1).clamp_min(0).long()
    previous = r.history[s.tables[s.owners.long(), before // PAGE].long(), before % PAGE].long()
    inside = torch.zeros(tokens, dtype=torch.bool, device=s.ids.device)
    inside[1:] = s.owners[1:] == s.owners[:-1]
    previous = torch.where(inside, s.ids.roll(1), previous)
    bigram = (previous * shape.mul_prev + s.ids * shape.mul_cur) % shape.buckets
    bigram = torch.where(s.positions == 0, shape.buckets, bigram)
    entry = torch.arange(shape.width, device=s.ids.device)
    angle = s.positions.double()[:, None] * 10000.0 ** (-2.0 * (entry // 2).double() / shape.width)
    x = w.embed[s.ids].double() * shape.embed_scale + w.bigram[bigram].double()
    x = x + torch.where(entry % 2 == 0, angle.sin(), angle.cos())
    first = None
    for index, (layer, lw) in enumerate(zip(shape.layers, w.layers)):
        qkv = x @ lw.qkv.double().t()
        if lw.qkv_bias is not None:
            qkv = qkv + lw.qkv_bias.double()
        q, k, v = qkv.split([layer.heads * layer.dim, layer.kv_heads * layer.dim, layer.kv_heads * layer.vdim], dim=-1)
        q = _rms(q.reshape(tokens, layer.heads, -1), shape.eps)
        k, v = _rms(k.reshape(tokens, layer.kv_heads, -1), shape.eps), v.reshape(tokens, layer.kv_heads, -1)
        if layer.temperature is not None:
            coef, every = layer.temperature
            q = q * (1.0 + coef * torch.log(((s.positions + 1) // every).double() + 1.0))[:, None, None]
        if layer.v_mix:
            first = v if first is None else first
            v = (1.0 - lw.lam) * v + lw.lam * first
        keys = Cache(s, r.key_blocks[index].double()).swap(k)
        values = Cache(s, r.value_blocks[index].double()).swap(v)
        mixed = _attend(s, q, keys, values, layer.scale, layer.window, lw.sinks).view(tokens, -1) @ lw.o.double().t()
        x = _rms(shape.alpha * x + mixed, shape.eps, 1.0 + lw.norm1.double())
        g, u = (x @ lw.gate_up.double().t()).chunk(2, dim=-1)
        g, u = g.clamp(max=layer.limit), u.clamp(-layer.limit, layer.limit)
        y = (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ lw.down.double().t()
        x = _rms(shape.alpha * x + y, shape.eps, 1.0 + lw.norm2.double())
    final = _rms(x[s.rows], shape.eps, 1.0 + w.final_norm.double())
    pages = {"keys": keys.pages, "values": values.pages} if s.chunks else {}
    return {"logits": final @ w.head.double().t(), **pages}


def _exact_ripesun(case, s):
    r = s.runner
    shape, w, tokens = r.shape, r.weights, s.ids.shape[0]
    spans, slots = s.decode + s.chunks, s.extra["state_slots"].long()
    state = r.state.rows.double()
    bounds, cursor = [], 0
    for start, count in spans:
        bounds.append((slice(cursor, cursor + count), start, count))
        cursor += count

    def gelu(z):
        return torch.nn.functional.gelu(z, approximate="tanh")

    def silu(z):
        return z * torch.sigmoid(z)

    def turn(x, mixer):
        inv = mixer.rot_base ** (-2.0 * torch.arange(mixer.rotated // 2, device=x.device).double() / mixer.rotated)
        angle = (s.positions.double()[:, None] * inv).view(tokens, *[1] * (x.ndim - 2), -1)
        u, v = x[..., 0:mixer.rotated:2], x[..., 1:mixer.rotated:2]
        both = torch.stack([u * angle.cos() - v * angle.sin(), v * angle.cos() + u * angle.sin()], dim=-1)
        return torch.cat([both.flatten(-2), x[..., mixer.rotated:]], dim=-1)

    def attention(index, mixer, lw, h):
        down = h @ lw.down.double().t()
        if mixer.kv_from is None:
            latent = _rms(down[:, mixer.q_rank:mixer.q_rank + mixer.kv_rank], shape.eps, lw.kv_norm.double())
            rows = torch.cat([latent, turn(down[:, mixer.q_rank + mixer.kv_rank:], mixer)], dim=-1)
            caches[index] = Cache(s, r.latents[index].double()).swap(rows[:, None])
        cache = caches[index if mixer.kv_from is None else mixer.kv_from]
        q = _rms(down[:, :mixer.q_rank], shape.eps, lw.q_norm.double()) @ lw.uq.double().t()
        q = q.view(tokens, mixer.heads, mixer.qk_dim)
        q = torch.cat([torch.einsum("thd,hdr->thr", q[..., :mixer.dim], lw.uk.double()), turn(q[..., mixer.dim:], mixer)], -1)
        values = Cache(s, cache.pages[..., :mixer.kv_rank])
        out = _attend(s, q, cache, values, mixer.scale, mixer.window, lw.sinks)
        return torch.einsum("thr,hvr->thv", out, lw.uv.double()).reshape(tokens, -1) @ lw.o.double().t()

    def lightning(index, mixer, lw, h):
        rows = h @ lw.inputs.double().t()
        keys, vals = mixer.heads * mixer.dim, mixer.heads * mixer.vdim
        q, k, v, gate = rows.split([keys, keys, vals, vals], dim=-1)
        q, k = (silu(y).view(tokens, mixer.heads, mixer.dim) for y in (q, k))
        v = silu(v).view(tokens, mixer.heads, mixer.vdim)
        decay, offset = lw.decay.double(), r.state.offsets[r._state_index[index]]
        out = torch.empty_like(v)
        for (rows_, start, count), slot in zip(bounds, slots.tolist()):
            old = state[slot, offset:offset + mixer.state_floats].view(mixer.heads, mixer.dim, mixer.vdim)
            carried = old * (0.0 if start == 0 else 1.0)
            for at in range(0, count, 512):  # 512 tokens at a time: a decayed product and the state before them
                part = slice(rows_.start + at, min(rows_.start + at + 512, rows_.stop))
                n = part.stop - part.start
                steps = torch.arange(n, device=h.device).double()
                apart = steps[:, None] - steps[None, :]
                falls = torch.where(apart >= 0, decay[:, None, None] ** apart.clamp_min(0), 0.0)
                qh, kh, vh = (y[part].transpose(0, 1) for y in (q, k, v))
                o = (torch.bmm(qh, kh.transpose(1, 2)) * falls) @ vh
                o = o + torch.bmm(qh, carried) * (decay[:, None] ** (steps + 1))[..., None]
                carried = carried * (decay ** n)[:, None, None] + torch.bmm(
                    (kh * (decay[:, None] ** (n - 1 - steps))[..., None]).transpose(1, 2), vh)
                out[part] = o.transpose(0, 1)
            old.copy_(carried)
        y = _rms(out.view(tokens, vals), shape.eps, lw.norm.double())
        return (y * torch.sigmoid(gate)) @ lw.o.double().t()

    def mingru(index, mixer, lw, h):
        z, u, gate = (h @ lw.inputs.double().t()).chunk(3, dim=-1)
        z, u = torch.sigmoid(z + lw.z_bias.double()), u + lw.u_bias.double()
        gain = z * torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
        offset = r.state.offsets[r._state_index[index]]
        out = torch.empty_like(gain)
        for (rows_, start, count), slot in zip(bounds, slots.tolist()):
            kept = state[slot, offset:offset + mixer.width]
            value = kept * (0.0 if start == 0 else 1.0)
            for t in range(rows_.start, rows_.stop):
                value = (1.0 - z[t]) * value + gain[t]
                out[t] = value
            kept.copy_(value)
        return (out * silu(gate)) @ lw.o.double().t()

    caches = {}
    x = w.embed[s.ids].double() * shape.embed_scale
    for index, (layer, lw) in enumerate(zip(shape.layers, w.layers)):
        h = _rms(x, shape.eps, lw.norm1.double())
        mixer = layer.mixer
        kind = attention if hasattr(mixer, "kv_rank") else lightning if hasattr(mixer, "decay") else mingru
        x = x + shape.residual_mult * _rms(kind(index, mixer, lw, h), shape.eps, lw.norm1b.double())
        h = _rms(x, shape.eps, lw.norm2.double())
        y = gelu(h @ lw.up.double().t()) @ lw.down_ff.double().t()
        x = x + shape.residual_mult * _rms(y, shape.eps, lw.norm2b.double())
        side = (gelu(x @ lw.side_gate.double().t()) * lw.side_table[s.ids].double()) @ lw.side_proj.double().t()
        x = x + shape.residual_mult * _rms(side, shape.eps, lw.side_norm.double())
    logits = _rms(x[s.rows], shape.eps, w.final_norm.double()) @ w.head.double().t()
    pages = {"latents": caches[max(caches)].pages} if s.chunks else {}
    return {"logits": shape.logit_softcap * torch.tanh(logits / shape.logit_softcap), **pages, "state": state}


def exact(case, seed):
    s = prepare(case, seed)
    s.graph = None
    design = {"tidelorn": _exact_tidelorn, "ripesun": _exact_ripesun}.get(case["design"], _exact_qwen3)
    return design(case, s)
