"""The work whose time is measured: what programs have this framework do, through its public engines.

Four kinds of work, over the registered shapes:

* ``step``    -- the next token of one sequence on a quantised decoder (``DecodeEngine``), its logits kept for a sampler;
* ``batch``   -- one step of several independent sequences (``BatchDecodeEngine``);
* ``prompt``  -- a prompt taken into the caches of a quantised decoder (``PrefillEngine``);
* ``layered`` -- prompts, portions of them and single steps on the layered decoders (``LayeredEngine``).

Weights and cache contents are the engines' synthetic ones, drawn from streams that the seed names, so every seed is another
model; ``_Conditioned`` gives them the proportions of trained ones where those matter to what errors do.  Greedy token ids are left out of the outputs: a head of random weights puts several of 152064 logits within one bf16 step
of the largest, so two correct runs may name different ones; the logits they come from are compared instead.

``exact`` restates the decoders in plain torch at 64 bits (weights regenerated from the same streams).
"""
import math
import random
from dataclasses import replace

import numpy as np
import torch

from fusekit_b200.batch import BatchDecodeEngine, PrefillEngine
from fusekit_b200.layered import LayeredEngine
from fusekit_b200.model_spec import ParallelMixerSpec, block_layout, config, stream_id, tensor_name
from fusekit_b200.runtime import DecodeEngine, Runtime

PROMPT_ROWS = 16          # positions that a PrefillEngine is made for
MOST_TOKENS = 1000        # longest drawn prompt of a quantised decoder


def listed():
    return [
        # the smallest call: a small model early in a chat, where launches and latency are most of the time
        {"name": "step 0.5b q4 ctx 32", "kind": "step", "model": "qwen2.5-0.5b", "bits": 4, "kv_bits": 0, "ctx": 32},
        # interactive generation on a 7B model, the shape of the headline benchmark
        {"name": "step 7b q4 ctx 512", "kind": "step", "model": "qwen2.5-7b", "bits": 4, "kv_bits": 0, "ctx": 512},
        # 8-bit weights and an 8-bit cache, chosen for quality and for long contexts; an odd context
        {"name": "step 7b q8 kv8 ctx 3999", "kind": "step", "model": "qwen2.5-7b", "bits": 8, "kv_bits": 8, "ctx": 3999},
        # sliding windows beside global layers, wide heads, a large vocabulary
        {"name": "step gemma q4 ctx 4096", "kind": "step", "model": "gemma3-4b", "bits": 4, "kv_bits": 0, "ctx": 4096},
        # a few short requests served together on a small model
        {"name": "batch 0.5b 5 rows ctx 300", "kind": "batch", "model": "qwen2.5-0.5b", "rows": 5, "ctx": 300},
        # a full batch of long sequences on the largest model
        {"name": "batch 32b 16 rows ctx 4096", "kind": "batch", "model": "qwen2.5-32b", "rows": 16, "ctx": 4096},
        # a short question to a small model; no multiple of the rows of a pass
        {"name": "prompt 0.5b 100", "kind": "prompt", "model": "qwen2.5-0.5b", "tokens": 100},
        # a document of some pages before a question
        {"name": "prompt 7b 1000", "kind": "prompt", "model": "qwen2.5-7b", "tokens": 1000},
        # generation on a mixture of experts with differential attention
        {"name": "fatulix-3584 step ctx 1024", "kind": "layered", "model": "fatulix-3584", "ctx": 1024, "tokens": 0, "forced": 1},
        # a full portion of a prompt on the looped mixture of experts
        {"name": "fatulix-2048 prompt 2048", "kind": "layered", "model": "fatulix-2048", "ctx": 0, "tokens": 2048, "forced": 0},
        # a short turn on parallel blocks: a prompt, then given tokens one by one (scoring, or a constrained reply)
        {"name": "kakunex-2048 turn 190 + 12", "kind": "layered", "model": "kakunex-2048", "ctx": 0, "tokens": 190, "forced": 12},
        # a long ragged prompt on the widest parallel blocks: windows, recurrences and matrix memories over rows
        {"name": "kakunex-5120 prompt 1500", "kind": "layered", "model": "kakunex-5120", "ctx": 0, "tokens": 1500, "forced": 0},
    ]


def _log(rng, low, high):
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    kind = rng.choice(("step", "batch", "prompt", "layered"))
    if kind == "step":
        model = rng.choice(("qwen2.5-0.5b", "qwen2.5-7b", "qwen2.5-7b", "gemma3-4b"))
        kv_bits = rng.choice((0, 0, 0, 4, 8)) if model == "qwen2.5-7b" else 0
        return {"kind": kind, "model": model, "bits": rng.choice((4, 4, 8, 16)), "kv_bits": kv_bits, "ctx": _log(rng, 20, 4096)}
    if kind == "batch":
        return {"kind": kind, "model": rng.choice(("qwen2.5-0.5b", "qwen2.5-7b")), "rows": rng.randint(2, 16), "ctx": _log(rng, 20, 4096)}
    if kind == "prompt":
        return {"kind": kind, "model": rng.choice(("qwen2.5-0.5b", "qwen2.5-7b")), "tokens": _log(rng, 9, MOST_TOKENS)}
    model = rng.choice(("fatulix-2048", "fatulix-3584", "fatulix-5120", "kakunex-2048", "kakunex-3584", "kakunex-5120"))
    if model.startswith("fatulix") and rng.random() < 0.5:
        return {"kind": kind, "model": model, "ctx": _log(rng, 20, 4000), "tokens": 0, "forced": 1}
    return {"kind": kind, "model": model, "ctx": 0, "tokens": _log(rng, 17, 2048), "forced": rng.choice((0, 0, rng.randint(1, 12)))}


# ---------------------------------------------------------------- what a program keeps
class _Owner:
    """An engine that is closed with the last thing that refers to it."""

    def __init__(self, engine):
        self.engine = engine

    def __del__(self):
        self.engine.close()


class _Memory:
    def __init__(self, owner, address, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": kind, "data": (address, False), "version": 3, "strides": None}


def _factors(spec):
    """Stream -> factor on the synthetic values.  In a trained decoder a sublayer adds little to the residual stream, so rounding
    errors are not multiplied from layer to layer; and a router is sharp, so the last of the chosen experts weighs little."""
    if hasattr(spec, "layers"):
        return {stream_id(spec.seed, "l%d.mlp.router" % i): 4.0 for i in range(len(spec.layers))}
    small, out = 0.5 / math.sqrt(2 * spec.n_layers), {}
    for l in range(spec.n_layers):
        for leaf in ("post_attention_norm", "post_feedforward_norm") if spec.arch == "gemma3" else ("o_proj", "down_proj"):
            out[stream_id(spec.seed, tensor_name(l, leaf))] = small
    if spec.arch != "gemma3":                           # its embedding rows are scaled by sqrt(hidden) when they are looked up
        out[stream_id(spec.seed, tensor_name(-1, "embed_tokens"))] = 50.0
    return out


class _Conditioned(Runtime):
    def __init__(self, spec):
        super().__init__()
        self.factors = _factors(spec)

    def weight_synth_rows(self, wid, dst_row0, nrows, stream, std, k_global, src_row0, k0):
        super().weight_synth_rows(wid, dst_row0, nrows, stream, std * self.factors.get(stream, 1.0), k_global, src_row0, k0)

    def synth_normal(self, dptr, stream, idx0, n, mean, std):
        f = self.factors.get(stream, 1.0)
        super().synth_normal(dptr, stream, idx0, n, mean * f, std * f)


def _view(owner, address, shape, dtype):
    """An engine's device buffer as a tensor; the engine lives as long as the tensor."""
    t = torch.as_tensor(_Memory(owner, address, shape, "<f4" if dtype == torch.float32 else "<i2"), device="cuda")
    return t if dtype == torch.float32 else t.view(dtype)


def _spec(case, seed):
    spec = replace(config(case["model"]), seed=int(seed))
    return spec.with_bits(case.get("bits", 4)) if case["kind"] != "layered" else spec


def _tokens(case, seed, count):
    rng = random.Random("tokens %d" % seed)
    vocab = config(case["model"]).vocab
    return [rng.randrange(vocab) for _ in range(count)]


def _quantised_cache(case, seed, which):
    """Packed words, scales and biases of every layer's cache rows: the digits, steps and lower edges that unit-variance rows have."""
    s, b, ctx = config(case["model"]), case["kv_bits"], case["ctx"]
    rng, top = np.random.default_rng([seed, which]), (1 << b) - 1
    for _ in range(s.n_layers):
        words = rng.integers(0, 1 << 32, (s.n_kv, ctx, s.head_dim * b // 32), np.uint32)
        step = rng.uniform(3.6, 5.0, (s.n_kv, ctx, s.head_dim // 64)).astype(np.float32) / top
        edge = -step * np.float32(top / 2.0)
        yield words, _bf16_bits(step), _bf16_bits(edge)


def _bf16_bits(a):
    return torch.from_numpy(a).to(torch.bfloat16).view(torch.int16).numpy().view(np.uint16)


def prepare(case, seed):
    spec = _spec(case, seed)
    return {"step": _prepare_step, "batch": _prepare_batch, "prompt": _prepare_prompt, "layered": _prepare_layered}[case["kind"]](case, spec, int(seed))


def _prepare_step(case, spec, seed):
    ctx = case["ctx"]
    eng = DecodeEngine(spec, ctx + 256, want_logits=True, runtime=_Conditioned(spec), kv_bits=case["kv_bits"])
    owner = _Owner(eng)
    eng.load_synthetic()
    if case["kv_bits"]:
        cap = ctx + 256
        for n, which in enumerate("kv"):
            for l, parts in enumerate(_quantised_cache(case, seed, n)):
                for name, a in zip((which, which + "_scales", which + "_biases"), parts):
                    for h in range(spec.n_kv):          # a head's rows lie `capacity` apart
                        eng.rt.upload(eng.cacheq[l][name] + h * cap * a[h, 0].nbytes, a[h])
    else:
        eng.prefill_kv_synthetic(ctx)
    eng.capture()
    return {"owner": owner, "case": case, "token": _tokens(case, seed, 1)[0],
            "logits": _view(owner, eng.logits, (spec.vocab,), torch.bfloat16),
            "stream": _view(owner, eng.x_ptr(0), (spec.n_layers + 1, spec.hidden), torch.bfloat16)}


def _prepare_batch(case, spec, seed):
    eng = BatchDecodeEngine(spec, case["ctx"] + 64, case["rows"], runtime=_Conditioned(spec))
    owner = _Owner(eng)
    eng.load_synthetic()
    eng.prefill_kv_synthetic(case["ctx"])
    eng.capture()
    return {"owner": owner, "case": case, "tokens": np.array(_tokens(case, seed, case["rows"]), np.uint32),
            "logits": _view(owner, eng.logits, (case["rows"], spec.vocab), torch.bfloat16),
            "stream": _view(owner, eng.x_ptr(0), (spec.n_layers + 1, case["rows"], spec.hidden), torch.bfloat16)}


def _prepare_prompt(case, spec, seed):
    n = case["tokens"]
    cap = -(-n // PROMPT_ROWS) * PROMPT_ROWS + 64
    eng = PrefillEngine(spec, cap, PROMPT_ROWS, runtime=_Conditioned(spec))
    owner = _Owner(eng)
    eng.load_synthetic()
    eng.capture()
    views = [[_view(owner, p, (spec.n_kv, cap, spec.head_dim), torch.bfloat16)[:, :n] for p in kv] for kv in eng.cache]
    return {"owner": owner, "case": case, "tokens": _tokens(case, seed, n), "caches": views,
            "logits": _view(owner, eng.logits, (PROMPT_ROWS, spec.vocab), torch.bfloat16)[:(n - 1) % PROMPT_ROWS + 1]}


def _prepare_layered(case, spec, seed):
    n, forced = case["tokens"], case["forced"]
    eng = LayeredEngine(spec, max(case["ctx"], n) + 256, runtime=_Conditioned(spec))
    owner = _Owner(eng)
    eng.load_synthetic()
    tokens = _tokens(case, seed, n + forced)
    if case["ctx"]:
        eng.prefill_kv_synthetic(case["ctx"])
    if forced:
        eng.capture()
    state = {"owner": owner, "case": case, "prompt": tokens[:n], "forced": tokens[n:]}
    if case["ctx"]:
        state["logits"] = _view(owner, eng.logits, (spec.vocab,), torch.float32)
        state["stream"] = _view(owner, eng.X, (len(spec.runs()) + 1, spec.hidden), torch.float32)
        return state
    state["memory"] = []
    for run, (i, _) in enumerate(spec.runs()):
        m, bufs, kept = spec.layers[i].mixer, eng.caches[eng.slot][run], {}
        a = m.left if isinstance(m, ParallelMixerSpec) else m
        for key, heads, d in (("layer_cache_k", getattr(a, "kv_heads", 0) * getattr(a, "maps", 1), a.dim), ("layer_cache_v", getattr(a, "kv_heads", 0), a.vdim)):
            if key in bufs:
                kept[key] = _view(owner, bufs[key], (heads, eng.capacity, d), torch.bfloat16)[:, :n + forced]
        state["memory"].append(kept)
    return state


def run(state):
    case, eng = state["case"], state["owner"].engine
    if case["kind"] == "step":
        eng.decode_chunk(case["ctx"], state["token"], 1)
        return {"logits": state["logits"], "stream": state["stream"]}
    if case["kind"] == "batch":
        eng.decode_chunk(case["ctx"], state["tokens"], 1)
        return {"logits": state["logits"], "stream": state["stream"]}
    if case["kind"] == "prompt":
        eng.prefill(state["tokens"])
        return {"logits": state["logits"], "caches": state["caches"]}
    if case["ctx"]:
        eng.decode_chunk(case["ctx"], state["forced"][0], 1)
        return {"logits": state["logits"], "stream": state["stream"]}
    seq = eng.open_sequence()
    out = [seq.append(state["prompt"], [len(state["prompt"]) - 1])]
    out += [seq.append([t], [0]) for t in state["forced"]]
    seq.close()
    return {"logits": out, "memory": state["memory"]}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    spec = _spec(case, 0)
    if case["kind"] == "layered":
        n, forced = case["tokens"], case["forced"]
        if case["ctx"]:
            return {"bytes": spec.bytes_per_token(case["ctx"] + 1), "flops": spec.flops_per_token(case["ctx"] + 1) + 2.0 * spec.hidden * spec.vocab}
        weights = 2 * sum(math.prod(shape) for shape in _matrices(spec).values())
        steps = forced * spec.bytes_per_token(n + 1)
        flops = n * spec.flops_per_token(n // 2) + forced * spec.flops_per_token(n) + 2.0 * (1 + forced) * spec.hidden * spec.vocab
        rows = [l.mixer.left if isinstance(l.mixer, ParallelMixerSpec) else l.mixer for l in (spec.layers[i] for i, _ in spec.runs())]
        rows = sum(2 * n * (m.k_rows + m.v_rows) for m in rows if hasattr(m, "k_rows"))       # keys and values, written once
        return {"bytes": weights + rows + steps + 4 * (1 + forced) * spec.vocab, "flops": flops}
    qkv = (spec.n_q + 2 * spec.n_kv) * spec.head_dim
    params = spec.n_layers * (spec.hidden * (qkv + spec.n_q * spec.head_dim + 3 * spec.inter)) + spec.hidden * spec.vocab
    rows = {"step": 1, "batch": case.get("rows", 1), "prompt": case.get("tokens", 1)}[case["kind"]]
    if case["kind"] == "prompt":
        kv, pairs = spec.kv_bytes_per_token(rows), rows * (rows + 1) / 2
    else:
        kv, pairs = rows * spec.kv_bytes_per_token(case["ctx"] + 1), rows * (case["ctx"] + 1)
        if case.get("kv_bits"):
            kv = kv * case["kv_bits"] / 16 * (1 + 32 / (64 * case["kv_bits"]))
    logits = 2 * spec.vocab * (rows if case["kind"] != "prompt" else 0)
    return {"bytes": spec.weight_bytes_per_token() + kv + logits, "flops": 2.0 * rows * params + 4.0 * pairs * spec.n_layers * spec.n_q * spec.head_dim}


def _matrices(spec):
    """Shapes of a layered decoder's matrices by name: every one is read for a prompt (all experts are, over many positions)."""
    out, D = {}, spec.hidden
    for i, l in enumerate(spec.layers):
        m, f, t = l.mixer, l.mlp, "l%d." % i
        if spec.block == "parallel":
            out.update({t + leaf: (n, D) for leaf, _, n in block_layout(l).sources})
            out.update({t + "mix.left.o": (D, m.left.out_rows), t + "mix.right.o": (D, m.right.out_rows)} if isinstance(m, ParallelMixerSpec) else {t + "mix.o": (D, m.out_rows)})
            if f is not None:
                out.update({t + "mlp.gate": (f.ff, D), t + "mlp.up": (f.ff, D), t + "mlp.down": (D, f.ff)})
            continue
        out.update({t + "mix.q": (m.q_rows, D), t + "mix.k": (m.k_rows, D), t + "mix.v": (m.v_rows, D), t + "mix.g": (m.heads, D), t + "mix.o": (D, m.heads * m.vdim)})
        out.update({t + "mlp.router": (f.experts, D), t + "mlp.shared.up": (f.shared_ff, D), t + "mlp.shared.down": (D, f.shared_ff)})
        for e in range(f.experts):
            out.update({"%smlp.e%d.up" % (t, e): (f.ff, D), "%smlp.e%d.down" % (t, e): (D, f.ff)})
    out["embed" if spec.block == "parallel" else "head"] = (spec.vocab, D)
    return out


def tolerance(case):
    """bf16 operands, caches and (on the quantised decoders) a bf16 residual through every layer: kernels that sum in another order
    flip roundings, which the layers carry on.  Seen between this library's two weight layouts and its two matrix products: 0.004 (24
    layers of the small model) to 0.023 (64 layers), largest single value 0.13; against 64 bits 0.011 to 0.016.  Layered decoders:
    against 64 bits 0.0002 (a step) to 0.017 (prompts, where a rounding may also pick another last expert for a position: single
    values up to 0.7 of the root mean square)."""
    return {"rel": 0.03, "max": 0.99 if case["model"].startswith("fatulix") and case["tokens"] else 0.5}


# ---------------------------------------------------------------- the same in 64 bits
_MASK = (1 << 64) - 1


def _signed(v):
    v &= _MASK
    return v - (1 << 64) if v >> 63 else v


def _shift(z, n):
    return (z >> n) & ((1 << (64 - n)) - 1)


def _mix(z):
    z = z + _signed(0x9E3779B97F4A7C15)
    z = (z ^ _shift(z, 30)) * _signed(0xBF58476D1CE4E5B9)
    z = (z ^ _shift(z, 27)) * _signed(0x94D049BB133111EB)
    return z ^ _shift(z, 31)


def _normal(stream, first, count):
    """Unit-variance values [first, first + count) of a stream: twelve 16-bit uniforms summed, exact in fp32."""
    base = _mix((torch.arange(first, first + count, device="cuda", dtype=torch.int64) * _signed(0xD1342543DE82EF95)) ^ _signed(stream))
    s = torch.zeros(count, device="cuda", dtype=torch.int64)
    for lane in range(3):
        h = _mix(base + lane)
        s += (h & 0xFFFF) + ((h >> 16) & 0xFFFF) + ((h >> 32) & 0xFFFF) + ((h >> 48) & 0xFFFF)
    return (s - 393210).to(torch.float32) * (1.0 / 65536.0)


def _bf16_stream(stream, first, count, mean, std):
    return (_normal(stream, first, count) * std + mean).to(torch.bfloat16).double()


def _weight(stream, rows, k, bits, std, first_row=0):
    """The rows of a synthetic weight as the numbers that its stored form stands for."""
    w = _normal(stream, first_row * k, rows * k) * std
    if bits == 16:
        return w.to(torch.bfloat16).double().view(rows, k)
    w = w.view(rows, k // 64, 64)
    top = torch.full((rows, k // 64, 1), float((1 << bits) - 1), device="cuda")
    low = w.amin(-1, keepdim=True)
    s = ((w.amax(-1, keepdim=True) - low) / top).to(torch.bfloat16).float()
    b = low.to(torch.bfloat16).float()
    q = torch.round((w - b) / s.expand_as(w)).clamp(0, (1 << bits) - 1)
    return (q.double() * s.double() + b.double()).view(rows, k)


def _times(x, stream, rows, k, bits, std=0.02):
    """x W^T in slices of rows."""
    step = max(1, (1 << 23) // k)
    return torch.cat([x @ _weight(stream, min(step, rows - r), k, bits, std, r).T for r in range(0, rows, step)], 1)


def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def exact(case, seed):
    if case["kind"] == "layered":
        return _exact_layered(case, _spec(case, seed), int(seed))
    if case["model"] == "qwen2.5-32b":
        return None                                     # 64 layers of weights and 17 GB of cache rows to regenerate
    with torch.no_grad():
        return _exact_quantised(case, _spec(case, seed), int(seed))


def _rope(x, positions, theta):
    """x [rows, heads, d]: dimensions d and d + half turned together."""
    half = x.shape[-1] // 2
    a = positions.double()[:, None] * theta ** (-torch.arange(half, device="cuda", dtype=torch.float64) / half)
    c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]
    lo, hi = x[..., :half], x[..., half:]
    return torch.cat([lo * c - hi * s, hi * c + lo * s], -1)


def _attend(q, k, v, scale, see=None):
    """q [heads, rows, d], k and v [kv heads, keys, d]; see [rows, keys]: which keys a row sees."""
    g = q.shape[0] // k.shape[0]
    out = []
    for h in range(q.shape[0]):
        s = q[h] @ k[h // g].T * scale
        out.append(torch.softmax(s if see is None else s.masked_fill(~see, -math.inf), -1) @ v[h // g])
    return torch.stack(out)


def _exact_quantised(case, s, seed):
    H, hd, nq, nkv, kind = s.hidden, s.head_dim, s.n_q, s.n_kv, case["kind"]
    gemma = s.arch == "gemma3"
    name = lambda l, leaf: stream_id(s.seed, tensor_name(l, leaf))                                     # noqa: E731
    by = _factors(s)
    fac = lambda l, leaf: by.get(name(l, leaf), 1.0)                                                   # noqa: E731
    lin = lambda x, l, leaf, rows: _times(x, name(l, leaf), rows, x.shape[1], s.bits, 0.02 * fac(l, leaf))                  # noqa: E731
    vec = lambda l, leaf, n, mean=1.0: _bf16_stream(name(l, leaf), 0, n, mean * fac(l, leaf), 0.02 * fac(l, leaf))          # noqa: E731
    rows = {"step": 1, "batch": case.get("rows", 1), "prompt": case.get("tokens", 1)}[kind]
    tokens, ctx = _tokens(case, seed, rows), case.get("ctx", 0)
    pos = torch.arange(rows, device="cuda") if kind == "prompt" else torch.full((rows,), ctx, device="cuda")
    x = torch.stack([_bf16_stream(name(-1, "embed_tokens"), t * H, H, 0.0, 0.02 * fac(-1, "embed_tokens")) for t in tokens])
    if gemma:
        x = x * float(torch.tensor(math.sqrt(H)).to(torch.bfloat16))
    stream, caches = [x], []
    packed = [list(_quantised_cache(case, seed, n)) for n in range(2)] if case.get("kv_bits") else None

    def cached(l, which, m):
        """Rows that the cache of sequence m holds before the pass, [kv heads, rows, hd]."""
        if packed is not None:
            words, step, edge = (torch.from_numpy(a.astype(np.int64)).cuda() for a in packed["kv".index(which)][l])
            b = case["kv_bits"]
            q = (words[..., None] >> (torch.arange(32 // b, device="cuda") * b)) & ((1 << b) - 1)
            real = lambda t: t.to(torch.int16).view(torch.bfloat16).double().repeat_interleave(64, -1)     # noqa: E731
            return q.reshape(nkv, ctx, hd).double() * real(step) + real(edge)
        n = min(ctx, s.window - 1) if s.is_sliding(l) else ctx
        st = stream_id(s.seed, f"layers.{l}.cache_{which}" + (f".seq{m}" if kind == "batch" else ""))
        return torch.stack([_bf16_stream(st, (h * 1048576 + ctx - n) * hd, n * hd, 0.0, 1.0).view(n, hd) for h in range(nkv)])

    for l in range(s.n_layers):
        h = _rms(x, vec(l, "input_norm", H), s.eps)
        q, k, v = lin(h, l, "q_proj", nq * hd), lin(h, l, "k_proj", nkv * hd), lin(h, l, "v_proj", nkv * hd)
        if not gemma:
            q, k, v = (a + vec(l, leaf, a.shape[1], 0.0) for a, leaf in ((q, "q_bias"), (k, "k_bias"), (v, "v_bias")))
        q, k, v = q.view(rows, nq, hd), k.view(rows, nkv, hd), v.view(rows, nkv, hd)
        if gemma:
            q, k = _rms(q, vec(l, "q_norm", hd), s.eps), _rms(k, vec(l, "k_norm", hd), s.eps)
        q, k = _rope(q, pos, s.layer_theta(l)), _rope(k, pos, s.layer_theta(l))
        if kind == "prompt":
            caches.append([k.transpose(0, 1), v.transpose(0, 1)])
            o = _attend(q.transpose(0, 1), k.transpose(0, 1), v.transpose(0, 1), hd ** -0.5, pos[:, None] >= pos[None]).transpose(0, 1)
        else:
            o = []
            for m in range(rows):
                kk, vv = (torch.cat([cached(l, which, m), a[m][:, None]], 1) for which, a in (("k", k), ("v", v)))
                o.append(_attend(q[m][:, None], kk, vv, hd ** -0.5)[:, 0])
            o = torch.stack(o)
        o = lin(o.reshape(rows, nq * hd), l, "o_proj", H)
        if gemma:
            x = x + _rms(o, vec(l, "post_attention_norm", H), s.eps)
            h = _rms(x, vec(l, "pre_feedforward_norm", H), s.eps)
        else:
            x = x + o
            h = _rms(x, vec(l, "post_attention_norm", H), s.eps)
        gate, up = lin(h, l, "gate_proj", s.inter), lin(h, l, "up_proj", s.inter)
        act = torch.nn.functional.gelu(gate, approximate="tanh") if gemma else torch.nn.functional.silu(gate)
        d = lin(act * up, l, "down_proj", H)
        x = x + (_rms(d, vec(l, "post_feedforward_norm", H), s.eps) if gemma else d)
        stream.append(x)
    if kind == "prompt":
        x = x[-((rows - 1) % PROMPT_ROWS + 1):]
    logits = lin(_rms(x, vec(-1, "final_norm", H), s.eps), -1, "lm_head", s.vocab)
    if kind == "prompt":
        return {"logits": logits, "caches": caches}
    return {"logits": logits[0] if kind == "step" else logits, "stream": torch.stack(stream)[:, 0] if kind == "step" else torch.stack(stream)}


class _Streams:
    """A layered decoder's tensors by name, made when they are asked for."""

    def __init__(self, spec):
        self.spec, self.shapes, self.factors = spec, _matrices(spec), _factors(spec)

    def times(self, x, name):
        rows, k = self.shapes[name]
        stream = stream_id(self.spec.seed, name)
        return _times(x, stream, rows, k, 16, 1.0 / math.sqrt(k) * self.factors.get(stream, 1.0))

    def vec(self, name, n, mean=1.0, std=0.02):
        return _bf16_stream(stream_id(self.spec.seed, name), 0, n, mean, std)


def _exact_layered(case, s, seed):
    n, ctx = case["tokens"] + case["forced"], case["ctx"]
    tokens = _tokens(case, seed, n)
    pos = ctx + torch.arange(n, device="cuda")
    t = _Streams(s)
    wanted = slice(n - 1 - case["forced"], n) if case["tokens"] else slice(0, n)
    with torch.no_grad():
        x, stream, memory = (_sandwich if s.block == "sandwich" else _parallel)(case, s, t, tokens, pos)
        if s.block == "sandwich":
            logits = t.times(_rms(x[wanted], t.vec("final.norm", s.hidden), s.eps), "head")
        else:
            h = torch.nn.functional.layer_norm(x[wanted], (s.hidden,), t.vec("final.norm", s.hidden), t.vec("final.norm.b", s.hidden, 0.0), s.eps)
            logits = _embedded(s, h)
    if ctx:
        return {"logits": logits[0], "stream": torch.stack(stream)[:, 0]}
    return {"logits": [r[None] for r in logits], "memory": memory}


def _sandwich(case, s, t, tokens, pos):
    D, ctx = s.hidden, case["ctx"]
    emb = torch.stack([_bf16_stream(stream_id(s.seed, "embed"), i * D, D, 0.0, 1.0) for i in tokens])
    x, stream, memory = emb, [], []
    for run, (i, again) in enumerate(s.runs()):
        m, f, p = s.layers[i].mixer, s.layers[i].mlp, f"l{i}."
        x = x + emb if again else x
        stream.append(x)
        h, T = _rms(x, t.vec(p + "norm1", D), s.eps), len(tokens)
        q = _rms(t.times(h, p + "mix.q").view(T, m.heads, m.maps, m.dim), t.vec(p + "mix.q.norm", m.dim), s.eps)
        k = _rms(t.times(h, p + "mix.k").view(T, m.kv_heads * m.maps, m.dim), t.vec(p + "mix.k.norm", m.dim), s.eps).transpose(0, 1)
        v = t.times(h, p + "mix.v").view(T, m.kv_heads, m.vdim).transpose(0, 1)
        memory.append({"layer_cache_k": k, "layer_cache_v": v})
        if ctx:
            k, v = (torch.cat([torch.stack([_bf16_stream(stream_id(s.seed, f"runs.{run}.cache_{w}"), hh * 1048576 * a.shape[2], ctx * a.shape[2], 0.0, 1.0).view(ctx, -1)
                                            for hh in range(a.shape[0])]), a], 1) for w, a in (("k", k), ("v", v)))
        see = pos[:, None] >= torch.arange(k.shape[1], device="cuda")[None]
        a = [_attend(q[:, :, j].transpose(0, 1), k[j::m.maps], v, m.scale, see) for j in range(m.maps)]
        o = a[0] - m.diff * a[1]                        # synthetic weights: lambda is its constant part
        o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + s.eps) * (1.0 - m.diff)
        o = (o.transpose(0, 1) * torch.sigmoid(t.times(h, p + "mix.g"))[..., None]).reshape(T, -1)
        x = x + _rms(t.times(o, p + "mix.o"), t.vec(p + "norm1b", D), s.eps)
        h = _rms(x, t.vec(p + "norm2", D), s.eps)
        value, chosen = torch.topk(t.times(h, p + "mlp.router"), f.top, -1)
        weight = torch.softmax(value, -1)
        y = t.times(torch.relu(t.times(h, p + "mlp.shared.up")) ** 2, p + "mlp.shared.down")
        for e in range(f.experts):
            row, place = torch.nonzero(chosen == e, as_tuple=True)
            if len(row):
                up = torch.relu(t.times(h[row], f"{p}mlp.e{e}.up")) ** 2
                y.index_add_(0, row, t.times(up, f"{p}mlp.e{e}.down") * weight[row, place][:, None])
        x = x + _rms(y, t.vec(p + "norm2b", D), s.eps)
    return x, stream + [x], memory


def _gate_up(t, p, f, h):
    """Gate and up rows are taken in turn from one stream."""
    st, k = stream_id(t.spec.seed, p + "mlp.gate+" + p + "mlp.up"), h.shape[1]
    both = _times(h, st, 2 * f.ff, k, 16, 1.0 / math.sqrt(k))
    return both[:, 0::2], both[:, 1::2]


def _embedded(s, h):
    return _times(h, stream_id(s.seed, "embed"), s.vocab, s.hidden, 16, 1.0 / math.sqrt(s.hidden)) * s.logit_scale


def _parallel(case, s, t, tokens, pos):
    D, T, eps = s.hidden, len(tokens), s.eps
    x = torch.cat([_weight(stream_id(s.seed, "embed"), 1, D, 16, 1.0 / math.sqrt(D), i) for i in tokens])
    stream, memory = [], []
    for i, l in enumerate(s.layers):
        m, f, p = l.mixer, l.mlp, f"l{i}."
        stream.append(x)
        h = torch.nn.functional.layer_norm(x, (D,), t.vec(p + "norm1", D), t.vec(p + "norm1.b", D, 0.0), eps)
        if isinstance(m, ParallelMixerSpec):
            a, r, freqs = m.left, m.right, torch.tensor(m.left.rotary.frequencies(), device="cuda", dtype=torch.float64)
            q = _rms(t.times(h, p + "mix.left.q"), t.vec(p + "mix.left.q.norm", a.q_rows), eps).view(T, a.heads, a.dim)
            k = _rms(t.times(h, p + "mix.left.k"), t.vec(p + "mix.left.k.norm", a.k_rows), eps).view(T, a.kv_heads, a.dim)
            v = t.times(h, p + "mix.left.v").view(T, a.kv_heads, a.vdim).transpose(0, 1)
            q, k = (_turn(z, pos, freqs).transpose(0, 1) for z in (q, k))
            memory.append({"layer_cache_k": k, "layer_cache_v": v})
            back = pos[:, None] - pos[None]
            o = _attend(q, k, v, a.scale, (back >= 0) & ((back < a.window) | (pos[None] < a.keep_first)))
            left = t.times(o.transpose(0, 1).reshape(T, -1), p + "mix.left.o")
            q, k, v = (torch.nn.functional.silu(t.times(h, p + "mix.right." + w)).view(T, r.heads, -1) for w in "qkv")
            decay, S, o = torch.tensor(r.decay, device="cuda", dtype=torch.float64)[:, None, None], 0.0, []
            for j in range(T):
                S = decay * S + k[j][:, :, None] * v[j][:, None]
                o.append(torch.einsum("hdv,hd->hv", S, q[j]))
            o = _rms(torch.stack(o).reshape(T, -1), t.vec(p + "mix.right.norm", r.out_rows), eps) * torch.sigmoid(t.times(h, p + "mix.right.g"))
            right = t.times(o, p + "mix.right.o")
            out = t.vec(p + "mix.left.out", D), t.vec(p + "mix.right.out", D)
            y = 0.5 * (_rms(left, out[0], eps) + _rms(right, out[1], eps))
        else:
            memory.append({})
            q = t.times(h, p + "mix.q").view(T, m.heads, -1) * m.dim ** -0.5
            k, v = (t.times(h, p + "mix." + w).view(T, m.heads, -1) for w in "kv")
            cap = lambda z: m.gate_cap * torch.tanh(z / m.gate_cap)                                    # noqa: E731
            gi = cap(t.times(h, p + "mix.i") + t.vec(p + "mix.i.b", m.heads, 1.0, 0.5))
            gf = torch.nn.functional.logsigmoid(cap(t.times(h, p + "mix.f") + t.vec(p + "mix.f.b", m.heads, 1.0, 0.5)))
            S, nrm, top, o = 0.0, 0.0, torch.zeros(m.heads, device="cuda", dtype=torch.float64), []
            for j in range(T):
                new = torch.maximum(gf[j] + top, gi[j])
                keep, add, top = torch.exp(gf[j] + top - new), torch.exp(gi[j] - new), new
                S = keep[:, None, None] * S + add[:, None, None] * k[j][:, :, None] * v[j][:, None]
                nrm = keep[:, None] * nrm + add[:, None] * k[j]
                den = torch.maximum((nrm * q[j]).sum(-1).abs(), torch.exp(-top)) + 1e-6
                o.append(torch.einsum("hdv,hd->hv", S, q[j]) / den[:, None])
            o = torch.stack(o)
            o = (o / torch.sqrt((o * o).mean(-1, keepdim=True) + eps)).reshape(T, -1) * t.vec(p + "mix.norm", m.out_rows)
            y = t.times(o * torch.sigmoid(t.times(h, p + "mix.g")), p + "mix.o")
        g, u = _gate_up(t, p, f, h)
        g, u = g.clamp(max=f.limit), u.clamp(-f.limit, f.limit)
        x = x + y + t.times(g * torch.sigmoid(1.702 * g) * (u + 1.0), p + "mlp.down")
    return x, stream + [x], memory


def _turn(x, pos, freqs):
    """Neighbouring dimensions (2i, 2i + 1) turned by position * freqs[i]."""
    a = pos.double()[:, None] * freqs
    c, s, out = torch.cos(a)[:, None], torch.sin(a)[:, None], x.clone()
    n = 2 * len(freqs)
    u, v = x[..., 0:n:2], x[..., 1:n:2]
    out[..., 0:n:2], out[..., 1:n:2] = u * c - v * s, v * c + u * s
    return out
