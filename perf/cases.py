"""The workloads this framework's speed is judged by: what a program that uses it does, through its public entry points.

`listed` names them, `draw` gives others of the same ranges, `prepare` makes what the program has in hand before the call, `run` is the
call, `work` is what it cannot do without, `exact` the same result in 64-bit arithmetic of plain torch, and `tolerance` how far two
correct implementations may be apart.

Models carry random weights. The norms of the Qwen3 ones are set so that the next token is a clear choice, as it is in a trained
model: norms of one leave 150 000 logits in which the largest two differ by less than 16-bit arithmetic resolves."""

import hashlib
import json
import math
import os
import pathlib
import struct
import tempfile
import weakref

import numpy as np
import torch

import brasa_b200 as B
from brasa_b200 import synth

KV = {"f16": B.KvType.F16, "q8_0": B.KvType.Q8_0, "f32": B.KvType.F32}
STD = 0.02  # of the weights
STACK = {"dunuzen": (synth.dunuzen_config, synth.dunuzen_shapes, ["latent_attention", "channel_delta"], synth.dunuzen_decode_bytes, synth.dunuzen_prefill_flops),
         "gugedra": (synth.gugedra_config, synth.gugedra_shapes, ["parallel", "delta"], synth.gugedra_decode_bytes, synth.gugedra_prefill_flops)}

QWEN_4B = dict(kind="qwen3", layers=36, hidden=2560, heads=32, kv_heads=8, ffn=9728, vocab=151936, tied=True)
# layers of the 32B architecture's shape, four of its 64 so that it loads quickly; tied, since a random head beside the table has no clear choice
QWEN_32B_4 = dict(kind="qwen3", layers=4, hidden=5120, heads=64, kv_heads=8, ffn=25600, vocab=151936, tied=True)
SMALL = dict(kind="qwen3", layers=3, hidden=512, heads=8, kv_heads=2, ffn=1536, vocab=1024, tied=True)
STACK_2560 = dict(width=2560, ff=9728, heads=32, kv_heads=16, window=1024, layers=8, vocab=32768)


def listed():
    return [
        # one product of the operator set with the gate / up matrix: what a caller of single operators pays
        dict(name="gemv-9728x2560", kind="gemv", rows=9728, cols=2560),
        # a short greedy answer of a small model: launches and host work are most of it
        dict(SMALL, name="small-chat-20", mode="chat", kv="f16", prompt=20, steps=12, chunk=32, temperature=0.0),
        # the headline workload: greedy tokens one at a time behind a 512-token prompt
        dict(QWEN_4B, name="4b-decode-512", mode="decode", kv="f16", prompt=512, steps=32, chunk=512),
        # the same over a long 8-bit cache
        dict(QWEN_4B, name="4b-decode-16k-q8", mode="decode", kv="q8_0", prompt=16384, steps=16, chunk=3584),
        # an ordinary prompt
        dict(QWEN_4B, name="4b-prefill-512", mode="prefill", kv="f16", prompt=512, chunk=512),
        # a document in runs of the default length, with a ragged end
        dict(QWEN_4B, name="4b-prefill-5000", mode="prefill", kv="f16", prompt=5000, chunk=1024),
        # the long-context workload: 16 384 tokens into an 8-bit cache
        dict(QWEN_4B, name="4b-prefill-16k-q8", mode="prefill", kv="q8_0", prompt=16384, chunk=3584),
        # a sampled chat turn behind a short odd prompt, through the session
        dict(QWEN_4B, name="4b-chat-37", mode="chat", kv="f16", prompt=37, steps=12, chunk=512, temperature=0.7),
        # agents: sequences behind one shared prompt, admitted and then decoded together with sampling
        dict(QWEN_4B, name="4b-serve-64", mode="serve", kv="f16", prefix=1024, prompt=100, steps=40, seqs=64, chunk=1024, temperature=0.7),
        # greedy tokens of a wide model whose feed-forward is beyond the one-kernel token
        dict(QWEN_32B_4, name="32b-layers-decode", mode="decode", kv="f16", prompt=300, steps=32, chunk=512),
        # layer-stack models: a prompt of several windows with a few tokens behind it, and a short prompt with a longer answer
        dict(STACK_2560, name="dunuzen-prefill-4096", kind="dunuzen", prompt=4096, steps=4, chunk=2048),
        dict(STACK_2560, name="gugedra-chat-300", kind="gugedra", prompt=300, steps=48, chunk=2048),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["gemv", "small", "decode", "prefill", "chat", "serve", "wide", "dunuzen", "gugedra"])
    if what == "gemv":
        return dict(kind="gemv", rows=32 * _log(rng, 16, 800), cols=256 * rng.randint(2, 38))
    if what in STACK:
        prompt = _log(rng, 16, 4096)
        return dict(STACK_2560, kind=what, prompt=prompt, steps=_log(rng, 2, 64), chunk=2048)
    if what == "small":
        kv_heads, group = rng.choice([1, 2, 4]), rng.choice([1, 2, 4, 8])
        model = dict(kind="qwen3", layers=rng.randint(2, 6), hidden=256 * rng.randint(2, 6), heads=kv_heads * group, kv_heads=kv_heads,
                     ffn=256 * rng.randint(3, 16), vocab=128 * rng.randint(8, 128), tied=True)
        kv, what = rng.choice(sorted(KV)), rng.choice(["decode", "prefill", "chat"])
    else:
        model, kv = (QWEN_32B_4 if what == "wide" else QWEN_4B), rng.choice(["f16", "f16", "q8_0"])
        what = "decode" if what == "wide" else what
    if what == "serve":
        return dict(model, mode="serve", kv=kv, prefix=16 * _log(rng, 4, 64), prompt=_log(rng, 9, 100), steps=_log(rng, 4, 40), seqs=_log(rng, 2, 64), chunk=1024,
                    temperature=rng.choice([0.0, 0.7]))
    if what == "prefill":
        return dict(model, mode="prefill", kv=kv, prompt=_log(rng, 9, 8192), chunk=rng.choice([512, 1024, 3584]))
    prompt = _log(rng, 16, 8192 if what == "decode" else 1024)
    case = dict(model, mode=what, kv=kv, prompt=prompt, steps=_log(rng, 4, 32), chunk=1024)
    return case if what == "decode" else dict(case, temperature=rng.choice([0.0, 0.7]))


# ---- models -------------------------------------------------------------------------------------------------------------


def _norms(c):
    """(layers' norm weight with which their sum is a few times the embedding, so that the input token stands out among the logits; final
    norm weight with which the others' standard deviation is 2)."""
    share = max(0.45, 16 / math.sqrt(c["hidden"]))
    goal = STD ** 2 * (1 / share ** 2 - 1)
    lo, hi = 0.0, 4.0
    for _ in range(40):
        w = (lo + hi) / 2
        g = STD * math.sqrt(c["hidden"]) * w
        ffn, attn = STD * math.sqrt(c["ffn"]) * g * g / 2, STD * math.sqrt(c["heads"] * 128) * g / 2
        lo, hi = (w, hi) if c["layers"] * (ffn ** 2 + attn ** 2) < goal else (lo, w)
    return lo, 2 / (STD * math.sqrt(c["hidden"]))


def _qwen_config(c):
    return dict(synth.QWEN3_4B, tie_word_embeddings=c["tied"], num_hidden_layers=c["layers"], hidden_size=c["hidden"], intermediate_size=c["ffn"],
                num_attention_heads=c["heads"], num_key_value_heads=c["kv_heads"], vocab_size=c["vocab"])


def _stack_config(c):
    make, shapes, kinds, _, _ = STACK[c["kind"]]
    size = {k: c[k] for k in ("width", "ff", "heads", "kv_heads", "vocab", "window")}
    cfg = make(layers=[kinds[i % 2] for i in range(c["layers"])], **size)
    return cfg, shapes(cfg)


def _model_file(c, ctx=None):
    """The model's file, written once on this machine."""
    keys = ("kind", "layers", "hidden", "heads", "kv_heads", "ffn", "vocab", "tied", "width", "ff", "window")
    tag = hashlib.sha256(json.dumps({k: c[k] for k in keys if k in c}, sort_keys=True).encode()).hexdigest()[:16]
    top = pathlib.Path(tempfile.gettempdir()) / f"brasa-perf-models-{os.getuid()}"
    path = top / (tag + (".brasa" if c["kind"] == "qwen3" else ""))
    if path.exists():
        return path
    top.mkdir(parents=True, exist_ok=True)
    tmp = top / f"{tag}.{os.getpid()}.tmp"
    if c["kind"] != "qwen3":
        cfg, shapes = _stack_config(c)
        synth.write_synthetic_stack(tmp, cfg, shapes, seed=1, std=STD)
    else:
        ctx = ctx or B.Context(0)
        meta = synth.write_synthetic_model(ctx, tmp, _qwen_config(c), seed=1, std=STD)
        with open(tmp, "r+b") as f:
            for t in meta["tensors"]:
                if t["name"].endswith("layernorm.weight") or t["name"] == "model.norm.weight":
                    data = np.full(t["shape"], _norms(c)[t["name"] == "model.norm.weight"], "<f4").tobytes()
                    t["sha256"] = hashlib.sha256(data).hexdigest()
                    f.seek(t["offset"])
                    f.write(data)
            meta["data_sha256"] = hashlib.sha256("".join(t["sha256"] for t in meta["tensors"]).encode()).hexdigest()
            js = json.dumps(meta, ensure_ascii=False, separators=(",", ":")).encode()
            f.seek(0)
            f.write(b"BRSA" + struct.pack("<IQ", 1, len(js)) + js)
    try:
        os.rename(tmp, path)
    except OSError:  # another process was first
        pass
    return path


class _Holder:
    """A context with a model or session on it, given back when the last state that uses it goes."""

    def __init__(self, c, positions):
        self.ctx = B.Context(0)
        path = _model_file(c, self.ctx)
        kv = KV[c["kv"]] if c["kind"] == "qwen3" else B.KvType.BF16
        limits = B.Limits(ctx=positions, max_tokens=c["chunk"], max_logit_rows=1, kv=kv)
        self.session = B.Session(self.ctx, path, limits) if c.get("mode") == "chat" else None
        self.model = self.session.model if self.session else B.model_class(path).load(self.ctx, path, limits)

    def __del__(self):
        if hasattr(self, "model") and B is not None:
            (self.session or self.model).free()
            self.ctx.close()


_shared = weakref.WeakValueDictionary()


def _holder(c, positions, own):
    """Prompts that start from nothing go through one loaded model, as in a program that serves them one after the other; `own`: a model for
    this state alone, since its cache is part of the state."""
    if own:
        return _Holder(c, positions)
    key = json.dumps(c, sort_keys=True)
    got = _shared.get(key)
    if got is None:
        got = _shared[key] = _Holder(c, positions)
    return got


class _OnDevice:
    """Device memory of a buffer as torch sees it."""

    def __init__(self, buf, shape):
        self.buf = buf
        self.__cuda_array_interface__ = {"data": (buf.ptr, False), "shape": tuple(shape), "typestr": "<f4", "version": 3, "strides": None}


def _ids(c, seed, n, stream=0):
    return np.random.default_rng([int(seed), stream]).integers(0, c["vocab"], size=n).astype(np.uint32)


def _feed(model, ids, chunk):
    logits = None
    for off in range(0, len(ids), chunk):
        logits, _ = model.forward(ids[off:off + chunk], off, want_logits=off + chunk >= len(ids))
    return logits


def _gemv_inputs(c, seed):
    g = torch.Generator("cuda").manual_seed(int(seed))
    w = torch.randn(c["rows"], c["cols"], device="cuda", generator=g) * STD
    return w, torch.randn(c["cols"], device="cuda", generator=g).half().float()


def prepare(case, seed):
    c = dict(case)
    c.pop("name", None)
    if c["kind"] == "gemv":
        w, x = _gemv_inputs(c, seed)
        ctx = B.Context(0)
        K, n = B.Kernels(ctx), w.numel()
        src, raw, tiled = ctx.buffer(4 * n), ctx.buffer(B.qtype_nbytes(B.WeightType.Q4_0, n)), ctx.buffer(B.qtype_nbytes(B.WeightType.Q4_0, n))
        xb, yb = ctx.buffer(4 * c["cols"]), ctx.buffer(4 * c["rows"])
        ctx.sync()
        torch.as_tensor(_OnDevice(src, w.shape), device="cuda").copy_(w)
        torch.as_tensor(_OnDevice(xb, x.shape), device="cuda").copy_(x)
        torch.cuda.synchronize()
        cmd = ctx.command()
        K.quantize(cmd, B.WeightType.Q4_0, src, raw, n)
        K.repack(cmd, B.WeightType.Q4_0, raw, tiled, c["rows"], c["cols"])
        cmd.wait()
        src.free()
        raw.free()
        return dict(case=c, ctx=ctx, K=K, w=B.QMatrix(tiled, B.WeightType.Q4_0, c["rows"], c["cols"], B.Layout.TILED), x=xb, y=yb,
                    out=torch.as_tensor(_OnDevice(yb, (c["rows"],)), device="cuda"))
    if c["kind"] != "qwen3":
        h = _holder(c, c["prompt"] + c["steps"], False)
        return dict(case=c, holder=h, ids=_ids(c, seed, c["prompt"]), fed=_ids(c, seed, c["steps"], 1))
    if c["mode"] == "serve":
        positions = -(-(c["prefix"] + c["prompt"] + c["steps"] + 1) // B.Batch.PAGE) * B.Batch.PAGE
        h = _holder(c, positions, False)
        return dict(case=c, holder=h, positions=positions, prefix=_ids(c, seed, c["prefix"]), own=[_ids(c, seed, c["prompt"], 1 + i) for i in range(c["seqs"])])
    positions, ids = c["prompt"] + c.get("steps", 0) + 2, _ids(c, seed, c["prompt"])
    h = _holder(c, positions, c["mode"] == "decode")
    state = dict(case=c, holder=h, ids=ids, seed=int(seed))
    if c["mode"] == "decode":
        state["first"] = int(np.argmax(_feed(h.model, ids, c["chunk"])))
    return state


def run(state):
    c = state["case"]
    if c["kind"] == "gemv":
        cmd = state["ctx"].command()
        state["K"].gemv(cmd, state["w"], state["x"], state["y"], 1)
        cmd.wait()
        return state["out"]
    h = state["holder"]
    if c["kind"] != "qwen3":
        out = [_feed(h.model, state["ids"], c["chunk"])]
        for i, t in enumerate(state["fed"]):
            out.append(h.model.forward([t], c["prompt"] + i)[0])
        return np.concatenate(out)
    if c["mode"] == "prefill":
        return _feed(h.model, state["ids"], c["chunk"])
    if c["mode"] == "decode":
        ids, _ = h.model.decode_greedy(state["first"], c["prompt"], c["steps"])
        return dict(ids=ids, logits=h.model.forward(ids[-1:], c["prompt"] + c["steps"])[0])
    params = B.SamplingParams(temperature=c["temperature"], top_k=0, top_p=0.95 if c["temperature"] else 1.0, seed=7)
    if c["mode"] == "chat":
        h.session.reset()
        ids, _ = h.session.generate(state["ids"], c["steps"], params)
        return dict(ids=ids, logits=h.model.forward(ids[-1:], c["prompt"] + len(ids) - 1)[0])
    page = B.Batch.PAGE
    pages = c["prefix"] // page + c["seqs"] * (state["positions"] // page - c["prefix"] // page)
    batch = B.Batch(h.model, c["seqs"], pages, state["positions"])
    try:
        batch.set_prefix(state["prefix"])
        for own in state["own"]:
            batch.add_sequence(own, params)
        ids, _ = batch.decode(c["steps"], params)
        return dict(ids=ids, logits=batch.peek_logits())
    finally:
        batch.free()


# ---- what a pass cannot do without --------------------------------------------------------------------------------------


def work(case):
    c = case
    if c["kind"] == "gemv":
        return dict(bytes=c["rows"] * c["cols"] // 32 * 18 + 4 * (c["rows"] + c["cols"]), flops=2 * c["rows"] * c["cols"])
    if c["kind"] != "qwen3":
        cfg, shapes = _stack_config(c)
        _, _, _, step_bytes, prompt_flops = STACK[c["kind"]]
        weights = 2 * sum(int(np.prod(s)) for n, s in shapes.items() if "embed" not in n)
        f = prompt_flops(cfg, c["prompt"])
        return dict(bytes=weights + sum(step_bytes(cfg, c["prompt"] + i) for i in range(c["steps"])),
                    flops=sum(f.values()) + weights * c["steps"])
    cfg = _qwen_config(c)
    weights, row = synth.weight_bytes_per_token(cfg), synth.kv_bytes_per_position(cfg, c["kv"])
    per_token = 2 * sum(int(np.prod(s)) for n, s in synth.tensor_shapes(cfg).items() if len(s) == 2 and "layers" in n)
    head, pair = 2 * c["vocab"] * c["hidden"], 4 * c["heads"] * 128 * c["layers"]

    def prompt(n, before=0):
        return n * per_token + head + pair * (n * before + n * (n + 1) // 2)

    n = c["prompt"]
    if c["mode"] == "prefill":
        return dict(bytes=weights * (n > 0) + row * n, flops=prompt(n))
    steps = c["steps"] + (c["mode"] == "decode")  # the logits behind the last token are one step more
    if c["mode"] == "serve":
        steps, s, p = c["steps"] + 1, c["seqs"], c["prefix"]
        kv = sum(row * (p + s * (n + i + 1)) for i in range(steps))
        flops = prompt(p) + s * prompt(n, p) + steps * s * (per_token + head) + sum(s * pair * (p + n + i + 1) for i in range(steps))
        return dict(bytes=weights * (1 + s + steps) + kv + s * row * (p + n), flops=flops)
    b, f = steps * weights + sum(row * (n + i + 1) for i in range(steps)), steps * (per_token + head) + sum(pair * (n + i + 1) for i in range(steps))
    if c["mode"] == "chat":
        b, f = b + weights + row * n, f + prompt(n)
    return dict(bytes=b, flops=f)


def tolerance(case):
    """About four times what the path is off its 64-bit value (f16 0.0008, 8-bit caches 0.004, bf16 stacks 0.005, one product 1e-7)."""
    if case["kind"] == "gemv":
        return dict(rel=1e-6)
    if case["kind"] != "qwen3":
        return dict(rel=2e-2, max=0.3)
    return dict(rel=1.6e-2, max=0.2) if case["kv"] == "q8_0" else dict(rel=3.5e-3, max=0.1)


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------


def _dequantize(raw, dtype, shape):
    """Blocks of 32 values with one scale, as float64 on the device."""
    size = {"q4_0": 18, "q6_0": 26}[dtype]
    b = torch.from_numpy(np.array(raw)).cuda().reshape(-1, size)
    d = b[:, :2].contiguous().view(torch.float16).double()
    lo = torch.cat([b[:, 2:18] & 15, b[:, 2:18] >> 4], 1)
    if dtype == "q4_0":
        return (d * (lo.double() - 8)).reshape(shape)
    hi = torch.cat([(b[:, 18:26] >> (2 * k)) & 3 for k in range(4)], 1)
    return (d * ((lo | (hi << 4)).double() - 32)).reshape(shape)


def _rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _rotate(x, dims, base, pos):
    """x [..., tokens, heads, n]: entry i of the first `dims` pairs with i + dims / 2."""
    half = dims // 2
    a = pos.double()[:, None] * base ** (-2.0 * torch.arange(half, device="cuda", dtype=torch.float64) / dims)
    cos, sin = a.cos()[:, None], a.sin()[:, None]
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * cos - v * sin, v * cos + u * sin, x[..., dims:]], -1)


class _Qwen64:
    """The Qwen3 forward over a `.brasa` file; the cache holds what a cache of type `kv` gives back."""

    def __init__(self, path, kv):
        raw = np.memmap(path, np.uint8, "r")
        n = struct.unpack("<Q", bytes(raw[8:16]))[0]
        meta = json.loads(bytes(raw[16:16 + n]))
        self.cfg, self.kv, self.cache, self.w = meta["model"]["config"], kv, {}, {}
        for t in meta["tensors"]:
            data = raw[t["offset"]:t["offset"] + t["nbytes"]]
            self.w[t["name"]] = torch.from_numpy(np.array(data).view("<f4")).cuda().double() if t["dtype"] == "f32" else _dequantize(data, t["dtype"], t["shape"])

    def stored(self, x):
        if self.kv == "f32":
            return x.float().double()
        if self.kv == "f16":
            return x.half().double()
        b = x.float().unflatten(-1, (-1, 32))
        d = (b.abs().amax(-1, keepdim=True) / 127).half().float()
        q = torch.where(d == 0, 0, (b / torch.where(d == 0, 1, d)).round().clamp(-127, 127))
        return (d.double() * q.double()).flatten(-2)

    def forward(self, ids, pos):
        """ids [sequences, tokens] from position pos; the logits of the last one of each."""
        c, w, eps = self.cfg, self.w, self.cfg["rms_norm_eps"]
        S, T = ids.shape
        hq, hk = c["num_attention_heads"], c["num_key_value_heads"]
        at = torch.arange(pos, pos + T, device="cuda")
        x = w["model.embed_tokens.weight"][ids.cuda()]
        for i in range(c["num_hidden_layers"]):
            def p(name):
                return w[f"model.layers.{i}.{name}.weight"]
            h = _rms(x, eps) * p("input_layernorm")
            q, k, v = ((h @ p(f"self_attn.{n}_proj").T).unflatten(-1, (-1, 128)) for n in "qkv")
            q = _rotate(_rms(q, eps) * p("self_attn.q_norm"), 128, c["rope_theta"], at)
            k = _rotate(_rms(k, eps) * p("self_attn.k_norm"), 128, c["rope_theta"], at)
            new = [self.stored(k), self.stored(v)]
            if pos:
                new = [torch.cat([old.expand(S, -1, -1, -1), n], 1) for old, n in zip(self.cache[i], new)]
            self.cache[i], o = new, torch.empty_like(q)
            hidden = torch.arange(pos + T, device="cuda")[None] > at[:, None]
            for g in range(hk):
                heads = slice(g * (hq // hk), (g + 1) * (hq // hk))
                s = torch.einsum("sthd,sld->shtl", q[:, :, heads], new[0][:, :, g]).mul_(128 ** -0.5).masked_fill_(hidden, -math.inf)
                o[:, :, heads] = torch.einsum("shtl,sld->sthd", torch.softmax(s, -1), new[1][:, :, g])
            x = x + o.flatten(-2) @ p("self_attn.o_proj").T
            h = _rms(x, eps) * p("post_attention_layernorm")
            x = x + (torch.nn.functional.silu(h @ p("mlp.gate_proj").T) * (h @ p("mlp.up_proj").T)) @ p("mlp.down_proj").T
        head = w["model.embed_tokens.weight" if c.get("tie_word_embeddings", True) else "lm_head.weight"]
        return (_rms(x[:, -1], eps) * w["model.norm.weight"]) @ head.T

    def feed(self, ids, pos=0, chunk=2048):
        for off in range(0, ids.shape[1], chunk):
            logits = self.forward(ids[:, off:off + chunk], pos + off)
        return logits


def _softplus(z):
    return torch.clamp(z, min=0) + torch.log1p(torch.exp(-z.abs()))


def _unit(x):
    return x * torch.rsqrt(x.square().sum(-1, keepdim=True) + 1e-6)


def _conv(x, w):
    taps = w.shape[1]
    x = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    return sum(x[i:i + len(x) - taps + 1] * w[:, i] for i in range(taps))


def _attend(q, k, v, window, scale, cap):
    """q [n, H, d], k [n, G, d], v [n, G, dv]: a query sees its own position and the window - 1 before it."""
    n, H, G = q.shape[0], q.shape[1], k.shape[1]
    d = torch.arange(n, device="cuda")[:, None] - torch.arange(n, device="cuda")[None]
    gone, out = (d < 0) | (d >= window), q.new_empty(n, H, v.shape[2])
    for h in range(H):
        s = q[:, h] @ k[:, h * G // H].T * scale
        s = cap * torch.tanh(s / cap) if cap else s
        out[:, h] = torch.softmax(s.masked_fill(gone, -math.inf), -1) @ v[:, h * G // H]
    return out


def _delta(q, k, v, g, beta):
    """The gated delta rule token by token: q, k, g [n, H, d], v [n, H, dv], beta [n, H]."""
    S, out = q.new_zeros(q.shape[1], q.shape[2], v.shape[2]), torch.empty_like(v)
    for t in range(len(q)):
        S = g[t][:, :, None] * S
        u = beta[t][:, None] * (v[t] - (k[t][:, None] @ S)[:, 0])
        S = torch.baddbmm(S, k[t][:, :, None], u[:, None])
        out[t] = (q[t][:, None] @ S)[:, 0]
    return out


def _delta_inputs(h, W, m):
    silu, rep = torch.nn.functional.silu, m["heads"] // m["kv_heads"]
    q, k, v = (silu(_conv(h @ W(n).T, W(n + ".conv"))) for n in "qkv")
    q, k = _unit(q.unflatten(-1, (-1, m["dim"]))) * m["dim"] ** -0.5, _unit(k.unflatten(-1, (-1, m["dim"])))
    return q.repeat_interleave(rep, 1), k.repeat_interleave(rep, 1), v.unflatten(-1, (-1, m["vdim"])), torch.sigmoid(h @ W("b").T)


def _dunuzen_mixer(kind, h, W, m, eps):
    pos = torch.arange(len(h), device="cuda")
    if kind == "latent_attention":
        H, d, kr, rot = m["heads"], m["dim"], m["kv_rank"], m["rot"]
        q, down = (h @ W("q").T).unflatten(-1, (H, -1)), h @ W("dkv").T
        c = _rms(down[:, :kr], eps) * W("dkv.norm")
        shared = _rotate(down[:, None, kr:], rot["dims"], rot["base"], pos).expand(-1, H, -1)
        k = torch.cat([(c @ W("uk").T).unflatten(-1, (H, d)), shared], -1)
        q = torch.cat([q[..., :d], _rotate(q[..., d:], rot["dims"], rot["base"], pos)], -1)
        o = _attend(q, k, (c @ W("uv").T).unflatten(-1, (H, -1)), m["mask"]["size"], m["scale"], None) * torch.sigmoid(h @ W("g").T)[..., None]
    else:
        q, k, v, beta = _delta_inputs(h, W, m)
        z = _softplus((h @ W("a1").T) @ W("a2").T + W("dt_bias")).unflatten(-1, (m["heads"], -1))
        o = _delta(q, k, v, torch.exp(-torch.exp(W("A_log"))[:, None] * z), beta)
        o = _rms(o, eps) * W("norm") * torch.sigmoid((h @ W("g1").T) @ W("g2").T).unflatten(-1, (m["heads"], -1))
    return o.flatten(1) @ W("o").T


def _gugedra_mixer(kind, h, W, m, eps):
    silu = torch.nn.functional.silu
    if kind == "delta":
        q, k, v, beta = _delta_inputs(h, W, m)
        g = torch.exp(-torch.exp(W("A_log")) * _softplus(h @ W("a").T + W("dt_bias")))
        o = _rms(_delta(q, k, v, g[..., None].expand_as(q), beta), eps) * W("norm") * silu((h @ W("g").T).unflatten(-1, (m["heads"], -1)))
        return o.flatten(1) @ W("o").T
    a, r, pos = m["left"], m["right"], torch.arange(len(h), device="cuda")
    q, k = (_rotate((h @ W(f"left.{n}").T).unflatten(-1, (-1, a["dim"])), a["rot"]["dims"], a["rot"]["base"], pos) for n in "qk")
    left = _attend(q, k, (h @ W("left.v").T).unflatten(-1, (-1, a["vdim"])), a["mask"]["size"], a["scale"], a["softcap"]).flatten(1) @ W("left.o").T
    H, N, G = r["heads"], r["state"], r["groups"]
    inner = H * r["vdim"]
    z, conv, dt = (h @ W("right.in").T).split([inner, inner + 2 * G * N, H], -1)
    x, b, c = silu(_conv(conv, W("right.conv")) + W("right.conv.b")).split([inner, G * N, G * N], -1)
    x, b, c = x.unflatten(-1, (H, -1)), b.unflatten(-1, (G, N)).repeat_interleave(H // G, 1), c.unflatten(-1, (G, N)).repeat_interleave(H // G, 1)
    dt = _softplus(dt + W("right.dt_bias"))
    decay, S, y = torch.exp(-torch.exp(W("right.A_log")) * dt), h.new_zeros(H, N, r["vdim"]), torch.empty_like(x)
    for t in range(len(h)):
        S = torch.baddbmm(decay[t][:, None, None] * S, b[t][:, :, None], (dt[t][:, None] * x[t])[:, None])
        y[t] = (c[t][:, None] @ S)[:, 0]
    y = (y + W("right.D")[:, None] * x).flatten(1) * silu(z)
    y = _rms(y.unflatten(-1, (r["norm_groups"], -1)), eps).flatten(1) * W("right.norm")
    return m["left_scale"] * left + m["right_scale"] * (y @ W("right.o").T)


def _stack64(c, ids, rows):
    path = _model_file(c)
    raw = np.memmap(path / "model.safetensors", np.uint8, "r")
    n = struct.unpack("<Q", bytes(raw[:8]))[0]
    where, cfg = json.loads(bytes(raw[8:8 + n])), json.loads((path / "config.json").read_text())

    def tensor(name):
        b, e = where[name]["data_offsets"]
        return torch.from_numpy(np.array(raw[8 + n + b:8 + n + e])).cuda().view(torch.bfloat16).double().reshape(where[name]["shape"])

    eps, F = cfg["norm"]["eps"], torch.nn.functional
    ids = torch.from_numpy(ids.astype(np.int64)).cuda()
    x = tensor("embed")[ids]
    dunuzen = c["kind"] == "dunuzen"
    x = x * cfg["embedding"]["scale"] if dunuzen else x
    side = None if dunuzen else tensor("side.embed")[ids].unflatten(-1, (len(cfg["layers"]), -1))

    def layer_norm(x, name):
        d = x - x.mean(-1, keepdim=True)
        return _rms(d, eps) * tensor(name) + tensor(name + ".b")

    def norm(x, name):
        return _rms(x, eps) * tensor(name)

    for i, layer in enumerate(cfg["layers"]):
        def W(name):
            return tensor(f"l{i}.{name}")

        def mix(name):
            return W("mix." + name)
        p = f"l{i}."
        if dunuzen:
            up = layer_norm(x, p + "norm2") @ W("mlp.up").T + W("mlp.up.b")
            x = x + _dunuzen_mixer(layer["type"], layer_norm(x, p + "norm1"), mix, layer["mixer"], eps) + up.clamp(min=0).square() @ W("mlp.down").T + W("mlp.down.b")
        else:
            x = x + norm(_gugedra_mixer(layer["type"], norm(x, p + "norm1"), mix, layer["mixer"], eps), p + "norm1b")
            h = norm(x, p + "norm2")
            x = x + norm((F.silu(h @ W("mlp.gate").T) * (h @ W("mlp.up").T)) @ W("mlp.down").T, p + "norm2b")
            x = x + norm((F.gelu(x @ W("side.gate").T, approximate="tanh") * side[:, i]) @ W("side.proj").T, p + "side.norm")
    if dunuzen:
        return layer_norm(x[rows], "final.norm") @ tensor("head").T * cfg["logit_scale"]
    return cfg["logit_softcap"] * torch.tanh(norm(x[rows], "final.norm") @ tensor("head").T / cfg["logit_softcap"])


def exact(case, seed):
    c = dict(case)
    c.pop("name", None)
    if c["kind"] == "gemv":
        w, x = _gemv_inputs(c, seed)
        b = w.reshape(-1, 32)
        d = (b.gather(1, b.abs().argmax(1, keepdim=True)) / -8).half().float()
        q = torch.where(d == 0, 8, ((b / torch.where(d == 0, 1, d)).round() + 8).clamp(0, 15))
        return (d.double() * (q.double() - 8)).reshape(w.shape) @ x.double()
    if c["kind"] != "qwen3":
        ids = np.concatenate([_ids(c, seed, c["prompt"]), _ids(c, seed, c["steps"], 1)])
        return _stack64(c, ids, slice(c["prompt"] - 1, None))
    model = _Qwen64(_model_file(c), c["kv"])

    def tokens(rows):
        return torch.from_numpy(np.stack(rows).astype(np.int64))

    if c["mode"] == "serve":
        model.feed(tokens([_ids(c, seed, c["prefix"])]))
        logits, at = model.feed(tokens([_ids(c, seed, c["prompt"], 1 + i) for i in range(c["seqs"])]), c["prefix"]), c["prefix"] + c["prompt"]
    else:
        logits, at = model.feed(tokens([_ids(c, seed, c["prompt"])])), c["prompt"]
    if c["mode"] == "prefill":
        return logits
    # drawn tokens are the likeliest ones: nothing else is left inside the nucleus of a clear choice
    for i in range(c["steps"] + (c["mode"] != "chat")):
        logits = model.forward(logits.argmax(-1, keepdim=True).cpu(), at + i)
    return dict(ids=None, logits=logits)
