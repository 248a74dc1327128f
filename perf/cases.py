"""What the speed of this package is measured on: calls that a program makes on a loaded model, from one token of a toy model to a
batch of 64 sequences and a prompt of a thousand tokens.

A case is a model, what is asked of it and how much. A process loads a model once and keeps it, as a server does (the checkpoint
belongs to the case); the seed makes the requests: prompts, forced tokens, contexts. Each state has KV slots of its own.

  decode   one step for `batch` sequences over contexts of ragged length, logits to the host (the caller samples there)
  greedy   `steps` tokens chosen on the device, one after the other; `penalty` above 1 is the reference's repetition penalty
  prompt   ingestion of one prompt, logits of its last token
  prompts  ingestion of `batch` ragged prompts in one call, logits of each last token
  session  a block model: ragged prompts from position 0 in one call, then `steps` steps with given tokens, logits of each
"""
import json
import math
import os
import shutil
import struct
import tempfile

import numpy as np
import torch

import __graft_entry__

pkg = __graft_entry__.load_package()

# Weights of every packed model are cut from one run of quantised N(0, 0.02) values per block type. The number of its
# 256-element blocks is a prime above every vocabulary, so that no two rows of a matrix are alike.
POOL_BLOCKS = 131071
# model -> (shape, scheme, most sequences of a call, positions a slot holds)
PACKED = {
    "tiny-q4km": ("tiny", 1, 64, 128),
    "tinyllama-q8": ("tinyllama-1.1b", 0, 64, 2048),
    "tinyllama-q4km": ("tinyllama-1.1b", 1, 64, 2048),
    "llama2-7b-q4km": ("llama2-7b", 1, 32, 1280),
    "llama3-8b-q6k": ("llama3-8b", 2, 64, 1280),
}
STATES = 4  # states alive at once
F32_MOST = 16  # most sequences over a 32-bit cache of the larger models
KV = {"f32": pkg.KV_F32, "i8": pkg.KV_I8}


def listed():
    return [
        # the smallest call there is: a step of a toy model; launches and latency
        {"name": "tiny-step", "model": "tiny-q4km", "kv": "f32", "do": "decode", "batch": 1, "context": 16},
        # a chat on a small model, everything on the device: plain greedy, and with the reference's default penalty for two users
        {"name": "1b-q8-greedy", "model": "tinyllama-q8", "kv": "f32", "do": "greedy", "batch": 1, "context": 128, "steps": 24, "penalty": 1.0},
        {"name": "1b-q4-penalty-2", "model": "tinyllama-q4km", "kv": "f32", "do": "greedy", "batch": 2, "context": 77, "steps": 16, "penalty": 1.3},
        # a long document, then several short questions at once, on a small model
        {"name": "1b-q4-prompts-7", "model": "tinyllama-q4km", "kv": "i8", "do": "prompts", "batch": 7, "context": 311},
        # the benchmark's model: one user sampling on the host after a thousand tokens, a few users, a full server
        {"name": "7b-q4-step-1", "model": "llama2-7b-q4km", "kv": "i8", "do": "decode", "batch": 1, "context": 1030},
        {"name": "7b-q4-step-5", "model": "llama2-7b-q4km", "kv": "i8", "do": "decode", "batch": 5, "context": 600},
        {"name": "7b-q4-step-16", "model": "llama2-7b-q4km", "kv": "i8", "do": "decode", "batch": 16, "context": 600},
        # a document for it
        {"name": "7b-q4-prompt-1024", "model": "llama2-7b-q4km", "kv": "i8", "do": "prompt", "batch": 1, "context": 1024},
        # grouped-query model with a large vocabulary: a full batch, and a question over the reference's default cache
        {"name": "8b-q6-step-64", "model": "llama3-8b-q6k", "kv": "i8", "do": "decode", "batch": 64, "context": 400},
        {"name": "8b-q6-prompt-37", "model": "llama3-8b-q6k", "kv": "f32", "do": "prompt", "batch": 1, "context": 37},
        # block models: prompts of three users and some tokens for each
        {"name": "nezolix-session-3", "model": "nezolix-w2048", "dtype": "bfloat16", "do": "session", "batch": 3, "context": 333, "steps": 8},
        {"name": "pizilix-session-8", "model": "pizilix-w2048", "dtype": "bfloat16", "do": "session", "batch": 8, "context": 200, "steps": 8},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    do = rng.choice(("decode", "decode", "decode", "greedy", "prompt", "prompts", "session"))
    if do == "session":
        dtype = "bfloat16" if rng.random() < 0.8 else "float32"
        batch = _log(rng, 1, 16)
        return {"model": rng.choice(("nezolix-w2048", "pizilix-w2048")), "dtype": dtype, "do": do, "batch": batch,
                "context": _log(rng, 2, 1200 // batch) if dtype == "bfloat16" else _log(rng, 2, max(3, 64 // batch)), "steps": rng.randint(1, 10)}
    if do == "greedy":
        model = rng.choice(("tiny-q4km", "tinyllama-q8", "tinyllama-q4km"))
        batch = _log(rng, 1, 8)
        return {"model": model, "kv": "f32", "do": do, "batch": batch, "context": _log(rng, 4, 90 if model == "tiny-q4km" else 200),
                "steps": rng.randint(2, max(3, 32 // batch)), "penalty": rng.choice((1.0, 1.1, 1.3))}
    model = rng.choice(("tiny-q4km", "tinyllama-q8", "tinyllama-q4km", "llama2-7b-q4km", "llama3-8b-q6k"))
    _, _, most, positions = PACKED[model]
    if model == "llama2-7b-q4km":  # a megabyte a position in 32 bits
        kv = "i8" if do == "decode" else rng.choice(("f32", "i8"))
    else:
        kv = rng.choice(("f32", "i8"))
    if kv == "f32" and not model.startswith("tiny"):
        most = F32_MOST
    if do == "decode":
        batch = _log(rng, 1, most)
        return {"model": model, "kv": kv, "do": do, "batch": batch, "context": _log(rng, 16, min(positions - 2, 16000 // batch))}
    if do == "prompt":
        return {"model": model, "kv": kv, "do": do, "batch": 1, "context": _log(rng, 16, min(positions - 2, 1024))}
    batch = rng.randint(2, 4 if model == "llama2-7b-q4km" else 12)
    return {"model": model, "kv": kv, "do": do, "batch": batch, "context": _log(rng, 8, min(positions - 2, 1024 // batch))}


# ---- inputs ------------------------------------------------------------------------------------------------------
def lengths(case):
    """Prompt or context length of each sequence: the first has `context` tokens, the others less, down to half of it."""
    n, b = case["context"], case["batch"]
    return [max(1, n - int(n // 2 * (0.618034 * i % 1))) for i in range(b)]


def vocab_of(case):
    m = case["model"]
    return pkg.synth.SHAPES[PACKED[m][0]]["vocab"] if m in PACKED else pkg.synth.BLOCK_SHAPES[m]["vocab"]


def requests(case, seed):
    """(prompt of each sequence, [steps][batch] tokens given after it)."""
    rng = np.random.default_rng([seed, 17])
    v = vocab_of(case)
    return [rng.integers(0, v, n).astype(np.int32) for n in lengths(case)], rng.integers(0, v, (max(1, case.get("steps", 1)), case["batch"])).astype(np.int32)


_pools = {}


def pool(kind, blocks):
    """At least `blocks` 256-element blocks of packed (or, kind 0, plain) N(0, 0.02) values."""
    if kind not in _pools:
        base = pkg.synth.fill_normal(POOL_BLOCKS * 256, 4321, stream=kind + 1)
        _pools[kind] = (pkg.synth.quantize(kind, base) if kind else base.view(np.uint8)).reshape(POOL_BLOCKS, -1)
    times = -(-blocks // POOL_BLOCKS)
    if len(_pools[kind]) < times * POOL_BLOCKS:
        _pools[kind] = np.concatenate([_pools[kind][:POOL_BLOCKS]] * times)
    return _pools[kind]


def tensors(model):
    """(name, type, rows, columns, first block in the pool) of every tensor of a packed model; norm vectors have type None."""
    shape, scheme, _, _ = PACKED[model]
    s = pkg.synth.SHAPES[shape]
    H, F, L, V = s["hidden"], s["ffn"], s["n_layers"], s["vocab"]
    kvd = H // s["n_heads"] * s["n_kv_heads"]
    main, alt = {0: (8, 8), 1: (12, 14), 2: (14, 14)}[scheme]
    out = [("token_embd.weight", 0, V, H)]
    for i in range(L):
        p = "blk.%d." % i
        out += [(p + "attn_norm.weight", None, 1, H), (p + "attn_q.weight", main, H, H), (p + "attn_k.weight", main, kvd, H), (p + "attn_v.weight", alt, kvd, H),
                (p + "attn_output.weight", main, H, H), (p + "ffn_norm.weight", None, 1, H), (p + "ffn_gate.weight", main, F, H), (p + "ffn_up.weight", main, F, H),
                (p + "ffn_down.weight", alt, H, F)]
    out += [("output_norm.weight", None, 1, H), ("output.weight", alt, V, H)]
    return [t + (11 + 7919 * i % POOL_BLOCKS,) for i, t in enumerate(out)]


def blocks_of(kind, rows, cols, first):
    n = rows * cols // 256
    return pool(kind, first + n)[first:first + n]


def norm_of(cols, first):
    return 1 + 0.1 * np.random.default_rng(first).standard_normal(cols).astype(np.float32)


class Model:
    """A loaded model and its free KV slots."""

    def __init__(self, case):
        name = case["model"]
        if name in PACKED:
            shape, scheme, most, positions = PACKED[name]
            if case["kv"] == "f32" and not name.startswith("tiny"):
                most = 4 if name == "llama2-7b-q4km" else F32_MOST
            self.engine = pkg.Engine.create(pkg.synth.SHAPES[shape], kv_dtype=KV[case["kv"]], max_seqs=STATES * most, max_ctx=positions)
            for t, kind, rows, cols, first in tensors(name):
                if kind is None:
                    self.engine.upload_tensor(t, 0, norm_of(cols, first), rows, cols)
                else:
                    self.engine.upload_tensor(t, kind, blocks_of(kind, rows, cols, first), rows, cols)
            self.engine.finalize()
        else:
            with block_folder(name) as folder:
                self.engine = pkg.Engine.from_model(folder, dtype=case["dtype"], max_seqs=STATES * 16, max_ctx=2048)
        self.free = list(range(self.engine.desc.max_seqs))

    def take(self, n):
        if len(self.free) < n:
            raise MemoryError("all KV slots are in use")
        got, self.free = self.free[:n], self.free[n:]
        return got


class block_folder:
    """A folder with config.json and model.safetensors of a block model, as long as the block lasts."""

    def __init__(self, shape):
        self.shape = shape

    def __enter__(self):
        self.path = tempfile.mkdtemp(dir="/dev/shm" if os.access("/dev/shm", os.W_OK) else None)
        return pkg.synth.write_block_model(self.path, self.shape)

    def __exit__(self, *_):
        shutil.rmtree(self.path, ignore_errors=True)


_loaded = {}


def model_of(case):
    key = (case["model"], case.get("kv"), case.get("dtype"))
    if key not in _loaded:
        for m in _loaded.values():  # one model at a time
            m.engine.close()
        _loaded.clear()
        _loaded[key] = Model(case)
    return _loaded[key]


class State:
    def __init__(self, case, seed):
        self.case, self.model = case, model_of(case)
        self.slots = self.model.take(case["batch"])
        self.prompts, self.given = requests(case, seed)
        self.lens = [len(p) for p in self.prompts]

    def __del__(self):
        try:
            self.model.free += self.slots
        except AttributeError:
            pass


def prepare(case, seed):
    s = State(case, seed)
    e = s.model.engine
    if case["do"] == "decode":  # contexts as ingestion leaves them
        e.prefill_batch(s.prompts, slots=s.slots, want_logits=False)
    elif case["do"] == "greedy":  # contexts as the decode path leaves them: the chosen ids don't hang on the prompt path's rounding
        for slot, p in zip(s.slots, s.prompts):
            for at in range(0, len(p), 15):
                e.prefill(p[at:at + 15], slot=slot, start_pos=at, want_logits=False)
    return s


def run(s):
    c, e = s.case, s.model.engine
    if c["do"] == "decode":
        return e.decode(s.given[0], s.lens, slots=s.slots, want_argmax=False)[0]
    if c["do"] == "greedy":
        if c["penalty"] > 1:
            ids, _ = e.generate_greedy_penalized(s.given[0], s.lens, c["steps"], c["penalty"], [[t] for t in s.given[0]], slots=s.slots)
        else:
            ids, _ = e.generate_greedy(s.given[0], s.lens, c["steps"], slots=s.slots)
        return ids, e.decode(ids[-1], [n + c["steps"] for n in s.lens], slots=s.slots, want_argmax=False)[0]
    if c["do"] == "prompt":
        return e.prefill(s.prompts[0], slot=s.slots[0])
    out = e.prefill_batch(s.prompts, slots=s.slots)
    if c["do"] == "prompts":
        return out
    return [out] + [e.decode(t, [n + i for n in s.lens], slots=s.slots, want_argmax=False)[0] for i, t in enumerate(s.given)]


# ---- what a pass cannot do without ---------------------------------------------------------------------------------
def work(case):
    lens, B, m = lengths(case), case["batch"], case["model"]
    passes = {"decode": 1, "greedy": case.get("steps", 0) + 1, "prompt": 0, "prompts": 0, "session": case.get("steps", 0)}[case["do"]]
    ingest = 0 if case["do"] in ("decode", "greedy") else 1
    V = vocab_of(case)
    if m in PACKED:
        s = pkg.synth.SHAPES[PACKED[m][0]]
        H, L = s["hidden"], s["n_layers"]
        kvd = H // s["n_heads"] * s["n_kv_heads"]
        size = {0: 4.0, 8: 34 / 32, 12: 144 / 256, 14: 210 / 256, None: 4.0}
        all_t = [t for t in tensors(m) if t[0] != "token_embd.weight"]
        weights = sum(r * c * size[k] for _, k, r, c, _ in all_t)
        head = V * H
        params = sum(r * c for _, k, r, c, _ in all_t if k is not None) - head
        row = L * 2 * kvd * (4 if case["kv"] == "f32" else 1) + (L * 2 * s["n_kv_heads"] * 4 if case["kv"] == "i8" else 0)
        seen = lambda n: (n, L * 4 * H * n)  # noqa: E731  (cache rows read, flops) of a token with n rows in sight
    else:
        cfg = pkg.synth.block_config(m)
        shapes = dict(pkg.synth.block_tensors(cfg, pkg.synth.BLOCK_SHAPES[m].get("decay_rank", 0)))
        H = cfg["width"]
        head = V * H
        params = sum(int(np.prod(v)) for k, v in shapes.items() if len(v) == 2 and k not in ("embed", "head"))
        weights = 2.0 * (params + head)
        el = 2 if case["dtype"] == "bfloat16" else 4
        row, per_key = 0, 0
        for l in cfg["layers"]:
            x = l["mixer"]
            if l["type"] == "latent_attention":
                row += (x["kv_rank"] + x["rot_dim"]) * el
                per_key += 2 * x["heads"] * (x["dim"] + x["rot_dim"] + x["vdim"])
            elif l["type"] == "attention":
                row += x["kv_heads"] * (x["dim"] + x["rot"]["dims"]) * el
                per_key += 4 * x["heads"] * x["dim"]
        seen = lambda n: (n, per_key * n)  # noqa: E731
    nbytes, flops = 0.0, 0.0
    if ingest:
        nbytes += weights + sum(lens) * (4 * H + row) + B * V * 4
        flops += 2.0 * params * sum(lens) + 2.0 * head * B + sum(seen(n)[1] * (n + 1) / 2 for n in lens)
    for i in range(passes):
        nbytes += weights + B * (4 * H + row) + sum(seen(n + i)[0] for n in lens) * row + (B * V * 4 if i == passes - 1 or case["do"] != "greedy" else B * 4)
        flops += 2.0 * (params + head) * B + sum(seen(n + i + 1)[1] for n in lens)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["do"] == "greedy":  # 24-bit activations against 32-bit sums
        return {"rel": 2e-4, "max": 2e-3, "differ": 0.0}
    if case.get("dtype") == "float32":
        return {"rel": 2e-4, "max": 2e-3}
    # Operands of the matrix products in 16 bits. An int8 cache's rounding follows them: every code next to a border moves by a
    # whole step, which measures 3 % of the logits in the 32-layer models, 1 % in the 22-layer one.
    return {"rel": 3e-2 if case.get("kv") == "i8" else 2e-2, "max": 0.3}


# ---- the same in 64 bits, in plain torch ----------------------------------------------------------------------------
def _half(b):
    return b.contiguous().view(torch.float16).double()


def unpack(kind, b):
    """Values of packed blocks (uint8 [blocks of 256][bytes])."""
    n = len(b)
    if kind == 8:
        b = b.reshape(n * 8, 34)
        return (_half(b[:, :2]).abs() * b[:, 2:].view(torch.int8).double()).reshape(n, 256)
    if kind == 12:
        d, dm = _half(b[:, 0:2]), _half(b[:, 2:4])
        lo, mid, hi = b[:, 4:8], b[:, 8:12], b[:, 12:16]
        sc = torch.cat([lo & 63, (hi & 15) | ((lo >> 6) << 4)], 1).double()
        mn = torch.cat([mid & 63, (hi >> 4) | ((mid >> 6) << 4)], 1).double()
        q = b[:, 16:].reshape(n, 4, 1, 32)
        q = torch.cat([q & 15, q >> 4], 2).reshape(n, 8, 32).double()
        return ((d * sc)[:, :, None] * q - (dm * mn)[:, :, None]).reshape(n, 256)
    ql, qh = b[:, :128].reshape(n, 2, 2, 32), b[:, 128:192].reshape(n, 2, 1, 32)
    low = torch.stack([ql & 15, ql >> 4], 2)  # [block][half][nibble][32-element run][32]
    high = torch.stack([qh >> 0, qh >> 2, qh >> 4, qh >> 6], 2).reshape(n, 2, 2, 2, 32) & 3
    q = (low | (high << 4)).double() - 32
    sc = b[:, 192:208].view(torch.int8).double().reshape(n, 2, 2, 2, 2, 1)
    return (_half(b[:, 208:210])[:, :, None, None, None, None] * sc * q.reshape(n, 2, 2, 2, 2, 16)).reshape(n, 256)


class Packed64:
    """A packed model's forward pass over several sequences, with their keys and values."""

    def __init__(self, case, keep):
        self.s = pkg.synth.SHAPES[PACKED[case["model"]][0]]
        self.i8, self.keep, self.made = case["kv"] == "i8", keep, {}
        self.t = {t[0]: t[1:] for t in tensors(case["model"])}
        self.kv = {}

    def w(self, name):
        if name in self.made:
            return self.made[name]
        kind, rows, cols, first = self.t[name]
        if kind is None:
            v = torch.from_numpy(norm_of(cols, first)).cuda().double()
        else:
            v = torch.empty(rows * cols // 256, 256, dtype=torch.float64, device="cuda")
            raw = blocks_of(kind, rows, cols, first)
            for at in range(0, len(v), 1 << 17):
                v[at:at + (1 << 17)] = unpack(kind, torch.from_numpy(raw[at:at + (1 << 17)]).cuda())
            v = v.reshape(rows, cols)
        if self.keep:
            self.made[name] = v
        return v

    def rows(self, x):
        """Cached rows [tokens][heads][dim] as the cache holds them."""
        if not self.i8:
            return x
        a = x.abs().amax(-1, keepdim=True)
        s = torch.where(a > 1e-8, a / 127, torch.ones_like(a))
        return (x / s).round().clamp(-127, 127) * s

    def norm(self, x, name):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-5) * self.w(name)

    def run(self, tokens, starts):
        """The next tokens of each sequence; logits of the last one of each."""
        s, lens = self.s, [len(t) for t in tokens]
        nq, nkv, hd = s["n_heads"], s["n_kv_heads"], s["hidden"] // s["n_heads"]
        ids = np.concatenate(tokens).astype(np.int64)
        _, _, cols, first = self.t["token_embd.weight"]
        at = first + ids[:, None] * (cols // 256) + np.arange(cols // 256)[None]
        x = torch.from_numpy(pool(0, int(at.max()) + 1)[at].view(np.float32).reshape(len(ids), cols)).cuda().double()
        pos = torch.cat([torch.arange(a, a + n, device="cuda") for a, n in zip(starts, lens)]).double()
        ang = pos[:, None] * s["theta"] ** (-2.0 * torch.arange(hd // 2, device="cuda").double() / hd)[None]
        c, sn = ang.cos()[:, None], ang.sin()[:, None]

        def turn(v):
            a, b = v[..., 0::2], v[..., 1::2]
            return torch.stack([a * c - b * sn, a * sn + b * c], -1).flatten(-2)

        for i in range(s["n_layers"]):
            p = "blk.%d." % i
            h = self.norm(x, p + "attn_norm.weight")
            q = turn((h @ self.w(p + "attn_q.weight").T).reshape(-1, nq, hd))
            k = self.rows(turn((h @ self.w(p + "attn_k.weight").T).reshape(-1, nkv, hd)))
            v = self.rows((h @ self.w(p + "attn_v.weight").T).reshape(-1, nkv, hd))
            o, at = torch.empty_like(q), 0
            for b, n in enumerate(lens):
                r = slice(at, at + n)
                kk, vv = (torch.cat([old, new[r]]) for old, new in zip(self.kv.get((i, b), (k[:0], v[:0])), (k, v)))
                if self.keep:
                    self.kv[i, b] = (kk, vv)
                g = q[r].reshape(n, nkv, nq // nkv, hd)
                a = torch.einsum("tghd,ngd->ghtn", g, kk) / math.sqrt(hd)
                late = torch.arange(len(kk), device="cuda")[None] > (len(kk) - n + torch.arange(n, device="cuda"))[:, None]
                a = a.masked_fill(late, -math.inf).softmax(-1)
                o[r] = torch.einsum("ghtn,ngd->tghd", a, vv).reshape(n, nq, hd)
                at += n
            x = x + o.reshape(len(ids), -1) @ self.w(p + "attn_output.weight").T
            h = self.norm(x, p + "ffn_norm.weight")
            x = x + (torch.nn.functional.silu(h @ self.w(p + "ffn_gate.weight").T) * (h @ self.w(p + "ffn_up.weight").T)) @ self.w(p + "ffn_down.weight").T
        last = x[torch.tensor(lens, device="cuda").cumsum(0) - 1]
        return self.norm(last, "output_norm.weight") @ self.w("output.weight").T


def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rotate(x, rot):
    """Rotation of x [tokens][...][n] at positions 0, 1, ...: adjacent pairs of the first rot.dims dimensions."""
    dims, base = rot["dims"], rot["base"]
    i = torch.arange(dims // 2, device="cuda").double()
    f, m = base ** (-2.0 * i / dims), 1.0
    s = rot.get("scaling")
    if s:
        where = lambda turns: dims * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
        lo, hi = max(math.floor(where(s["fast"])), 0), min(math.ceil(where(s["slow"])), dims - 1)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        f, m = f / s["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(s["factor"]) + 1.0
    a = (torch.arange(len(x), device="cuda").double()[:, None] * f).reshape((len(x),) + (1,) * (x.ndim - 2) + (len(f),))
    c, sn = a.cos() * m, a.sin() * m
    u, v = x[..., 0:dims:2], x[..., 1:dims:2]
    return torch.cat([torch.stack([u * c - v * sn, v * c + u * sn], -1).flatten(-2), x[..., dims:]], -1)


def _latent(h, W, m, eps):
    T, H, D, R = len(h), m["heads"], m["dim"], m["rot_dim"]
    q = (_rms(h @ W("dq").T, W("dq.norm"), eps) @ W("uq").T).reshape(T, H, D + R)
    low = h @ W("dkv").T
    c, kr = _rms(low[:, :m["kv_rank"]], W("dkv.norm"), eps), _rotate(low[:, m["kv_rank"]:], m["rot"])
    k, v = (c @ W("uk").T).reshape(T, H, D), (c @ W("uv").T).reshape(T, H, m["vdim"])
    s = (torch.einsum("thd,nhd->htn", q[..., :D], k) + torch.einsum("thr,nr->htn", _rotate(q[..., D:], m["rot"]), kr)) * m["scale"]
    t = torch.arange(T, device="cuda")
    s = s.masked_fill((t[None] > t[:, None]) | (t[None] <= t[:, None] - m["mask"]["size"]), -math.inf).softmax(-1)
    o = torch.einsum("htn,nhv->thv", s, v).reshape(T, -1)
    return (o * torch.sigmoid(h @ W("g").T)) @ W("o").T


def _wkv(h, W, m, eps):
    T, H, D = len(h), m["heads"], m["dim"]
    prev = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
    mix = {s: h + (prev - h) * W("mu." + s) for s in "rkvgw"}
    r, k, v = ((mix[s] @ W(s).T).reshape(T, H, D) for s in "rkv")
    w = torch.exp(-torch.exp(torch.tanh(mix["w"] @ W("w1").T) @ W("w2").T + W("w0"))).reshape(T, H, D)
    S, o = torch.zeros(H, D, D, dtype=torch.float64, device="cuda"), []
    for t in range(T):
        kv = k[t][:, :, None] * v[t][:, None, :]
        o.append(torch.einsum("hk,hkv->hv", r[t], S + W("u")[:, :, None] * kv))
        S = w[t][:, :, None] * S + kv
    o = torch.stack(o)
    o = (o * torch.rsqrt(o.square().mean(-1, keepdim=True) + eps)).reshape(T, -1) * W("norm")
    return (o * torch.nn.functional.silu(mix["g"] @ W("g").T)) @ W("o").T


def _shared_kv(h, W, m):
    T, H, G, D = len(h), m["heads"], m["kv_heads"], m["dim"]
    q = _rotate((h @ W("q").T).reshape(T, H, D), m["rot"]).reshape(T, G, H // G, D)
    v = (h @ W("k").T).reshape(T, G, D)
    s = torch.einsum("tgxd,ngd->gxtn", q, _rotate(v, m["rot"])) * m["scale"]
    s = m["softcap"] * torch.tanh(s / m["softcap"])
    t = torch.arange(T, device="cuda")
    s = s.masked_fill((t[None] > t[:, None]) | (t[None] < (t // m["mask"]["size"] * m["mask"]["size"])[:, None]), -math.inf)
    s = torch.cat([s, torch.zeros_like(s[..., :1])], -1).softmax(-1)[..., :-1]  # the sink: one more score of zero
    return torch.einsum("gxtn,ngd->tgxd", s, v).reshape(T, -1) @ W("o").T


def _rglru(h, W, m):
    T, N, B = len(h), m["width"], m["blocks"]
    y = torch.nn.functional.gelu(h @ W("y").T + W("y.b"), approximate="tanh")
    x, w = h @ W("x").T + W("x.b"), W("conv")
    x = torch.cat([torch.zeros(m["conv"] - 1, N, dtype=torch.float64, device="cuda"), x])
    u = sum(x[k:k + T] * w[:, k] for k in range(m["conv"])) + W("conv.b")
    ub = u.reshape(T, B, N // B)
    r, i = (torch.sigmoid(torch.einsum("boi,tbi->tbo", W(n), ub) + W(n + ".b")).reshape(T, N) for n in ("ra", "ri"))
    la = -8.0 * r * torch.nn.functional.softplus(W("lam"), threshold=100.0)
    a, x = la.exp(), torch.sqrt(-torch.expm1(2 * la)) * i * u
    S, o = torch.zeros(N, dtype=torch.float64, device="cuda"), []
    for t in range(T):
        S = a[t] * S + x[t]
        o.append(S)
    return (torch.stack(o) * y) @ W("o").T


class Block64:
    def __init__(self, case):
        with block_folder(case["model"]) as folder:
            self.cfg = json.load(open(os.path.join(folder, "config.json")))
            raw = np.fromfile(os.path.join(folder, "model.safetensors"), np.uint8)
        n = struct.unpack("<Q", raw[:8].tobytes())[0]
        self.t = {}
        for name, t in json.loads(raw[8:8 + n].tobytes()).items():
            lo, hi = (8 + n + v for v in t["data_offsets"])
            self.t[name] = torch.from_numpy(raw[lo:hi].copy()).cuda().view(torch.bfloat16).double().reshape(t["shape"])

    def run(self, tokens):
        """Logits of every token of one sequence from its start."""
        cfg, t, eps = self.cfg, self.t, self.cfg["norm"]["eps"]
        piz = cfg["architecture"] == "Pizilix"
        x = t["embed"][torch.from_numpy(tokens.astype(np.int64)).cuda()] * (1.0 if piz else cfg["embedding"]["scale"])
        act = torch.nn.functional.silu if piz else torch.relu
        for i, l in enumerate(cfg["layers"]):
            norm = lambda v, n: _rms(v, t["l%d.%s" % (i, n)] + (1 if piz else 0), eps)  # noqa: E731, B023
            W = lambda n: t["l%d.mix.%s" % (i, n)]  # noqa: E731, B023
            h, m = norm(x, "norm1"), l["mixer"]
            y = {"latent_attention": lambda: _latent(h, W, m, eps), "wkv": lambda: _wkv(h, W, m, eps), "attention": lambda: _shared_kv(h, W, m),
                 "rglru": lambda: _rglru(h, W, m)}[l["type"]]()
            x = x + (y if piz else norm(y, "norm1b"))
            h = norm(x, "norm2")
            M = lambda n: t["l%d.mlp.%s" % (i, n)].T  # noqa: E731, B023
            y = (act(h @ M("gate")) * (h @ M("up"))) @ M("down")
            x = x + (y if piz else norm(y, "norm2b"))
        if piz:
            z = _rms(x, 1 + t["final.norm"], eps) @ t["embed"].T
            return cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"])
        return _rms(x, t["final.norm"], eps) @ t["head"].T


def exact(case, seed):
    prompts, given = requests(case, seed)
    do, starts = case["do"], [0] * case["batch"]
    if do == "session":
        m, steps = Block64(case), []
        for b, p in enumerate(prompts):
            steps.append(m.run(np.concatenate([p, given[:, b]]))[len(p) - 1:])
        return [torch.stack([s[i] for s in steps]) for i in range(len(given) + 1)]
    params = sum(r * c for n, k, r, c, _ in tensors(case["model"]) if k is not None and n not in ("token_embd.weight", "output.weight"))
    if 2.0 * params * sum(map(len, prompts)) > 3e14:  # 20 seconds and more
        return None
    m = Packed64(case, keep=do == "greedy")
    if do in ("prompt", "prompts"):
        out = m.run(prompts, starts)
        return out[0] if do == "prompt" else out
    if do == "decode":
        return m.run([np.append(p, t) for p, t in zip(prompts, given[0])], starts)
    m.run(prompts, starts)
    at, now, window, ids = [len(p) for p in prompts], given[0], [[int(t)] for t in given[0]], []
    for _ in range(case["steps"]):
        z = m.run([[t] for t in now], at)
        for b, hist in enumerate(window):
            for t in hist[-64:] if case["penalty"] > 1 else ():
                z[b, t] = z[b, t] / case["penalty"] if z[b, t] > 0 else z[b, t] * case["penalty"]
        now, at = z.argmax(-1).tolist(), [a + 1 for a in at]
        window = [hist + [t] for hist, t in zip(window, now)]
        ids.append(now)
    return np.array(ids, np.int32), m.run([[t] for t in now], at)
