"""The work this library is measured on: its public entry points over the sizes, types and options that programs
use them with.  Sizes of the named configurations are those of the repository's benchmark; the others are generic.

    listed()          the cases that are always measured
    draw(rng)         one more case of the same ranges
    prepare(case, s)  what a program holds before the call: seeded inputs, outputs, checkpoints, scratch
    run(state)        one pass through the public entry points; returns its outputs whole
    work(case)        bytes and floating-point operations the pass cannot do without
    tolerance(case)   how far two correct implementations at the same precision may lie apart

A training pass is the forward call that saves its checkpoints followed by the backward call that reads them.
"""
import importlib.util
import math
import random
import sys
from pathlib import Path

import torch

ROOT = Path(__file__).resolve().parent.parent
TYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
SIZE = {"bf16": 2, "f16": 2, "f32": 4}
DEV = "cuda"


def _load_package():
    """The package directory's name holds a dot, so it is loaded by path."""
    if "tylo_b200" not in sys.modules:
        pkg = ROOT / "tylo.jl_b200"
        spec = importlib.util.spec_from_file_location("tylo_b200", pkg / "__init__.py", submodule_search_locations=[str(pkg)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["tylo_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["tylo_b200"]


tylo = _load_package()


# ---------------------------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------------------------
def attention(name, dtype, batch, heads, kv_heads, q_len, k_len, head_dim, *, causal, ragged=False, backward=False):
    return dict(name=name, kind="attention", dtype=dtype, batch=batch, heads=heads, kv_heads=kv_heads, q_len=q_len,
                k_len=k_len, head_dim=head_dim, causal=causal, ragged=ragged, backward=backward)


def flex(name, mods, dtype, batch, heads, kv_heads, length, head_dim, *, window=0, docs=0, backward=True):
    return dict(name=name, kind="flex", mods=mods, dtype=dtype, batch=batch, heads=heads, kv_heads=kv_heads, length=length,
                head_dim=head_dim, window=window, docs=docs, backward=backward)


def decode(name, dtype, batch, heads, kv_heads, head_dim, min_len, max_len, *, page=0):
    return dict(name=name, kind="decode", dtype=dtype, batch=batch, heads=heads, kv_heads=kv_heads, head_dim=head_dim,
                min_len=min_len, max_len=max_len, page=page)


def norm(name, op, dtype, hidden, tokens, *, backward=True):
    return dict(name=name, kind="norm", op=op, dtype=dtype, hidden=hidden, tokens=tokens, backward=backward)


def softmax(name, dtype, length, rows, *, backward=True):
    return dict(name=name, kind="softmax", dtype=dtype, length=length, rows=rows, backward=backward)


def listed():
    return [
        # serving: the prompt of a batch of requests, grouped-query attention, statistics saved (benchmark config 3)
        attention("prefill_4k", "bf16", 4, 32, 8, 4096, 4096, 128, causal=True),
        # training: the same layer, forward and backward (benchmark config 3)
        attention("train_4k", "bf16", 4, 32, 8, 4096, 4096, 128, causal=True, backward=True),
        # an encoder over a padded batch: no causal mask, odd length, per-entry lengths, half precision, head dim 64
        attention("encoder_ragged", "f16", 8, 16, 16, 777, 777, 64, causal=False, ragged=True),
        # Float32 arrays, the element type the library's users start from (benchmark config 1), forward and backward
        attention("train_fp32", "f32", 2, 8, 8, 512, 512, 64, causal=False, backward=True),
        # packed documents with a sliding window and a soft cap, forward and backward (benchmark config 4)
        flex("flex_docs_train", "docs_softcap", "bf16", 2, 16, 16, 8192, 128, window=1024, docs=8),
        # a learned position bias with its gradient (the benchmark's bias variant)
        flex("flex_bias_train", "bias", "bf16", 2, 8, 8, 2048, 128),
        # one token for each of a full batch of conversations of very different lengths (benchmark config 5a)
        decode("decode_batch", "bf16", 64, 64, 8, 128, 1024, 32768),
        # one token for a single user with a short context: launch and host latency
        decode("decode_single", "bf16", 1, 32, 8, 128, 1537, 1537),
        # one token over a million-token context (benchmark config 5b)
        decode("decode_1m", "bf16", 1, 64, 8, 128, 1 << 20, 1 << 20),
        # the norm of a wide layer over a training batch (benchmark config 2)
        norm("rms_train", "rms", "bf16", 8192, 16384),
        # the norm of a small Float32 layer on an odd number of tokens: launch and host latency
        norm("layer_fp32_small", "layer", "f32", 768, 333),
        # rows of logits (benchmark config 2)
        softmax("softmax_train", "bf16", 32768, 4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shrink(case, key, limit, cost):
    """Halves case[key] until the pass costs no more than `limit`."""
    while cost(case) > limit and case[key] > 1:
        case[key] = max(1, case[key] // 2)
    return case


def _blocks(length):
    """Causal layers with one query head per KV head: sequences padded to whole blocks of 256 rows."""
    return -(-length // 256) * 256


MAX_FLOPS, MAX_FLOPS_F32, MAX_BYTES = 1.8e12, 5e10, 4e9


def draw(rng):
    kind = rng.choice(["prefill", "train", "encoder", "fp32", "flex", "flex", "decode", "decode", "norm", "norm", "softmax"])
    flops = lambda c: work(c)["flops"]
    size = lambda c: work(c)["bytes"]
    if kind in ("prefill", "train", "encoder", "fp32"):
        f32 = kind == "fp32"
        kv_heads = rng.choice([1, 2, 4, 8, 16])
        heads = kv_heads * rng.choice([1, 1, 2, 4, 8])
        k_len = _log_int(rng, 33, 1500 if f32 else 16384)
        # a chunk of a longer prompt sees the keys before it too
        q_len = max(1, k_len // rng.choice([2, 4, 8])) if kind == "prefill" and rng.random() < 0.3 else k_len
        c = attention("", "f32" if f32 else rng.choice(["bf16", "bf16", "f16"]), rng.choice([1, 2, 3, 4, 8, 16]), heads, kv_heads,
                      q_len, k_len, rng.choice([32, 64, 64, 128] if f32 else [64, 96, 128, 128]),
                      causal=kind in ("prefill", "train") or (f32 and rng.random() < 0.5), ragged=kind == "encoder",
                      backward=kind == "train" or (f32 and rng.random() < 0.7))
        limit = MAX_FLOPS_F32 if f32 else MAX_FLOPS
        c = _shrink(_shrink(c, "batch", limit, flops), "q_len", limit, flops)
        if kind in ("prefill", "train") and heads == kv_heads:
            c["q_len"], c["k_len"] = _blocks(c["q_len"]), _blocks(c["k_len"])
        if kind != "prefill":
            c["k_len"] = c["q_len"]
    elif kind == "flex":
        mods = rng.choice(["docs_softcap", "alibi", "bias", "window"])
        kv_heads = rng.choice([2, 4, 8, 16])
        heads = kv_heads * rng.choice([1, 1, 2, 4])
        length = _log_int(rng, 100, 3000 if mods == "bias" else 16384)
        c = flex("", mods, rng.choice(["bf16", "bf16", "f16"]), rng.choice([1, 2, 4]), heads, kv_heads, length, rng.choice([64, 128, 128]),
                 window=max(16, _log_int(rng, length // 32 + 16, length // 2 + 32)) if mods in ("docs_softcap", "window") else 0,
                 docs=rng.randint(2, 12) if mods == "docs_softcap" else 0, backward=rng.random() < 0.7)
        c = _shrink(_shrink(_shrink(c, "batch", MAX_FLOPS, flops), "batch", MAX_BYTES / 4, size), "length", MAX_FLOPS, flops)
        if mods in ("alibi", "bias") and heads == kv_heads:
            c["length"] = _blocks(c["length"])
    elif kind == "decode":
        kv_heads = rng.choice([1, 2, 4, 8, 8])
        heads = kv_heads * rng.choice([1, 4, 8, 8, 16])
        hi = _log_int(rng, 100, 262144)
        c = decode("", rng.choice(["bf16", "bf16", "f16"]), _log_int(rng, 1, 128), heads, kv_heads, rng.choice([64, 128, 128]),
                   rng.choice([hi, max(1, hi // 2), max(1, hi // 32)]), hi, page=rng.choice([0, 0, 64, 256]))
        c = _shrink(c, "batch", MAX_BYTES, size)
    elif kind == "norm":
        hidden = _log_int(rng, 64, 2048) * 8 if rng.random() < 0.85 else _log_int(rng, 100, 16384)
        c = norm("", rng.choice(["rms", "layer"]), rng.choice(["bf16", "bf16", "f16", "f32"]), hidden, _log_int(rng, 1, 65536),
                 backward=rng.random() < 0.6)
        c = _shrink(c, "tokens", MAX_BYTES / 3, size)
    else:
        length = _log_int(rng, 8, 16384) * 8 if rng.random() < 0.7 else _log_int(rng, 50, 131072)
        c = softmax("", rng.choice(["bf16", "bf16", "f16", "f32"]), length, _log_int(rng, 1, 65536), backward=rng.random() < 0.6)
        c = _shrink(c, "rows", MAX_BYTES / 3, size)
    del c["name"]
    return c


# ---------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------
def _lengths(lo, hi, n, g):
    """n lengths evenly spread over [lo, hi], in a seeded order."""
    return torch.linspace(lo, hi, n, dtype=torch.float64).round().to(torch.int32)[torch.randperm(n, generator=g)].to(DEV)


def _documents(batch, length, docs, seed):
    """(batch, length) document ids: every sequence cut at docs - 1 uniformly drawn places."""
    ids = torch.zeros(batch, length, dtype=torch.int32)
    rng = random.Random(seed)
    for b in range(batch):
        for cut in _cuts(rng, length, docs):
            ids[b, cut:] += 1
    return ids.to(DEV)


def _cuts(rng, length, docs):
    return sorted(rng.randrange(1, length) for _ in range(docs - 1)) if length > 1 else []


def _slopes(heads):
    return torch.tensor([2.0 ** (-8.0 * (h + 1) / heads) for h in range(heads)], dtype=torch.float32, device=DEV)


def _mods(c, seed):
    m = c["mods"]
    if m == "docs_softcap":
        ids = _documents(c["batch"], c["length"], c["docs"], seed)
        return tylo.SoftCapScore(50.0), tylo.CausalMask() & tylo.SlidingWindowMask(c["window"]) & tylo.DocumentMask(ids)
    if m == "window":
        return None, tylo.CausalMask() & tylo.SlidingWindowMask(c["window"])
    if m == "alibi":
        return tylo.AliBiScore(_slopes(c["heads"])), tylo.CausalMask()
    g = torch.Generator(DEV).manual_seed(seed + 1)
    return tylo.BiasScore(torch.randn(1, c["heads"], c["length"], c["length"], generator=g, device=DEV)), tylo.CausalMask()


def prepare(case, seed):
    c = case
    dt = TYPES[c["dtype"]]
    g, gc = torch.Generator(DEV).manual_seed(seed), torch.Generator().manual_seed(seed)

    def normal(*shape, scale=1.0, shift=0.0):
        x = torch.randn(*shape, generator=g, device=DEV, dtype=torch.float32 if math.prod(shape) < 1 << 28 else dt)
        return (x if scale == 1.0 and shift == 0.0 else x * scale + shift).to(dt)

    kind = c["kind"]
    s = dict(case=c)
    if kind in ("attention", "flex"):
        B, H, Hkv, D = c["batch"], c["heads"], c["kv_heads"], c["head_dim"]
        Sq, Sk = (c["q_len"], c["k_len"]) if kind == "attention" else (c["length"], c["length"])
        s["Q"], s["K"], s["V"] = normal(B, H, Sq, D), normal(B, Hkv, Sk, D), normal(B, Hkv, Sk, D)
        s["O"] = torch.zeros_like(s["Q"])
        s["checkpoints"] = tylo.allocate_checkpoints_attention(s["Q"], s["K"], s["V"])
        if kind == "attention":
            s["options"] = dict(causal=c["causal"], input_pos=Sk - Sq if c["causal"] else 0)
            if c["ragged"]:
                n = _lengths(max(1, Sk // 2), Sk, B, gc)
                s["options"].update(k_lengths=n, q_lengths=n)
                s["checkpoints"].M.zero_(), s["checkpoints"].L.zero_()      # rows beyond a length are left as they are
        else:
            score, mask = _mods(c, seed)
            s["options"] = dict(score_mod=score, mask_mod=mask)
        if c["backward"]:
            s["dO"] = normal(B, H, Sq, D)
            s["dQ"], s["dK"], s["dV"] = (torch.empty_like(s[k]) for k in "QKV")
            s["scratch"] = tylo.allocate_scratchspace_grad_attention(s["Q"], s["K"], s["V"], s["O"])
            if kind == "flex" and c["mods"] in ("alibi", "bias"):
                s["d_score_mod"] = tylo.grad_shadow(s["options"]["score_mod"])
    elif kind == "decode":
        B, H, Hkv, D = c["batch"], c["heads"], c["kv_heads"], c["head_dim"]
        s["Q"] = normal(B, H, D)
        s["O"] = torch.empty_like(s["Q"])
        s["lengths"] = _lengths(c["min_len"], c["max_len"], B, gc)
        if c["page"]:
            pages = -(-c["max_len"] // c["page"])
            s["K"], s["V"] = normal(B * pages, Hkv, c["page"], D), normal(B * pages, Hkv, c["page"], D)
            s["table"] = torch.randperm(B * pages, generator=gc).to(torch.int32).reshape(B, pages).to(DEV)
            keys = pages * c["page"]
        else:
            keys = c["max_len"]
            s["K"], s["V"] = normal(B, Hkv, keys, D), normal(B, Hkv, keys, D)
        s["scratch"] = tylo.allocate_scratchspace_decode_attention(s["O"], s["Q"], n_splits=tylo.decode_suggest_splits(keys, Hkv, B))
    elif kind == "norm":
        M, N = c["hidden"], c["tokens"]
        s["X"], s["W"] = normal(N, M), normal(M, scale=0.02, shift=1.0)
        s["Y"] = torch.empty_like(s["X"])
        layer = c["op"] == "layer"
        if layer:
            s["B"] = normal(M, scale=0.02)
        weights = (s["W"], s["B"]) if layer else (s["W"],)
        s["checkpoints"] = (tylo.allocate_checkpoints_layer_norm if layer else tylo.allocate_checkpoints_rms_norm)(s["X"], *weights)
        if c["backward"]:
            s["dY"], s["dX"], s["dW"] = normal(N, M), torch.empty_like(s["X"]), torch.empty_like(s["W"])
            if layer:
                s["dB"] = torch.empty_like(s["B"])
            s["scratch"] = (tylo.allocate_scratchspace_grad_layer_norm if layer else tylo.allocate_scratchspace_grad_rms_norm)(s["X"], *weights)
    else:
        M, N = c["length"], c["rows"]
        s["X"] = normal(N, M, scale=2.0)
        s["Y"] = torch.empty_like(s["X"])
        if c["backward"]:
            s["dY"], s["dX"] = normal(N, M), torch.empty_like(s["X"])
    return s


# ---------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------
def run(state):
    s, c = state, state["case"]
    dup = tylo.Duplicated
    kind = c["kind"]
    if kind in ("attention", "flex"):
        forward, backward = ((tylo.attention_, tylo.grad_attention_) if kind == "attention"
                             else (tylo.flex_attention_, tylo.grad_flex_attention_))
        forward(s["O"], s["Q"], s["K"], s["V"], checkpoints=s["checkpoints"], **s["options"])
        out = dict(O=s["O"], M=s["checkpoints"].M, L=s["checkpoints"].L)
        if c["backward"]:
            extra = {}
            d = s.get("d_score_mod")
            if d is not None:       # parameter gradients are accumulated, so every step starts them at zero
                param = d.bias if c["mods"] == "bias" else d.slopes
                param.zero_()
                extra = dict(d_score_mod=d)
                out["d_param"] = param
            backward(dup(s["O"], s["dO"]), dup(s["Q"], s["dQ"]), dup(s["K"], s["dK"]), dup(s["V"], s["dV"]),
                     checkpoints=s["checkpoints"], scratch=s["scratch"], **s["options"], **extra)
            out.update(dQ=s["dQ"], dK=s["dK"], dV=s["dV"])
        return out
    if kind == "decode":
        if c["page"]:
            tylo.paged_decode_attention_(s["O"], s["Q"], s["K"], s["V"], block_table=s["table"], lengths=s["lengths"], scratch=s["scratch"])
        else:
            tylo.decode_attention_(s["O"], s["Q"], s["K"], s["V"], lengths=s["lengths"], scratch=s["scratch"])
        return s["O"]
    if kind == "norm":
        out = dict(Y=s["Y"], checkpoints=list(s["checkpoints"]))
        if c["op"] == "rms":
            tylo.rms_norm_(s["Y"], s["X"], s["W"], eps=1e-6, checkpoints=s["checkpoints"])
            if c["backward"]:
                tylo.grad_rms_norm_(dup(s["Y"], s["dY"]), dup(s["X"], s["dX"]), dup(s["W"], s["dW"]),
                                    checkpoints=s["checkpoints"], scratch=s["scratch"])
                out.update(dX=s["dX"], dW=s["dW"])
        else:
            tylo.layer_norm_(s["Y"], s["X"], s["W"], s["B"], eps=1e-6, checkpoints=s["checkpoints"])
            if c["backward"]:
                tylo.grad_layer_norm_(dup(s["Y"], s["dY"]), dup(s["X"], s["dX"]), dup(s["W"], s["dW"]), dup(s["B"], s["dB"]),
                                      checkpoints=s["checkpoints"], scratch=s["scratch"])
                out.update(dX=s["dX"], dW=s["dW"], dB=s["dB"])
        return out
    tylo.softmax_(s["Y"], s["X"])
    if not c["backward"]:
        return s["Y"]
    tylo.grad_softmax_(dup(s["Y"], s["dY"]), dup(s["X"], s["dX"]))
    return dict(Y=s["Y"], dX=s["dX"])


# ---------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------
def _band(length, window):
    """Pairs with 0 <= q - kv <= window among `length` positions."""
    w = min(window, length - 1)
    return (w + 1) * length - w * (w + 1) // 2


def _pairs(c):
    """Unmasked (query, key) pairs of all batch entries and heads.  Where lengths or documents come from the seed:
    lengths have one sum for every seed, documents are averaged over 32 drawings."""
    B, H = c["batch"], c["heads"]
    if c["kind"] == "attention":
        Sq, Sk = c["q_len"], c["k_len"]
        if c["ragged"]:
            ends = [round(x) for x in torch.linspace(max(1, Sk // 2), Sk, B, dtype=torch.float64).tolist()]
            return H * sum(n * n for n in ends)
        return B * H * (Sq * Sk - Sq * (Sq - 1) // 2 if c["causal"] else Sq * Sk)
    n, w = c["length"], c["window"] or c["length"]
    if not c["docs"]:
        return B * H * _band(n, w)
    rng, total = random.Random(0), 0
    for _ in range(32):
        edges = [0] + _cuts(rng, n, c["docs"]) + [n]
        total += sum(_band(b - a, w) for a, b in zip(edges, edges[1:]) if b > a)
    return B * H * total / 32


def work(case):
    c = case
    e = SIZE[c["dtype"]]
    kind = c["kind"]
    if kind in ("attention", "flex"):
        B, H, Hkv, D = c["batch"], c["heads"], c["kv_heads"], c["head_dim"]
        Sq, Sk = (c["q_len"], c["k_len"]) if kind == "attention" else (c["length"], c["length"])
        q, kv, stats = B * H * Sq * D * e, B * Hkv * Sk * D * e, 2 * B * H * Sq * 4
        bias = H * Sq * Sk * 4 if kind == "flex" and c["mods"] == "bias" else 0
        nbytes, flops = 2 * q + 2 * kv + stats + bias, 4 * D * _pairs(c)
        if c["backward"]:       # reads Q, K, V, O, dO, statistics (and the table); writes the gradients
            nbytes += 4 * q + 4 * kv + stats + 2 * bias
            flops += 10 * D * _pairs(c)
        return dict(bytes=nbytes, flops=flops)
    if kind == "decode":
        n = c["batch"] * (c["min_len"] + c["max_len"]) / 2 if c["batch"] > 1 else c["min_len"]
        D = c["head_dim"]
        return dict(bytes=2 * n * c["kv_heads"] * D * e + 2 * c["batch"] * c["heads"] * D * e, flops=4 * n * c["heads"] * D)
    x = c["hidden"] * c["tokens"] if kind == "norm" else c["length"] * c["rows"]
    nbytes, flops = 2 * x * e, 4 * x
    if c["backward"]:
        nbytes += 3 * x * e
        flops += 8 * x
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    """Four times the largest relative error of any output against float64 on the same inputs, over the listed and sixty
    drawn cases.  Attention and decode: 3.2e-3 in bf16 and 4.3e-4 in f16 (P and dS are rounded to the storage type before
    the second product), 4.0e-7 in f32.  Row kernels: the rounding of the result, 1.8e-3 in bf16 and 2.1e-4 in f16; in f32
    sums over a row or over all tokens, 2.5e-7."""
    if case["dtype"] == "f32":
        return {"rel": 1.6e-6}
    if case["kind"] in ("attention", "flex"):
        return {"rel": 1.2e-2 if case["dtype"] == "bf16" else 1.7e-3}
    if case["kind"] == "decode":
        return {"rel": 9e-3 if case["dtype"] == "bf16" else 1.1e-3}
    return {"rel": 7e-3 if case["dtype"] == "bf16" else 8.5e-4}
