"""The work a user has this framework do, as measurable cases: whole calls through the public entry points.

Kinds of work (`case["kind"]`):

  forward   `nsa_forward` on device tensors (prefill; Tq < Tk is a chunk of a longer prefill)
  train     `nsa_forward` and the gradients of Q, K, V and the gate logits through autograd
  decode    one decoding step: `KVCache.append` of the new keys and values, then `nsa_decode`
  fp8       `nsa_forward_fp8` on e4m3 tensors with per-tensor scales
  layer     `nsa_attention_token_major`: projection outputs in, rotary embedding inside, [B,T,H*D] out

Shapes: the reference's benchmark model (16 heads with their own keys, D=64, 64/64 pooling, one block list per
head), the headline model (64 query heads over 4 KV heads, D=64 or 128, 32/16 pooling, one list per KV head), the
CPU-runnable configuration (16 over 1, D=64), the training shape (12 over 1, D=64) and the small grouped shape of
the tests (8 over 2).  Values are N(0,1); gate logits come from a random Linear(D,3) on Q.
"""
import math

import numpy as np
import torch

import nsa_from_scratch_b200 as nsa

DEFAULTS = {
    "kind": "forward", "B": 1, "H": 64, "Hkv": 4, "D": 128, "Tq": 1024, "Tk": 1024, "dtype": "bf16",
    "cmp_block": 32, "cmp_stride": 16, "top_k": 16, "window": 512, "force_first": 1, "force_local": 2,
    "per_group": True, "gate": "sigmoid", "scorer": "mean",
}
# The reference's own model: a KV head per query head, no overlap in the pooling, nothing forced, a list per head.
MHA = {"H": 16, "Hkv": 16, "D": 64, "cmp_block": 64, "cmp_stride": 64, "force_first": 0, "force_local": 0, "per_group": False}


def _case(name=None, T=None, **kw):
    c = dict(DEFAULTS)
    c.update(kw)
    if T is not None:
        c["Tq"] = c["Tk"] = T
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # A short prompt on the reference's benchmark model: launches and host time count.
        _case("forward_mha_1k", T=1024, **MHA),
        # The same model at a common context length.
        _case("forward_mha_16k", T=16384, **MHA),
        # Two prompts of an odd length, fp16, softmax gates, one list per query head of a grouped model.
        _case("forward_ragged_fp16", B=2, H=16, Hkv=1, D=64, T=4001, dtype="fp16", gate="softmax", per_group=False),
        # The headline workload: the largest call.
        _case("forward_gqa_64k", T=65536),
        # Chunked prefill: the next 2048 positions of a prompt, 30000 already there.
        _case("prefill_chunk", Tq=2048, Tk=32048),
        # Selection scored by the compressed branch's own probabilities.
        _case("forward_scorer_16k", T=16384, scorer="compressed"),
        # fp8 storage, with the outliers that such tensors have.
        _case("fp8_32k", kind="fp8", T=32768),
        # The attention layer between its projections.
        _case("layer_16k", kind="layer", T=16384),
        # One token of one long conversation; one token of eight shorter ones.
        _case("decode_b1_64k", kind="decode", Tq=1, Tk=65536),
        _case("decode_b8_8k", kind="decode", B=8, Tq=1, Tk=8200),
        # Training at the training shape, and a short batch of the reference's model.
        _case("train_gqa_32k", kind="train", B=2, H=12, Hkv=1, D=64, T=32768),
        _case("train_mha_2k", kind="train", B=2, T=2048, **MHA),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges.  The longest length of a kind keeps its cost below the headline workload's."""
    kind = rng.choice(["forward", "forward", "forward", "chunk", "fp8", "layer", "decode", "decode", "train", "train"])
    H, Hkv, D = rng.choice([(16, 16, 64), (64, 4, 128), (64, 4, 64), (16, 1, 64), (12, 1, 64), (8, 2, 128)])
    grouped = H != Hkv
    c = _case(H=H, Hkv=Hkv, D=D, dtype=rng.choice(["bf16", "bf16", "bf16", "fp16"]), gate=rng.choice(["sigmoid", "sigmoid", "softmax"]),
              top_k=rng.choice([8, 16, 16, 16]), window=rng.choice([256, 512, 512]), per_group=grouped and rng.random() < 0.75)
    if not grouped or rng.random() < 0.2:
        c.update(cmp_block=64, cmp_stride=64)
    if rng.random() < 0.3:
        c.update(force_first=0, force_local=0)
    heavy = H == 64 and (D == 128 or not c["per_group"])
    if kind == "decode":
        c.update(kind="decode", B=rng.choice([1, 2, 4, 8]), Tq=rng.choice([1, 1, 1, 2, 4]))
        c["Tk"] = _log(rng, 1024, 65536)
        return c
    if kind == "chunk":
        c["Tq"] = _log(rng, 256, 4096)
        c["Tk"] = c["Tq"] + _log(rng, 1024, 32768)
        return c
    if kind == "fp8":
        c.update(kind="fp8", dtype="e4m3", per_group=grouped)
        top = 32768
    elif kind == "layer":
        c["kind"] = "layer"
        top = 32768
    elif kind == "train":
        c["kind"] = "train"
        top = 4096 if H == 64 else 16384
    else:
        if grouped and rng.random() < 0.2:
            c.update(scorer="compressed")
        top = 16384 if c["scorer"] == "compressed" else 49152
    if heavy and not c["per_group"]:
        top = min(top, 16384)
    T = _log(rng, 512, top)
    if rng.random() < 0.5:
        T = max(512, T // 64 * 64)
    c["Tq"] = c["Tk"] = T
    c["B"] = 2 if T <= 8192 and rng.random() < 0.4 else 1
    return c


def _cfg(c):
    return nsa.NSAConfig(
        block_size_c=c["cmp_block"], stride_c=None if c["cmp_stride"] == c["cmp_block"] else c["cmp_stride"], top_k=c["top_k"],
        window_size=c["window"], force_first=c["force_first"], force_local=c["force_local"], select_per_group=c["per_group"],
        gate_activation=c["gate"], scorer=c["scorer"])


def prepare(case, seed):
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(int(seed))
    B, H, Hkv, D, Tq, Tk, kind = (case[k] for k in ("B", "H", "Hkv", "D", "Tq", "Tk", "kind"))
    dt = torch.float16 if case["dtype"] == "fp16" else torch.bfloat16
    s = {"kind": kind, "cfg": _cfg(case)}

    def normal(*shape):
        return torch.randn(shape, generator=g, device=dev, dtype=dt)

    w = torch.randn((3, D), generator=g, device=dev) / D ** 0.5

    def gates(q):
        return (q @ w.to(q.dtype).T).contiguous()

    if kind == "layer":
        s["q"], s["k"], s["v"] = normal(B, Tq, H, D), normal(B, Tq, Hkv, D), normal(B, Tq, Hkv, D)
        s["gates"] = gates(s["q"])
        s["cos"], s["sin"] = nsa.rope_cache(Tq, D, 10000.0, dev)
        s["dtype"] = dt
    elif kind == "decode":
        # a cache that holds all but the step's own positions, and room for more
        cache = nsa.KVCache(B, Hkv, D, Tk + 256, s["cfg"], dtype=dt, device=dev)
        cache.append(normal(B, Hkv, Tk - Tq, D), normal(B, Hkv, Tk - Tq, D))
        s.update(cache=cache, filled=cache.length, q=normal(B, H, Tq, D), k=normal(B, Hkv, Tq, D), v=normal(B, Hkv, Tq, D))
        s["gates"] = gates(s["q"])
    else:
        q, k, v = normal(B, H, Tq, D), normal(B, Hkv, Tk, D), normal(B, Hkv, Tk, D)
        s["gates"] = gates(q)
        if kind == "fp8":
            for x in (q, k, v):        # one value in a thousand is an outlier of twenty times the size
                x.mul_(1.0 + 19.0 * (torch.rand(x.shape, generator=g, device=dev) < 0.001).to(dt))
            (q, s["sq"]), (k, s["sk"]), (v, s["sv"]) = (nsa.quantize_to_fp8(x) for x in (q, k, v))
        s.update(q=q, k=k, v=v)
        if kind == "train":
            s["do"] = normal(B, H, Tq, D)
            for n in ("q", "k", "v", "gates"):
                s[n].requires_grad_(True)
    return s


def run(s):
    kind, cfg = s["kind"], s["cfg"]
    if kind == "forward":
        return nsa.nsa_forward(s["q"], s["k"], s["v"], cfg, gate_logits=s["gates"])
    if kind == "train":
        leaves = (s["q"], s["k"], s["v"], s["gates"])
        out = nsa.nsa_forward(*leaves[:3], cfg, gate_logits=leaves[3])
        return (out.detach(), *torch.autograd.grad(out, leaves, s["do"]))
    if kind == "fp8":
        return nsa.nsa_forward_fp8(s["q"], s["k"], s["v"], s["sq"], s["sk"], s["sv"], cfg, gate_logits=s["gates"])
    if kind == "layer":
        return nsa.nsa_attention_token_major(s["q"], s["k"], s["v"], s["cos"], s["sin"], cfg, gate_logits=s["gates"], dtype=s["dtype"])
    cache = s["cache"]
    cache.length = s["filled"]         # the step's positions are taken back, as after a rejected draft token
    cache.append(s["k"], s["v"])
    out = nsa.nsa_decode(s["q"], cache, gate_logits=s["gates"])
    return out, cache.K, cache.V, cache.Kc, cache.Vc, cache.Kb


def _pairs(c):
    """(query, key) pairs of the three branches for one head: pooled tokens whose window has ended, keys of the
    listed blocks (the query's own block among them), keys of the window."""
    Tq, Tk = c["Tq"], c["Tk"]
    p = np.arange(Tk - Tq, Tk, dtype=np.int64)
    cmp_ = np.maximum((p + 1 - c["cmp_block"]) // c["cmp_stride"] + 1, 0).sum()
    own = p % 64 + 1
    sel = (np.minimum(p // 64, c["top_k"] - 1) * 64 + own).sum()
    return int(cmp_ + sel + np.minimum(p + 1, c["window"]).sum())


def work(case):
    c = case
    B, H, Hkv, D, Tq, Tk = (c[k] for k in ("B", "H", "Hkv", "D", "Tq", "Tk"))
    isz = 1 if c["kind"] == "fp8" else 2
    rows, keys = B * H * Tq, B * Hkv * Tk
    flops = 4.0 * D * B * H * _pairs(c)
    nbytes = rows * D * (isz + 2) + 2 * keys * D * isz + rows * 3 * 2
    if c["kind"] == "train":
        flops *= 3.5                    # five products of the forward's size for the gradients, two in the forward
        nbytes += rows * D * 4 + 2 * keys * D * 2 + rows * 3 * 2
    elif c["kind"] == "layer":
        nbytes += 2 * Tq * D * 4
    elif c["kind"] == "decode":
        # pooled keys and values, block means, at most the listed blocks and the window of the cache; the new rows
        listed_rows = min(Tk, c["top_k"] * 64) + min(Tk, c["window"])
        nbytes = rows * D * 4 + B * Hkv * D * 2 * (2 * (Tk // c["cmp_stride"]) + Tk // 64 + 2 * listed_rows + 4 * Tq)
    return {"bytes": float(nbytes), "flops": flops}


def tolerance(case):
    # 16-bit operands, probabilities and results.  `max`: the lists are chosen inside the call, so where two blocks
    # score the same to fp32 rounding, either may be taken and single rows differ by their own size.
    return {"rel": 1e-2, "max": 0.9}
