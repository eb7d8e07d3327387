"""Measured workloads of the NVFP4 attention package, as a user's program calls it.

Six kinds of pass, each through the public entry points:

  decode     one serving step: append a token to an ``NVFP4KVCache``, attend over the packed cache
  hybrid     the same step with a high-precision recent window (``hybrid_decode``)
  prefill    attention over a prompt and packing of its K / V into the layer's cache
  producers  prompt attention with rotary and V-projection fused into the packers
  cross      attention without a causal mask, padded keys (bias), ``[Z, S, H, D]`` output
  train      forward and backward of ``nvfp4_flash_attn_func`` (dense or packed samples)

Sizes are those of the repository's benchmark, demo and tests or lie between them.  Keys carry a
constant offset on eight channels, as the benchmark's inputs do.
"""

import math

import torch

import sageattention_b200.nvfp4 as nv

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # One chat request on one GPU: the smallest call, latency and launches are all there is.
        dict(name="decode_one_request", kind="decode", z=1, h=32, hk=8, d=128, s=1021, dtype="bf16"),
        # A few requests at head dim 256 in fp16, ragged cache length.
        dict(name="decode_d256_fp16", kind="decode", z=4, h=16, hk=4, d=256, s=6007, dtype="fp16"),
        # A full serving batch at 32k context (the benchmark's decode configuration).
        dict(name="decode_batch_32k", kind="decode", z=16, h=32, hk=8, d=128, s=32768, dtype="bf16"),
        # A serving batch that keeps the last 512 tokens exact.
        dict(name="hybrid_batch_8k", kind="hybrid", z=8, h=32, hk=8, d=128, s=8190, window=512, dtype="bf16"),
        # A short prompt of a small model (the demo's head counts), cache with a recent window.
        dict(name="prefill_short", kind="prefill", z=1, h=8, hk=2, d=128, s=777, window=128, dtype="bf16"),
        # The benchmark's prefill configuration.
        dict(name="prefill_batch_8k", kind="prefill", z=4, h=32, hk=8, d=128, s=8192, window=0, dtype="bf16"),
        # One long prompt at head dim 256, odd length.
        dict(name="prefill_d256_12k", kind="prefill", z=1, h=16, hk=4, d=256, s=12289, window=0, dtype="bf16"),
        # A decoder layer's prompt with the packers fused into rotary and the V projection.
        dict(name="producers_2k", kind="producers", z=1, h=32, hk=8, d=128, s=2048, hidden=4096, dtype="bf16"),
        # Cross attention to a padded context.
        dict(name="cross_bias_fp16", kind="cross", z=2, h=32, hk=8, d=128, sq=1029, s=2309, dtype="fp16"),
        # A training step of a short sequence, default backward (bf16 gradient products below 4096 tokens).
        dict(name="train_1k", kind="train", z=1, h=16, hk=4, d=128, s=1024, samples=0, dtype="bf16"),
        # The benchmark's packed training step: samples of 256 to 4096 tokens in a row of 16384.
        dict(name="train_packed_16k", kind="train", z=1, h=32, hk=8, d=128, s=16384, samples=8, dtype="bf16"),
        # Long-sequence training at head dim 256, default backward (all-FP4 from 4096 tokens on).
        dict(name="train_d256_8k", kind="train", z=1, h=16, hk=4, d=256, s=8192, samples=0, dtype="bf16"),
    ]


_MOST_FLOPS = 2.2e12      # prefill_batch_8k
_MOST_BYTES = 6.1e8       # decode_batch_32k


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    while True:
        kind = rng.choice(("decode", "decode", "hybrid", "prefill", "prefill", "producers", "cross", "train", "train", "train"))
        d = 128 if rng.random() < 0.7 else 256
        h, hk = rng.choice(((32, 8), (32, 8), (32, 4), (16, 4), (8, 2), (8, 8)))
        c = dict(kind=kind, z=1, h=h, hk=hk, d=d, dtype="bf16" if rng.random() < 0.75 else "fp16")
        if kind in ("decode", "hybrid"):
            c["z"] = _log_int(rng, 1, 16)
            c["s"] = _log_int(rng, 256, 32768)
            if kind == "hybrid":
                c["window"] = rng.choice((128, 256, 512))
                c["s"] = max(c["s"], 2 * c["window"] + 1)
        elif kind == "prefill":
            c["z"] = _log_int(rng, 1, 4)
            c["s"] = _log_int(rng, 128, 16384)
            c["window"] = rng.choice((0, 0, 128, 512))
        elif kind == "producers":
            c["s"] = _log_int(rng, 128, 8192)
            c["hidden"] = rng.choice((1024, 2048, 4096))
        elif kind == "cross":
            c["z"] = _log_int(rng, 1, 4)
            c["sq"] = _log_int(rng, 64, 8192)
            c["s"] = _log_int(rng, 64, 8192)
        else:
            c["z"] = rng.choice((1, 1, 2))
            c["s"] = _log_int(rng, 256, 16384)
            c["samples"] = rng.choice((0, 0, 4, 8, 16)) if c["z"] == 1 and c["s"] >= 2048 else 0
        w = work(c)
        if w["flops"] <= _MOST_FLOPS and w["bytes"] <= _MOST_BYTES:
            return c


def _lengths(case):
    """Sample lengths of a packed row: `samples` of them, spread between a sixth and twice the mean."""
    n, total = case["samples"], case["s"]
    if not n:
        return [total]
    weights = [0.16 + 1.84 * ((i * 0.618034 + 0.31) % 1.0) for i in range(n)]
    lens = [max(16, int(total * w / sum(weights))) for w in weights]
    lens[-1] += total - sum(lens)
    return lens


def prepare(case, seed):
    c = dict(case)
    dev = torch.device("cuda")
    dt = _DTYPES[c["dtype"]]
    gen = torch.Generator(device=dev).manual_seed(seed)

    def rn(*shape, dtype=dt):
        return torch.randn(*shape, device=dev, dtype=dtype, generator=gen)

    z, h, hk, d, s = c["z"], c["h"], c["hk"], c["d"], c["s"]
    st = {"kind": c["kind"], "s": s, "g": h // hk, "scaling": d ** -0.5, "case": c}
    offset = torch.zeros(d, device=dev, dtype=dt)
    offset[torch.randperm(d, device=dev, generator=gen)[:8]] = rn(8) * 2.0
    if c["kind"] in ("decode", "hybrid"):
        cache = nv.NVFP4KVCache(z, hk, d, s + 128, dev, dt, recent_window=c.get("window", 0))
        cache.prefill(rn(z, hk, s, d) + offset, rn(z, hk, s, d))
        st.update(cache=cache, fill=(s, cache.partial_len), q=rn(z, h, 1, d), k=rn(z, hk, 1, d) + offset,
                  v=rn(z, hk, 1, d))
    elif c["kind"] == "prefill":
        st.update(cache=nv.NVFP4KVCache(z, hk, d, s + 128, dev, dt, recent_window=c["window"]), q=rn(z, h, s, d),
                  k=rn(z, hk, s, d) + offset, v=rn(z, hk, s, d))
    elif c["kind"] == "producers":
        angle = torch.arange(s, device=dev)[:, None] / 10000.0 ** (torch.arange(0, d, 2, device=dev) / d)
        st.update(x=rn(z, s, c["hidden"]), q=rn(z * h, s, d), k=rn(z * hk, s, d) + offset,
                  w=rn(hk * d, c["hidden"]) * c["hidden"] ** -0.5, cos=angle.cos(), sin=angle.sin(), dtype=dt)
    elif c["kind"] == "cross":
        bias = torch.zeros(z, s, device=dev, dtype=torch.float32)
        for i in range(z):                      # every entry of the batch has its own number of valid keys
            bias[i, s - (i + 1) * s // 9:] = float("-inf")
        st.update(q=rn(z, h, c["sq"], d), k=rn(z, hk, s, d) + offset, v=rn(z, hk, s, d), bias=bias)
    else:
        st.update(q=rn(z, h, s, d).requires_grad_(True), k=(rn(z, hk, s, d) + offset).requires_grad_(True),
                  v=rn(z, hk, s, d).requires_grad_(True), do=rn(z, h, s, d), cu=None)
        if c["samples"]:
            st["cu"] = torch.tensor([0] + _lengths(c), device=dev).cumsum(0).to(torch.int32)
    return st


def run(st):
    kind, g, scaling = st["kind"], st["g"], st["scaling"]
    if kind in ("decode", "hybrid"):
        cache = st["cache"]
        cache.length, cache.partial_len = st["fill"]          # every pass appends the same next token
        cache.append(st["k"], st["v"])
        if kind == "decode":
            return (nv.nvfp4_flash_decode_prequant(st["q"], cache.get_packed(), scaling, g),) + _buffers(cache)
        return (cache.hybrid_decode(st["q"], scaling, g),) + _buffers(cache)
    if kind == "prefill":
        out = nv.nvfp4_flash_attention(st["q"], st["k"], st["v"], scaling, causal=True, num_key_value_groups=g)
        st["cache"].prefill(st["k"], st["v"])
        return (out,) + _buffers(st["cache"])
    if kind == "producers":
        c = st["case"]
        qnv, qsc = nv.rope_quant_nvfp4(st["q"], st["cos"], st["sin"])
        knv, ksc = nv.rope_quant_nvfp4(st["k"], st["cos"], st["sin"])
        vnv, vsc, value = nv.vproj_quant_nvfp4(st["x"], st["w"], None, c["hk"], c["d"])
        out = nv.nvfp4_flash_attention_packed(qnv, qsc, knv, ksc, vnv, vsc, c["z"], c["h"], c["hk"], c["s"], c["s"],
                                              c["d"], scaling, st["dtype"], causal=True)
        return out, value
    if kind == "cross":
        return nv.nvfp4_flash_attention(st["q"], st["k"], st["v"], scaling, num_key_value_groups=g,
                                        key_pad_bias=st["bias"], out_layout="zshd")
    out = nv.nvfp4_flash_attn_func(st["q"], st["k"], st["v"], scaling, causal=True, num_key_value_groups=g,
                                   cu_seqlens=st["cu"])
    return (out,) + torch.autograd.grad(out, (st["q"], st["k"], st["v"]), st["do"])


def _buffers(cache):
    """The cache's state after a pass."""
    ring = (cache.rk, cache.rv) if cache.recent_window > 0 else ()
    return (cache.knv, cache.ksc.view(torch.uint8), cache.vnv, cache.vsc.view(torch.uint8), cache.v_partial_bf16) + ring


def work(case):
    """Bytes: inputs read once, outputs written once (packed cache: 9/16 byte a value).  FLOPs: the visible
    part of Q K^T and P V, 2.5 times that again for a backward, and the V projection where the path has it."""
    c = case
    z, h, hk, d, s = c["z"], c["h"], c["hk"], c["d"], c["s"]
    q_val, kv_val, packed = z * h * d, z * hk * d, 9.0 / 16.0
    if c["kind"] in ("decode", "hybrid"):
        recent = min(s, c.get("window", 0))
        nbytes = 2 * kv_val * (s - recent) * packed + 2 * 2 * kv_val * recent + 2 * 2 * q_val + 2 * 2 * kv_val
        return {"bytes": nbytes, "flops": 4.0 * q_val * s}
    if c["kind"] == "prefill":
        return {"bytes": 2.0 * 2 * q_val * s + 2 * 2 * kv_val * s + 2 * kv_val * s * packed, "flops": 2.0 * q_val * s * s}
    if c["kind"] == "producers":
        nbytes = 2.0 * 2 * q_val * s + 2 * 2 * kv_val * s + 2.0 * z * s * c["hidden"] + 2.0 * hk * d * c["hidden"]
        return {"bytes": nbytes, "flops": 2.0 * q_val * s * s + 2.0 * z * s * c["hidden"] * hk * d}
    if c["kind"] == "cross":
        return {"bytes": 2.0 * 2 * q_val * c["sq"] + 2 * 2 * kv_val * s, "flops": 4.0 * q_val * c["sq"] * s}
    pairs = sum(float(n) * n for n in _lengths(c)) / 2.0
    return {"bytes": 2.0 * 4 * q_val * s + 2 * 4 * kv_val * s, "flops": 3.5 * 4.0 * q_val * pairs}


def tolerance(case):
    """16-bit results of sums over FP4 operands.  Packed bytes and cached rows are the same to the bit.  A probability
    next to a rounding boundary of the FP4 grid may fall to either side, which moves single values by up to half."""
    return {"rel": 1e-2, "max": 0.5}
