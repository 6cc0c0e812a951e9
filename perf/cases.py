"""The work that programs have this framework do, as cases that can be timed and compared.

Six kinds of call, all through the package's public entry points:

  decode    ``PackedKVCache.attend`` with one query token per sequence over a filled compressed cache (one layer)
  prefill   ``PackedKVCache.attend`` with a chunk of prompt tokens that the cache already holds (causal, bottom-right)
  generate  one request batch from an empty ``PackedKVCache``: the prompt of every layer is appended and attended, then
            tokens one at a time, layers alternating between full and sliding-window attention
  encode    ``HQMQ.encode`` of a prompt's keys and values to fresh compressed planes
  fakequant ``quantize_K`` / ``quantize_V``, the quantizer plugin interface: dense in, dense out
  tuple     ``fused_attention`` on the packed tuple (indices, radius codes, scales, joint tables), a decode query over the
            whole cache or a causal prompt

Shapes: 32 query heads on 8 KV heads and 28 on 4 at head dim 128 with codebooks s24_r3, s96_r4 and s192_r6, 64 on 8 at head
dim 64 with s96_r4 (whose rows are whole words there); with outlier extraction (C = 3) and without; bf16 and fp16."""
import math

import torch

import hqmq_b200 as hqmq

HEADS = ((32, 8, 128), (28, 4, 128), (64, 8, 64))        # query heads, KV heads, head dim
CODEBOOKS = ((24, 3), (96, 4), (192, 6))                  # secondary codebook size, radius bits
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
# share of the chunks that a threshold of three medians flags, per value distribution
FLAGGED = {"randn": 0.0, "hot": 0.06, "student": 0.06, "spiky": 0.005, "onehot": 0.04}
# ... and a share that every (sequence, head) is sure to reach
FLAGGED_LEAST = {"randn": 0.0, "hot": 0.012, "student": 0.012, "spiky": 0.001, "onehot": 0.0}


def listed():
    return [
        # a single user's decode step at a short context: a launch-bound call
        dict(name="decode_1x4k", kind="decode", B=1, Hq=32, Hkv=8, d=128, T=4096, S=24, rb=3, C=0.0, kk="randn", vk="randn",
             window=0, dtype="fp16"),
        # a serving batch at long context: the cache of one layer is 650 MB
        dict(name="decode_16x32k", kind="decode", B=16, Hq=32, Hkv=8, d=128, T=32768, S=96, rb=4, C=3.0, kk="hot", vk="randn",
             window=0, dtype="bf16"),
        # seven query heads per KV head, 19-bit fields, heavy-tailed key channels, a ragged context
        dict(name="decode_32x8k_g7", kind="decode", B=32, Hq=28, Hkv=4, d=128, T=8111, S=192, rb=6, C=3.0, kk="student",
             vk="randn", window=0, dtype="bf16"),
        # one very long document: few units, split over the whole chip
        dict(name="decode_1x128k", kind="decode", B=1, Hq=32, Hkv=8, d=128, T=131072, S=24, rb=3, C=3.0, kk="spiky", vk="spiky",
             window=0, dtype="bf16"),
        # head dim 64 with eight query heads per KV head, an outlier channel in every head, a large batch
        dict(name="decode_64x16k_d64", kind="decode", B=64, Hq=64, Hkv=8, d=64, T=16384, S=96, rb=4, C=3.0, kk="onehot",
             vk="onehot", window=0, dtype="bf16"),
        # chunked prefill: the last 2048 tokens of an 8 k prompt attend over the compressed cache
        dict(name="prefill_2k_of_8k", kind="prefill", B=1, Hq=32, Hkv=8, d=128, T=8192, Tq=2048, S=96, rb=4, C=3.0, kk="hot",
             vk="randn", window=0, dtype="bf16"),
        # a short request through four layers, every second one with a 128-token window: prompt, then twelve tokens
        dict(name="generate_4x500_12", kind="generate", B=4, Hq=64, Hkv=8, d=64, T=500, layers=4, steps=12, S=96, rb=4, C=3.0,
             kk="onehot", vk="onehot", window=128, layout="tokens", dtype="bf16"),
        # prompts of a batch compressed: 131072 tokens of keys and values
        dict(name="encode_16x8k", kind="encode", B=16, Hq=32, Hkv=8, d=128, T=8192, S=96, rb=4, C=3.0, kk="hot", vk="randn",
             layout="heads", dtype="bf16"),
        # the plugin interface on a prompt, and on the token of a decode step
        dict(name="fakequant_1x4k", kind="fakequant", B=1, Hq=32, Hkv=8, d=128, T=4096, S=24, rb=3, C=3.0, kk="hot", vk="randn",
             layout="heads", dtype="fp16"),
        dict(name="fakequant_16x1", kind="fakequant", B=16, Hq=32, Hkv=8, d=128, T=1, S=96, rb=4, C=3.0, kk="hot", vk="randn",
             layout="tokens", dtype="bf16"),
        # the drop-in attention call on the packed tuple: a decode query over 16 k tokens, a causal prompt of 2048
        dict(name="tuple_decode_1x16k", kind="tuple", B=1, Hq=32, Hkv=8, d=128, T=16384, Tq=1, S=192, rb=6, C=0.0, kk="randn",
             vk="randn", dtype="fp16"),
        dict(name="tuple_prefill_2k", kind="tuple", B=1, Hq=32, Hkv=8, d=128, T=2048, Tq=2048, S=192, rb=6, C=0.0, kk="randn",
             vk="randn", dtype="fp16"),
    ]


def _log_int(rng, lo, hi):
    hi = max(lo, int(hi))
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "prefill", "generate", "encode", "fakequant", "tuple"))
    Hq, Hkv, d = rng.choice(HEADS)
    S, rb = rng.choice(CODEBOOKS if d == 128 else CODEBOOKS[1:2])
    # (four hot or two heavy-tailed channels are a configuration of head dim 128: at 64 they would flag most chunks)
    kk, vk = rng.choice((("hot", "randn"), ("student", "randn"), ("spiky", "spiky")) if d == 128 else
                        (("onehot", "onehot"), ("spiky", "spiky")))
    C = rng.choice((3.0, 3.0, 0.0))
    if C == 0.0:
        kk = vk = "randn"
    c = dict(kind=kind, Hq=Hq, Hkv=Hkv, d=d, S=S, rb=rb, C=C, kk=kk, vk=vk, dtype=rng.choice(("bf16", "bf16", "fp16")))
    row = Hkv * d
    if kind == "decode":
        c["B"] = _log_int(rng, 1, 64)
        c["T"] = _log_int(rng, 200, min(131072, 500_000_000 // (c["B"] * row)))
        c["window"] = 128 if rng.random() < 0.2 else 0
    elif kind == "prefill":
        c["B"] = _log_int(rng, 1, 4)
        c["Tq"] = _log_int(rng, 16, 2048)
        c["T"] = _log_int(rng, c["Tq"], min(32768, 130_000_000 // (c["B"] * Hkv * c["Tq"])))
        c["window"] = 128 if rng.random() < 0.2 else 0
    elif kind == "generate":
        c["B"] = _log_int(rng, 1, 16)
        c["layers"] = rng.choice((2, 4))
        c["steps"] = _log_int(rng, 4, 12)
        c["T"] = _log_int(rng, 16, min(1024, 2000 // c["B"]))
        c["window"] = rng.choice((0, 128))
        c["layout"] = rng.choice(("tokens", "heads"))
    elif kind == "encode":
        c["B"] = _log_int(rng, 1, 32)
        c["T"] = _log_int(rng, 100, 130_000_000 // (c["B"] * row))
        c["layout"] = rng.choice(("tokens", "heads"))
    elif kind == "fakequant":
        c["B"] = _log_int(rng, 1, 64)
        c["T"] = 1 if rng.random() < 0.5 else _log_int(rng, 2, 32_000_000 // (c["B"] * row))
        c["layout"] = rng.choice(("tokens", "heads"))
    else:
        c.update(C=0.0, kk="randn", vk="randn")
        c["B"] = _log_int(rng, 1, 4)
        if rng.random() < 0.5:
            c["Tq"] = 1
            c["T"] = _log_int(rng, 200, 130_000_000 // (4 * c["B"] * row))
        else:
            c["T"] = c["Tq"] = _log_int(rng, 60, min(2048, int(math.sqrt(33_000_000 / (c["B"] * Hkv)))))
    return c


def _values(kind, B, H, T, d, gen, dtype, layout="heads"):
    """Keys or values (B, H, T, d): normal, with a head's outlier channels ("hot", "onehot", "student") or single spikes.
    layout "tokens": the memory order is (B, T, H, d), as a model's projection leaves it."""
    x = torch.randn(B, H, T, d, generator=gen, device="cuda", dtype=torch.float32)

    def channels(n):
        at = torch.rand(H, d, generator=gen, device="cuda").argsort(dim=1)[:, :n]          # n channels of every head
        return torch.zeros(H, d, device="cuda").scatter_(1, at, 1.0).bool().view(1, H, 1, d)

    if kind == "hot":
        x *= torch.where(channels(4), 8.0, 1.0)
    elif kind == "onehot":
        size = torch.exp(torch.rand(1, H, 1, 1, generator=gen, device="cuda") * math.log(200.0))
        x *= torch.where(channels(1), size, torch.ones_like(size))
    elif kind == "student":                                                                 # t with two degrees of freedom
        heavy = 100.0 / torch.empty(B, H, T, 1, device="cuda").exponential_(1.0, generator=gen).clamp_(min=1e-6).sqrt()
        x *= torch.where(channels(2), heavy, torch.ones_like(heavy))
    elif kind == "spiky":
        spike = torch.rand(B, H, T, d // 4, 1, generator=gen, device="cuda") < 0.005
        x = (x.view(B, H, T, d // 4, 4) * torch.where(spike, 20.0, 1.0)).view(B, H, T, d)
    x = x.to(dtype)
    return x.transpose(1, 2).contiguous().transpose(1, 2) if layout == "tokens" else x


def _quantizer(c, layers=1):
    q = hqmq.HQMQ(n_layers=layers, n_heads=c["Hkv"], secondary_size=c["S"], radius_bits=c["rb"], device="cuda")
    for layer in range(layers):
        for kv in (0, 1):
            q.tables(layer, kv, "cuda")                                                     # codebook tables: laid out once
    return hqmq.with_outlier_extraction(q, C=c["C"]) if c["C"] else q


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    dt, B, Hq, Hkv, d, T = DTYPES[c["dtype"]], c["B"], c["Hq"], c["Hkv"], c["d"], c["T"]
    s = {"case": c, "q": _quantizer(c, c.get("layers", 1))}

    def queries(n):
        return (torch.randn(B, Hq, n, d, generator=gen, device="cuda") / math.sqrt(d)).to(dt)

    if c["kind"] in ("decode", "prefill"):
        s["cache"] = hqmq.PackedKVCache(s["q"], max_tokens=T, sliding_window={0: c["window"]} if c["window"] else None)
        k = _values(c["kk"], B, Hkv, T, d, gen, dt)
        v = _values(c["vk"], B, Hkv, T, d, gen, dt)
        s["cache"].update(k, v, 0)
        s["Q"] = queries(c.get("Tq", 1))
    elif c["kind"] == "generate":
        def step(n):
            return (_values(c["kk"], B, Hkv, n, d, gen, dt, c["layout"]), _values(c["vk"], B, Hkv, n, d, gen, dt, c["layout"]),
                    queries(n))
        s["steps"] = [[step(n) for _ in range(c["layers"])] for n in [T] + [1] * c["steps"]]
    elif c["kind"] in ("encode", "fakequant"):
        s["K"] = _values(c["kk"], B, Hkv, T, d, gen, dt, c["layout"])
        s["V"] = _values(c["vk"], B, Hkv, T, d, gen, dt, c["layout"])
    else:
        def packed(kind, kv):
            idx, rq, rs, _ = s["q"].encode(_values(kind, B, Hkv, T, d, gen, dt), 0, kv).to_reference()
            return idx, rq, rs.to(dt), s["q"].tables(0, kv, "cuda")["joint"].to(dt)
        s["args"] = (queries(c["Tq"]), *packed(c["kk"], 0), *packed(c["vk"], 1), (1 << c["rb"]) - 1)
    return s


def _planes(pk, kind):
    """What an encode call wrote: the rows of the T tokens, and of the outliers' values the entries every head has."""
    held = int(FLAGGED_LEAST[kind] * pk.T * pk.n_chunks)
    rows = (pk.B, pk.H, pk.T_cap)
    out = [pk.codes[:pk.B * pk.H * pk.T_cap * pk.row_bytes].view(*rows, pk.row_bytes)[:, :, :pk.T],
           pk.rs[:pk.B * pk.H * pk.T_cap].view(rows)[:, :, :pk.T]]
    if pk.with_outliers:
        out += [pk.flags[:pk.B * pk.H * pk.T_cap].view(rows)[:, :, :pk.T], pk.out_count,
                pk.out_off.view(pk.B, pk.H, -1)[:, :, :(pk.T + 15) // 16 + 1],
                pk.out_vals[:pk.B * pk.H * pk.out_cap * 4].view(pk.B, pk.H, pk.out_cap, 4)[:, :, :held]]
    return out


def run(s):
    c = s["case"]
    if c["kind"] in ("decode", "prefill"):
        return s["cache"].attend(s["Q"], 0)
    if c["kind"] == "generate":
        windows = {layer: c["window"] for layer in range(1, c["layers"], 2)} if c["window"] else None
        cache = hqmq.PackedKVCache(s["q"], max_tokens=c["T"] + c["steps"], sliding_window=windows)
        out = []
        for step in s["steps"]:
            for layer, (k, v, query) in enumerate(step):
                cache.update(k, v, layer)
                out.append(cache.attend(query, layer))
        return out
    if c["kind"] == "encode":
        q = getattr(s["q"], "inner", s["q"])
        k = q.encode(s["K"], 0, 0, median_mult=c["C"] or None)
        v = q.encode(s["V"], 0, 1, median_mult=c["C"] or None)
        return _planes(k, c["kk"]), _planes(v, c["vk"])
    if c["kind"] == "fakequant":
        return s["q"].quantize_K(s["K"], 0), s["q"].quantize_V(s["V"], 0)
    return hqmq.fused_attention(*s["args"], causal=c["Tq"] > 1)


def _packed_bytes(c, tokens):
    """Compressed bytes of the keys and values of so many tokens of one sequence."""
    n = c["d"] // 4
    per = 2 * (n * (math.ceil(math.log2(24 * c["S"])) + c["rb"]) / 8 + 2)
    if c["C"]:
        per += 2 * n / 8 + 8 * n * (FLAGGED[c["kk"]] + FLAGGED[c["vk"]])
    return c["Hkv"] * tokens * per


def _attend_work(c, Tq, T, window):
    """(keys read, query-key pairs) of Tq queries that are the last positions of T keys."""
    span = window or T
    pairs = sum(min(T - Tq + i + 1, span) for i in range(Tq))
    return min(T, span + Tq - 1), pairs


def work(case):
    c = case
    B, Hq, Hkv, d, T = c["B"], c["Hq"], c["Hkv"], c["d"], c["T"]
    if c["kind"] in ("decode", "prefill"):
        Tq = c.get("Tq", 1)
        keys, pairs = _attend_work(c, Tq, T, c["window"])
        return {"bytes": B * (_packed_bytes(c, keys) + 4 * Hq * Tq * d), "flops": 4 * B * Hq * d * pairs}
    if c["kind"] == "generate":
        total = {"bytes": 0.0, "flops": 0.0}
        for layer in range(c["layers"]):
            window = c["window"] if layer % 2 else 0
            for n, held in [(T, T)] + [(1, T + i + 1) for i in range(c["steps"])]:
                keys, pairs = _attend_work(c, n, held, window)
                total["bytes"] += B * (4 * Hkv * n * d + _packed_bytes(c, n) + (_packed_bytes(c, keys) if n == 1 else 0)
                                       + 4 * Hq * n * d)
                total["flops"] += B * (4 * Hq * d * pairs + 40 * Hkv * n * d)
        return total
    if c["kind"] == "encode":
        return {"bytes": B * (4 * Hkv * T * d + _packed_bytes(c, T)), "flops": 40 * B * Hkv * T * d}
    if c["kind"] == "fakequant":
        return {"bytes": 8 * B * Hkv * T * d, "flops": 44 * B * Hkv * T * d}
    pairs = sum(i + 1 for i in range(T)) if c["Tq"] > 1 else T
    return {"bytes": B * (2 * Hkv * T * (8 * d // 4 + 2) + 4 * Hq * c["Tq"] * d), "flops": 4 * B * Hq * d * pairs}


def tolerance(case):
    # the codes, scales, flags and the dense values rebuilt from them are defined bit by bit; attention is a sum over 16-bit
    # weights and values, rounded to a 16-bit output
    if case["kind"] in ("encode", "fakequant"):
        return "exact"
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 3e-3}
