"""Decode attention of small problems (a unit per thread-block cluster, merged through distributed shared memory) against a
plain fp32 evaluation on the dense reconstruction: one to eight CTAs per unit, CTAs without a tile, warps without a tile,
one key, windows, partial results."""
import math

import pytest
import torch

import hqmq_b200 as hqmq
from tests.test_gpu_prefill import _check, _dense_attention
from tests.util import make_kv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Hq,Hkv,d,T,Tq,window", [
    (1, 4, 1, 128, 1, 1, None),            # one key
    (1, 8, 8, 128, 4096, 1, None),         # eight CTAs per unit, two rounds of tiles per warp
    (1, 7, 1, 128, 4095, 1, None),
    (2, 8, 2, 128, 2000, 1, None),         # the last CTA of a unit has fewer tiles
    (1, 8, 1, 128, 1100, 1, None),         # 69 tiles over eight CTAs of nine: the last has six
    (4, 64, 8, 64, 513, 1, None),          # four CTAs per unit
    (3, 8, 1, 64, 777, 1, 128),            # one CTA per unit, nine tiles for sixteen warps
    (1, 16, 2, 64, 3000, 3, None),         # a few query positions
    (37, 16, 4, 64, 300, 1, None),         # 148 units
    (2, 8, 8, 128, 1900, 1, None),         # 16, 20, 29, 37 and 48 units: more than clusters of 148 / units CTAs fit at once
    (5, 8, 4, 128, 1000, 1, None),
    (29, 4, 1, 128, 700, 1, None),
    (37, 4, 1, 64, 1001, 1, None),
    (12, 8, 4, 128, 640, 1, None),
    (1, 8, 2, 128, 10239, 1, None),        # five rounds of tiles per warp, the most of a cluster, and one tile more
    (1, 8, 2, 128, 10241, 1, None),
    (1, 8, 1, 64, 4097, 1, None),          # one unit: two rounds and one tile
    (6, 16, 8, 64, 2600, 1, None),         # four rounds in clusters of three
    (1, 32, 8, 128, 7001, 1, 5001),        # a window that starts inside a tile
])
@pytest.mark.parametrize("S,br,outliers", [(96, 4, True), (96, 4, False), (24, 3, True), (192, 6, False)])
def test_small_decode(B, Hq, Hkv, d, T, Tq, window, S, br, outliers):
    if d == 64 and S != 96:
        pytest.skip("rows with padding bits take the generic kernel")
    q = hqmq.HQMQ(1, Hkv, S, br, device="cuda")
    K = make_kv("hot" if d == 128 and outliers else "spiky", (B, Hkv, T, d), seed=71, dtype=torch.bfloat16).cuda()
    V = make_kv("spiky" if outliers else "randn", (B, Hkv, T, d), seed=72, dtype=torch.bfloat16).cuda()
    mult = 3.0 if outliers else None
    Kp, Vp = q.encode(K, 0, 0, median_mult=mult), q.encode(V, 0, 1, median_mult=mult)
    tk, tv = q.tables(0, 0, "cuda")["table16"], q.tables(0, 1, "cuda")["table16"]
    Q = (torch.randn(B, Hq, Tq, d, generator=torch.Generator().manual_seed(73)) / math.sqrt(d)).bfloat16().cuda()
    causal = "bottom_right" if Tq > 1 else False
    want = _dense_attention(Q, q.decode(Kp, 0, 0), q.decode(Vp, 0, 1), causal, window)
    O = torch.empty(Q.shape, dtype=torch.float32, device="cuda")
    for _ in range(2):
        hqmq.fused_attention_packed(Q, Kp, Vp, tk, tv, causal=causal, window=window, out=O.fill_(7))
        _check(O, want)
    parts = torch.full((1, B, Hq, Tq, d + 2), float("nan"), device="cuda")
    hqmq.fused_attention_packed(Q, Kp, Vp, tk, tv, causal=causal, window=window, partials=parts[0])
    _check(hqmq.combine_partials(parts), want)


@pytest.mark.parametrize("B,Hq,Hkv,d,T,Tq,window", [
    (1, 1, 1, 128, 1, 1, None),            # one key
    (1, 28, 4, 128, 3001, 1, None),        # units cut into many CTAs, the last with fewer tiles
    (2, 16, 2, 64, 517, 3, None),
    (40, 8, 4, 64, 75, 1, None),           # more units than SMs: CTAs that hold several
    (1, 8, 2, 128, 900, 1, 333),
])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
def test_tuple_decode(B, Hq, Hkv, d, T, Tq, window, dtype):
    """The packed tuple at its usual types, and with 64-bit indices and strided planes (loaded field by field)."""
    from hqmq_b200 import kernels
    q = hqmq.HQMQ(1, Hkv, 192, 6, device="cuda")
    args, dense = [], []
    for kv in (0, 1):
        x = make_kv("randn", (B, Hkv, T, d), seed=74 + kv, dtype=torch.bfloat16).cuda()
        idx, rq, rs, _ = q.encode(x, 0, kv).to_reference()
        args += [idx, rq, rs.to(dtype), q.tables(0, kv, "cuda")["joint"].to(dtype)]
        dense.append(kernels.decode_dequant(idx, rq, args[-2].float(), args[-1].float(), 63))
    Q = (torch.randn(B, Hq, Tq, d, generator=torch.Generator().manual_seed(76)) / math.sqrt(d)).to(dtype).cuda()
    want = _dense_attention(Q, *dense, False, window)
    O, O2 = torch.empty(Q.shape, dtype=torch.float32, device="cuda"), torch.empty(Q.shape, dtype=torch.float32, device="cuda")
    for _ in range(2):
        hqmq.fused_attention(Q, *args, 63, causal=False, window=window, out=O.fill_(7))
        _check(O, want)
    args[0], args[5] = args[0].long(), args[5].transpose(1, 2).contiguous().transpose(1, 2)
    hqmq.fused_attention(Q, *args, 63, causal=False, window=window, out=O2)
    assert torch.equal(O, O2)
