"""Attention of many query positions (tensor-core path) against a plain fp32 evaluation of the same operation on the
dense reconstruction: edges of the 128-token tiles and of the row blocks, ragged groups, every mask, units cut between CTAs."""
import math
import os
import subprocess
import sys

import pytest
import torch

import hqmq_b200 as hqmq
from hqmq_b200 import _lib, kernels
from tests.util import make_kv, rel_l2

pytestmark = pytest.mark.gpu


def _dense_attention(Q, K, V, causal, window):
    """fp32 softmax(scale Q K^T + mask) V and softmax(..) |V|; causal as fused_attention_packed takes it; rows that see no key
    are zero."""
    B, Hq, Tq, d = Q.shape
    T, G = K.shape[2], Hq // K.shape[1]
    K, V = K.float().repeat_interleave(G, 1), V.float().repeat_interleave(G, 1)
    i, t = torch.arange(Tq, device=Q.device)[:, None], torch.arange(T, device=Q.device)[None, :]
    end = (i + 1).clamp(max=T) if causal is True else (T - Tq + i + 1).clamp(min=0) if causal == "bottom_right" else torch.full_like(i, T)
    ok = (t < end) & (t >= (end - window if window else torch.zeros_like(end)))
    s = (Q.half().float() @ K.transpose(-1, -2)) / math.sqrt(d)
    p = torch.softmax(s.masked_fill(~ok, float("-inf")), -1).nan_to_num(0.0)
    return p @ V, p @ V.abs()


def _check(got, want):
    """2e-3 max-abs where the values that a row averages are about 1 in size, 1e-3 relative L2.  A value is an fp16 codeword times
    an fp16 product, two roundings of 2^-11: rows that see a few keys of a spike's size are off by that share of what they average."""
    want, size = want
    assert ((got - want).abs() <= 1e-3 + size * 2.0 ** -10).all() and rel_l2(got, want) < 1e-3


@pytest.mark.parametrize("B,Hq,Hkv,d,T,Tq,causal,window", [
    (1, 32, 8, 128, 1024, 16, "bottom_right", None),     # one stream, units over many CTAs
    (2, 8, 2, 128, 700, 33, "bottom_right", None),       # the second stream holds one position
    (1, 14, 2, 128, 519, 37, "bottom_right", None),      # seven heads per group: 18 positions in 126 rows
    (2, 16, 2, 64, 129, 129, "bottom_right", None),      # a prompt from empty, one key in the last tile
    (1, 8, 1, 64, 128, 100, False, None),                # no mask, exactly one tile
    (1, 32, 8, 128, 3000, 200, "bottom_right", 128),     # window: early tiles untouched
    (3, 8, 2, 64, 640, 40, False, 77),
    (1, 16, 1, 128, 300, 20, True, None),                # sixteen heads per group, top-left mask
    (1, 4, 2, 128, 40, 64, "bottom_right", None),        # more queries than keys: the first rows see nothing
])
@pytest.mark.parametrize("outliers", [True, False])
def test_packed_prompt_attention(B, Hq, Hkv, d, T, Tq, causal, window, outliers):
    S, br = (96, 4) if d == 64 or outliers else (192, 6)
    q = hqmq.HQMQ(1, Hkv, S, br, device="cuda")
    K = make_kv("hot" if d == 128 and outliers else "spiky", (B, Hkv, T, d), seed=81, dtype=torch.bfloat16).cuda()
    V = make_kv("spiky", (B, Hkv, T, d), seed=82, dtype=torch.bfloat16).cuda()
    mult = 3.0 if outliers else None
    Kp, Vp = q.encode(K, 0, 0, median_mult=mult), q.encode(V, 0, 1, median_mult=mult)
    tk, tv = q.tables(0, 0, "cuda"), q.tables(0, 1, "cuda")
    Q = (torch.randn(B, Hq, Tq, d, generator=torch.Generator().manual_seed(83)) / math.sqrt(d)).bfloat16().cuda()
    want = _dense_attention(Q, q.decode(Kp, 0, 0), q.decode(Vp, 0, 1), causal, window)
    O = torch.empty(Q.shape, dtype=torch.float32, device="cuda")
    hqmq.fused_attention_packed(Q, Kp, Vp, tk["table16"], tv["table16"], causal=causal, window=window, out=O)
    _check(O, want)
    # the 16-bit output of a strided query tensor is that result rounded once
    Qs = Q.transpose(1, 2).contiguous().transpose(1, 2)
    O16 = hqmq.fused_attention_packed(Qs, Kp, Vp, tk["table16"], tv["table16"], causal=causal, window=window)
    assert torch.equal(O16, O.bfloat16())


@pytest.mark.parametrize("Hq,Hkv,d,T,Tq,causal", [(32, 8, 128, 257, 257, True), (7, 1, 64, 127, 127, True), (8, 2, 128, 390, 50, False)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_tuple_prompt_attention(Hq, Hkv, d, T, Tq, causal, dtype):
    q = hqmq.HQMQ(1, Hkv, 192, 6, device="cuda")
    args, dense = [], []
    for kv in (0, 1):
        idx, rq, rs, _ = q.encode(make_kv("randn", (1, Hkv, T, d), seed=84 + kv, dtype=torch.bfloat16).cuda(), 0, kv).to_reference()
        args += [idx, rq, rs.to(dtype), q.tables(0, kv, "cuda")["joint"].to(dtype)]
        dense.append(kernels.decode_dequant(idx, rq, args[-2].float(), args[-1].float(), 63))
    Q = (torch.randn(1, Hq, Tq, d, generator=torch.Generator().manual_seed(86)) / math.sqrt(d)).to(dtype).cuda()
    O = torch.empty(Q.shape, dtype=torch.float32, device="cuda")
    hqmq.fused_attention(Q, *args, 63, causal=causal, out=O)
    _check(O, _dense_attention(Q, *dense, causal, None))


@pytest.mark.parametrize("scale_dtype,G", [(torch.bfloat16, 4), (torch.float32, 4), (torch.bfloat16, 16)])
def test_prompt_keeps_fp32_outliers(scale_dtype, G):
    """Outliers kept in fp32 (without fp16 records) weigh into scores and sums in fp32 whatever the number of query positions.
    The keys differ by about 1 around 1000 in a flagged chunk: rounding them to 11 bits moves the scores by 2e-2."""
    B, Hkv, T, Tq, d = 1, 2, 1100, 70, 128
    g = torch.Generator().manual_seed(87)
    K, V = torch.randn(B, Hkv, T, d, generator=g), torch.randn(B, Hkv, T, d, generator=g)
    K[..., :4] += 1000.0
    V[..., 20:24] *= 50.0
    q = hqmq.HQMQ(1, Hkv, 96, 4, device="cuda")
    Kp, Vp = (q.encode(x.cuda(), 0, kv, median_mult=3.0, scale_dtype=scale_dtype, ofrag=False) for kv, x in ((0, K), (1, V)))
    assert Kp.out_dtype == torch.float32 and Kp.n_outliers() >= B * Hkv * T
    Q = torch.randn(B, Hkv * G, Tq, d, generator=g).half().float().cuda()
    O = torch.empty(Q.shape, dtype=torch.float32, device="cuda")
    hqmq.fused_attention_packed(Q, Kp, Vp, q.tables(0, 0, "cuda")["table16"], q.tables(0, 1, "cuda")["table16"], causal=True, out=O)
    Kd, Vd = (q.decode(pk, 0, kv).double().repeat_interleave(G, 1) for kv, pk in ((0, Kp), (1, Vp)))
    s = Q.double() @ Kd.transpose(-1, -2) / math.sqrt(d)
    want = torch.softmax(s.masked_fill(~torch.ones(Tq, T, dtype=torch.bool, device="cuda").tril(), float("-inf")), -1) @ Vd
    assert rel_l2(O, want) < 1e-3
    if scale_dtype == torch.bfloat16 and G == 4:
        # the first position returns its one key's values; of a flagged chunk all 24 bits but the roundings of P x / P
        x = V[:, :, 0, 20:24].repeat_interleave(G, 1).cuda()
        assert ((O[:, :, 0, 20:24] - x).abs() <= 2e-6 * x.abs()).all()


@pytest.mark.parametrize("Tq", [1, 100])
def test_repeated_calls_pass_the_workspace_that_their_key_count_needs(Tq, monkeypatch):
    """One call shape over a growing cache, a key at a time: the cut of the work changes with single keys."""
    L, Hkv = _lib.lib(), 8
    q = hqmq.HQMQ(1, Hkv, 96, 4, device="cuda")
    Kp, Vp = (q.encode(make_kv("randn", (1, Hkv, 1700, 128), seed=88 + kv, dtype=torch.bfloat16).cuda(), 0, kv) for kv in (0, 1))
    tk, tv = q.tables(0, 0, "cuda")["table16"], q.tables(0, 1, "cuda")["table16"]
    Q = torch.randn(1, 32, Tq, 128, device="cuda").bfloat16()
    short, real = [], L.hqmq_attn_decode

    def attn_decode(a, ws, nbytes, st):
        if nbytes < L.hqmq_attn_workspace_bytes(a):
            short.append(T)
        return real(a, ws, nbytes, st)
    monkeypatch.setattr(L, "hqmq_attn_decode", attn_decode)
    for T in list(range(1520, 1700)) + [1600, 1100, 1023, 1024]:
        hqmq.fused_attention_packed(Q, Kp, Vp, tk, tv, causal="bottom_right", T_kv=T)
    assert not short


def test_prompt_calls_leave_no_workspace_behind():
    """A cache that exists to save memory holds no dense copy of itself after a prompt attended over it."""
    q = hqmq.HQMQ(1, 8, 96, 4, device="cuda")
    Kp, Vp = (q.encode(make_kv("randn", (1, 8, 4096, 128), seed=88 + kv, dtype=torch.bfloat16).cuda(), 0, kv) for kv in (0, 1))
    tk, tv = q.tables(0, 0, "cuda")["table16"], q.tables(0, 1, "cuda")["table16"]
    for Tq in (200, 300, 200):
        Q = (torch.randn(1, 32, Tq, 128, device="cuda") / 11).bfloat16()
        O = [torch.empty_like(Q), torch.empty_like(Q)]
        before = torch.cuda.memory_allocated()
        for out in O:
            hqmq.fused_attention_packed(Q, Kp, Vp, tk, tv, causal=False, out=out)
        assert torch.cuda.memory_allocated() - before < 1 << 20 and torch.equal(*O)


@pytest.mark.parametrize("form", ["native", torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shift", [0, 4])
def test_tables_of_every_alignment(form, shift):
    """Codeword tables 16 bytes aligned are copied in one piece, others (4 elements further on) entry by entry; T ends inside a tile
    and inside the tiles of one CTA."""
    Hq, Hkv, d, T, Tq = 8, 2, 128, 1100, 40
    q = hqmq.HQMQ(1, Hkv, 24, 3, device="cuda")

    def moved(t):
        room = torch.empty(t.numel() + 8, dtype=t.dtype, device="cuda")
        out = room[shift:shift + t.numel()].view(t.shape).copy_(t)
        assert (out.data_ptr() % 16 != 0) == (shift * t.element_size() % 16 != 0)
        return out

    Q = (torch.randn(1, Hq, Tq, d, generator=torch.Generator().manual_seed(87)) / math.sqrt(d)).half().cuda()
    O = torch.empty(Q.shape, dtype=torch.float32, device="cuda")
    packed = [q.encode(make_kv("randn", (1, Hkv, T, d), seed=88 + kv, dtype=torch.bfloat16).cuda(), 0, kv) for kv in (0, 1)]
    if form == "native":
        dense = [q.decode(pk, 0, kv) for kv, pk in enumerate(packed)]
        tabs = [moved(q.tables(0, kv, "cuda")["table16"]) for kv in (0, 1)]
        hqmq.fused_attention_packed(Q, *packed, *tabs, causal="bottom_right", out=O)
        causal = "bottom_right"
    else:
        args, dense, causal = [], [], False
        for kv, pk in enumerate(packed):
            idx, rq, rs, _ = pk.to_reference()
            args += [idx, rq, rs.to(form), moved(q.tables(0, kv, "cuda")["joint"].to(form))]
            dense.append(kernels.decode_dequant(idx, rq, args[-2].float(), args[-1].float(), 7))
        hqmq.fused_attention(Q, *args, 7, causal=False, out=O)
    _check(O, _dense_attention(Q, *dense, causal, None))


@pytest.mark.parametrize("d,Tq,window", [(128, 70, None), (64, 33, 50)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_queries_and_outputs_of_any_stride(d, Tq, window, dtype):
    """Rows that are 16 bytes aligned are read and written 16 bytes at a time, others an element at a time: same bits.  Seven heads
    to a group (rows of a block without a query), positions that end inside a stream, masks inside 32-key groups at both ends."""
    Hq, Hkv, T = 14, 2, 333
    q = hqmq.HQMQ(1, Hkv, 96, 4, device="cuda")
    packed = [q.encode(make_kv("spiky", (2, Hkv, T, d), seed=91 + kv, dtype=torch.bfloat16).cuda(), 0, kv, median_mult=3.0) for kv in (0, 1)]
    tabs = [q.tables(0, kv, "cuda")["table16"] for kv in (0, 1)]
    Q = (torch.randn(2, Hq, Tq, d, generator=torch.Generator().manual_seed(93)) / math.sqrt(d)).to(dtype).cuda()
    want = torch.empty_like(Q)
    hqmq.fused_attention_packed(Q, *packed, *tabs, causal="bottom_right", window=window, out=want)
    odd = torch.zeros(2, Hq, Tq, d + 4, dtype=dtype, device="cuda")
    Qo, O = odd[..., 4:].copy_(Q), torch.zeros(2, Hq, Tq, d + 4, dtype=dtype, device="cuda")
    hqmq.fused_attention_packed(Qo, *packed, *tabs, causal="bottom_right", window=window, out=O[..., :d])
    assert torch.equal(O[..., :d], want) and not O[..., d:].any()
    O32 = torch.empty(Q.shape, dtype=torch.float32, device="cuda")
    hqmq.fused_attention_packed(Qo, *packed, *tabs, causal="bottom_right", window=window, out=O32)
    _check(O32, _dense_attention(Q, q.decode(packed[0], 0, 0), q.decode(packed[1], 0, 1), "bottom_right", window))


@pytest.mark.parametrize("B,Hq,Hkv,d,T", [(32, 32, 8, 128, 80), (64, 64, 8, 64, 80), (40, 32, 8, 128, 96), (24, 14, 2, 128, 128)])
@pytest.mark.parametrize("causal", ["bottom_right", False])
def test_many_prompts_of_one_tile(B, Hq, Hkv, d, T, causal):
    """A batch of prompts with all keys in one tile: several units to a CTA, and in the last row block of each a second stream that
    holds no query (or few), which is through with a unit before the first stream has loaded its queries.  Queries 16 bytes at a time,
    in fp32 and at odd addresses (an element at a time, the slowest load)."""
    q = hqmq.HQMQ(1, Hkv, 96, 4, device="cuda")
    packed = [q.encode(make_kv("spiky", (B, Hkv, T, d), seed=94 + kv, dtype=torch.bfloat16).cuda(), 0, kv, median_mult=3.0) for kv in (0, 1)]
    tabs = [q.tables(0, kv, "cuda")["table16"] for kv in (0, 1)]
    Q = (torch.randn(B, Hq, T, d, generator=torch.Generator().manual_seed(96)) / math.sqrt(d)).half().cuda()
    O = torch.full(Q.shape, float("nan"), device="cuda")
    hqmq.fused_attention_packed(Q, *packed, *tabs, causal=causal, out=O)
    _check(O, _dense_attention(Q, q.decode(packed[0], 0, 0), q.decode(packed[1], 0, 1), causal, None))
    odd = torch.zeros(B, Hq, T, d + 4, dtype=Q.dtype, device="cuda")[..., 4:].copy_(Q)
    for queries in (Q.float(), odd):
        same = torch.full_like(O, float("nan"))
        hqmq.fused_attention_packed(queries, *packed, *tabs, causal=causal, out=same)
        assert torch.equal(same, O)


_LOST_CALL = '''
import torch
import hqmq_b200 as hqmq
from hqmq_b200 import _lib
L, calls, lost = _lib.lib(), 0, 0
real = L.hqmq_attn_decode
def attn_decode(a, ws, nbytes, st):
    # the calls of a process are numbered from 0x5eed0001
    global calls
    calls += 1
    held = torch.zeros((nbytes + 3) // 4, dtype=torch.int32, device="cuda")
    held[0] = 0x5eed0000 + calls - 1 + lost
    return real(a, held.data_ptr(), nbytes, st)
L.hqmq_attn_decode = attn_decode
for B, Hq, T, Tq in ((2, 4, 80, 80), (20, 32, 300, 40), (1, 8, 3000, 64)):
    q = hqmq.HQMQ(1, 2, 96, 4, device="cuda")
    packed = [q.encode(torch.randn(B, 2, T, 128, device="cuda").bfloat16(), 0, kv) for kv in (0, 1)]
    tabs = [q.tables(0, kv, "cuda")["table16"] for kv in (0, 1)]
    for lost in (1, 0):
        O = hqmq.fused_attention_packed(torch.randn(B, Hq, Tq, 128, device="cuda").half(), *packed, *tabs, causal="bottom_right")
        assert (O.isnan() if lost else O.isfinite()).all(), (B, T, lost)
'''


def test_call_whose_expansion_gave_up_is_all_nan():
    """The status word of a call, raised ahead of the attention kernel as the expansion does when it goes on without a codeword
    table: every row is NaN, of units that one CTA does whole and of those that are merged.  The word of another call does nothing."""
    subprocess.run([sys.executable, "-c", _LOST_CALL], check=True, timeout=300, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
