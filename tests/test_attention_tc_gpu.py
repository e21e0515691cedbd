"""Attention of prompt portions on tcgen05 (sllm_seq_attention / sllm_seq_attention_out, bf16 pools): portions that end anywhere in a tile, several at once and
behind a cached context, one, two and four query heads of a kv head in a CTA, pages of other lengths than a tile, every option, shares merged by the caller
and results written by the launch, maxima that keep growing. Cache rows beyond a portion hold NaN. Against float64 on the bf16-rounded queries: the
weights keep 2^-24 (three bf16 terms), the sums of at most 1400 keys a few 2^-23 a tile; 2e-5 of the result's norm is generous (tighter:
test_attention_forms_gpu.py)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(segs, heads, kv_heads, dim, page, seed, rising):
    """segs: (first position, tokens) of each sequence."""
    import torch

    from simplellminference_b200._lib import SeqBatch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n, ends = len(segs), [p + x for p, x in segs]
    held = [-(-x // page) for x in ends]
    order = torch.randperm(sum(held) + 2, generator=torch.Generator().manual_seed(seed)).tolist()
    table, at = np.full((n, max(held)), -1, np.int32), 0
    for i, h in enumerate(held):
        table[i, :h] = order[at:at + h]
        at += h
    T = sum(x for _, x in segs)
    q = torch.randn(T, heads * dim + 4, generator=g, device="cuda")
    k, v = (torch.full((sum(held) + 2, kv_heads, page, dim), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(2))
    if rising:
        q[:, :heads * dim:dim] = 6.0
    rows = []
    for i, x in enumerate(ends):
        ki, vi = (torch.randn(kv_heads, x, dim, generator=g, device="cuda") for _ in range(2))
        if rising:
            ki[:, :, 0] = torch.linspace(0.0, 8.0 * dim ** 0.5, x, device="cuda")
        ki, vi = ki.to(k.dtype), vi.to(k.dtype)
        for p in range(held[i]):
            m = min(page, x - p * page)
            k[table[i, p], :, :m], v[table[i, p], :, :m] = ki[:, p * page:p * page + m], vi[:, p * page:p * page + m]
        rows.append((ki.double(), vi.double()))
    tiles = sorted([(i, o) for i, (_, x) in enumerate(segs) for o in range(0, x, 32)], key=lambda t: -(segs[t[0]][0] + t[1]))
    ints = lambda x: torch.tensor(np.asarray(x, np.int32), device="cuda")   # noqa: E731
    lens = [x for _, x in segs]
    keep = [ints(np.repeat(range(n), lens)), ints(np.concatenate([np.arange(p, p + x) for p, x in segs])), ints(np.cumsum([0] + lens[:-1])), ints(lens), ints(range(n)),
            ints([p for p, _ in segs]), ints(table), ints([t[0] for t in tiles]), ints([t[1] for t in tiles]), ints(np.cumsum([0] + [-(-x // 32) for x in lens[:-1]]))]
    b = SeqBatch(T, n, *[t.data_ptr() for t in keep[:6]], keep[6].data_ptr(), table.shape[1], page, len(tiles), keep[7].data_ptr(), keep[8].data_ptr(), keep[9].data_ptr())
    return q, k, v, rows, b, keep


def _want(q, rows, segs, heads, kv_heads, dim, scale, window=0, keep_first=0, softcap=0.0, slopes=None, logdist=None, chunk=0):
    import torch
    out, at = [], 0
    for (k, v), (p, n) in zip(rows, segs):
        pos = torch.arange(p, p + n, device="cuda")[:, None]
        key = torch.arange(p + n, device="cuda")[None]
        back = pos - key
        sees = back >= 0
        if chunk:
            sees = sees & (pos // chunk == key // chunk)
        if window:
            sees = sees & ((back < window) | (key < keep_first))
        o = []
        for h in range(heads):
            gk = h // (heads // kv_heads)
            s = (q[at:at + n, h * dim:(h + 1) * dim].to(torch.bfloat16).double() @ k[gk].T) * scale
            if softcap:
                s = softcap * torch.tanh(s / softcap)
            if slopes is not None:
                s = s - slopes[h].double() * back
            if logdist is not None:
                s = s - logdist[0, h].double() * torch.log1p(logdist[1, h].double() * back.clamp(min=0))
            o.append(torch.softmax(s.masked_fill(~sees, -math.inf), -1) @ v[gk])
        out.append(torch.cat(o, 1))
        at += n
    return torch.cat(out)


def _check(segs, heads, kv_heads, dim, page=64, rising=False, **o):
    segs = segs + [(3, 517)]        # a portion that makes the step large enough for this body
    import torch

    from simplellminference_b200.config import BF16
    from simplellminference_b200.seqops import Ops
    ops, T, st = Ops(BF16), sum(x for _, x in segs), torch.cuda.current_stream().cuda_stream
    q, k, v, rows, b, keep = _case(segs, heads, kv_heads, dim, page, T + heads, rising)
    if "slopes" in o:
        o["slopes"] = 0.01 * torch.arange(1, heads + 1, device="cuda").float()
    if "logdist" in o:
        o["logdist"] = torch.stack([0.3 * torch.arange(heads, device="cuda").float(), torch.full((heads,), 0.1, device="cuda")]).contiguous()
    want, opts = _want(q, rows, segs, heads, kv_heads, dim, dim ** -0.5, **o), ops.attention_options(**o)
    for nsplit in (1, 3):
        ws, out = torch.full((T * heads * nsplit * (dim + 2),), float("nan"), device="cuda"), torch.full((T, heads * dim), float("nan"), device="cuda")
        ops.attention(b, q.data_ptr(), q.stride(0), heads, kv_heads, dim, dim, dim ** -0.5, k, v, nsplit, ws, st, opts=opts)
        ops.attention_finish(b, ws, nsplit, heads, dim, None, 0, None, 0, out, heads * dim, st)
        assert float((out.double() - want).norm() / want.norm()) < 2e-5, nsplit
        out, out16 = torch.full_like(out, float("nan")), torch.full((T, heads * dim), float("nan"), device="cuda", dtype=torch.bfloat16)
        ops.attention_out(b, q.data_ptr(), q.stride(0), heads, kv_heads, dim, dim, dim ** -0.5, k, v, nsplit, ws, out, heads * dim, st, opts=opts, out16=out16)
        assert float((out.double() - want).norm() / want.norm()) < 2e-5, nsplit
        assert torch.equal(out16, out.to(torch.bfloat16))


@pytest.mark.parametrize("heads,kv_heads,dim,page", [(8, 2, 128, 64), (6, 3, 128, 32), (3, 3, 64, 64), (16, 2, 64, 96), (5, 1, 128, 128)])
@pytest.mark.parametrize("segs", [[(0, 2)], [(0, 64), (0, 65), (31, 33)], [(0, 700)], [(1000, 130), (5, 1), (0, 31), (64, 257)]], ids=str)
def test_portions_and_heads(heads, kv_heads, dim, page, segs):
    _check(segs, heads, kv_heads, dim, page)


@pytest.mark.parametrize("o", [dict(window=1), dict(window=100), dict(window=40, keep_first=70), dict(softcap=2.0, window=257), dict(slopes=True), dict(logdist=True, window=300), dict(chunk=100),
                               dict(chunk=64, softcap=5.0)], ids=str)
@pytest.mark.parametrize("heads,kv_heads", [(8, 2), (4, 2), (2, 2)])
def test_options(heads, kv_heads, o):
    _check([(0, 500), (130, 333), (700, 40)], heads, kv_heads, 128, **o)


@pytest.mark.parametrize("dim", [64, 128])
def test_maxima_that_keep_growing(dim):
    _check([(0, 900), (300, 200)], 4, 1, dim, rising=True)
