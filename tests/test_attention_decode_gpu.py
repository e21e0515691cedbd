"""Attention of single-token steps (sllm_seq_attention / sllm_seq_attention_out with one query per sequence): over fp32 pools in the body that reads them straight
into registers, over bf16 pools in the one whose tensor-core products take three bf16 terms. Contexts that end anywhere in a run, a tile or a page, every number
of query heads a CTA can hold, every way in which a score can be changed or hidden, shares merged by the caller and results written by the launch. Cache rows
beyond a context hold NaN. Against float64 on the same operands; fp32 sums over at most 3000 keys stay within 2e-6."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PAGE = 64


def _case(lens, heads, kv_heads, dim, dtype, seed):
    import torch

    from simplellminference_b200._lib import SeqBatch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n, held = len(lens), [-(-x // PAGE) for x in lens]
    pages = torch.randperm(sum(held) + 3, generator=torch.Generator().manual_seed(seed)).tolist()
    table, at = np.full((n, max(held)), -1, np.int32), 0
    for i, h in enumerate(held):
        table[i, :h] = pages[at:at + h]
        at += h
    q = torch.randn(n, heads * dim + 4, generator=g, device="cuda")
    k, v = (torch.full((sum(held) + 3, kv_heads, PAGE, dim), float("nan"), device="cuda", dtype=getattr(torch, dtype)) for _ in range(2))
    rows = []
    for i, x in enumerate(lens):
        ki, vi = (torch.randn(kv_heads, x, dim, generator=g, device="cuda").to(k.dtype) for _ in range(2))
        for p in range(held[i]):
            m = min(PAGE, x - p * PAGE)
            k[table[i, p], :, :m], v[table[i, p], :, :m] = ki[:, p * PAGE:p * PAGE + m], vi[:, p * PAGE:p * PAGE + m]
        rows.append((ki.double(), vi.double()))
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")   # noqa: E731
    own, zero, one, pos, tab = ints(list(range(n))), ints([0] * n), ints([1] * n), ints([x - 1 for x in lens]), torch.tensor(table, device="cuda")
    b = SeqBatch(n, n, own.data_ptr(), pos.data_ptr(), own.data_ptr(), one.data_ptr(), own.data_ptr(), pos.data_ptr(), tab.data_ptr(), tab.shape[1], PAGE, n, own.data_ptr(),
                 zero.data_ptr(), own.data_ptr())
    return q, k, v, rows, b, (own, zero, one, pos, tab)


def _want(q, rows, heads, kv_heads, dim, scale, window=0, keep_first=0, softcap=0.0, slopes=None, logdist=None, chunk=0):
    import torch
    out = []
    for i, (k, v) in enumerate(rows):
        x, pos = k.shape[1], k.shape[1] - 1
        back = pos - torch.arange(x, device="cuda")
        sees = back >= 0
        if chunk:
            sees &= back <= pos % chunk
        if window:
            sees &= (back < window) | (torch.arange(x, device="cuda") < keep_first)
        for h in range(heads):
            gk = h // (heads // kv_heads)
            s = (k[gk] @ q[i, h * dim:(h + 1) * dim].double()) * scale
            if softcap:
                s = softcap * torch.tanh(s / softcap)
            if slopes is not None:
                s = s - slopes[h].double() * back
            if logdist is not None:
                s = s - logdist[0, h].double() * torch.log1p(logdist[1, h].double() * back)
            out.append(torch.softmax(s.masked_fill(~sees, -math.inf), 0) @ v[gk])
    return torch.stack(out).view(len(rows), heads * dim)


def _run(ops, b, q, k, v, heads, kv_heads, dim, nsplit, opts, merged):
    import torch
    n, st = q.shape[0], torch.cuda.current_stream().cuda_stream
    ws, out = torch.full((n * heads * nsplit * (dim + 2),), float("nan"), device="cuda"), torch.full((n, heads * dim), float("nan"), device="cuda")
    if merged:
        ops.attention_out(b, q.data_ptr(), q.stride(0), heads, kv_heads, dim, dim, dim ** -0.5, k, v, nsplit, ws, out, heads * dim, st, opts=opts)
    else:
        ops.attention(b, q.data_ptr(), q.stride(0), heads, kv_heads, dim, dim, dim ** -0.5, k, v, nsplit, ws, st, opts=opts)
        ops.attention_finish(b, ws, nsplit, heads, dim, None, 0, None, 0, out, heads * dim, st)
    return out


@pytest.mark.parametrize("heads,kv_heads,dim", [(8, 2, 128), (6, 2, 128), (4, 2, 64), (2, 2, 128), (16, 2, 64), (3, 3, 64), (12, 2, 128)])
@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("lens", [[1], [31, 32, 33, 64, 65, 1], [2999], [700, 3, 129] * 7], ids=["one", "edges", "long", "many"])
def test_contexts_and_heads(heads, kv_heads, dim, dtype, lens):
    from simplellminference_b200.config import BF16, F32
    from simplellminference_b200.seqops import Ops
    ops = Ops(BF16 if dtype == "bfloat16" else F32)
    q, k, v, rows, b, keep = _case(lens, heads, kv_heads, dim, dtype, len(lens) + heads)
    want = _want(q, rows, heads, kv_heads, dim, dim ** -0.5)
    for nsplit, merged in ((1, False), (5, False), (3, True)):
        got = _run(ops, b, q, k, v, heads, kv_heads, dim, nsplit, None, merged).double()
        assert float((got - want).norm() / want.norm()) < 2e-6, (nsplit, merged)


@pytest.mark.parametrize("opts", [dict(window=1), dict(window=100), dict(window=40, keep_first=70), dict(softcap=2.0, window=257), dict(slopes=True), dict(logdist=True, window=300),
                                  dict(chunk=100), dict(chunk=64, softcap=5.0)], ids=str)
@pytest.mark.parametrize("heads,kv_heads", [(8, 2), (4, 2), (2, 2)])
def test_hidden_and_changed_scores(heads, kv_heads, opts):
    import torch

    from simplellminference_b200.config import BF16
    from simplellminference_b200.seqops import Ops
    ops, dim = Ops(BF16), 128
    q, k, v, rows, b, keep = _case([500, 1, 64, 101, 1000, 200], heads, kv_heads, dim, "bfloat16", 3)
    o = dict(opts)
    if "slopes" in o:
        o["slopes"] = 0.01 * torch.arange(1, heads + 1, device="cuda").float()
    if "logdist" in o:
        o["logdist"] = torch.stack([0.3 * torch.arange(heads, device="cuda").float(), torch.full((heads,), 0.1, device="cuda")]).contiguous()
    want = _want(q, rows, heads, kv_heads, dim, dim ** -0.5, **o)
    for nsplit, merged in ((4, False), (4, True)):
        got = _run(ops, b, q, k, v, heads, kv_heads, dim, nsplit, ops.attention_options(**o), merged).double()
        assert float((got - want).norm() / want.norm()) < 2e-6, merged
