"""What the attention bodies for heads of 64 and 128 accept beyond the usual: pages of other lengths than the tiles, changed scores with heads of 64, query rows
that do not start at a multiple of 16 bytes, and how far off sums over long contexts are. Against float64 on bf16-exact queries. Single tokens: fp32 sums, 2e-6.
Portions: weights to 2^-24, exponentials and their arguments to 5e-7; the tensor core truncates a sum by up to 2^-23 per product it adds, 12 tiles of 12 products
at most before it is rounded into fp32, on average half of that from a sum half as large: 4e-6."""
import math

import numpy as np
import pytest
from test_attention_tc_gpu import _case, _want

pytestmark = pytest.mark.gpu

OPTIONS = [dict(window=100), dict(window=40, keep_first=70), dict(softcap=2.0, window=257), dict(slopes=True), dict(logdist=True), dict(chunk=100)]


def _options(o, heads):
    import torch
    o = dict(o)
    if "slopes" in o:
        o["slopes"] = 0.01 * torch.arange(1, heads + 1, device="cuda").float()
    if "logdist" in o:
        o["logdist"] = torch.stack([0.3 * torch.arange(heads, device="cuda").float(), torch.full((heads,), 0.1, device="cuda")]).contiguous()
    return o


def _ops():
    from simplellminference_b200.config import BF16
    from simplellminference_b200.seqops import Ops
    return Ops(BF16)


def _inputs(segs, heads, kv_heads, dim, page):
    """As the other file's, with queries that bf16 holds exactly."""
    import torch
    q, k, v, rows, b, keep = _case(segs, heads, kv_heads, dim, page, heads + len(segs), False)
    return q.to(torch.bfloat16).float(), k, v, rows, b, keep


def _run(ops, b, q, k, v, heads, kv_heads, dim, opts, ldq=None, offset=0, nsplit=2):
    import torch
    T = q.shape[0]
    ws, out = torch.full((T * heads * nsplit * (dim + 2),), float("nan"), device="cuda"), torch.full((T, heads * dim), float("nan"), device="cuda")
    ops.attention_out(b, q.data_ptr() + 4 * offset, ldq or q.stride(0), heads, kv_heads, dim, dim, dim ** -0.5, k, v, nsplit, ws, out, heads * dim,
                      torch.cuda.current_stream().cuda_stream, opts=opts)
    return out


def _close(got, want, bound=2e-6):
    return float((got.double() - want).norm() / want.norm()) < bound


@pytest.mark.parametrize("o", [{}] + OPTIONS, ids=str)
@pytest.mark.parametrize("heads,kv_heads,dim,page", [(8, 2, 64, 32), (6, 2, 64, 96), (3, 3, 128, 160), (8, 2, 128, 32)])
def test_decoding_over_pages_of_other_lengths(heads, kv_heads, dim, page, o):
    segs = [(x - 1, 1) for x in (500, 1, 33, 97, 1000)]
    q, k, v, rows, b, keep = _inputs(segs, heads, kv_heads, dim, page)
    o, ops = _options(o, heads), _ops()
    assert _close(_run(ops, b, q, k, v, heads, kv_heads, dim, ops.attention_options(**o)), _want(q, rows, segs, heads, kv_heads, dim, dim ** -0.5, **o))


@pytest.mark.parametrize("o", OPTIONS, ids=str)
@pytest.mark.parametrize("heads,kv_heads,dim", [(8, 2, 64), (4, 2, 64), (3, 3, 64), (6, 3, 128)])
@pytest.mark.parametrize("offset", [0, 1], ids=["aligned", "unaligned"])
def test_portions_with_changed_scores(heads, kv_heads, dim, o, offset):
    segs = [(0, 500), (130, 333), (700, 40), (9, 1)]
    q, k, v, rows, b, keep = _inputs(segs, heads, kv_heads, dim, 64)
    o, ops = _options(o, heads), _ops()
    want = _want(q[:, offset:], rows, segs, heads, kv_heads, dim, dim ** -0.5, **o)
    assert _close(_run(ops, b, q, k, v, heads, kv_heads, dim, ops.attention_options(**o), offset=offset), want, 4e-6)


@pytest.mark.parametrize("segs,heads,kv_heads,dim", [([(6000, 256), (0, 300)], 16, 4, 128), ([(3000, 600)], 4, 4, 64), ([(5000, 1)] * 20 + [(2000, 300)], 40, 8, 128)], ids=str)
@pytest.mark.parametrize("nsplit", [1, 3])
def test_sums_over_long_contexts(segs, heads, kv_heads, dim, nsplit):
    q, k, v, rows, b, keep = _inputs(segs, heads, kv_heads, dim, 64)
    ops, want = _ops(), _want(q, rows, segs, heads, kv_heads, dim, dim ** -0.5)
    out = _run(ops, b, q, k, v, heads, kv_heads, dim, None, nsplit=nsplit)
    at = 0
    for _, n in segs:        # each portion by itself: the norms of long contexts' results are small
        assert _close(out[at:at + n], want[at:at + n], 4e-6)
        at += n


@pytest.mark.parametrize("cap", [0.5, 9.0, 14.0, 60.0])
@pytest.mark.parametrize("heads,kv_heads,dim", [(8, 2, 64), (3, 3, 128), (8, 2, 128)])
def test_portions_with_caps_near_and_far_from_the_scores(heads, kv_heads, dim, cap):
    """Scores of up to about five: all tiles beyond a quarter of the cap, some, hardly any, none (the two loops of the capped body)."""
    segs = [(0, 500), (130, 333), (700, 40)]
    q, k, v, rows, b, keep = _inputs(segs, heads, kv_heads, dim, 64)
    ops = _ops()
    want = _want(q, rows, segs, heads, kv_heads, dim, dim ** -0.5, softcap=cap)
    assert _close(_run(ops, b, q, k, v, heads, kv_heads, dim, ops.attention_options(softcap=cap)), want, 4e-6)
