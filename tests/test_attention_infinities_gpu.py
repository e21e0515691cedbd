"""Infinite values in a bf16 cache while decoding."""
import math

import pytest
from test_attention_forms_gpu import _close, _inputs, _ops, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,dim", [(8, 2, 128), (3, 3, 64)])
def test_infinite_cache_values_while_decoding(heads, kv_heads, dim):
    """An infinite value comes out infinite with its sign and a key whose score is -inf is not seen, as fp32 products give it."""
    import torch
    n, ops = 900, _ops()
    segs = [(n - 1, 1), (300, 1)]
    q, k, v, rows, b, keep = _inputs(segs, heads, kv_heads, dim, 64)
    q = q + 2.0 ** -13 * torch.rand(q.shape, device="cuda")        # second and third terms in the queries too
    table = keep[6]
    group = heads // kv_heads
    at = lambda pool, g, pos: pool[table[0, pos // 64], g, pos % 64]   # noqa: E731
    at(v, 0, 17)[3], at(v, 0, 640)[5] = math.inf, -math.inf
    rows[0][1][0, 17, 3], rows[0][1][0, 640, 5] = math.inf, -math.inf
    h = (kv_heads - 1) * group           # first query head of the last kv head: a key it sees at -inf, the others of the group at whatever comes of it
    at(k, kv_heads - 1, 33)[0] = -math.inf
    q[0, h * dim:(h + group) * dim:dim] = 1.0 + 2.0 ** -10 + 2.0 ** -20
    got = _run(ops, b, q, k, v, heads, kv_heads, dim, None)
    rows[0][0][kv_heads - 1, 33, 0] = -math.inf
    for i in range(2):
        for hh in range(heads):
            s = rows[i][0][hh // group] @ q[i, hh * dim:(hh + 1) * dim].double() * dim ** -0.5
            want, have = torch.softmax(s, 0) @ rows[i][1][hh // group], got[i, hh * dim:(hh + 1) * dim].double()
            fine = torch.isfinite(want)
            assert torch.equal(torch.where(fine, 0.0, want), torch.where(fine, 0.0, have)), (i, hh)
            assert _close(have[fine], want[fine], 5e-6), (i, hh)
