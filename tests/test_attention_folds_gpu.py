"""Decode attention over bf16 pools whose clusters serve one request each or two, side by side in equal or unequal parts or in turns: requests alike, one long one among short ones, a number of items that does not fill the last
cluster, shares and results, more requests than a CTA has threads. Against float64; fp32 sums of at most 3000 keys stay within 2e-6."""
import pytest
from test_attention_decode_gpu import _case, _run, _want

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,dim", [(8, 2, 128), (3, 3, 64), (9, 3, 128), (32, 8, 64)])
@pytest.mark.parametrize("lens", [[300] * 13, [3000] + [40] * 12, [2500, 100] * 5, [257] * 2, [64] * 37, [20] * 130], ids=["alike", "one long", "two kinds", "two", "many", "130"])
def test_contexts(heads, kv_heads, dim, lens):
    from simplellminference_b200.config import BF16
    from simplellminference_b200.seqops import Ops
    ops = Ops(BF16)
    q, k, v, rows, b, keep = _case(lens, heads, kv_heads, dim, "bfloat16", len(lens) + heads)
    want = _want(q, rows, heads, kv_heads, dim, dim ** -0.5)
    for nsplit, merged in ((1, True), (3, False), (2, True)):
        got = _run(ops, b, q, k, v, heads, kv_heads, dim, nsplit, None, merged).double()
        assert float((got - want).norm() / want.norm()) < 2e-6, (nsplit, merged)


@pytest.mark.parametrize("heads,kv_heads,dim", [(32, 8, 64), (8, 8, 128)])
@pytest.mark.parametrize("lens", [[2500, 1200, 600, 300, 20], [2900, 2100] + [70] * 10, [3000, 1000] + [70] * 17, [3000] + [40] * 36, [17, 3000, 900, 40, 2000, 300, 33, 16]],
                         ids=["five", "twelve", "nineteen", "odd", "in no order"])
@pytest.mark.parametrize("window,softcap", [(0, 0.0), (700, 20.0)])
def test_pairs(heads, kv_heads, dim, lens, window, softcap):
    """Eight, four and two CTAs a pair, a request in the middle that has no partner, parts of one to seven CTAs and turns."""
    from simplellminference_b200.config import BF16
    from simplellminference_b200.seqops import Ops
    ops = Ops(BF16)
    q, k, v, rows, b, keep = _case(lens, heads, kv_heads, dim, "bfloat16", len(lens))
    want = _want(q, rows, heads, kv_heads, dim, dim ** -0.5, window=window, softcap=softcap)
    opts = ops.attention_options(window=window, softcap=softcap) if window else None
    for nsplit, merged in ((1, True), (2, False)):
        got = _run(ops, b, q, k, v, heads, kv_heads, dim, nsplit, opts, merged).double()
        assert float((got - want).norm() / want.norm()) < 2e-6, (nsplit, merged)
