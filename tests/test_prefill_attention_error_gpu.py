"""What prompt attention over a bf16 cache is off by, beyond the rounding of its result: the weights are rounded to bf16 relative to the largest one so far and
divided by the sum of the rounded ones, so that attention on few keys loses next to nothing by them. Against float64: the norm of the error is held to 1.06 of
the result's own rounding where the scores are wide (1.04 seen; 1.28 with weights relative to a reference that lags) and to 1.41 where they are not (1.38 seen)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,bound", [(4.0, 1.06), (1.0, 1.41)])
@pytest.mark.parametrize("T,pos0,heads,kv_heads,hd", [(512, 3000, 16, 4, 128), (1024, 1234, 32, 4, 64)])
def test_error_against_the_rounding_of_the_result(T, pos0, heads, kv_heads, hd, scale, bound):
    import torch

    from simplellminference_b200 import kernels as K
    g = torch.Generator(device="cuda").manual_seed(T)
    n = pos0 + T
    q = (scale * torch.randn(T, heads * hd, device="cuda", generator=g)).to(torch.bfloat16)
    k, v = (torch.randn(kv_heads, n, hd, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    got = K.prefill_attention(q, k, v, pos0, heads, kv_heads).double().view(T, heads, hd)
    hidden = torch.arange(n, device="cuda")[None] > (pos0 + torch.arange(T, device="cuda"))[:, None]
    off = rounding = 0.0
    for h in range(heads):
        s = (q.view(T, heads, hd)[:, h].double() @ k[h // (heads // kv_heads)].double().T) / hd ** 0.5
        want = torch.softmax(s.masked_fill(hidden, float("-inf")), -1) @ v[h // (heads // kv_heads)].double()
        off += float((got[:, h] - want).square().sum())
        rounding += float((want.to(torch.bfloat16).double() - want).square().sum())
    assert off ** 0.5 < bound * rounding ** 0.5
