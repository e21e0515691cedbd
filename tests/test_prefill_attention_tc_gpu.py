"""Causal attention of prompt portions on tcgen05 (bf16 caches): one and two query tiles per CTA, two heads of a kv head or two tiles of a head sharing it,
tiles that end anywhere, portions behind a long context, scores whose maximum keeps growing along the keys (the accumulator is rescaled) and scores
that start at their maximum. Against float64 on the same operands: weights and result are rounded to bf16 (2^-9 each), 4e-3 of the result's norm at most."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("T,pos0,heads,kv_heads", [(1, 0, 1, 1), (127, 1, 2, 2), (128, 0, 2, 1), (129, 300, 3, 1), (700, 513, 40, 40), (385, 129, 64, 32), (257, 0, 66, 22), (1100, 0, 20, 5)])
@pytest.mark.parametrize("shape", ["plain", "rising", "falling"])
def test_tiles_heads_and_rescaling(T, pos0, heads, kv_heads, hd, shape):
    import torch

    from simplellminference_b200 import kernels as K
    g = torch.Generator(device="cuda").manual_seed(T + 7 * pos0 + heads)
    n, S = pos0 + T, pos0 + T + 9
    q = torch.randn(T, heads * hd, device="cuda", generator=g)
    k, v = (torch.randn(kv_heads, S, hd, device="cuda", generator=g) for _ in range(2))
    if shape != "plain":        # a common direction that grows or shrinks along the keys: scores move by some 80 over the context
        ramp = torch.linspace(0.0, 1.0, S, device="cuda") if shape == "rising" else torch.linspace(1.0, 0.0, S, device="cuda")
        q[:, ::hd] = 10.0
        k[:, :, 0] = 8.0 * hd ** 0.5 * ramp
    q, k, v = (t.to(torch.bfloat16) for t in (q, k, v))
    k[:, n:], v[:, n:] = float("nan"), float("nan")
    got = K.prefill_attention(q, k, v, pos0, heads, kv_heads).double().view(T, heads, hd)
    hidden = torch.arange(n, device="cuda")[None] > (pos0 + torch.arange(T, device="cuda"))[:, None]
    for h in range(heads):
        kh, vh = k[h // (heads // kv_heads), :n].double(), v[h // (heads // kv_heads), :n].double()
        s = (q.view(T, heads, hd)[:, h].double() @ kh.T) / hd ** 0.5
        want = torch.softmax(s.masked_fill(hidden, float("-inf")), -1) @ vh
        assert float((got[:, h] - want).norm() / want.norm()) < 4e-3, h
