"""Causal attention of prompt portions with scratch, where every CTA has an equal share of all key tiles: work items in two and in many shares, shares of several items,
shares that end in front of keys that only some queries of an item see (a row without any in that share, a whole tile without any), items whose second tile is missing. The
scratch starts as NaN, so that nothing of it counts that was not written. Against float64 as in test_prefill_attention_tc_gpu.py (4e-3 of the result's norm: weights and
result are rounded to bf16); without enough scratch the call is the one that has none, bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("T,pos0,heads,kv_heads", [(1, 6000, 8, 2), (300, 5000, 3, 1), (129, 4095, 5, 5), (128, 3969, 2, 1), (257, 2300, 99, 33), (1500, 3000, 16, 4), (2048, 900, 20, 5)])
@pytest.mark.parametrize("shape", ["plain", "rising", "falling"])
def test_shares(T, pos0, heads, kv_heads, hd, shape):
    import torch

    from simplellminference_b200 import _lib
    lib = _lib.load()
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
    need = lib.sllm_prefill_attention_scratch(1, T, pos0, hd, heads, kv_heads)
    assert need > 0 and need % 4 == 0
    scratch = torch.full((need // 4,), float("nan"), device="cuda")

    def run(short=0):
        out = torch.full((T, heads * hd), 7.0, device="cuda", dtype=torch.bfloat16)
        _lib.check(lib.sllm_prefill_attention_in(q.data_ptr(), k.data_ptr(), v.data_ptr(), 1, out.data_ptr(), T, pos0, S, hd, heads, kv_heads, scratch.data_ptr(), need - short,
                                                 torch.cuda.current_stream().cuda_stream))
        return out
    got = run().double().view(T, heads, hd)
    hidden = torch.arange(n, device="cuda")[None] > (pos0 + torch.arange(T, device="cuda"))[:, None]
    for h in range(heads):
        kh, vh = k[h // (heads // kv_heads), :n].double(), v[h // (heads // kv_heads), :n].double()
        s = (q.view(T, heads, hd)[:, h].double() @ kh.T) / hd ** 0.5
        want = torch.softmax(s.masked_fill(hidden, float("-inf")), -1) @ vh
        assert float((got[:, h] - want).norm() / want.norm()) < 4e-3, h
    none = torch.empty_like(q)
    _lib.check(lib.sllm_prefill_attention(q.data_ptr(), k.data_ptr(), v.data_ptr(), 1, none.data_ptr(), T, pos0, S, hd, heads, kv_heads, torch.cuda.current_stream().cuda_stream))
    assert torch.equal(run(4), none)


@pytest.mark.parametrize("T,pos0,heads,kv_heads,hd", [(1, 0, 8, 2, 128), (64, 0, 8, 8, 128), (65, 100, 6, 2, 128), (300, 5000, 3, 1, 128), (700, 33, 16, 4, 128), (1, 128, 8, 2, 64),
                                                      (257, 60, 5, 5, 64), (300, 4000, 24, 8, 64)])
def test_fp32_rows_are_rounded_once(T, pos0, heads, kv_heads, hd):
    """A cache in fp32 is rounded as the kernel without scratch rounds it: the results are those of the rounded cache, bit for bit."""
    import torch

    from simplellminference_b200 import _lib, kernels as K
    g = torch.Generator(device="cuda").manual_seed(T + pos0)
    n, S = pos0 + T, pos0 + T + 9
    q = torch.randn(T, heads * hd, device="cuda", generator=g).to(torch.bfloat16)
    k, v = (torch.randn(kv_heads, S, hd, device="cuda", generator=g) for _ in range(2))
    k[:, n:], v[:, n:] = float("nan"), float("nan")
    assert _lib.load().sllm_prefill_attention_scratch(0, T, pos0, hd, heads, kv_heads) >= 4 * kv_heads * n * hd
    got = K.prefill_attention(q, k, v, pos0, heads, kv_heads)
    assert torch.equal(got, K.prefill_attention(q, k.to(torch.bfloat16), v.to(torch.bfloat16), pos0, heads, kv_heads))
    plain = torch.empty_like(q)
    _lib.check(_lib.load().sllm_prefill_attention(q.data_ptr(), k.data_ptr(), v.data_ptr(), 0, plain.data_ptr(), T, pos0, S, hd, heads, kv_heads, torch.cuda.current_stream().cuda_stream))
    assert float((got.double() - plain.double()).norm() / plain.double().norm()) < 8e-3      # two results within 4e-3 of the same sums


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("T,pos0,heads,kv_heads", [(1, 6000, 8, 2), (300, 5000, 3, 1), (1500, 3000, 16, 4)])
def test_keys_at_minus_infinity(T, pos0, heads, kv_heads, hd):
    """A long run of keys whose scores are -inf, with whole shares in it: they count for nothing, with scratch as without."""
    import torch

    from simplellminference_b200 import _lib
    lib, g = _lib.load(), torch.Generator(device="cuda").manual_seed(T + hd)
    n = pos0 + T
    q = torch.randn(T, heads * hd, device="cuda", generator=g)
    k, v = (torch.randn(kv_heads, n, hd, device="cuda", generator=g) for _ in range(2))
    q[:, ::hd] = 1.0
    k[:, 700:2900, 0] = float("-inf")
    q, k, v = (t.to(torch.bfloat16) for t in (q, k, v))
    need = lib.sllm_prefill_attention_scratch(1, T, pos0, hd, heads, kv_heads)
    assert need > 0
    scratch = torch.full((need // 4,), float("nan"), device="cuda")
    hidden = torch.arange(n, device="cuda")[None] > (pos0 + torch.arange(T, device="cuda"))[:, None]
    for room in (need, 0):
        out = torch.full((T, heads * hd), 7.0, device="cuda", dtype=torch.bfloat16)
        _lib.check(lib.sllm_prefill_attention_in(q.data_ptr(), k.data_ptr(), v.data_ptr(), 1, out.data_ptr(), T, pos0, n, hd, heads, kv_heads, scratch.data_ptr(), room,
                                                 torch.cuda.current_stream().cuda_stream))
        for h in range(heads):
            kh, vh = k[h // (heads // kv_heads)].double(), v[h // (heads // kv_heads)].double()
            s = (q.view(T, heads, hd)[:, h].double() @ kh.T) / hd ** 0.5
            want = torch.softmax(s.masked_fill(hidden, float("-inf")), -1) @ vh
            assert float((out.double().view(T, heads, hd)[:, h] - want).norm() / want.norm()) < 4e-3, (room, h)
