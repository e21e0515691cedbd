"""Operands and results at addresses that wide accesses cannot use: fp32 rows in front of a tensor-core product, and the result of prompt attention over a bf16
cache. Products of bf16 values summed in fp32 (K = 200: 2e-6); attention rounds weights and result to bf16 (4e-3, as in test_prefill_attention_tc_gpu.py)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset,pad", [(0, 0), (1, 0), (0, 3), (1, 4)])
def test_rows_of_a_product(offset, pad):
    import torch

    from simplellminference_b200.config import BF16
    from simplellminference_b200.seqops import Ops
    ops, T, N, K = Ops(BF16), 70, 96, 200
    g = torch.Generator(device="cuda").manual_seed(1)
    lda = K + pad
    flat = torch.randn(T * lda + 8, device="cuda", generator=g)
    A = flat[offset:offset + T * lda].view(T, lda)[:, :K]
    W = torch.randn(N, K, device="cuda", generator=g).to(torch.bfloat16)
    C = torch.full((T, N), float("nan"), device="cuda")
    scratch = torch.empty(T * K * 2 + 256 + T * N * 4 + 256, dtype=torch.uint8, device="cuda")
    ops.linear(flat.data_ptr() + 4 * offset, lda, W, K, None, C.data_ptr(), N, T, N, K, torch.cuda.current_stream().cuda_stream, scratch=scratch)
    want = A.to(torch.bfloat16).double() @ W.double().T
    assert float((C.double() - want).norm() / want.norm()) < 2e-6


@pytest.mark.parametrize("hd,heads,kv_heads,T,pos0", [(128, 4, 2, 300, 77), (64, 2, 2, 130, 0), (128, 2, 1, 40, 0), (64, 40, 8, 300, 50)])
@pytest.mark.parametrize("shift", [0, 2, 6])
def test_result_of_prompt_attention(hd, heads, kv_heads, T, pos0, shift):
    import torch

    from simplellminference_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(T)
    n = pos0 + T
    q = torch.randn(T, heads * hd, device="cuda", generator=g).to(torch.bfloat16)
    k, v = (torch.randn(kv_heads, n, hd, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    flat = torch.full((T * heads * hd + 16,), float("nan"), device="cuda", dtype=torch.bfloat16)
    _lib.check(_lib.load().sllm_prefill_attention(q.data_ptr(), k.data_ptr(), v.data_ptr(), 1, flat.data_ptr() + 2 * shift, T, pos0, n, hd, heads, kv_heads,
                                                  torch.cuda.current_stream().cuda_stream))
    got = flat[shift:shift + T * heads * hd].view(T, heads, hd).double()
    hidden = torch.arange(n, device="cuda")[None] > (pos0 + torch.arange(T, device="cuda"))[:, None]
    for h in range(heads):
        s = (q.view(T, heads, hd)[:, h].double() @ k[h // (heads // kv_heads)].double().T) / hd ** 0.5
        want = torch.softmax(s.masked_fill(hidden, float("-inf")), -1) @ v[h // (heads // kv_heads)].double()
        assert float((got[:, h] - want).norm() / want.norm()) < 4e-3, h
    assert bool(torch.isnan(flat[:shift]).all()) and bool(torch.isnan(flat[shift + T * heads * hd:]).all())
