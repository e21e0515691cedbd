"""Waits inside the tcgen05 kernels that run out: the report, and that nothing of it stays behind."""
import pytest
from test_attention_forms_gpu import _close, _inputs, _ops, _run
from test_attention_tc_gpu import _want

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", ["paged", "contiguous"])
def test_waits_that_run_out_are_reported(which):
    """With no polls allowed the tcgen05 kernels give up their first waits; the library's next call says so, once, and later launches are whole again."""
    import torch

    from simplellminference_b200 import _lib, kernels
    ops, lib = _ops(), _lib.load()
    heads, kv_heads, dim, segs = 8, 2, 128, [(0, 517)]
    q, k, v, rows, b, keep = _inputs(segs, heads, kv_heads, dim, 64)
    q16 = q[:, :heads * dim].to(torch.bfloat16).contiguous()
    kc, vc = (rows[0][i].to(torch.bfloat16).contiguous() for i in (0, 1))

    def call():
        if which == "paged":
            return _run(ops, b, q, k, v, heads, kv_heads, dim, None)
        return kernels.prefill_attention(q16, kc, vc, 0, heads, kv_heads).float()
    want = _want(q, rows, segs, heads, kv_heads, dim, dim ** -0.5)
    assert lib.sllm_status() == 0
    assert lib.sllm_tune(10, 0) == 0
    try:
        call()
        torch.cuda.synchronize()
    finally:
        assert lib.sllm_tune(10, 1 << 24) == 0
    with pytest.raises(_lib.SllmError) as e:
        call()
    assert e.value.code == _lib.ETIMEOUT
    torch.cuda.synchronize()
    assert lib.sllm_status() == 0
    assert _close(call(), want, 4e-6 if which == "paged" else 4e-3)


@pytest.mark.parametrize("T", [100, 700], ids=["one SM", "two SMs a tile"])
def test_waits_of_a_product_that_run_out_are_reported(T):
    """The same for the product, whose roles all give up and whose CTAs of a pair leave together."""
    import torch

    from simplellminference_b200 import _lib, kernels
    lib, g = _lib.load(), torch.Generator(device="cuda").manual_seed(T)
    a = torch.randn(T, 512, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(4100, 512, generator=g, device="cuda").to(torch.bfloat16)
    want = a.double() @ w.double().T
    assert lib.sllm_status() == 0
    assert lib.sllm_tune(10, 0) == 0
    try:
        kernels.prefill_gemm(a, w)
        torch.cuda.synchronize()
    finally:
        assert lib.sllm_tune(10, 1 << 24) == 0
    with pytest.raises(_lib.SllmError) as e:
        kernels.prefill_gemm(a, w)
    assert e.value.code == _lib.ETIMEOUT
    torch.cuda.synchronize()
    assert lib.sllm_status() == 0
    for _ in range(3):                  # tensor memory and barriers of the SMs are free again
        assert float((kernels.prefill_gemm(a, w).double() - want).norm() / want.norm()) < 1e-6
