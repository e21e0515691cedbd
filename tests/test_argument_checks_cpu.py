"""Addresses the kernels cannot read or write at the width they use are refused on the host, before anything is launched (no device)."""
import pytest

from simplellminference_b200 import _lib

BASE = 0x7F0000000000       # never dereferenced: the checks come first


@pytest.mark.parametrize("kv_dtype", [0, 1], ids=["f32", "bf16"])
@pytest.mark.parametrize("q,k,v,out", [(2, 0, 0, 0), (8, 0, 0, 0), (0, 4, 0, 0), (0, 0, 8, 0), (0, 0, 0, 2)])
def test_prompt_attention(kv_dtype, q, k, v, out):
    rc = _lib.load().sllm_prefill_attention(BASE + q, BASE + (1 << 20) + k, BASE + (2 << 20) + v, kv_dtype, BASE + (3 << 20) + out, 64, 0, 64, 128, 8, 2, None)
    assert rc == _lib.EINVAL


def test_bf16_rows_left_by_the_caller():
    rc = _lib.load().sllm_seq_linear(BASE, 64, BASE + (1 << 20), 1, 64, None, BASE + (2 << 20), 64, 64, 64, 64, 1.0, 0, 1, 1, 0, 0, 0, 0, BASE + (3 << 20) + 2, 1, None, None)
    assert rc == _lib.EINVAL
