"""State-space duality in blocks of tokens (sllm_seq_ssd_blocks) keeps what the token-by-token form (sllm_seq_ssd_scan) has: its accuracy, which tokens a value
reaches, and an error where index arrays and counts contradict each other. Three bf16 terms per operand leave 2^-24 of a product; fp32 sums of up to 128 + 64
products and 16 blocks of carried state stay within 5e-7."""
import math

import pytest
from test_ssd_blocks_gpu import _batch

pytestmark = pytest.mark.gpu


def _inputs(lens, heads, groups, state, dv, rate):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(sum(lens) + heads * state)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")   # noqa: E731
    T, inner, gn = sum(lens), heads * dv, groups * state
    return dict(x=rnd(T, inner), B=rnd(T, gn), C=rnd(T, gn), step=rnd(T, heads), a=rate + 0.5 * rnd(heads), bias=rnd(heads) - 1.5, D=rnd(heads), S=rnd(len(lens), heads, state, dv))


def _run(t, lens, heads, groups, state, dv, n_qtiles=None, blocks=True):
    import torch

    from simplellminference_b200.config import BF16
    from simplellminference_b200.seqops import Ops
    ops, T, inner, gn = Ops(BF16), sum(lens), heads * dv, groups * state
    b, keep = _batch(lens, list(range(len(lens))))
    if n_qtiles:
        b.n_qtiles = n_qtiles
    S, y = t["S"].clone(), torch.full((T, inner), float("nan"), device="cuda")
    args = (b, t["x"].data_ptr(), inner, t["B"].data_ptr(), gn, t["C"].data_ptr(), gn, t["step"].data_ptr(), heads, t["a"], t["bias"], t["D"], heads, groups, state, dv, S, y, inner,
            None, 0, 0, 0, None, torch.cuda.current_stream().cuda_stream)
    if blocks:
        ws = torch.full((ops.ssd_block_ws_floats(b.n_qtiles, b.nseg, heads, groups, state),), float("nan"), device="cuda")
        ops.ssd_blocks(*args, block_ws=ws)
    else:
        ops.ssd_scan(*args)
    torch.cuda.synchronize()
    return y, S


def _want(t, lens, heads, groups, state, dv):
    import torch
    T = sum(lens)
    x, dt = t["x"].double().view(T, heads, dv), torch.nn.functional.softplus(t["step"].double() + t["bias"].double())
    B, C = (t[k].double().view(T, groups, state).repeat_interleave(heads // groups, 1) for k in "BC")
    decay, S, y, at = torch.exp(-torch.exp(t["a"].double()) * dt), t["S"].double(), torch.empty(T, heads, dv, dtype=torch.float64, device="cuda"), 0
    for i, n in enumerate(lens):
        for k in range(at, at + n):
            S[i] = decay[k][:, None, None] * S[i] + (dt[k][:, None] * B[k])[:, :, None] * x[k][:, None]
            y[k] = torch.bmm(C[k][:, None], S[i])[:, 0]
        at += n
    return (y + t["D"].double()[:, None] * x).view(T, heads * dv), S


@pytest.mark.parametrize("shape", [(4, 2, 128, 64), (3, 1, 64, 32), (2, 2, 70, 36), (2, 1, 33, 7)], ids=str)
@pytest.mark.parametrize("lens", [[64, 65, 2], [1000]], ids=str)
@pytest.mark.parametrize("rate", [0.0, 4.0, -6.0])
def test_accuracy(shape, lens, rate):
    t = _inputs(lens, *shape, rate)
    for got, want in zip(_run(t, lens, *shape), _want(t, lens, *shape)):
        assert float((got.double() - want).norm() / want.norm()) < 5e-7


@pytest.mark.parametrize("value", [math.nan, math.inf, -math.inf])
def test_a_value_that_is_not_finite_reaches_no_earlier_token(value):
    import torch
    lens, shape = [200, 70], (2, 1, 64, 64)
    heads, groups, state, dv = shape
    t = _inputs(lens, *shape, 0.0)
    clean = _run(t, lens, *shape)
    at, col = 75, 64 + 5                       # in the middle of a block; column 5 of the second head
    t["x"][at, col] = value
    y, S = _run(t, lens, *shape)
    y2, S2 = _run(t, lens, *shape, blocks=False)
    touched = torch.zeros_like(y, dtype=torch.bool)
    touched[at:200, col] = True
    assert torch.equal(y[~touched], clean[0][~touched])
    rest = torch.ones_like(S, dtype=torch.bool)
    rest[0, 1, :, 5] = False
    assert torch.equal(S[rest], clean[1][rest])
    assert torch.equal(torch.isfinite(y[at:128, col]), torch.isfinite(y2[at:128, col]))      # (infinite or no number: the two forms sum in different orders)


def test_a_tile_count_that_leaves_tokens_out_is_reported():
    from simplellminference_b200 import _lib
    lens, shape = [33] * 16, (2, 1, 64, 32)
    t = _inputs(lens, *shape, 0.0)
    with pytest.raises(_lib.SllmError) as e:          # fewer tiles than tokens need at all: refused at once
        _run(t, lens, *shape, n_qtiles=16)
    assert e.value.code == _lib.EINVAL
    lib = _lib.load_seq()
    assert lib.sllm_status() == 0
    _run(t, lens, *shape, n_qtiles=17)                # two tiles a segment are needed: seen on the device
    assert lib.sllm_status() == _lib.EINVAL and lib.sllm_status() == 0
