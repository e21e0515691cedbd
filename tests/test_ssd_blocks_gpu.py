"""State-space duality in blocks of 64 tokens on the tensor cores (sllm_seq_ssd_blocks): portions that end anywhere in a block, several portions in one
step that go on from a state, states and columns that are multiples of nothing, groups, with and without the skip term, decays that forget within a
token and ones that hardly forget. Against float64 on the same fp32 inputs; three bf16 terms per operand leave 2^-24 of each product:
2e-5 of the result is generous (tighter: test_ssd_blocks_terms_gpu.py). The ring afterwards is that of sllm_seq_ssd_scan, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(lens, slots):
    import torch

    from simplellminference_b200._lib import SeqBatch
    ints = lambda x: torch.tensor(np.asarray(x, np.int32), device="cuda")   # noqa: E731
    T, starts = sum(lens), np.cumsum([0] + list(lens[:-1]))
    tiles = [(i, off) for i, n in enumerate(lens) for off in range(0, n, 32)]
    order = sorted(tiles, key=lambda t: -t[1])
    tile0 = np.cumsum([0] + [-(-n // 32) for n in lens[:-1]])
    keep = [ints(np.repeat(slots, lens)), ints(np.concatenate([np.arange(n) for n in lens])), ints(starts), ints(lens), ints(slots), ints([0] * len(lens)), ints([t[0] for t in order]),
            ints([t[1] for t in order]), ints(tile0)]
    b = SeqBatch()
    b.T, b.nseg, b.n_qtiles = T, len(lens), len(tiles)
    b.tok_slot, b.tok_pos, b.seg_start, b.seg_len, b.seg_slot, b.seg_pos0, b.qt_seg, b.qt_off, b.seg_tile0 = [k.data_ptr() for k in keep]
    return b, keep


@pytest.mark.parametrize("lens", [[1], [63], [64, 65, 2], [200, 1, 33, 128], [1000]], ids=str)
@pytest.mark.parametrize("heads,groups,state,dv", [(4, 2, 128, 64), (3, 1, 64, 32), (2, 2, 70, 36), (4, 1, 16, 130), (2, 1, 33, 7)])
@pytest.mark.parametrize("rate,skip", [(0.0, True), (4.0, False), (-6.0, True)], ids=["usual", "forgetful", "long memory"])
def test_blocks_against_float64(lens, heads, groups, state, dv, rate, skip):
    import torch

    from simplellminference_b200.config import BF16
    from simplellminference_b200.seqops import Ops
    ops, T, taps = Ops(BF16), sum(lens), 4
    g = torch.Generator(device="cuda")
    g.manual_seed(T + heads * state)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")   # noqa: E731
    inner, gn = heads * dv, groups * state
    channels = inner + 2 * gn
    ld = channels + heads + 1
    u, step = rnd(T, channels), rnd(T, ld)
    a_log, bias, D = rate + 0.5 * rnd(heads), rnd(heads) - 1.0, rnd(heads)
    slots = list(range(len(lens)))[::-1]
    S0, ring0 = rnd(len(lens), heads, state, dv), rnd(len(lens), taps - 1, channels)
    b, keep = _batch(lens, slots)
    st = torch.cuda.current_stream().cuda_stream
    outs = []
    for blocks in (True, False):
        S, ring, y = S0.clone(), ring0.clone(), torch.full((T, inner), float("nan"), device="cuda")
        args = (b, u.data_ptr(), channels, u.data_ptr() + 4 * inner, channels, u.data_ptr() + 4 * (inner + gn), channels, step.data_ptr(), ld, a_log, bias, D if skip else None, heads,
                groups, state, dv, S, y, inner, u.data_ptr(), channels, channels, taps, ring, st)
        if blocks:
            n = ops.ssd_block_ws_floats(b.n_qtiles, b.nseg, heads, groups, state)
            ops.ssd_blocks(*args, block_ws=torch.full((n,), float("nan"), device="cuda"))
        else:
            ops.ssd_scan(*args)
        outs.append((S, ring, y))
    assert torch.equal(outs[0][1], outs[1][1])
    S, y, at = S0.double(), torch.empty(T, heads, dv, dtype=torch.float64, device="cuda"), 0
    x = u[:, :inner].double().view(T, heads, dv)
    B, C = (u[:, inner + i * gn:inner + (i + 1) * gn].double().view(T, groups, state).repeat_interleave(heads // groups, 1) for i in (0, 1))
    dt = torch.nn.functional.softplus(step[:, :heads].double() + bias.double())
    decay = torch.exp(-torch.exp(a_log.double()) * dt)
    for i, n in enumerate(lens):
        s = S[slots[i]].clone()
        for t in range(at, at + n):
            s = decay[t][:, None, None] * s + (dt[t][:, None] * B[t])[:, :, None] * x[t][:, None]
            y[t] = torch.bmm(C[t][:, None], s)[:, 0]
        S[slots[i]] = s
        at += n
    if skip:
        y = y + D.double()[:, None] * x
    y = y.view(T, inner)
    for got, want in ((outs[0][2], y), (outs[0][0], S)):
        assert float((got.double() - want).norm() / want.norm()) < 2e-5
