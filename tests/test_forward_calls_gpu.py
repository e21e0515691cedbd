"""sllm_engine_forward on the persistent kernels: token and position come with the launch. The same logits and tokens as a greedy run, positions out of order, and the
state it leaves for steps that follow; contexts cut into more splits than the merge takes in one go, at positions on both sides of a split's border."""
import numpy as np
import pytest

from simplellminference_b200.config import BF16, F32, INT8, ModelShape
from simplellminference_b200.engine import Engine

pytestmark = pytest.mark.gpu

MODES = {"mega": dict(mega=True), "mega_v2": dict(mega=True, mega_v2=True), "mega_v2_fuse": dict(mega=True, mega_v2=True, mega_fuse_down=True)}
V1, V1F, V2, V2F = "megakernel", "megakernel(fused-down)", "megakernel(v2)", "megakernel(v2,fused-down)"
# (shape, weights, the kernel each mode gets: the one with per-head counters takes neither int8 weights nor kv head groups of more than 128 16-byte
# chunks, nor the largest plans): one kv head,
# 16 splits of it, eight query heads; 8 kv heads, 16 splits; two query heads a kv head; a merge whose pieces are as many as its threads; one with twice as many, 9 splits
SHAPES = [(ModelShape(320, 32, 256, 32, 512, 1024, 2, 8, 1), F32, (V1, V2, V2F)), (ModelShape(512, 64, 512, 512, 768, 1024, 2, 8, 8), INT8, (V1, V1, V1)),
          (ModelShape(512, 64, 1024, 512, 512, 1024, 2, 16, 8), BF16, (V1, V2, V2F)), (ModelShape(300, 128, 2048, 256, 256, 600, 1, 16, 2), F32, (V1, V1, V1F)),
          (ModelShape(300, 128, 4096, 512, 512, 576, 1, 32, 4), BF16, (V1, V1, V1F))]


@pytest.mark.parametrize("mode", list(MODES))
@pytest.mark.parametrize("shape,wd,kernels", SHAPES)
def test_calls_follow_a_greedy_run(mode, shape, wd, kernels):
    kw = dict(w_dtype=wd, kv_dtype=F32, group=64)
    a = Engine(shape, **kw, **MODES[mode]).load_synthetic(5)
    assert a.mode == kernels[list(MODES).index(mode)], a.mode
    b = Engine(shape, **kw).load_synthetic(5)             # the kernels of one op each, in a graph
    prompt, n = np.arange(1, 40, dtype=np.int32), 90
    want = b.greedy(prompt, n)
    fed = np.concatenate([prompt[:1], want])
    for pos in range(n - 1):
        logits, nxt = a.forward(int(fed[pos]), pos)
        ref, ref_next = b.forward(int(fed[pos]), pos)
        # fp32 sums of at most a few thousand products in another order: 3e-4 of the largest logit is the bound of every decode test of this repository
        assert np.abs(logits - ref).max() <= 3e-4 * max(1.0, np.abs(ref).max()), pos
        assert nxt == int(np.argmax(logits)) and (nxt == ref_next or ref[nxt] > ref.max() - 1e-3)
    assert np.array_equal(logits, a.buffer("model_pred").cpu().numpy())
    # an earlier position again, without logits, then steps that go on from there
    none, nxt = a.forward(int(fed[50]), 50, want_logits=False)
    b.forward(int(fed[50]), 50)
    assert none is None
    a.enqueue_steps(3)
    b.enqueue_steps(3)
    got, ref = a.read_tokens(4), b.read_tokens(4)
    assert got[0] == nxt and np.array_equal(got, ref)


def test_bad_calls_are_refused_and_leave_the_engine_usable():
    from simplellminference_b200._lib import SllmError
    e = Engine(SHAPES[0][0], w_dtype=F32, kv_dtype=F32, mega=True, mega_v2=True).load_synthetic(5)
    first = e.forward(3, 0)[0]
    for token, pos in ((-1, 0), (320, 0), (3, -1), (3, 1024)):
        with pytest.raises(SllmError):
            e.forward(token, pos)
    assert np.abs(e.forward(3, 0)[0] - first).max() < 1e-4
