"""Prompts of several engines at once, each engine on a stream of its own.

The products of a prompt run as pairs of CTAs that share their tensor memory, one CTA per SM, and the SMs that one engine's kernel leaves are taken by another's at any moment: set-up and
teardown of a pair must hold whoever comes next. What an engine computes must not depend on the others: it is compared with the same prompt run alone. Rows are rounded to bf16 in front of
every product and split sums are added in any order, so two runs may differ by roundings: the bound of the whole prompt against the oracle, 3e-3 of the largest logit.
"""
import numpy as np
import pytest
import torch

from simplellminference_b200 import _lib
from simplellminference_b200.config import BF16, ModelShape
from simplellminference_b200.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [129, 300])   # the fewest tokens that pairs take, and a last tile that is not full
def test_engines_on_streams_of_their_own(T):
    shape = ModelShape(4096, 128, 1024, 512, 2816, 512, 2, 8, 4)
    engines = [Engine(shape, w_dtype=BF16, kv_dtype=BF16, mega=True).load_synthetic(seed) for seed in (1, 2, 3)]
    rng = np.random.default_rng(T)
    prompts = [rng.integers(0, shape.vocab, T + 7 * i).astype(np.int32) for i in range(3)]
    alone = []
    for e, prompt in zip(engines, prompts):
        e.prefill(prompt)
        torch.cuda.synchronize()
        alone.append(e.buffer("model_pred").float().cpu().clone())
    for _ in range(200):
        for e, prompt in zip(engines, prompts):
            e.prefill(prompt)
    torch.cuda.synchronize()
    _lib.check(_lib.load().sllm_status())
    for e, want in zip(engines, alone):
        got = e.buffer("model_pred").float().cpu()
        assert torch.isfinite(want).all() and float((got - want).abs().max()) <= 3e-3 * float(want.abs().max())
