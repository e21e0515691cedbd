"""Which form of state-space duality a step takes, from its counts alone (no device): blocks of tokens on the tensor cores for portions that fill them."""
import types

import pytest
import torch

from simplellminference_b200.seqengine import Step


@pytest.mark.parametrize("tensor_cores,T,nseg,heads,state,dv,blocks", [
    (True, 2048, 1, 64, 128, 64, True), (False, 2048, 1, 64, 128, 64, False), (True, 32, 1, 64, 128, 64, False), (True, 64, 1, 64, 128, 64, True), (True, 8, 8, 64, 128, 64, False),
    (True, 8 + 64, 9, 64, 128, 64, False), (True, 8 + 128, 9, 64, 128, 64, True), (True, 32 + 256, 33, 64, 128, 64, False), (True, 677, 4, 64, 128, 64, True),
    (True, 2048, 1, 8, 128, 64, False), (True, 700, 1, 8, 64, 128, True), (True, 2048, 1, 16, 64, 128, True)])
def test_blocks_of_state_space_duality(tensor_cores, T, nseg, heads, state, dv, blocks):
    class Engine:
        max_len, device = 4096, torch.device("cpu")
        ops = types.SimpleNamespace(ssd_block_ws_floats=lambda n_qtiles, nseg, heads, groups, n_state: 4)

        def _scratch(self, name, n_floats):
            return name

    engine = Engine()
    engine.tensor_cores = tensor_cores
    step = Step(engine)
    step.T, step.nseg = T, nseg
    assert (step.ssd_block_scratch(heads, 1, state, dv) is not None) == blocks
