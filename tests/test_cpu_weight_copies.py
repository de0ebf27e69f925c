"""The registry of transposed weight copies: an entry belongs to its copy, not to the address the copy had."""
import gc

import torch

import genesis_b200 as genesis
from genesis_b200 import amp_state


def test_twin_is_found_by_its_copy_only():
    lp, twin = torch.zeros(4, 6, dtype=torch.bfloat16), torch.ones(6, 4, dtype=torch.bfloat16)
    amp_state.keep_transposed(lp, twin)
    assert amp_state.transposed_of(lp) is twin
    other = lp.view(4, 6)                       # another tensor at the same address
    assert other.data_ptr() == lp.data_ptr() and amp_state.transposed_of(other) is None
    key = lp.data_ptr()
    del lp, other
    gc.collect()
    assert key not in amp_state.transposed


def test_twins_leave_with_their_optimizer():
    lin = genesis.nn.Linear(64, 96, bias=False)
    lin.weight.wants_transposed_copy = True
    opt = genesis.optim.AdamW(lin.parameters(), lr=1e-3)
    before = len(amp_state.transposed)
    opt.enable_shadows(genesis.bfloat16)
    assert len(amp_state.transposed) == before + 1
    copy, twin = opt._transposed[0]
    assert amp_state.transposed_of(copy) is twin and torch.equal(twin, copy.t())
    del opt, copy, twin
    gc.collect()
    assert len(amp_state.transposed) == before
