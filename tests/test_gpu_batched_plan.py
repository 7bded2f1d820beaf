"""Batched runs on the gate-list plan (jq_batched_plan_build,
jq_simulate_batched_planned): every stream against the CPU oracle in each
item form and layout, and the prepared-script kernels that serve scripts
without a plan."""
import numpy as np
import pytest
import torch

import cases
from jacquard_b200 import batched
from test_gpu_batched import BatchedCase, SPLIT4

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,nb,split,parts,xprop,lanes,per_item,grid,form", [
    ("tiny", 8, (5,), 0, False, 3, 0, 0, (1, 0)),        # odd lanes, no X
    ("tiny", 8, (5,), 0, False, 4, 0, 0, (2, 0)),
    ("sram", 16, (8,), 4, False, 8, 0, 0, (2, 0)),       # too few items for octets
    ("soc_mini", 148, SPLIT4, 37, False, 8, 0, 0, (8, 3)),   # 2-state octets, SRAMs
    ("small", 148, (8, 16, 24), 37, False, 8, 0, 0, (8, 3)),
    ("sram", 16, (8,), 0, True, 8, 0, 0, (2, 1)),        # cone partitions, SRAM port items
    ("sram", 16, (8,), 0, True, 5, 0, 2, (1, 1)),        # more items than CTAs
    ("soc_mini", 296, SPLIT4, 296, True, 8, 8, 0, (8, 2)),   # more items than SMs
    # deep cones whose octet slots do not fit even when split: lane pairs
    ("soc_mini", 148, (20, 40, 60), 0, True, 16, 0, 0, (2, 1)),
    ("soc_mini", 148, SPLIT4, 37, True, 16, 0, 0, (8, 2)),   # two octet groups, split
])
def test_batched_plan_forms_match_oracle(kind, nb, split, parts, xprop, lanes, per_item, grid, form):
    s = cases.script(kind, nb, split, xprop=xprop, target_parts=parts)
    c = BatchedCase(kind, s, lanes, per_item=per_item, grid=grid, cycles=7)
    assert c.B.plan is not None
    assert (c.B.plan.lanes_per_item, c.B.x_interleaved) == form
    c.launch()
    assert c.B.status() == 0
    c.verify()


@pytest.mark.parametrize("kind,nb,split,parts,xprop,lanes,per_item", [
    ("tiny", 8, (5,), 0, False, 4, 2),
    ("sram", 16, (8,), 0, True, 2, 1),
    ("soc_mini", 148, SPLIT4, 37, True, 8, 8),
])
def test_prepared_script_kernels_match_oracle(monkeypatch, kind, nb, split, parts, xprop, lanes,
                                              per_item):
    """The kernels that run scripts without a plan (planned=False)."""
    init = batched.BatchedSim.__init__
    monkeypatch.setattr(batched.BatchedSim, "__init__",
                        lambda self, *a, **k: init(self, *a, planned=False, **k))
    s = cases.script(kind, nb, split, xprop=xprop, target_parts=parts)
    c = BatchedCase(kind, s, lanes, per_item=per_item, cycles=5)
    assert c.B.plan is None
    c.launch()
    assert c.B.status() == 0
    c.verify()


@pytest.mark.parametrize("lanes,signals,layout", [(8, 96, 3), (16, 7, 3), (8, 64, 2), (3, 50, 0)])
def test_state_layouts_round_trip(lanes, signals, layout):
    from jacquard_b200 import sim
    L = batched.lib()
    x = torch.randint(-2**31, 2**31 - 1, (lanes, signals), dtype=torch.int32, device="cuda")
    st = torch.zeros(L.jq_batched_state_words(lanes, signals), dtype=torch.int32, device="cuda")
    y = torch.zeros_like(x)
    q = torch.cuda.current_stream().cuda_stream
    assert L.jq_batched_pack_state(x.data_ptr(), lanes, signals, layout, st.data_ptr(), q) == 0
    assert L.jq_batched_unpack_state(st.data_ptr(), lanes, signals, layout, y.data_ptr(), q) == 0
    assert torch.equal(x, y)
    if layout == 3:  # word ((l >> 3) * signals + s) * 8 + (l & 7)
        assert torch.equal(st[:lanes * signals].view(lanes // 8, signals, 8).permute(0, 2, 1)
                           .reshape(lanes, signals), x)
    assert sim.lib().jq_sim_status(q) == 0
