"""Planned runs (one-stream and batched) where their memory layout, the order
of their CTAs or their choice of form can go wrong, against the CPU oracle."""
import pytest

import cases
import test_gpu_batched as tgb
from jacquard_b200 import batched

pytestmark = pytest.mark.gpu


def test_timed_single_lane_items_without_x_of_any_slot_count():
    """Setup/hold checks in single-lane items without X, whose slots are one
    word each: the tables behind them (8-byte accesses) start on 16 bytes."""
    for lanes, per_item, parts in [(1, 1, 0), (3, 0, 0), (1, 0, 4), (2, 1, 16), (1, 1, 2)]:
        s = cases.script("sram", 16, (8,), xprop=False, timing_seed=9, target_parts=parts)
        plan = batched.BatchedSim(s, lanes, lanes_per_item=per_item).plan
        assert plan is not None and plan.lanes_per_item == 1
        assert plan.max_slots % 4 == 0  # before any launch
        tgb.test_batched_setup_hold_events_match_oracle_per_stream(False, lanes, per_item, parts)
