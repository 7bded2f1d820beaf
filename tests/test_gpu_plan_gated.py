"""Clock enables that clear between cycles, in every planned form, against the
CPU oracle: a random clock flag, a second clock and enables gated by an input,
so that registers keep their values (and X) over many cycles."""
import functools

import numpy as np
import pytest
import torch

import cases
import test_gpu_batched as tgb
from jacquard_b200 import frontend, sim, state
from test_gpu_plain import run_gpu, run_oracle

pytestmark = pytest.mark.gpu


def gated_design(params):
    """A generated design whose registers are enabled by its clock flag, by
    that flag AND an input, or by a second clock flag."""
    d = frontend.Design(params)
    lib = frontend._lib()
    an_input = int(np.nonzero(d.kind == 2)[0][-1])  # (2: input; not the reset)
    clk2 = lib.jqf_builder_clock_flag(d._h)
    gated = lib.jqf_builder_and(d._h, d.clock_flag_pin << 1, an_input << 1)
    for i, div in enumerate(d.dff_d.tolist()):
        if i % 3:
            assert lib.jqf_builder_set_dff(d._h, i, div, clk2 << 1 if i % 3 == 1 else gated) == 0
    d._load_info()
    return d


def gated_stimulus(kind, s, cycles, seed=3, p_toggle=0.5, reset_cycles=2, x_init=False):
    d = cases.design(kind)
    vals = state.stimulus_inputs(s, d, cycles, seed, p_toggle, reset_cycles)
    col = np.asarray(s.input_layout) == d.clock_flag_pin
    rng = np.random.default_rng(seed + 77)
    vals[:, col] = rng.integers(0, 2, size=(cycles + 1, 1), dtype=np.uint8)
    v = state.pack_inputs(s, vals)
    if s.xprop_enabled:
        v = state.expand_states_for_xprop(v, s)
        if not x_init:
            v[0, s.reg_io_state_size:] = 0
    if s.timing_arrivals_enabled:
        v = state.expand_states_for_arrivals(v, s)
    return np.ascontiguousarray(v)


@pytest.fixture
def gated(monkeypatch):
    """tests/cases.py with gated designs and clocks."""
    params = {k: cases.design(k).params for k in ("small", "sram", "soc_mini")}
    design = functools.lru_cache(None)(lambda kind, seed=11: gated_design(params[kind]))
    monkeypatch.setattr(cases, "design", design)
    monkeypatch.setattr(cases, "script", functools.lru_cache(None)(cases.script.__wrapped__))
    monkeypatch.setattr(cases, "stimulus", gated_stimulus)


@pytest.mark.parametrize("xprop", [True, False])
@pytest.mark.parametrize("kind,nb,split,parts,form", [
    ("small", 64, (), 3, "flow"),               # one item a CTA and cycle, no hint
    ("sram", 16, (), 4, "flow"),
    ("soc_mini", 148, (20, 40, 60), 37, "hint"),  # more than 64 items a stage
    ("small", 64, (8, 16, 24), 0, "mirror"),
])
def test_kept_registers_match_oracle(gated, kind, nb, split, parts, form, xprop):
    s = cases.script(kind, nb, split, xprop=xprop, target_parts=parts)
    cycles = 200 if kind != "soc_mini" else 24
    states = cases.stimulus(kind, s, cycles, x_init=xprop)
    want, wsram, wsx, _ = run_oracle(s, states, cycles)
    plan = sim.DeviceScript(s).plan()
    assert (bool(plan.mirrored), plan.widest > 64) == (form == "mirror", form == "hint")
    for legacy in (False, True):
        for _ in range(3):
            got, sram, sram_x, _ = run_gpu(s, states, cycles, legacy=legacy)
            assert np.array_equal(got, want)
            assert np.array_equal(sram[:wsram.size], wsram)
            if xprop:
                assert np.array_equal(sram_x[:wsx.size], wsx)
    ds = sim.DeviceScript(s)  # the script's own form
    st = sim.u32_to_dev(states.reshape(-1))
    n = max(1, s.sram_storage_size)
    sim.simulate(ds, st, cycles, states.shape[1], torch.zeros(n, dtype=torch.int32, device="cuda"),
                 torch.full((n,), -1, dtype=torch.int32, device="cuda"), planned=False)
    assert sim.status() == 0
    assert np.array_equal(sim.dev_to_u32(st).reshape(states.shape), want)


@pytest.mark.parametrize("kind,nb,split,parts,xprop,lanes,per_item,layout", [
    ("sram", 16, (8,), 0, False, 3, 0, 0),
    ("sram", 16, (8,), 0, False, 2, 2, 0),
    ("sram", 16, (8,), 0, True, 3, 0, 1),
    ("sram", 16, (8,), 4, True, 4, 2, 1),
    ("sram", 16, (8,), 16, True, 8, 8, 2),
    ("sram", 16, (8,), 16, False, 32, 0, 3),
])
def test_kept_registers_batched_match_oracle(gated, kind, nb, split, parts, xprop, lanes, per_item,
                                             layout):
    s = cases.script(kind, nb, split, xprop=xprop, target_parts=parts)
    c = tgb.BatchedCase(kind, s, lanes, per_item=per_item, cycles=24)
    assert c.B.plan is not None and c.B.x_interleaved == layout
    c.launch()
    assert c.B.status() == 0
    c.verify()


@pytest.mark.parametrize("xprop,lanes,per_item,parts", [
    (False, 3, 0, 0), (False, 2, 2, 0), (True, 3, 0, 0), (True, 2, 2, 4), (True, 8, 8, 16),
    (False, 32, 0, 16)])
def test_kept_registers_batched_checks_match_oracle(gated, xprop, lanes, per_item, parts):
    """Setup/hold records per stream: only streams whose enable is set."""
    tgb.test_batched_setup_hold_events_match_oracle_per_stream(xprop, lanes, per_item, parts)
