"""The gate-list plan of one-stream runs (jq_plain_plan_build,
jq_simulate_planned) against the CPU oracle: snapshots, SRAM contents,
arrivals and violations bit for bit, in both of its forms and where its
sizes and rules can go wrong."""
import numpy as np
import pytest
import torch

import cases
import oracle_lib
from jacquard_b200 import sim
from test_gpu_plain import run_oracle, sorted_events

pytestmark = pytest.mark.gpu


def planned(s, target):
    ds = sim.DeviceScript(s)
    return ds, ds.plan(target)


def run(ds, s, states, cycles, cons=None, cap=0, off=0, stream=None, first_cycle=0):
    st = sim.u32_to_dev(states.reshape(-1))
    n = max(1, s.sram_storage_size)
    sram = torch.zeros(n, dtype=torch.int32, device="cuda")
    sram_x = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    c = sim.u32_to_dev(cons) if cons is not None else None
    ev = sim.new_event_buffer(cap) if cons is not None else None
    torch.cuda.synchronize()
    sim.simulate(ds, st, cycles, states.shape[1], sram, sram_x, constraints=c, events=ev,
                 event_capacity=cap, arrival_state_offset=off, stream=stream,
                 first_cycle=first_cycle)
    return st, sram, sram_x, ev


@pytest.mark.parametrize("target", [0, 1, 5, sim.PLAN_NO_MIRROR])
@pytest.mark.parametrize("kind,nb,split,parts,xprop,cycles", [
    ("tiny", 4, (), 0, False, 1),             # one cycle, one major stage
    ("tiny", 148, (5,), 0, True, 9),
    ("small", 64, (8, 16, 24), 0, False, 40),  # one partition a stage: mirrored
    ("small", 148, (8, 16, 24), 37, False, 7),
    ("sram", 16, (8,), 0, True, 33),           # SRAMs, duplicates
    ("sram", 3, (), 0, False, 6),
    ("soc_mini", 148, (20, 40, 60), 37, True, 12),
    ("soc_mini", 296, (4, 8, 12, 40), 296, True, 4),  # 40 boomerang stages a partition
    ("soc_mini", 296, (20, 40, 60), 296, True, 4),  # more items than SMs
])
def test_plan_matches_oracle(kind, nb, split, parts, xprop, cycles, target):
    s = cases.script(kind, nb, split, xprop=xprop, target_parts=parts)
    ds, plan = planned(s, target)
    assert plan is not None
    if target == 0:
        per = np.bincount(s.stage_block_part[:, 0]).max()
        assert bool(plan.mirrored) == (per <= 2)
    if target == sim.PLAN_NO_MIRROR:
        assert not plan.mirrored
    states = cases.stimulus(kind, s, cycles, x_init=xprop)
    want, wsram, wsx, _ = run_oracle(s, states, cycles)
    st, sram, sram_x, _ = run(ds, s, states, cycles)
    assert sim.status() == 0
    assert np.array_equal(sim.dev_to_u32(st).reshape(states.shape), want)
    assert np.array_equal(sim.dev_to_u32(sram)[:wsram.size], wsram)
    if xprop:
        assert np.array_equal(sim.dev_to_u32(sram_x)[:wsx.size], wsx)


@pytest.mark.parametrize("target", [0, sim.PLAN_NO_MIRROR])
@pytest.mark.parametrize("kind,nb,split", [("sram", 16, (8,)), ("tiny", 4, (5,))])
def test_plan_timing_matches_oracle(kind, nb, split, target):
    s = cases.script(kind, nb, split, timing_seed=9)
    s.enable_timing_arrivals()
    try:
        states = cases.stimulus(kind, s, 24)
        cons = cases.constraint_buffer(kind, s, clock_ps=120, setup=30, hold=150)
        off = s.arrival_state_offset
        want, _, _, (wev, wcnt) = run_oracle(s, states, 24, constraints=cons, cap=1 << 16,
                                             arrival_off=off)
        ds, plan = planned(s, target)
        assert plan is not None
        st, _, _, ev = run(ds, s, states, 24, cons, 1 << 16, off)
        assert sim.status() == 0
    finally:
        s.timing_arrivals_enabled = False
        s.arrival_state_offset = 0
    rec, cnt, _ = sim.read_events(ev)
    assert np.array_equal(sim.dev_to_u32(st).reshape(states.shape), want)
    assert cnt == wcnt and wcnt > 0
    assert sorted_events(rec) == sorted_events(wev.view(np.uint32))


def test_plan_launches_on_two_streams_and_graph_replay():
    """One script's plan, launches that may overlap on two streams (each with
    its own exchange buffer), and a captured launch replayed."""
    s = cases.script("soc_mini", 148, (20, 40, 60), xprop=True, target_parts=37)
    ds, plan = planned(s, 0)
    assert plan is not None and not plan.mirrored
    states = cases.stimulus("soc_mini", s, 12, x_init=True)
    want, _, _, _ = run_oracle(s, states, 12)
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = [run(ds, s, states, 12, stream=k) for k in streams]
    for k, o in zip(streams, outs):
        assert sim.status(k) == 0
        assert np.array_equal(sim.dev_to_u32(o[0]).reshape(states.shape), want)
    st, sram, sram_x, _ = outs[0]
    fresh = sim.u32_to_dev(states.reshape(-1))
    torch.cuda.synchronize()
    with torch.cuda.stream(streams[0]):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=streams[0]):
            sim.simulate(ds, st, 12, states.shape[1], sram, sram_x)
        for _ in range(2):
            st.copy_(fresh)
            sram.zero_()
            sram_x.fill_(-1)
            g.replay()
        streams[0].synchronize()
    assert np.array_equal(sim.dev_to_u32(st).reshape(states.shape), want)
    del g


@pytest.mark.parametrize("spoil", ["stale slot", "same stage", "two writers"])
def test_plan_refuses_what_it_does_not_represent(spoil):
    """A writeout slot nothing writes, a read of a word of the own major
    stage, and two writers of a word depend on the order of a block's
    partitions: no plan, and the script runs in its own form as before."""
    s = cases.script("tiny", 8, (5,))

    class Spoiled:
        def __init__(self):
            self.__dict__.update(s.__dict__)
            self.blocks_data = s.blocks_data.copy()

    b = Spoiled()
    bd = b.blocks_data
    offs = []
    for e in range(s.num_blocks * s.num_major_stages):
        off = int(s.blocks_start[e])
        if bd[off]:
            offs.append((e // s.num_blocks, off))
    (_, off), (_, off2) = offs[0], offs[1]
    if spoil == "stale slot":
        bd[off + 128] |= 0xFFFF  # slot 0 without a hook
    elif spoil == "same stage":
        ms0 = [o for m, o in offs if m == 0]
        g = bd[ms0[0] + 256: ms0[0] + 256 + 512].reshape(-1, 2)
        k = int(np.nonzero(g[:, 1])[0][0])
        g[k, 0] = 0x80000000 | int(bd[ms0[0] + 3])  # its own first word, staged
    else:
        bd[off2 + 3] = bd[off + 3]
    ds = sim.DeviceScript(b)
    assert ds.plan() is None
    states = cases.stimulus("tiny", s, 3)
    st, _, _, _ = run(ds, s, states, 3)
    assert sim.status() == 0
    want = run(ds, s, states, 3)[0] if spoil == "two writers" else None
    assert want is None or want.shape == st.shape


@pytest.mark.parametrize("cycles", [7, 8, 20])
def test_legacy_symbol_around_the_plan_rule(cycles):
    """The reference-compatible symbol builds the plan from 8 cycles on."""
    s = cases.script("sram", 16, (8,), xprop=True)
    states = cases.stimulus("sram", s, cycles, x_init=True)
    want, wsram, wsx, _ = run_oracle(s, states, cycles)
    ds = sim.DeviceScript(s)
    st = sim.u32_to_dev(states.reshape(-1))
    n = max(1, s.sram_storage_size)
    sram = torch.zeros(n, dtype=torch.int32, device="cuda")
    sram_x = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    sim.lib().simulate_v1_noninteractive_simple_scan_cuda(
        s.num_blocks, s.num_major_stages, ds.blocks_start.data_ptr(), ds.blocks_data.data_ptr(),
        sram.data_ptr(), sram_x.data_ptr(), cycles, states.shape[1], st.data_ptr(), 0)
    assert np.array_equal(sim.dev_to_u32(st).reshape(states.shape), want)
    assert np.array_equal(sim.dev_to_u32(sram)[:wsram.size], wsram)
    assert np.array_equal(sim.dev_to_u32(sram_x)[:wsx.size], wsx)


def test_first_timed_launch_on_another_stream_and_two_threads():
    """The plan and the arrival tables are made inside the first launch; it may
    be on another stream than the current one, and two threads may share the
    script."""
    import threading
    s = cases.script("sram", 16, (8,), timing_seed=9)
    s.enable_timing_arrivals()
    try:
        states = cases.stimulus("sram", s, 12)
        cons = cases.constraint_buffer("sram", s, clock_ps=120, setup=30, hold=150)
        off = s.arrival_state_offset
        want, _, _, _ = run_oracle(s, states, 12, constraints=cons, cap=1 << 16, arrival_off=off)
        ds = sim.DeviceScript(s)
        streams = [torch.cuda.Stream() for _ in range(2)]
        outs = [None, None]

        def work(k):
            outs[k] = run(ds, s, states, 12, cons, 1 << 16, off, stream=streams[k])

        threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for k in range(2):
            assert sim.status(streams[k]) == 0
            assert np.array_equal(sim.dev_to_u32(outs[k][0]).reshape(states.shape), want)
    finally:
        s.timing_arrivals_enabled = False
        s.arrival_state_offset = 0
