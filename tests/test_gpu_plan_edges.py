"""Planned runs (one-stream and batched) where their memory layout, the order
of their CTAs or their choice of form can go wrong, against the CPU oracle."""
import threading

import numpy as np
import pytest
import torch

import cases
import test_gpu_batched as tgb
from jacquard_b200 import batched, frontend, sim, state
from test_gpu_plain import run_gpu, run_oracle

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


def one_way_design(n_src=512, n_sink=512, depth=64, seed=5):
    """Registers that only depend on themselves (shift and XOR), and registers
    that nothing reads behind `depth` levels of gates over them."""
    lib = frontend._lib()
    rng = np.random.default_rng(seed)
    b = lib.jqf_builder_new()
    clk = lib.jqf_builder_clock_flag(b)
    x = lib.jqf_builder_input(b) << 1
    q = [lib.jqf_builder_dff(b) << 1 for _ in range(n_src + n_sink)]

    def and_(u, v):
        return lib.jqf_builder_and(b, u, v)

    for i in range(n_src):
        u, v = q[i - 1] if i else x, q[(i * 7 + 3) % n_src]
        assert lib.jqf_builder_set_dff(b, i, and_(and_(u, v) ^ 1, and_(u ^ 1, v ^ 1) ^ 1), clk << 1) == 0
    for k in range(n_sink):
        s = q[k % n_src]
        for _ in range(depth):
            s = and_(s ^ int(rng.integers(2)), q[int(rng.integers(n_src))] ^ int(rng.integers(2))) ^ 1
        assert lib.jqf_builder_set_dff(b, n_src + k, s, clk << 1) == 0
    lib.jqf_builder_output(b, q[n_src])
    assert lib.jqf_builder_finish(b, clk, 0) == 0
    return frontend.Design.from_handle(b), n_src


@pytest.mark.parametrize("xprop", [False, True])
@pytest.mark.parametrize("parts", [3, 6])
def test_producers_do_not_run_ahead_of_consumers(parts, xprop):
    """One-way dependencies in the flow form: nothing but the ring's own count
    holds the CTAs of the sources back from those of the much slower sinks,
    whose words they overwrite four cycles later."""
    d, n_src = one_way_design()
    s = d.build_script(num_blocks=16, xprop=xprop, target_parts=parts, merge_passes=0)
    assert s.num_major_stages == 1
    word = state.dff_positions(s, d) >> 5
    src, sink = set(word[:n_src].tolist()), set(word[n_src:].tolist())
    assert len(src - sink) >= 8  # words (and so items) of sources alone
    cycles = 400
    states = state.random_stimulus_states(s, d, cycles, 3)
    if xprop:
        states = state.expand_states_for_xprop(states, s)
    states[0, :s.reg_io_state_size] |= np.random.default_rng(1).integers(
        0, 2**32, s.reg_io_state_size, dtype=np.uint32)
    want, _, _, _ = run_oracle(s, states, cycles)
    ds = sim.DeviceScript(s)
    assert not ds.plan(sim.PLAN_NO_MIRROR).mirrored
    for _ in range(3):
        st = sim.u32_to_dev(states.reshape(-1))
        z = torch.zeros(1, dtype=torch.int32, device="cuda")
        sim.simulate(ds, st, cycles, states.shape[1], z, z)
        assert sim.status() == 0
        assert np.array_equal(sim.dev_to_u32(st).reshape(states.shape), want)


@pytest.mark.parametrize("cycles", [1, 2, 3, 5])
def test_short_mirrored_launches_in_a_row(cycles):
    """The cluster form's CTAs end only when the words sent to them have
    arrived: many short launches, each on the state the last one left."""
    s = cases.script("small", 64, (8, 16, 24))
    ds = sim.DeviceScript(s)
    assert ds.plan().mirrored
    n = 40 * cycles
    states = cases.stimulus("small", s, n)
    want, _, _, _ = run_oracle(s, states, n)
    st = sim.u32_to_dev(states.reshape(-1))
    z = torch.zeros(1, dtype=torch.int32, device="cuda")
    eff = states.shape[1]
    for k in range(0, n, cycles):
        sim.simulate(ds, st[k * eff:], cycles, eff, z, z)
    assert sim.status() == 0
    assert np.array_equal(sim.dev_to_u32(st).reshape(states.shape), want)


def _threads(*works):
    errors = []

    def guard(w):
        try:
            w()
        except Exception as e:  # reported by the caller's assertion
            errors.append(e)

    ts = [threading.Thread(target=guard, args=(w,)) for w in works]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors


def test_two_threads_launch_plans_of_different_size():
    """Two threads launch the same kernel for scripts whose plans need very
    different shared memory, each on its own stream; then the same for
    batched runs.  No launch is refused."""
    scripts = [cases.script("tiny", 8, (5,), xprop=True),
               cases.script("soc_mini", 148, (20, 40, 60), xprop=True, target_parts=37)]
    kinds, works, check = ("tiny", "soc_mini"), [], []
    dss = [sim.DeviceScript(s) for s in scripts]
    plans = [ds.plan(sim.PLAN_NO_MIRROR) for ds in dss]
    assert plans[0].paired == plans[1].paired and plans[1].max_slots > 2 * plans[0].max_slots
    for k, s, ds in zip(kinds, scripts, dss):
        states = cases.stimulus(k, s, 2, x_init=True)
        st = sim.u32_to_dev(states.reshape(-1))
        n = max(1, s.sram_storage_size)
        sram, sram_x = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
        q = torch.cuda.Stream()

        def work(ds=ds, st=st, eff=states.shape[1], sram=sram, sram_x=sram_x, q=q):
            for _ in range(400):
                sim.simulate(ds, st, 2, eff, sram, sram_x, stream=q)

        works.append(work)
        check.append(q)
    torch.cuda.synchronize()
    _threads(*works)
    for q in check:
        assert sim.status(q) == 0
    works = []
    sims = [batched.BatchedSim(s, 2, lanes_per_item=2) for s in scripts]
    assert sims[0].plan.paired == sims[1].plan.paired
    for B in sims:
        B.load_state(np.zeros((2, B.sig), np.uint32))
        q = torch.cuda.Stream()

        def work(B=B, q=q):
            for _ in range(400):
                B.run(None, 2, stream=q)
            assert B.status(q) == 0

        works.append(work)
    torch.cuda.synchronize()
    _threads(*works)


class Edited:
    """A script with its own copy of the instruction words."""

    def __init__(self, s):
        self.__dict__.update(s.__dict__)
        self.blocks_data = s.blocks_data.copy()

    def partitions(self):
        """(major stage, block, word offset) in script order."""
        bd, out = self.blocks_data, []
        for e in range(self.num_major_stages * self.num_blocks):
            off = int(self.blocks_start[e])
            while bd[off]:
                out.append((e // self.num_blocks, e % self.num_blocks, off))
                if bd[off + 1]:
                    break
                off += 256 + 512 * int(bd[off + 6]) + 5120 * (int(bd[off]) + 2)
        return out


def script_form(b, states, cycles):
    """(snapshots, SRAM, SRAM X) of a run of the script's own form."""
    st = sim.u32_to_dev(states.reshape(-1))
    n = max(1, b.sram_storage_size)
    sram = torch.zeros(n, dtype=torch.int32, device="cuda")
    sram_x = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    sim.simulate(sim.DeviceScript(b), st, cycles, states.shape[1], sram, sram_x, planned=False)
    assert sim.status() == 0
    return sim.dev_to_u32(st).reshape(states.shape), sim.dev_to_u32(sram), sim.dev_to_u32(sram_x)


def check_without_plan(b, states, cycles, want):
    """No plan of either kind, and every entry point gives the script's result."""
    assert sim.DeviceScript(b).plan() is None
    for legacy in (False, True):
        got = run_gpu(b, states, cycles, legacy=legacy)[:3]
        for g, w in zip(got, want):
            assert np.array_equal(g[:w.size] if g.ndim == 1 else g, w)
    assert batched.BatchedSim(b, 2).plan is None


def test_shared_sram_and_x_words_read_as_values_have_no_plan():
    """Two partitions of a block on one SRAM run in the block's order, and a
    read of another partition's X word as a value needs the barrier of its
    major stage: the plan orders neither, so the script runs in its own form."""
    s = cases.script("sram", 1, (), xprop=True, target_parts=4)
    states = cases.stimulus("sram", s, 40, x_init=True)
    b = Edited(s)
    ports = [off for _, _, off in b.partitions() if b.blocks_data[off + 4]]
    assert len(ports) == 3
    b.blocks_data[ports[1] + 5] = b.blocks_data[ports[0] + 5]
    check_without_plan(b, states, 40, run_oracle(b, states, 40)[:3])

    s = cases.script("sram", 16, (8,), xprop=True, target_parts=4)
    states = cases.stimulus("sram", s, 40, x_init=True)
    b = Edited(s)
    bd = b.blocks_data
    first, second = [[o for m, _, o in b.partitions() if m == k] for k in (0, 1)]
    g = bd[first[0] + 256:first[0] + 256 + 512].reshape(-1, 2)
    k = int(np.nonzero(g[:, 1])[0][0])
    g[k, 0] = bd[second[0] + 9] + bd[second[0] + 3] + 1  # an X word stage 1 writes
    check_without_plan(b, states, 40, script_form(b, states, 40))


def test_each_asked_for_plan_is_its_own():
    """plan(target) gives the plan of that target whatever was built before,
    and simulate() runs the one asked for last."""
    s = cases.script("small", 64, (8, 16, 24))
    states = cases.stimulus("small", s, 20)
    want, _, _, _ = run_oracle(s, states, 20)
    ds = sim.DeviceScript(s)
    z = torch.zeros(1, dtype=torch.int32, device="cuda")

    def run():
        st = sim.u32_to_dev(states.reshape(-1))
        sim.simulate(ds, st, 20, states.shape[1], z, z)
        assert sim.status() == 0
        assert np.array_equal(sim.dev_to_u32(st).reshape(states.shape), want)

    run()
    first = ds.plan()
    assert first.mirrored
    for target, items in [(sim.PLAN_NO_MIRROR, None), (5, 5), (0, 16)]:
        plan = ds.plan(target)
        assert bool(plan.mirrored) == (target != sim.PLAN_NO_MIRROR)
        assert items is None or plan.widest == items
        run()
    assert ds.plan() is first


def test_no_memory_for_a_plan(monkeypatch):
    """A plan's workspace that cannot be allocated: the script's own form (one
    stream) and the prepared script (batched) run, and a later plan() builds it."""
    huge = 1 << 42  # words
    monkeypatch.setattr(sim.lib(), "jq_plain_plan_words", lambda *a: huge)
    monkeypatch.setattr(batched.lib(), "jq_batched_plan_words", lambda *a: huge)
    s = cases.script("sram", 16, (8,), xprop=True)
    states = cases.stimulus("sram", s, 10, x_init=True)
    want, _, _, _ = run_oracle(s, states, 10)
    ds = sim.DeviceScript(s)

    def run():
        st = sim.u32_to_dev(states.reshape(-1))
        n = s.sram_storage_size
        sim.simulate(ds, st, 10, states.shape[1], torch.zeros(n, dtype=torch.int32, device="cuda"),
                     torch.full((n,), -1, dtype=torch.int32, device="cuda"))
        assert sim.status() == 0
        assert np.array_equal(sim.dev_to_u32(st).reshape(states.shape), want)

    run()
    assert ds.plan() is None
    c = tgb.BatchedCase("sram", s, 2)
    assert c.B.plan is None
    c.launch()
    assert c.B.status() == 0
    c.verify()
    monkeypatch.undo()
    assert ds.plan() is not None
    run()


def test_plain_stream_handles_and_bare_launch_arrays():
    """simulate() takes any object with a cuda_stream handle as the stream, and
    a DeviceScript of nothing but the launch arrays."""
    class Handle:
        def __init__(self, stream):
            self.cuda_stream = stream.cuda_stream

    class Arrays:
        def __init__(self, s):
            for f in ("num_blocks", "num_major_stages", "blocks_start", "blocks_data"):
                setattr(self, f, getattr(s, f))

    s = cases.script("sram", 16, (8,), timing_seed=9)
    n = s.sram_storage_size
    for script, off in [(s, 0), (Arrays(s), 0), (Arrays(s), s.reg_io_state_size)]:
        states = cases.stimulus("sram", s, 10)
        if off:
            states = state.expand_states_for_arrivals(states, s)
        want, _, _, _ = run_oracle(s, states, 10, arrival_off=off)
        q = torch.cuda.Stream()
        for handle in (q, Handle(q), Handle(torch.cuda.default_stream())):
            st = sim.u32_to_dev(states.reshape(-1))
            sram = torch.zeros(n, dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            sim.simulate(sim.DeviceScript(script), st, 10, states.shape[1], sram, sram,
                         arrival_state_offset=off, stream=handle)
            assert sim.status(handle) == 0
            assert np.array_equal(sim.dev_to_u32(st).reshape(states.shape), want)


def test_two_threads_call_the_reference_symbol():
    """Calls on one device take turns and keep to their own scripts."""
    works = []
    for kind, nb, split in (("tiny", 8, (5,)), ("sram", 16, (8,))):
        s = cases.script(kind, nb, split)
        states = cases.stimulus(kind, s, 20)
        want, _, _, _ = run_oracle(s, states, 20)

        def work(s=s, states=states, want=want):
            for _ in range(10):
                assert np.array_equal(run_gpu(s, states, 20, legacy=True)[0], want)

        works.append(work)
    _threads(*works)


def spoiled(spoil):
    """A script that has no plan, whose result the order of its blocks decides."""
    s = cases.script("tiny", 1, (5,), target_parts=4)
    b = Edited(s)
    bd = b.blocks_data
    offs = [o for m, _, o in b.partitions() if m == 0]
    last = offs[-1]
    if spoil == "stale slot":
        bd[last + 128] |= 0xFFFF  # slot 0 without a hook
    elif spoil == "same stage":
        g = bd[last + 256:last + 256 + 512].reshape(-1, 2)
        k = int(np.nonzero(g[:, 1])[0][0])
        g[k, 0] = 0x80000000 | int(bd[offs[0] + 3])  # the first partition's word, staged
    else:
        bd[last + 3] = bd[offs[0] + 3]
    return s, b


@pytest.mark.parametrize("spoil", ["stale slot", "same stage", "two writers"])
def test_refused_scripts_give_the_oracles_result(spoil):
    """Scripts that the plan does not represent, each spoiled in its last
    partition, in one block (so that the result is defined): one-stream runs,
    the script form and the reference symbol give the oracle's snapshots."""
    s, b = spoiled(spoil)
    states = cases.stimulus("tiny", s, 20)
    want = run_oracle(b, states, 20)[0]
    assert sim.DeviceScript(b).plan() is None
    assert batched.BatchedSim(b, 2).plan is None
    assert np.array_equal(run_gpu(b, states, 20)[0], want)
    assert np.array_equal(script_form(b, states, 20)[0], want)
    assert np.array_equal(run_gpu(b, states, 20, legacy=True)[0], want)


@pytest.mark.parametrize("kind,nb,split,cycles", [
    ("tiny", 4, (), 8), ("tiny", 4, (), 11), ("tiny", 4, (), 12), ("tiny", 8, (5,), 7),
    ("tiny", 8, (5,), 8)])
def test_reference_symbol_around_the_stage_rule(kind, nb, split, cycles):
    """The symbol builds the plan from 8 cycles and 12 stages on."""
    s = cases.script(kind, nb, split)
    states = cases.stimulus(kind, s, cycles)
    want, _, _, _ = run_oracle(s, states, cycles)
    assert np.array_equal(run_gpu(s, states, cycles, legacy=True)[0], want)


def test_planned_octets_do_not_keep_the_prepared_script():
    """Asking for octet items checks the prepared script's capacity; a run on
    the plan does not read that script, and it is made again where it is."""
    s = cases.script("sram", 16, (8,), xprop=True, target_parts=16)
    B = batched.BatchedSim(s, 8, lanes_per_item=8)
    assert B.plan is not None and B._prep is None
    assert B.prepared.numel() == B.ds.blocks_data.numel()
    assert B.octet_need() <= batched.octet_capacity()


@pytest.mark.parametrize("parts,split_into", [(37, 4), (148, 1)])
def test_items_of_split_partitions(parts, split_into):
    """Octet items of the training family: every partition of a full stage in
    as many items as fill the SMs, and part_cycles their sum."""
    s = cases.script("soc_mini", 148, (20, 40, 60), xprop=True, target_parts=parts)
    B = batched.BatchedSim(s, 8, lanes_per_item=0)
    per = B.items_per_partition()
    stage = np.asarray(s.stage_block_part)[:, 0]
    assert per.sum() == B.plan.stage_item[32] and per.min() >= 1
    groups = 8 // B.plan.lanes_per_item
    for ms in range(s.num_major_stages):
        n = int((stage == ms).sum())
        want = max(1, min(16, (148 // groups) // n))
        assert (per[stage == ms] == want).all()
    if B.plan.lanes_per_item == 8:
        assert per.max() == split_into
    pc = torch.zeros(s.num_partitions, dtype=torch.int64, device="cuda")
    B.load_state(np.zeros((8, B.sig), np.uint32))
    B.run(None, 3, part_cycles=pc)
    assert B.status() == 0
    assert (pc > 0).all()
    assert (batched.BatchedSim(s, 8, lanes_per_item=0, planned=False).items_per_partition() == 1).all()
