"""Performance cases of the interpreter: what a program that simulates designs
with this package has it do, through the package's public entry points.

A case names a design (clusters of levelized random ANDs, DFFs, SRAMs), the
script built for it (logic levels per major stage, script blocks, cone or
balanced partitions, X-propagation), a launch form and a window of cycles:

  plain    one stimulus stream, sim.simulate (jq_simulate); with `timed` the
           arrivals are written and setup/hold violations are drained
  legacy   one stimulus stream through the reference-compatible symbol
  batched  32 * lanes streams, batched.BatchedSim.run; with `timed` the
           setup/hold checks run per stream and the records are drained
  multi    several designs of uneven size in one batched launch

The script of a design is built once and kept, as a program that loads a
design and then simulates many stimuli does.  The stimulus (and so every
output) comes from the seed.  All outputs are words and counts, compared bit
by bit; they have no more exact value than the one the interpreter gives.
"""
import functools
import math

import numpy as np
import torch

from jacquard_b200 import batched, frontend, sim, state, timing

P_TOGGLE_BITS = 2  # an input toggles with probability 2^-2 per cycle
RESET_CYCLES = 16
CLOCK_PS, SETUP_PS, HOLD_PS = 10_000, 30, 10


def _case(path, clusters, cycles, *, nodes=4096, depth=80, dffs=None, pis=128, pos=128, srams=0,
          split=4, blocks=148, parts=0, xprop=True, timed=False, lanes=0, per_item=0, designs=1):
    return {"path": path, "clusters": clusters, "nodes": nodes, "depth": depth,
            "dffs": max(64, 200_000 * clusters // 512) if dffs is None else dffs,
            "pis": pis, "pos": pos, "srams": srams, "split": split, "blocks": blocks,
            "parts": parts, "xprop": xprop, "timed": timed, "lanes": lanes, "per_item": per_item,
            "designs": designs, "cycles": cycles}


def _small(path, cycles, **kw):
    """16,384 ANDs to depth 32, 1,024 DFFs, 32 inputs and outputs, 2-state."""
    return _case(path, 1, cycles, nodes=16384, depth=32, dffs=1024, pis=32, pos=32, split=8,
                 xprop=False, **kw)


def listed():
    return [
        # a small block under test, one stimulus: launches and latency count
        dict(_small("plain", 64, blocks=64), name="small-1"),
        # the 2M-gate SoC with X-propagation, one stimulus, as a single
        # waveform run of a large design has it
        dict(_case("plain", 512, 16, srams=16, blocks=296), name="soc2M-1"),
        # a mid-size 2-state design called through the reference's symbol by a
        # host that was written for the reference
        dict(_case("legacy", 64, 32, srams=2, xprop=False), name="soc256k-1-legacy"),
        # timing sign-off of one stimulus: arrivals and setup/hold violations
        dict(_case("plain", 64, 16, srams=2, timed=True, blocks=296), name="soc256k-1-timed"),
        # 32 seeds of the small block (one lane word)
        dict(_small("batched", 64, parts=37, lanes=1), name="small-32"),
        # 64 seeds of a mid-size design, lane pairs, one round of items
        dict(_case("batched", 64, 32, srams=2, parts=148, lanes=2), name="soc256k-64"),
        # 160 seeds (an odd number of lane words: single-lane items), on the
        # cone partitions that serve the one-stimulus run too
        dict(_case("batched", 64, 8, srams=2, lanes=5), name="soc256k-160-cone"),
        # 256 seeds of a 2-state design (no X words): the library's own choice
        dict(_case("batched", 128, 32, srams=4, parts=37, xprop=False, lanes=8),
             name="soc512k-256-2state"),
        # the regression of the 2M-gate SoC: 256 streams, octet items
        dict(_case("batched", 512, 64, srams=16, parts=148, lanes=8, per_item=8),
             name="soc2M-256"),
        # twice the streams of a mid-size design (two octet groups)
        dict(_case("batched", 128, 32, srams=4, parts=74, lanes=16, per_item=8),
             name="soc512k-512"),
        # setup/hold checks on 256 streams, violations drained
        dict(_case("batched", 128, 8, srams=4, parts=148, lanes=8, per_item=8, timed=True),
             name="soc512k-256-timed"),
        # several designs of uneven size sharing one launch (more items than CTAs)
        dict(_case("multi", 160, 16, srams=2, parts=1, lanes=8, per_item=8, designs=5),
             name="mixed5-256"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    path = rng.choice(["plain", "plain", "legacy", "batched", "batched", "batched", "multi"])
    clusters = log(1, 96)
    kw = dict(nodes=log(900, 4097), depth=rng.randrange(12, 81), pis=rng.randrange(9, 140),
              pos=rng.randrange(7, 140), srams=rng.choice([0, 1, 2, 3]),
              split=rng.choice([3, 4, 4, 5]), xprop=rng.random() < 0.65)
    kw["dffs"] = max(40, log(150, 500) * clusters)
    cycles = 2 * log(3, 24)  # even windows: the batched state ends in its first buffer
    if path in ("plain", "legacy"):
        return _case(path, clusters, cycles, blocks=rng.choice([37, 148, 296]),
                     timed=path == "plain" and rng.random() < 0.3, **kw)
    if path == "multi":
        kw.update(xprop=True)
        return _case(path, clusters, cycles, parts=1, lanes=8, per_item=8,
                     designs=rng.randrange(2, 5), **kw)
    form = rng.choice(["lanes", "cone", "octets", "octets"])
    if form == "octets":
        lanes = rng.choice([8, 8, 16])
        kw.update(xprop=True)
        timed = rng.random() < 0.25  # a window's violations fit the event buffer
        return _case(path, clusters, min(cycles, 8) if timed else cycles,
                     parts=148 // (lanes // 8), lanes=lanes, per_item=8, timed=timed, **kw)
    lanes = rng.randrange(1, 9)
    return _case(path, clusters, cycles, lanes=lanes,
                 parts=0 if form == "cone" else 148 // max(1, (lanes + 1) // 2), **kw)


# ------------------------------------------------------------------ designs

def _sizes(case):
    """Clusters of each design of the case (halving from the largest)."""
    return [max(1, case["clusters"] >> k) for k in range(case["designs"])]


def _key(case):
    return tuple(case[k] for k in ("path", "clusters", "nodes", "depth", "dffs", "pis", "pos",
                                   "srams", "split", "blocks", "parts", "xprop", "timed",
                                   "designs"))


@functools.lru_cache(maxsize=1)
def _design(clusters, nodes, depth, dffs, pis, pos, srams, seed):
    return frontend.Design(frontend.DesignParams(
        seed=seed, n_clusters=clusters, nodes_per_cluster=nodes, depth=depth, fanin_window=4,
        intra_frac=0.9 if clusters > 1 else 1.0, n_dff=dffs, n_pi=pis, n_po=pos, n_sram=srams,
        sram_addr_bits=10, with_reset=1 if clusters > 1 else 0))


@functools.lru_cache(maxsize=32)
def _load(key):
    """[(design facts, script, constraint buffer or None)] of a case."""
    path, clusters, nodes, depth, dffs, pis, pos, srams, split, blocks, parts, xprop, timed, n = key
    out = []
    for k, c in enumerate(max(1, clusters >> j) for j in range(n)):
        d = _design(c, nodes, depth, max(40, dffs * c // clusters), pis, pos, srams, 2 + k)
        if timed:  # per-gate delays U[20, 200] ps
            r = np.random.default_rng(3).integers(20, 201, size=d.num_pins + 1).astype(np.uint32)
            r[d.kind != 1] = 0
            d.set_delays(r, r)
        levels = tuple(range(split, depth, split))
        p = parts
        if path == "multi":  # about 650 gates per partition and major stage
            p = max(1, -(-int(d.num_and) // (len(levels) + 1) // 650))
        s = d.build_script(num_blocks=blocks, xprop=xprop, level_split=levels, target_cone=6000,
                           target_parts=p, merge_passes=0 if p else 1)
        cons = None
        if timed:
            zero = np.zeros(d.num_pins + 1, np.uint32)
            d.set_delays(zero, zero)
            ca = np.random.default_rng(5).integers(0, 301, size=int(d.num_dffs)).astype(np.int16)
            cons = timing.constraint_buffer(d, s, CLOCK_PS, SETUP_PS, HOLD_PS, ca)
            if path == "plain":
                s.enable_timing_arrivals()
        lay = np.asarray(s.input_layout)
        out.append({"script": s, "cons": cons, "in_pos": state.input_positions(s),
                    "clock": lay == d.clock_flag_pin,
                    "reset": lay == d.reset_pin if d.reset_pin else np.zeros(lay.size, bool),
                    "po": state.po_positions(s, d)})
    return out


def _lane_inputs(rng, d, cycles, lanes):
    """(cycles + 1, lanes, inputs) u32 lane words: every input toggles with
    probability 2^-P_TOGGLE_BITS per cycle and stream, the clock flag is set,
    the reset is held for the first RESET_CYCLES snapshots."""
    n = d["in_pos"].size
    flip = rng.integers(0, 2**32, size=(cycles + 1, lanes, n), dtype=np.uint32)
    for _ in range(P_TOGGLE_BITS - 1):
        flip[1:] &= rng.integers(0, 2**32, size=(cycles, lanes, n), dtype=np.uint32)
    vals = np.bitwise_xor.accumulate(flip, axis=0)
    vals[:, :, d["clock"]] = 0xFFFFFFFF
    vals[:, :, d["reset"]] = 0
    vals[:RESET_CYCLES, :, d["reset"]] = 0xFFFFFFFF
    return vals


# ------------------------------------------------------------------- states

def _prepare_single(case, rng):
    d = _load(_key(case))[0]
    s, cycles = d["script"], case["cycles"]
    bits = (_lane_inputs(rng, d, cycles, 1)[:, 0, :] & 1).astype(np.uint8)
    v = state.pack_inputs(s, bits)
    if s.xprop_enabled:
        v = state.expand_states_for_xprop(v, s)
        v[0, s.reg_io_state_size:] = state.xmask_all_state_x(s)
    if s.timing_arrivals_enabled:
        v = state.expand_states_for_arrivals(v, s)
    n = max(1, s.sram_storage_size)
    st = {"path": case["path"], "cycles": cycles, "eff": v.shape[1], "ds": sim.DeviceScript(s),
          "states": sim.u32_to_dev(np.ascontiguousarray(v).reshape(-1)),
          "sram": torch.zeros(n, dtype=torch.int32, device="cuda"),
          "sram_x": torch.full((n,), -1, dtype=torch.int32, device="cuda"),
          "arrivals": s.arrival_state_offset, "cons": None}
    if case["timed"]:
        st["cons"] = sim.u32_to_dev(d["cons"])
        st["capacity"] = 1 << 18
        st["events"] = sim.new_event_buffer(st["capacity"])
    return st


def _prepare_batched(case, rng):
    ds = _load(_key(case))
    lanes, cycles = case["lanes"], case["cycles"]
    if case["path"] == "multi":
        script = batched.CombinedScript([d["script"] for d in ds])
        po = np.concatenate([[script.signal(i, int(p)) for p in d["po"]]
                             for i, d in enumerate(ds)]).astype(np.int64)
    else:
        script, po = ds[0]["script"], ds[0]["po"]
    try:
        B = batched.BatchedSim(script, lanes, po_signals=po, lanes_per_item=case["per_item"])
    except ValueError:  # partitions too large for the asked-for items: the library's choice
        B = batched.BatchedSim(script, lanes, po_signals=po)
    stim = np.zeros((cycles + 1, lanes, B.in_sigs), np.uint32)
    col = 0
    for d in ds:
        stim[:, :, col + d["in_pos"]] = _lane_inputs(rng, d, cycles, lanes)
        col += batched.input_words(d["script"]) * 32
    # snapshot 0: the inputs of cycle 0, every register X (multi: all known 0)
    snap = np.zeros((lanes, B.sig), np.uint32)
    if case["path"] != "multi":
        snap[:, :B.in_sigs] = stim[0]
        if script.xprop_enabled:
            x = np.unpackbits(state.xmask_all_state_x(script).view(np.uint8), bitorder="little")
            snap[:, B.sig // 2:] = np.where(x, np.uint32(0xFFFFFFFF), np.uint32(0))
    B.load_state(snap)
    B.reset_sram(x=True)
    st = {"path": case["path"], "cycles": cycles, "B": B, "timing": None,
          "stim": sim.u32_to_dev(stim.reshape(-1)),
          "wave": torch.empty(cycles * len(po) * lanes, dtype=torch.int32, device="cuda")}
    if case["timed"]:
        st["timing"] = batched.Timing(script, ds[0]["cons"], 1 << 23)
    return st


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    return (_prepare_single if case["path"] in ("plain", "legacy") else _prepare_batched)(case, rng)


# --------------------------------------------------------------------- runs

def _violations(events, capacity):
    """The buffer's records in (cycle, word, kind, stream) order, and its count."""
    count = int(events[0].item()) & 0xFFFFFFFF
    n = min(count, capacity)
    rec = events[4:4 + 8 * n].view(n, 8)
    r = rec.to(torch.int64)
    key = ((r[:, 2] << 32 | r[:, 4]) << 3 | r[:, 0]) << 10 | r[:, 3]
    return rec[torch.argsort(key)], count


def run(st):
    if st["path"] == "legacy":
        d = st["ds"]
        sim.lib().simulate_v1_noninteractive_simple_scan_cuda(
            d.num_blocks, d.num_major_stages, d.blocks_start.data_ptr(), d.blocks_data.data_ptr(),
            st["sram"].data_ptr(), st["sram_x"].data_ptr(), st["cycles"], st["eff"],
            st["states"].data_ptr(), 0)
        return {"states": st["states"], "sram": st["sram"]}
    if st["path"] == "plain":
        if st["cons"] is None:
            sim.simulate(st["ds"], st["states"], st["cycles"], st["eff"], st["sram"], st["sram_x"])
            return {"states": st["states"], "sram": st["sram"], "sram_x": st["sram_x"]}
        st["events"][:2].zero_()
        sim.simulate(st["ds"], st["states"], st["cycles"], st["eff"], st["sram"], st["sram_x"],
                     constraints=st["cons"], events=st["events"], event_capacity=st["capacity"],
                     arrival_state_offset=st["arrivals"])
        records, count = _violations(st["events"], st["capacity"])
        return {"states": st["states"], "sram": st["sram"], "sram_x": st["sram_x"],
                "violations": records, "count": count}
    B, tm = st["B"], st["timing"]
    if tm is not None:
        tm.reset_events()
    B.run(st["stim"], st["cycles"], wave=st["wave"], timing=tm)
    out = {"wave": st["wave"], "state": B.final_state(st["cycles"]), "sram": B.sram,
           "sram_x": B.sram_x}
    if tm is not None:
        out["violations"], out["count"] = _violations(tm.events, tm.capacity)
    return out


def work(case):
    """Gate evaluations (one per AND, stream and cycle; with X a second plane
    that takes three) and the bytes in and out: the netlist (two 4-byte
    operands per AND), the registers, inputs and outputs of each snapshot a
    one-stream run writes, or of the first and last one, the stimulus and the
    waveform of a batched run."""
    planes = 2 if case["xprop"] else 1
    streams = 32 * case["lanes"] if case["lanes"] else 1
    sizes = _sizes(case)
    ands = case["nodes"] * sum(sizes)
    regs = sum(max(40, case["dffs"] * c // case["clusters"]) for c in sizes)
    ports = (case["pis"] + case["pos"]) * len(sizes)
    snaps = 2 if case["lanes"] else case["cycles"] + 1
    bits = snaps * regs * planes + (case["cycles"] + 1) * ports
    return {"bytes": 8 * ands + bits * streams / 8,
            "flops": ands * (4 if case["xprop"] else 1) * streams * case["cycles"]}


def exact(case, seed):
    return None
