"""Host driver of the interpreter: the `sim_cuda` step of the reference
(src/bin/jacquard.rs:1089-1256) over this library's C ABI.

Device buffers are torch tensors (int32 storage for u32 words); every kernel
call goes through libjacquard_b200.so -- there is no other execution path.
"""
import ctypes
import threading

import numpy as np
import torch

from ._native import load

vp = ctypes.c_void_p


class SimArgs(ctypes.Structure):
    _fields_ = [("num_blocks", ctypes.c_size_t), ("num_major_stages", ctypes.c_size_t),
                ("blocks_start", vp), ("blocks_data", vp), ("sram_data", vp),
                ("sram_xmask", vp), ("num_cycles", ctypes.c_size_t),
                ("state_size", ctypes.c_size_t), ("states", vp), ("timing_constraints", vp),
                ("events", vp), ("event_capacity", ctypes.c_uint32),
                ("arrival_state_offset", ctypes.c_int32), ("first_cycle", ctypes.c_uint32),
                ("barrier_timeout_cycles", ctypes.c_uint64), ("stream", vp),
                ("stage_depth", vp), ("stage_depth_base", vp)]


class PlainPlan(ctypes.Structure):
    _fields_ = [("num_blocks", ctypes.c_size_t), ("num_major_stages", ctypes.c_size_t),
                ("supported", ctypes.c_uint32), ("max_blob", ctypes.c_uint32),
                ("max_slots", ctypes.c_uint32), ("max_gw", ctypes.c_uint32),
                ("stage_item", ctypes.c_uint32 * 33), ("widest", ctypes.c_uint32),
                ("nbuf", ctypes.c_uint32), ("paired", ctypes.c_uint32), ("mirrored", ctypes.c_uint32), ("rio", ctypes.c_uint32),
                ("xoff", ctypes.c_uint32), ("n_unwritten", ctypes.c_uint32),
                ("stage_words", ctypes.c_uint32 * 32), ("unwritten", vp),
                ("exchange_words", ctypes.c_size_t), ("used_words", ctypes.c_size_t),
                ("blob", vp), ("item_off", vp), ("item_words", vp)]


PLAN_NO_MIRROR = 0xFFFFFFFF
EVENT_WORDS = 8
EVENT_HEADER_WORDS = 4


def lib():
    L = load("libjacquard_b200.so")
    if not getattr(L, "_jq_typed", False):
        L.jq_simulate.restype = ctypes.c_int
        L.jq_simulate.argtypes = [ctypes.POINTER(SimArgs)]
        L.jq_sim_status.restype = ctypes.c_int
        L.jq_sim_status.argtypes = [vp]
        L.jq_max_blocks.restype = ctypes.c_int
        L.jq_max_blocks.argtypes = [ctypes.c_int, ctypes.POINTER(ctypes.c_size_t)]
        L.jq_plain_prepare.restype = ctypes.c_int
        L.jq_plain_prepare.argtypes = [vp, vp, ctypes.c_size_t, ctypes.c_size_t, vp, vp,
                                       ctypes.c_size_t, ctypes.POINTER(ctypes.c_size_t), vp]
        L.jq_plain_plan_words.restype = ctypes.c_size_t
        L.jq_plain_plan_words.argtypes = [ctypes.c_size_t] * 4
        L.jq_plain_plan_build.restype = ctypes.c_int
        L.jq_plain_plan_build.argtypes = [vp, vp, ctypes.c_size_t, ctypes.c_size_t, ctypes.c_size_t,
                                          ctypes.c_uint32, vp, ctypes.c_size_t,
                                          ctypes.POINTER(PlainPlan), vp]
        L.jq_simulate_planned.restype = ctypes.c_int
        L.jq_simulate_planned.argtypes = [ctypes.POINTER(SimArgs), ctypes.POINTER(PlainPlan), vp, vp, vp]
        L.jq_strerror.restype = ctypes.c_char_p
        L.jq_strerror.argtypes = [ctypes.c_int]
        sz, u32p, i32 = ctypes.c_size_t, vp, ctypes.c_int32
        L.simulate_v1_noninteractive_simple_scan_cuda.restype = None
        L.simulate_v1_noninteractive_simple_scan_cuda.argtypes = [sz, sz, vp, vp, vp, vp, sz, sz, vp, i32]
        L.simulate_v1_noninteractive_timed_cuda.restype = None
        L.simulate_v1_noninteractive_timed_cuda.argtypes = [sz, sz, vp, vp, vp, vp, sz, sz, vp, vp, vp, i32]
        L._jq_typed = True
    return L


def u32_to_dev(a, device="cuda"):
    a = np.ascontiguousarray(a, dtype=np.uint32)
    return torch.from_numpy(a.view(np.int32)).to(device)


def dev_to_u32(t):
    return t.cpu().numpy().view(np.uint32)


class DeviceScript:
    """Script arrays resident on the device.  The plan, stage depths and
    arrivals made from them on first use are kept: a changed script takes a new
    DeviceScript."""

    def __init__(self, script, device="cuda"):
        self.script = script
        self.num_blocks = script.num_blocks
        self.num_major_stages = script.num_major_stages
        self.blocks_start = torch.from_numpy(
            np.ascontiguousarray(script.blocks_start, dtype=np.uint64).view(np.int64)).to(device)
        self.blocks_data = u32_to_dev(script.blocks_data, device)
        self._depth = None
        self._plan = None  # the plan in use: (plan, its workspace)
        self._plans = {}   # by target_items
        self._arrivals = None
        self._exchange = {}
        # the tables below are made once, also when threads share the script
        self._lock = threading.RLock()

    def plan(self, target_items=0):
        """The script's gate-list plan (jq_plain_plan_build) that simulate()
        runs from then on, or None when the script is not one it represents
        or its workspace cannot be allocated; built on first use.
        target_items is jq_plain_plan_build's (0: its default, PLAN_NO_MIRROR:
        never the form that keeps the state in shared memory); simulate()
        alone uses the default."""
        with self._lock:
            if target_items not in self._plans:
                try:
                    self._plans[target_items] = self._make_plan(target_items)
                except torch.cuda.OutOfMemoryError:
                    # the script's own form runs in less; plan() tries again
                    self._plan = (None, None)
                    return None
            self._plan = self._plans[target_items]
            return self._plan[0]

    def plan_in_use(self):
        """The plan simulate() runs: the last one asked for, else the default."""
        with self._lock:
            return self.plan() if self._plan is None else self._plan[0]

    def _make_plan(self, target_items):
        """(plan or None, its workspace)"""
        L = lib()
        dev = self.blocks_data.device
        rio = getattr(self.script, "reg_io_state_size", None)
        if rio is None:  # launch arrays alone (the layout is the caller's)
            return None, None
        n = L.jq_plain_plan_words(self.blocks_data.numel(), self.num_blocks,
                                  self.num_major_stages, rio)
        ws = torch.empty(n, dtype=torch.int32, device=dev)
        p = PlainPlan()
        rc = L.jq_plain_plan_build(self.blocks_start.data_ptr(), self.blocks_data.data_ptr(),
                                   self.num_blocks, self.num_major_stages, rio, target_items,
                                   ws.data_ptr(), n, ctypes.byref(p), torch.cuda.current_stream(dev).cuda_stream)
        if rc:
            raise RuntimeError("jq_plain_plan_build: " + L.jq_strerror(rc).decode())
        if p.supported:  # keep the used part only
            used = ws[:p.used_words].clone()
            for f in ("blob", "item_off", "item_words", "unwritten"):
                setattr(p, f, getattr(p, f) - ws.data_ptr() + used.data_ptr())
            torch.cuda.current_stream(dev).synchronize()
            return p, used
        return None, None

    def exchange(self, stream=None, plan=None):
        """Device pointer of the exchange buffer for launches of `plan` (the
        one in use) on this stream (one per stream, allocated on it, so launches
        on two streams may overlap; kept with the script, as large for each of
        its plans that needs one), or None when the plan needs none."""
        n = (plan or self.plan_in_use()).exchange_words
        if not n:
            return None
        if stream is None:
            stream = torch.cuda.current_stream(self.blocks_data.device)
        with self._lock:
            buf = self._exchange.get(stream.cuda_stream)
            if buf is None:
                with torch.cuda.stream(_torch_stream(stream, self.blocks_data.device)):
                    buf = torch.empty(n, dtype=torch.int32, device=self.blocks_data.device)
                self._exchange[stream.cuda_stream] = buf
            return buf.data_ptr()

    def arrivals(self):
        """(first cycle's, later cycles') u16 arrival of every state word, in
        int32 device tensors; computed on first use."""
        with self._lock:
            if self._arrivals is None:
                tables = arrival_tables(self)
                # complete before a launch on any stream reads them
                torch.cuda.current_stream(self.blocks_data.device).synchronize()
                self._arrivals = tables
            return self._arrivals

    def depth(self, stream=None):
        """(stage depth codes, per-entry base) on the device
        (jq_plain_prepare), computed on first use."""
        if self._depth is None:
            L = lib()
            st = stream.cuda_stream if stream is not None else torch.cuda.current_stream().cuda_stream
            entries = self.num_blocks * self.num_major_stages
            base = torch.empty(entries, dtype=torch.int32, device=self.blocks_data.device)
            n = ctypes.c_size_t()
            rc = L.jq_plain_prepare(self.blocks_start.data_ptr(), self.blocks_data.data_ptr(),
                                    self.num_blocks, self.num_major_stages, base.data_ptr(),
                                    None, 0, ctypes.byref(n), st)
            if rc:
                raise RuntimeError("jq_plain_prepare: " + lib().jq_strerror(rc).decode())
            depth = torch.empty(max(1, n.value), dtype=torch.uint8, device=self.blocks_data.device)
            rc = L.jq_plain_prepare(self.blocks_start.data_ptr(), self.blocks_data.data_ptr(),
                                    self.num_blocks, self.num_major_stages, base.data_ptr(),
                                    depth.data_ptr(), depth.numel(), None, st)
            if rc:
                raise RuntimeError("jq_plain_prepare: " + lib().jq_strerror(rc).decode())
            self._depth = (depth, base)
        return self._depth


def max_blocks(device=0):
    n = ctypes.c_size_t()
    rc = lib().jq_max_blocks(device, ctypes.byref(n))
    if rc:
        raise RuntimeError(lib().jq_strerror(rc).decode())
    return n.value


def _torch_stream(stream, device):
    """`stream` as a torch stream; any object with a cuda_stream handle does."""
    if isinstance(stream, torch.cuda.Stream):
        return stream
    if not stream.cuda_stream:
        return torch.cuda.default_stream(device)
    return torch.cuda.ExternalStream(stream.cuda_stream, device=device)


def _capturing(stream, device):
    if stream is None:
        return torch.cuda.is_current_stream_capturing()
    with torch.cuda.stream(_torch_stream(stream, device)):
        return torch.cuda.is_current_stream_capturing()


def simulate(ds, states, num_cycles, state_size, sram, sram_x=None, constraints=None,
             events=None, event_capacity=0, arrival_state_offset=0, first_cycle=0,
             stream=None, barrier_timeout_cycles=0, skip_dead_levels=True, planned=True):
    """Launch the plain interpreter (asynchronous, but for the first call on a
    script: it builds the script's plan in a workspace larger than the script,
    or its stage-depth tables, and waits for them; a first call with arrivals
    or constraints also runs two cycles for the arrival tables).  All tensors
    on device.
    skip_dead_levels: pass the script's stage-depth tables, so tree levels
    whose outputs nothing reads are skipped (False runs every level).
    planned: run the script's gate-list plan when it has one, the memory for it
    is there and the barrier wait is not bounded by the caller
    (skip_dead_levels only)."""
    a = SimArgs(ds.num_blocks, ds.num_major_stages, ds.blocks_start.data_ptr(),
                ds.blocks_data.data_ptr(), sram.data_ptr(),
                sram_x.data_ptr() if sram_x is not None else None, num_cycles, state_size,
                states.data_ptr(), constraints.data_ptr() if constraints is not None else None,
                events.data_ptr() if events is not None else None, event_capacity,
                arrival_state_offset, first_cycle, barrier_timeout_cycles,
                stream.cuda_stream if stream is not None else torch.cuda.current_stream().cuda_stream)
    if skip_dead_levels and planned and not barrier_timeout_cycles:
        tracked = bool(arrival_state_offset) or constraints is not None
        # the plan and the arrival tables are made on first use, which a
        # stream capture cannot record: such a call runs the script's own form
        ready = ds._plan is not None and (ds._arrivals is not None or not tracked)
        plan = ds.plan_in_use() if ready or not _capturing(stream, ds.blocks_data.device) else None
        if plan is not None:
            first = steady = None
            try:
                if tracked:
                    first, steady = (t.data_ptr() for t in ds.arrivals())
                buf = ds.exchange(stream, plan)
            except torch.cuda.OutOfMemoryError:
                plan = None
        if plan is not None:
            rc = lib().jq_simulate_planned(ctypes.byref(a), ctypes.byref(plan), first, steady, buf)
            if rc:
                raise RuntimeError("jq_simulate: " + lib().jq_strerror(rc).decode())
            return
    if skip_dead_levels:
        depth, base = ds.depth(stream)
        a.stage_depth = depth.data_ptr()
        a.stage_depth_base = base.data_ptr()
    rc = lib().jq_simulate(ctypes.byref(a))
    if rc:
        raise RuntimeError("jq_simulate: " + lib().jq_strerror(rc).decode())


def arrival_tables(ds, stream=None):
    """The u16 arrival of every state word in the first cycle of a launch
    and in later cycles (int32 device tensors of reg_io_state_size words):
    the arrival sections of snapshots 1 and 2 of a two-cycle run of the
    script itself.  Arrivals follow from the script's delays and each block's
    execution order, not from the stimulus, so an all-zero state serves."""
    s = ds.script
    rio = s.reg_io_state_size
    eff = rio * (2 if s.xprop_enabled else 1) + rio  # + arrival section
    dev = ds.blocks_data.device
    st = torch.zeros(3 * eff, dtype=torch.int32, device=dev)
    n_sram = max(1, s.sram_storage_size)
    sram = torch.zeros(n_sram, dtype=torch.int32, device=dev)
    sram_x = torch.zeros(n_sram, dtype=torch.int32, device=dev)
    off = eff - rio
    simulate(ds, st, 2, eff, sram, sram_x, arrival_state_offset=off, stream=stream, planned=False)
    rc = status(stream)
    if rc:
        raise RuntimeError("arrival tables: " + lib().jq_strerror(rc).decode())
    snaps = st.view(3, eff)
    return snaps[1, off:].clone(), snaps[2, off:].clone()


def status(stream=None):
    s = stream.cuda_stream if stream is not None else torch.cuda.current_stream().cuda_stream
    return lib().jq_sim_status(s)


def new_event_buffer(capacity, device="cuda"):
    buf = torch.zeros(EVENT_HEADER_WORDS + EVENT_WORDS * capacity, dtype=torch.int32, device=device)
    buf[2] = capacity
    return buf


def read_events(buf):
    h = dev_to_u32(buf[:EVENT_HEADER_WORDS])
    count, overflow, cap = int(h[0]), int(h[1]), int(h[2])
    n = min(count, cap)
    ev = dev_to_u32(buf[EVENT_HEADER_WORDS:EVENT_HEADER_WORDS + EVENT_WORDS * n]).reshape(n, EVENT_WORDS)
    return ev, count, overflow
