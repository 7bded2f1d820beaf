// Batched executor of the gate-list plan (plan_build.cuh), sm_100a: 32 * LW
// streams per work item, one slot of LW lane words (with their X words) per
// signal, gates evaluated level by level on whole slots.
//
// An item is one plan item (a partition, or a range of its writeout slots)
// for one lane group.  Per item: copy the signals it reads into slots 1..,
// evaluate the gates (two slot reads, one slot write), run the SRAM ports,
// and write each writeout signal from its reference.  A signal whose clock
// enable is the constant 0 is never written (both state buffers start with
// snapshot 0), one whose enable is the constant 1 needs no enable or old
// value.  The next item's blob (about 9 KB) is copied by TMA one item ahead.
//
// What bounds it: the chain of a major stage.  2M gates x 256 streams (907
// gates and 856 signals per item, one item per SM), SM clocks of a stage's
// 12,050: release fence of the arrival 1,550, barrier wait 1,200 (last CTA) to
// 2,700 (mean), reads 1,400 + 750 (55 KB from L2), gates 3,640 (16 to 19
// shared-memory wavefronts per warp and gate round), commit 1,640.  256k x 64
// (121 gates per item): 6,300, of which 2,900 are fence and barrier.  us per
// pass, prepared script / plan: 2M x 256 x 64 cycles 12,317 / 7,490, 512k x 512
// x 32 5,232 / 2,740, 256k x 64 x 32 4,297 / 1,805, 16k x 32 x 64 2,395 / 805.
//
// 512 threads: 128 registers, no spills; 1024 threads (64, spills) ran 1.2 to
// 1.3 times slower, 768 2 to 15%, 384 5% slower on the large and 2% faster on the
// smallest items, 256 20% slower on the large.
#pragma once
#include "plan_build.cuh"

namespace jqk {

// Gates of a level up to which a script's items take two levels per barrier:
// half a round of the CTA (512 threads, 16 bytes of a slot each), so that a
// pair of levels is one round.  All of a plan's items or none, so that the
// kernel has one of the two loops: with both, items that do not use the second
// ran 1 to 2.5% slower.  16k gates x 32 streams 908 / 812 us a pass, 256k x 64
// 1950 / 1815, 16k x 256 (octets, levels of 16) 526 / 497.
constexpr uint32_t bplan_pair_gates(uint32_t lw, bool x) {
  return lw == 8 ? (x ? 64 : 128) : 256;
}

struct BPlanParams {
  const uint32_t *blob;
  const unsigned long long *item_off;
  const uint32_t *item_words;
  uint32_t stage_item[33];
  // shared memory layout (slots: a multiple of 16 bytes)
  uint32_t blob_cap, nbuf, slots;
};

// The part of a slot one thread handles: (value, X) words of its lane words,
// or values only.
template <int LW, bool X>
struct LaneVec {
  using T = uint4;
};
template <>
struct LaneVec<1, true> {
  using T = uint2;
};
template <>
struct LaneVec<2, false> {
  using T = uint2;
};
template <>
struct LaneVec<1, false> {
  using T = uint32_t;
};

__device__ __forceinline__ void bp_xand(uint32_t a, uint32_t ax, uint32_t b, uint32_t bx,
                                        uint32_t &r, uint32_t &rx) {
  r = a & b;
  rx = (ax | bx) & (a | ax) & (b | bx);
}
// values inverted under mask m
template <bool X>
__device__ __forceinline__ uint4 bp_inv(uint4 v, uint32_t m) {
  return X ? make_uint4(v.x ^ m, v.y, v.z ^ m, v.w)
           : make_uint4(v.x ^ m, v.y ^ m, v.z ^ m, v.w ^ m);
}
template <bool X>
__device__ __forceinline__ uint2 bp_inv(uint2 v, uint32_t m) {
  return X ? make_uint2(v.x ^ m, v.y) : make_uint2(v.x ^ m, v.y ^ m);
}
template <bool X>
__device__ __forceinline__ uint32_t bp_inv(uint32_t v, uint32_t m) {
  return v ^ m;
}
template <bool X>
__device__ __forceinline__ uint4 bp_and(uint4 a, uint4 b) {
  uint4 r;
  if (X) {
    bp_xand(a.x, a.y, b.x, b.y, r.x, r.y);
    bp_xand(a.z, a.w, b.z, b.w, r.z, r.w);
  } else {
    r = make_uint4(a.x & b.x, a.y & b.y, a.z & b.z, a.w & b.w);
  }
  return r;
}
template <bool X>
__device__ __forceinline__ uint2 bp_and(uint2 a, uint2 b) {
  uint2 r;
  if (X)
    bp_xand(a.x, a.y, b.x, b.y, r.x, r.y);
  else
    r = make_uint2(a.x & b.x, a.y & b.y);
  return r;
}
template <bool X>
__device__ __forceinline__ uint32_t bp_and(uint32_t a, uint32_t b) {
  return a & b;
}
// DFF commit of new value n (X words with it) over the old one under enable e
__device__ __forceinline__ void bp_keep(uint32_t &n, uint32_t o, uint32_t e) { n = (o & ~e) | (n & e); }
__device__ __forceinline__ void bp_keepx(uint32_t &n, uint32_t &nx, uint32_t o, uint32_t ox, uint32_t e,
                                         uint32_t ex) {
  n = (o & ~e) | (n & e);
  nx = (ox & ~e & ~ex) | (nx & e & ~ex) | ex;
}
template <bool X>
__device__ __forceinline__ uint4 bp_commit(uint4 n, uint4 o, uint4 e) {
  if (X) {
    bp_keepx(n.x, n.y, o.x, o.y, e.x, e.y);
    bp_keepx(n.z, n.w, o.z, o.w, e.z, e.w);
  } else {
    bp_keep(n.x, o.x, e.x);
    bp_keep(n.y, o.y, e.y);
    bp_keep(n.z, o.z, e.z);
    bp_keep(n.w, o.w, e.w);
  }
  return n;
}
template <bool X>
__device__ __forceinline__ uint2 bp_commit(uint2 n, uint2 o, uint2 e) {
  if (X) {
    bp_keepx(n.x, n.y, o.x, o.y, e.x, e.y);
  } else {
    bp_keep(n.x, o.x, e.x);
    bp_keep(n.y, o.y, e.y);
  }
  return n;
}
template <bool X>
__device__ __forceinline__ uint32_t bp_commit(uint32_t n, uint32_t o, uint32_t e) {
  bp_keep(n, o, e);
  return n;
}
// AND over the value words: all ones when every stream's enable is set
template <bool X>
__device__ __forceinline__ uint32_t bp_all(uint4 e) {
  return X ? e.x & e.z : e.x & e.y & e.z & e.w;
}
template <bool X>
__device__ __forceinline__ uint32_t bp_all(uint2 e) {
  return X ? e.x : e.x & e.y;
}
template <bool X>
__device__ __forceinline__ uint32_t bp_all(uint32_t e) {
  return e;
}
__device__ __forceinline__ uint32_t bp_any_x(uint4 e) { return e.y | e.w; }
__device__ __forceinline__ uint32_t bp_any_x(uint2 e) { return e.y; }
__device__ __forceinline__ uint32_t bp_any_x(uint32_t) { return 0; }
// values written, X words left
__device__ __forceinline__ void bp_store_values(uint4 *p, uint4 v) {
  uint32_t *w = reinterpret_cast<uint32_t *>(p);
  w[0] = v.x;
  w[2] = v.z;
}
__device__ __forceinline__ void bp_store_values(uint2 *p, uint2 v) {
  *reinterpret_cast<uint32_t *>(p) = v.x;
}
__device__ __forceinline__ void bp_store_values(uint32_t *p, uint32_t v) { *p = v; }
__device__ __forceinline__ uint4 bp_no_x(uint4 v) { return make_uint4(v.x, 0, v.z, 0); }
__device__ __forceinline__ uint2 bp_no_x(uint2 v) { return make_uint2(v.x, 0); }
__device__ __forceinline__ uint32_t bp_no_x(uint32_t v) { return v; }
// words of a thread's part, by index
__device__ __forceinline__ uint32_t bp_word(uint4 v, int i) {
  return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w;
}
__device__ __forceinline__ uint32_t bp_word(uint2 v, int i) { return i ? v.y : v.x; }
__device__ __forceinline__ uint32_t bp_word(uint32_t v, int) { return v; }

// Setup/hold checks of one state word for the lane words of an item, with the
// plain interpreter's predicate (csrc/kernel_v1_impl.cuh:536-558) per stream:
// arrival a and constraint cv are the word's, clk[l] the streams of lane word
// l whose clock enable is set on any of its signals.  One warp; one atomic
// claims the records of a kind.
__device__ __noinline__ void bp_check(const BatchParams &P, uint32_t word, uint32_t a, uint32_t cv,
                                      const uint32_t *clk, uint32_t lw, uint32_t lane0,
                                      uint32_t cyc) {
  const uint32_t clock_ps = __ldg(P.constraints), su = cv >> 16, ho = cv & 0xffffu;
  const bool v[2] = {a > 0 && a + su > clock_ps, a < ho};
  if (!cv || !(v[0] || v[1])) return;
  const uint32_t lane = threadIdx.x & 31, below = (1u << lane) - 1u;
  // records as two 16-byte stores where the buffer's alignment allows it
  const bool wide = (reinterpret_cast<size_t>(P.events->events) & 15) == 0;
  uint32_t n = 0;
  for (uint32_t l = 0; l < lw; ++l) n += __popc(clk[l]);
  if (!n) return;
#pragma unroll 1
  for (int kind = 0; kind < 2; ++kind) {
    if (!v[kind]) continue;
    const uint32_t slack = kind == 0 ? (uint32_t)((int32_t)clock_ps - (int32_t)a - (int32_t)su)
                                     : (uint32_t)((int32_t)a - (int32_t)ho);
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(&P.events->count, n);
    base = __shfl_sync(0xffffffffu, base, 0);
#pragma unroll 1
    for (uint32_t l = 0; l < lw; ++l) {
      const uint32_t m = clk[l], idx = base + __popc(m & below);
      if ((m >> lane) & 1u) {
        if (wide && idx < P.event_cap) {
          uint4 *e = reinterpret_cast<uint4 *>(&P.events->events[idx]);
          e[0] = make_uint4(4 + kind, word, P.first_cycle + cyc, 32 * (lane0 + l) + lane);
          e[1] = make_uint4(word, slack, a, kind == 0 ? su : ho);
        } else {
          put_event(P, idx, 4 + kind, word, P.first_cycle + cyc, slack, a, kind == 0 ? su : ho,
                    32 * (lane0 + l) + lane);
        }
      }
      base += __popc(m);
    }
  }
}

// Outputs and the optional record of the cycle that ended (state `in`), and
// the stimulus of the next snapshot into `out`: a CTA takes the elements of
// its rank, so no CTA has more than a few.
__device__ __noinline__ void bp_io(const BatchParams &P, const uint32_t *in, uint32_t *out, size_t c,
                                   uint32_t rank, uint32_t ctas, uint32_t lane_lo, uint32_t lane_n) {
  if (c) {
    const uint32_t n = P.n_po * lane_n;
    for (uint32_t q = rank + ctas * threadIdx.x; q < n; q += ctas * blockDim.x) {
      const uint32_t po = q / lane_n, l = lane_lo + q % lane_n;
      P.wave[((c - 1) * P.n_po + po) * P.lanes + l] = ldcg(in + phys(P, l, P.po_sig[po]));
    }
    if (P.record) {  // lane-major [lane][signal]
      uint32_t *dst = P.record + c * P.sig_per_snap * P.lanes + (size_t)lane_lo * P.sig_per_snap;
      for (size_t q = (size_t)rank * blockDim.x + threadIdx.x; q < P.sig_per_snap * lane_n;
           q += (size_t)ctas * blockDim.x)
        dst[q] = ldcg(in + phys(P, lane_lo + (uint32_t)(q / P.sig_per_snap), q % P.sig_per_snap));
    }
  }
  if (P.stim && c < P.num_cycles) {
    const uint32_t sigs = (uint32_t)P.input_sigs, n = sigs * lane_n;
    const uint32_t *src = P.stim + (c + 1) * P.input_sigs * P.lanes;
    for (uint32_t q = rank + ctas * threadIdx.x; q < n; q += ctas * blockDim.x) {
      const uint32_t l = lane_lo + q / sigs, i = q % sigs;
      uint32_t dst = i;
      if (P.input_regions)
        for (uint32_t r = 0; r < P.n_input_regions; ++r) {
          const uint32_t d0 = P.input_regions[3 * r], s0 = P.input_regions[3 * r + 1],
                         k = P.input_regions[3 * r + 2];
          if (i >= s0 && i < s0 + k) dst = d0 + (i - s0);
        }
      out[phys(P, l, dst)] = src[(size_t)l * sigs + i];
    }
  }
}

template <int LW, bool X, bool TIMED, bool PAIR>
__global__ void __launch_bounds__(BT, 1)
    jq_bplan_kernel(const __grid_constant__ BatchParams P, const __grid_constant__ BPlanParams Q) {
  using V = typename LaneVec<LW, X>::T;
  constexpr uint32_t WPS = LW * (X ? 2 : 1);      // words of a slot
  constexpr uint32_t TPE = WPS * 4 / sizeof(V);   // threads per slot
  constexpr uint32_t NE = BT / TPE;               // slots per round
  constexpr uint32_t PV = X ? 2 : 1;              // words per lane word
  // a signal's parts in the state are GS apart (single lanes skip the other
  // lane of their pair)
  constexpr uint32_t GS = LW == 1 ? 2 : TPE;
  constexpr uint32_t PT = BT - 32;                // the thread that issues the blob copies
  extern __shared__ __align__(128) uint8_t dyn[];
  __shared__ uint64_t bar[2];
  uint32_t *const buf0 = reinterpret_cast<uint32_t *>(dyn);
  V *const S = reinterpret_cast<V *>(dyn + 4 * (size_t)Q.nbuf * Q.blob_cap);
  uint32_t *const Sw = reinterpret_cast<uint32_t *>(S);
  // setup/hold checks: clock enables [256][LW], then (arrival, constraint) [256]
  uint32_t *const clk_or = Sw + (size_t)Q.slots * WPS;
  uint2 *const chk = reinterpret_cast<uint2 *>(clk_or + 256 * LW);
  const uint32_t t = threadIdx.x, k = t % TPE, el = t / TPE, warp = t >> 5, ln = t & 31;
  const uint32_t groups = P.lanes / LW, rank = blockIdx.x, G = gridDim.x, nms = P.num_major_stages;
  const bool two = Q.nbuf == 2;
  // Lane groups share no state.  When every stage has at most one item per
  // CTA and a grid of a multiple of the groups, a CTA always runs one group,
  // and each group has its own barrier, stimulus and outputs.
  bool grouped = groups > 1 && groups <= MAX_GROUPS && G >= groups;
  for (unsigned ms = 0; ms < nms; ++ms)
    grouped &= (Q.stage_item[ms + 1] - Q.stage_item[ms]) * groups <= G;
  const uint32_t my_group = grouped ? rank % groups : 0;
  const uint32_t g_rank = grouped ? rank / groups : rank;
  const uint32_t g_ctas = grouped ? (G - my_group + groups - 1) / groups : G;
  const uint32_t lane_lo = grouped ? LW * my_group : 0, lane_n = grouped ? LW : P.lanes;
  unsigned long long *const bcount =
      grouped ? &g_bgroup[(size_t)P.slot * MAX_GROUPS + my_group] : &g_bcount[P.slot];
  if (t == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (t < WPS) Sw[t] = 0;  // slot 0: the constant
  __syncthreads();
  // blob copies, one item ahead over all cycles (thread PT): copy n lands in
  // buffer n mod nbuf, in phase n / nbuf of its mbarrier; the next item's
  // descriptor is loaded when the copy before it is issued
  uint32_t f_n = 0, f_idx = rank, f_words = 0;
  unsigned f_ms = 0;
  size_t f_c = 0;
  unsigned long long f_off = 0;
  auto buf_of = [&](uint32_t n) { return two ? n & 1u : 0u; };
  auto par_of = [&](uint32_t n) { return two ? (n >> 1) & 1u : n & 1u; };
  auto settle = [&]() {
    uint32_t wraps = 0;
    while (f_c < P.num_cycles &&
           f_idx >= (Q.stage_item[f_ms + 1] - Q.stage_item[f_ms]) * groups) {
      if (++f_ms == nms) {
        f_ms = 0;
        ++f_c;
        if (++wraps == 2) f_c = P.num_cycles;  // this CTA has no item at all
      }
      f_idx = rank;
    }
    if (f_c < P.num_cycles) {
      const uint32_t i = Q.stage_item[f_ms] + f_idx / groups;
      f_off = Q.item_off[i];
      f_words = Q.item_words[i];
    }
  };
  auto issue = [&]() {
    if (f_c >= P.num_cycles) return;
    const uint32_t b = buf_of(f_n);
    mbar_expect_tx(&bar[b], 4 * f_words);
    tma_load_1d(buf0 + (size_t)b * Q.blob_cap, Q.blob + f_off, 4 * f_words, &bar[b]);
    ++f_n;
    f_idx += G;
    settle();
  };
  if (t == PT) {
    settle();
    issue();
  }
  uint32_t n_run = 0;
  unsigned long long target = 0;  // arrivals that complete the barrier ahead
  bool failed = false;
  // the barrier that ends the stage before (thread 0); bounded
  auto wait_stage = [&]() {
    const uint64_t t0 = clock64();
    while (ld_acquire64(bcount) < target) {
      if (*((volatile int *)&g_status[P.slot]) != 0) return false;
      if ((uint64_t)(clock64() - t0) > P.timeout) {
        atomicCAS(&g_status[P.slot], 0, JQ_ERR_BARRIER_TIMEOUT);
        return false;
      }
    }
    return true;
  };
  for (size_t c = 0; c < P.num_cycles && !failed; ++c) {
    const uint32_t *in = (c & 1) ? P.state_b : P.state_a;
    uint32_t *out = (c & 1) ? P.state_a : P.state_b;
    for (unsigned ms = 0; ms < nms; ++ms) {
      const uint32_t total = (Q.stage_item[ms + 1] - Q.stage_item[ms]) * groups;
      bool opened = false;
      for (uint32_t idx = rank; idx < total || !opened; idx += G) {
        const bool have = idx < total;
        const uint32_t *B = buf0 + (size_t)buf_of(n_run) * Q.blob_cap;
        bool ok = !have || plan_mbar_wait(&bar[buf_of(n_run)], par_of(n_run));
        if (!opened && t == 0) ok = wait_stage() && ok;
        // (also: the last item is done with the slots)
        if (__syncthreads_or(!ok)) {
          failed = true;
          break;
        }
        const bool io = !opened && ms == 0;
        opened = true;
        if (!have) {
          if (io) bp_io(P, in, out, c, g_rank, g_ctas, lane_lo, lane_n);
          break;
        }
        const long long t_start = clock64();
        const uint32_t group = groups == 1 ? 0 : idx % groups, ngr = B[PH_NGR], nw = B[PH_NW];
        const bool isx = X && B[PH_ISX] != 0;
        // the group's part of signal 0, in V units
        const size_t g0 = LW == 8   ? (size_t)group * P.vsig * TPE + k
                          : LW == 2 ? (size_t)group * P.vsig
                                    : (size_t)(group >> 1) * P.vsig * 2 + (group & 1);
        const V *vin = reinterpret_cast<const V *>(in) + g0;
        V *vout = reinterpret_cast<V *>(out) + g0;
        // ---- read signals into slots 1..
        {
          const uint32_t *gr = B + B[PH_OEXP];
          if (sizeof(V) == 16 && (!X || isx)) {
#pragma unroll 1
            for (uint32_t i = el; i < ngr; i += NE) {
              const uint32_t e = gr[i];
              const V *src = ((e >> 31) ? vout : vin) + (size_t)(e & 0x7fffffffu) * GS;
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                               smem_u32(S + (1 + i) * TPE + k)),
                           "l"(src)
                           : "memory");
            }
          } else {
            for (uint32_t i0 = el; i0 < ngr; i0 += 4 * NE) {
              V v[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const uint32_t i = i0 + j * NE;
                if (i < ngr) {
                  const uint32_t e = gr[i];
                  v[j] = __ldcg(((e >> 31) ? vout : vin) + (size_t)(e & 0x7fffffffu) * GS);
                }
              }
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const uint32_t i = i0 + j * NE;
                if (i < ngr) S[(1 + i) * TPE + k] = X && !isx ? bp_no_x(v[j]) : v[j];
              }
            }
          }
          if constexpr (TIMED) {
            for (uint32_t i = t; i < nw * LW; i += BT) clk_or[i] = 0;
            if (t < nw) {
              const uint32_t o = B[PH_IO] + t;
              chk[t] = make_uint2(__ldg((c ? P.arr_steady : P.arr_first) + o) & 0xffffu,
                                  __ldg(P.constraints + 1 + o));
            }
          }
        }
        if (two && t == PT) issue();  // into the other buffer, free since the barrier above
        if (io) bp_io(P, in, out, c, g_rank, g_ctas, lane_lo, lane_n);
        if (sizeof(V) == 16) asm volatile("cp.async.wait_all;" ::: "memory");
        // ---- gates, one level per CTA barrier; a thread's first gate of a
        // level is loaded before the barrier that opens the level
        if constexpr (!PAIR) {
          const uint32_t *ends = B + B[PH_OLEV], *gates = B + B[PH_OGATE];
          const uint32_t nlev = B[PH_NLEV];
          V *dst = S + (1 + ngr) * TPE + k;
          uint32_t g = el, g1 = nlev ? ends[0] : 0u;
          uint32_t e = g < g1 ? gates[g] : 0u;
          __syncthreads();
          for (uint32_t l = 0; l < nlev; ++l) {
            const uint32_t g2 = l + 1 < nlev ? ends[l + 1] : 0u;
#pragma unroll 1
            while (g < g1) {
              const V a = S[((e >> 1) & 0x7fffu) * TPE + k], b = S[(e >> 17) * TPE + k];
              dst[g * TPE] = bp_and<X>(bp_inv<X>(a, 0u - (e & 1u)),
                                       bp_inv<X>(b, 0u - ((e >> 16) & 1u)));
              g += NE;
              if (g < g1) e = gates[g];
            }
            g = g1 + el;
            g1 = g2;
            if (g < g1) e = gates[g];
            __syncthreads();
          }
        }
        else {
          // two levels per barrier (plan_build.cuh)
          const uint32_t *ends = B + B[PH_OLEV];
          const uint2 *gates = reinterpret_cast<const uint2 *>(B + B[PH_OGATE]);
          const uint32_t nph = B[PH_NLEV];
          V *dst = S + (1 + ngr) * TPE + k;
          uint32_t g = el, g1 = nph ? ends[0] : 0u;
          uint2 e = g < g1 ? gates[g] : make_uint2(0, 0);
          __syncthreads();
          for (uint32_t l = 0; l < nph; ++l) {
            const uint32_t g2 = l + 1 < nph ? ends[l + 1] : 0u;
#pragma unroll 1
            while (g < g1) {
              auto half = [&](uint32_t h) {
                const V x = S[((h >> 1) & 0x3fffu) * TPE + k], y = S[((h >> 16) & 0x3fffu) * TPE + k];
                return bp_inv<X>(bp_and<X>(bp_inv<X>(x, 0u - (h & 1u)),
                                           bp_inv<X>(y, 0u - ((h >> 15) & 1u))),
                                 0u - ((h >> 30) & 1u));
              };
              dst[g * TPE] = bp_and<X>(half(e.x), half(e.y));
              g += NE;
              if (g < g1) e = gates[g];
            }
            g = g1 + el;
            g1 = g2;
            if (g < g1) e = gates[g];
            __syncthreads();
          }
        }
        // ---- SRAM ports: a warp per (SRAM, lane word), lane = stream; staged
        // rows (read address 0..15, write address 16..31, write enable
        // 32..63, data 64..95) to per-stream bits by warp transposes
        if (const uint32_t nsr = B[PH_NSR]) {
          const uint32_t *sr = B + B[PH_OSRAM];
          const uint32_t rd = B[PH_SRSLOT], sram_off = B[PH_SRAM_OFF];
#pragma unroll 1
          for (uint32_t ih = warp; ih < nsr * LW; ih += BT / 32) {
            const uint32_t i = ih / LW, lw = ih % LW;
            uint32_t w[3], wx = 0;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
              const uint32_t r = sr[96 * i + 32 * j + ln];
              const uint32_t *p = Sw + (size_t)(r >> 1) * WPS + PV * lw;
              w[j] = warp_transpose32(p[0] ^ (0u - (r & 1u)));
              if (X && j == 2) wx = warp_transpose32(p[1]);
            }
            const uint32_t ra = w[0] & 0xffffu, wa = w[0] >> 16, en = w[1], data = w[2];
            const size_t stream = (size_t)(group * LW + lw) * 32 + ln;
            const size_t at = stream * P.sram_words + sram_off + (size_t)i * SRAM_WORDS;
            const bool hx = isx && P.sram_x != nullptr;
            const uint32_t r = ldcg(P.sram + at + ra), w0 = ldcg(P.sram + at + wa);
            uint32_t rx = 0, w0x = 0;
            if (hx) {
              rx = ldcg(P.sram_x + at + ra);
              w0x = ldcg(P.sram_x + at + wa);
            }
            P.sram[at + wa] = (w0 & ~en) | (data & en);
            if (hx) P.sram_x[at + wa] = (w0x & ~en) | (wx & en);
            uint32_t *o = Sw + (size_t)(rd + 32 * i + ln) * WPS + PV * lw;
            o[0] = warp_transpose32(r);
            if (X) {
              const uint32_t x = warp_transpose32(rx);
              o[1] = isx ? x : 0u;
            }
          }
          __syncthreads();
        }
        // ---- commit
        {
          const uint32_t *com = B + B[PH_OCOM];
          const uint32_t nq = 32 * nw;
          const size_t s0 = (size_t)B[PH_IO] * 32;
#pragma unroll 1
          for (uint32_t q = el; q < nq; q += NE) {
            const uint32_t e = com[q], cr = e >> 16;
            if (cr == 0) continue;  // never enabled
            V v = bp_inv<X>(S[((e >> 1) & 0x7fffu) * TPE + k], 0u - (e & 1u));
            const size_t at = (s0 + q) * GS;
            if (cr != 1) {  // not always enabled
              const V en = bp_inv<X>(S[(cr >> 1) * TPE + k], 0u - (cr & 1u));
              // (every stream enabled: only X enables change the value)
              if (bp_all<X>(en) != 0xffffffffu)
                v = bp_commit<X>(v, __ldcg(vin + at), en);
              else if (X && bp_any_x(en))
                v = bp_commit<X>(v, v, en);
              if constexpr (TIMED) {
#pragma unroll
                for (int j = 0; j < (int)(sizeof(V) / 4 / PV); ++j)
                  atomicOr(&clk_or[(q >> 5) * LW + k * (sizeof(V) / 4 / PV) + j],
                           bp_word(en, j * PV));
              }
            } else if constexpr (TIMED) {
#pragma unroll
              for (int j = 0; j < (int)(sizeof(V) / 4 / PV); ++j)
                clk_or[(q >> 5) * LW + k * (sizeof(V) / 4 / PV) + j] = 0xffffffffu;
            }
            if (X && !isx)
              bp_store_values(vout + at, v);
            else
              vout[at] = v;
          }
          if constexpr (TIMED) {
            __syncthreads();
            for (uint32_t j = warp; j < nw; j += BT / 32)
              bp_check(P, B[PH_IO] + j, chk[j].x, chk[j].y, clk_or + j * LW, LW, group * LW,
                       (uint32_t)c);
          }
        }
        if (P.part_cycles) {
          __syncthreads();
          if (t == 0)
            atomicAdd(&P.part_cycles[B[PH_PART]], (unsigned long long)(clock64() - t_start));
        }
        ++n_run;
        if (!two) {
          __syncthreads();
          if (t == PT) issue();
        }
      }
      if (failed) break;
      // ---- arrive
      __syncthreads();
      if (t == 0) {
        target += g_ctas;
        asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(bcount) : "memory");
      }
    }
  }
  if (!failed && P.num_cycles) {  // the last cycle's outputs
    bool ok = t != 0 || wait_stage();
    if (!__syncthreads_or(!ok))
      bp_io(P, (P.num_cycles & 1) ? P.state_b : P.state_a, nullptr, P.num_cycles, g_rank, g_ctas,
            lane_lo, lane_n);
  }
  if (failed && t == 0) atomicCAS(&g_status[P.slot], 0, JQ_ERR_BARRIER_TIMEOUT);
  if (t == PT)  // copies in flight land before the CTA leaves
    for (uint32_t n = n_run; n < f_n; ++n) plan_mbar_wait(&bar[buf_of(n)], par_of(n));
}

}  // namespace jqk
