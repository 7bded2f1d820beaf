// Executors of the gate-list plan (plan_build.cuh) for one stimulus stream
// (sm_100a).  Per item and cycle: one load per state word, one byte per needed
// bit, two byte reads and one byte write per gate with one CTA barrier per
// logic level, and ballots that pack the writeouts.  Values are bytes (bit 0
// value, bit 1 X) in shared memory, one per slot.
//
// What bounds it: latency.  A major stage of one stream is a chain of state
// word exchange, a few gate levels and the commit; an item's blob (up to
// about 60 KB) is copied by TMA one item ahead.  us per pass, script form / plan:
// 16k gates x 64 cycles 2721 / 532, 2M gates x 16 cycles 5742 / 1156, 256k
// gates x 32 cycles 4918 / 1486.
#pragma once
#include "plan_build.cuh"

namespace jqk {

// Threads of the executors.  A logic level has 50 to 500 gates of a split
// partition, so more threads only add warps that issue the loop and the
// barrier; 1024 (64 registers, spills) measured 1.1 to 1.4 times slower on
// every design, 256 within 1% on the small design and 8% slower on the
// 2M-gate one.
constexpr int EB = 512;
constexpr uint32_t PT = EB - 32;  // the thread that issues the blob copies

struct PlanParams {
  unsigned num_major_stages;
  const uint32_t *blob;
  const unsigned long long *item_off;
  const uint32_t *item_words;
  uint32_t stage_item[33];  // first item of each major stage
  uint32_t blob_cap, nbuf, slot_bytes, gw_cap;  // shared memory layout
  // mirrored form: words of a mirrored snapshot, words each stage writes, the
  // X offset (0: no X words), the words no partition writes
  uint32_t rio, stage_words[32], xoff, active;  // active: CTAs that run items
  const uint32_t *unwritten;
  uint32_t n_unwritten;
  void *exchange;      // flow form: published words of four snapshots
  uint32_t hint_slack; // flow form: see plan_flow_kernel; 0 = no hint
  uint32_t *sram, *sram_x;
  size_t num_cycles, state_size;
  uint32_t *states;
  const uint32_t *constraints;
  jq_event_buffer *events;
  uint32_t event_cap;
  int32_t arrival_off;
  const uint32_t *arr_first, *arr_steady;
  uint32_t first_cycle;
  uint64_t timeout;
  int slot;
};

// g_plan_count[slot][k]: arrivals of cycles c with c mod 4 = k (see plan_flow_kernel)
static __device__ unsigned long long g_plan_count[BAR_SLOTS][4], g_plan_hint[BAR_SLOTS];

// plan_mbar_wait for words other CTAs of the cluster sent.
__device__ __forceinline__ bool plan_mbar_wait_cluster(uint64_t *bar, uint32_t parity) {
  uint32_t done = 0;
  const uint64_t t0 = clock64();
  for (;;) {
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(plan_smem(bar)), "r"(parity)
        : "memory");
    if (done) return true;
    if ((uint64_t)(clock64() - t0) > DEFAULT_BARRIER_TIMEOUT) return false;
  }
}

// Copies each item's blob one item ahead (with one buffer: when the last
// item is done with it), over all cycles.  Copy k lands in buffer k mod nbuf,
// in phase k / nbuf of that buffer's mbarrier.  The next item's descriptor is
// loaded when the copy before it is issued, so no copy waits for a load.
// One thread (the first of the last warp, which the
// writeouts and small levels reach last) issues them.
struct PlanFetch {
  const PlanParams &P;
  uint32_t *buf;
  uint64_t *bar;
  uint32_t rank, G;
  unsigned ms;
  uint32_t item, n;  // next item to copy, copies issued
  size_t cyc;
  unsigned long long off;
  uint32_t words;  // as loaded: nothing waits for it before the next issue
  __device__ PlanFetch(const PlanParams &p, uint32_t *b, uint64_t *mb, uint32_t r, uint32_t g)
      : P(p), buf(b), bar(mb), rank(r), G(g), ms(0), item(p.stage_item[0] + r), n(0), cyc(0) {
    settle();
  }
  __device__ uint32_t buf_of(uint32_t k) const { return P.nbuf == 2 ? k & 1u : 0u; }
  __device__ uint32_t par_of(uint32_t k) const { return P.nbuf == 2 ? (k >> 1) & 1u : k & 1u; }
  // moves to the next existing item and loads its descriptor
  __device__ void settle() {
    uint32_t wraps = 0;
    while (cyc < P.num_cycles && item >= P.stage_item[ms + 1]) {
      if (++ms == P.num_major_stages) {
        ms = 0;
        ++cyc;
        if (++wraps == 2) cyc = P.num_cycles;  // this CTA has no item at all
      }
      item = P.stage_item[ms] + rank;
    }
    if (cyc < P.num_cycles) {
      off = P.item_off[item];
      words = P.item_words[item];
    }
  }
  __device__ void issue() {
    if (cyc >= P.num_cycles) return;
    const uint32_t b = buf_of(n), bytes = 4 * words;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(plan_smem(&bar[b])),
                 "r"(bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(plan_smem(buf + (size_t)b * P.blob_cap)),
        "l"(P.blob + off), "r"(bytes), "r"(plan_smem(&bar[b]))
        : "memory");
    ++n;
    item += G;
    settle();
  }
  // copies not consumed yet (k: items consumed) land before the CTA leaves
  __device__ void drain(uint32_t k) const {
    for (; k < n; ++k) plan_mbar_wait(&bar[buf_of(k)], par_of(k));
  }
};

// AND of two slot bytes (bit 0 value, bit 1 X).
template <bool X>
__device__ __forceinline__ uint32_t plan_and2(uint32_t a, uint32_t b) {
  return X ? (a & b & 1u) | ((a | b) & (a << 1 | a) & (b << 1 | b) & 2u) : a & b;
}

// Gates of an item, two logic levels per CTA barrier (plan_build.cuh); ends
// with one.  A thread's first gate of a phase is loaded before the barrier
// that opens it.  A phase is latency: two levels in one cost four byte reads
// a gate instead of two but one chain and one barrier instead of two.
template <bool X>
__device__ __forceinline__ void plan_phases(const uint32_t *B, uint8_t *slots, uint32_t ngr) {
  const uint32_t *ends = B + B[PH_OLEV];
  const uint2 *gates = reinterpret_cast<const uint2 *>(B + B[PH_OGATE]);
  const uint32_t nph = B[PH_NLEV];
  uint8_t *dst = slots + 1 + ngr;
  uint32_t g = threadIdx.x, g1 = nph ? ends[0] : 0u;
  uint2 e = g < g1 ? gates[g] : make_uint2(0, 0);
  __syncthreads();
  for (uint32_t l = 0; l < nph; ++l) {
    const uint32_t g2 = l + 1 < nph ? ends[l + 1] : 0u;
    while (g < g1) {
      const uint32_t a = slots[(e.x >> 1) & 0x3fffu] ^ (e.x & 1u);
      const uint32_t b = slots[(e.x >> 16) & 0x3fffu] ^ ((e.x >> 15) & 1u);
      const uint32_t c = slots[(e.y >> 1) & 0x3fffu] ^ (e.y & 1u);
      const uint32_t d = slots[(e.y >> 16) & 0x3fffu] ^ ((e.y >> 15) & 1u);
      dst[g] = (uint8_t)plan_and2<X>(plan_and2<X>(a, b) ^ ((e.x >> 30) & 1u),
                                     plan_and2<X>(c, d) ^ ((e.y >> 30) & 1u));
      g += EB;
      if (g < g1) e = gates[g];
    }
    g = g1 + threadIdx.x;
    g1 = g2;
    if (g < g1) e = gates[g];
    __syncthreads();
  }
}
// The same for items listed by level.
template <bool X>
__device__ __forceinline__ void plan_levels(const uint32_t *B, uint8_t *slots, uint32_t ngr) {
  const uint32_t *ends = B + B[PH_OLEV], *gates = B + B[PH_OGATE];
  const uint32_t nlev = B[PH_NLEV];
  uint8_t *dst = slots + 1 + ngr;
  uint32_t g = threadIdx.x, g1 = nlev ? ends[0] : 0u;
  uint32_t e = g < g1 ? gates[g] : 0u;
  __syncthreads();
  for (uint32_t l = 0; l < nlev; ++l) {
    const uint32_t g2 = l + 1 < nlev ? ends[l + 1] : 0u;
    while (g < g1) {
      const uint32_t a = slots[(e >> 1) & 0x7fffu] ^ (e & 1u);
      const uint32_t b = slots[e >> 17] ^ ((e >> 16) & 1u);
      dst[g] = (uint8_t)plan_and2<X>(a, b);
      g += EB;
      if (g < g1) e = gates[g];
    }
    g = g1 + threadIdx.x;
    g1 = g2;
    if (g < g1) e = gates[g];
    __syncthreads();
  }
}
// PAIRS: every item of the plan is listed by pairs, so the kernel has one loop
// (16k gates, 64 cycles: 555 us a pass with both, 537 with one).
template <bool X, bool PAIRS>
__device__ __forceinline__ void plan_gates(const uint32_t *B, uint8_t *slots, uint32_t ngr) {
  if (PAIRS || B[PH_PAIR])
    plan_phases<X>(B, slots, ngr);
  else
    plan_levels<X>(B, slots, ngr);
}

// SRAM ports of an item: a warp per SRAM, lane = bit of each staged word;
// ends with a CTA barrier.
__device__ __forceinline__ void plan_srams(const PlanParams &P, const uint32_t *B, uint8_t *slots,
                                           bool isx) {
  const uint32_t nsr = B[PH_NSR];
  if (!nsr) return;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t *sr = B + B[PH_OSRAM];
  uint8_t *rd = slots + B[PH_SRSLOT];
  for (uint32_t i = threadIdx.x >> 5; i < nsr; i += EB / 32) {
    uint32_t w[3], wx = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const uint32_t r = sr[96 * i + 32 * k + lane];
      const uint32_t s = slots[r >> 1];
      w[k] = __ballot_sync(0xffffffffu, (s ^ r) & 1u);
      if (k == 2) wx = __ballot_sync(0xffffffffu, (s >> 1) & 1u);
    }
    const uint32_t ra = w[0] & 0xffffu, wa = w[0] >> 16, en = w[1], data = w[2];
    const size_t base = (size_t)B[PH_SRAM_OFF] + (size_t)i * SRAM_WORDS;
    const bool hx = isx && P.sram_x != nullptr;
    const uint32_t r = ldcg(P.sram + base + ra), w0 = ldcg(P.sram + base + wa);
    uint32_t rx = 0, w0x = 0;
    if (hx) {
      rx = ldcg(P.sram_x + base + ra);
      w0x = ldcg(P.sram_x + base + wa);
    }
    __syncwarp();
    if (lane == 0) {
      P.sram[base + wa] = (w0 & ~en) | (data & en);
      if (hx) P.sram_x[base + wa] = (w0x & ~en) | (wx & en);
    }
    rd[32 * i + lane] = (uint8_t)(((r >> lane) & 1u) | (((rx >> lane) & 1u) << 1));
  }
  __syncthreads();
}

// Setup/hold checks and the arrival word of state word o (one thread).
__device__ __forceinline__ void plan_timing(const PlanParams &P, uint32_t *out, size_t o,
                                            uint32_t cp, size_t c) {
  const uint32_t a = __ldg((c ? P.arr_steady : P.arr_first) + o) & 0xffffu;
  if (P.arrival_off) out[(size_t)(uint32_t)P.arrival_off + o] = a;
  const uint32_t cv = P.constraints && cp ? __ldg(P.constraints + 1 + o) : 0u;
  if (!cv) return;
  const uint32_t su = cv >> 16, ho = cv & 0xffffu, clk = __ldg(P.constraints);
  const uint32_t cyc = P.first_cycle + (uint32_t)c;
  if (a > 0 && a + su > clk)
    push_event(P.events, P.event_cap, 4, (uint32_t)o, cyc,
               (uint32_t)((int32_t)clk - (int32_t)a - (int32_t)su), a, su);
  if (a < ho)
    push_event(P.events, P.event_cap, 5, (uint32_t)o, cyc, (uint32_t)((int32_t)a - (int32_t)ho), a,
               ho);
}

// New value and X word of writeout j of an item, and the streams' clock
// enable: packed from the slot bytes by ballots (whole warp).
struct PlanWord {
  uint32_t v, x, cp, cx;
};
__device__ __forceinline__ PlanWord plan_word(const uint32_t *com, const uint8_t *slots, uint32_t j,
                                              bool isx) {
  const uint32_t e = com[32 * j + (threadIdx.x & 31)];
  const uint32_t s = slots[(e >> 1) & 0x7fffu], k = slots[e >> 17];
  PlanWord w;
  w.v = __ballot_sync(0xffffffffu, (s ^ e) & 1u);
  w.cp = __ballot_sync(0xffffffffu, (k ^ (e >> 16)) & 1u);
  w.x = w.cx = 0;
  if (isx) {
    w.x = __ballot_sync(0xffffffffu, s & 2u);
    w.cx = __ballot_sync(0xffffffffu, k & 2u);
  }
  return w;
}

// State word of a snapshot as producers publish it: (value, snapshot number)
// and (X word, snapshot number), each one 8-byte access, so a consumer that
// reads its number has the word, without a barrier or a fence.
__device__ __forceinline__ uint4 plan_poll(const uint4 *p) {
  unsigned long long a, b;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
  return make_uint4((uint32_t)a, (uint32_t)(a >> 32), (uint32_t)b, (uint32_t)(b >> 32));
}
__device__ __forceinline__ uint2 plan_poll(const uint2 *p) {
  unsigned long long a;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
  return make_uint2((uint32_t)a, (uint32_t)(a >> 32));
}

// The plan on a grid of co-resident CTAs, as a data flow: an item waits for
// the state words it reads, not for its major stage.  Snapshot k's words are
// published in buffer k mod 4 with the number k (zeroed before the launch;
// words that no partition writes are read from the snapshot itself).  The
// buffer of snapshot c + 1 held snapshot c - 3, so a CTA starts cycle c when
// every CTA is done with the loads of cycle c - 3.  Each CTA arrives once per
// cycle, in the counter of the cycle mod 4: nothing holds a CTA back from one
// that only reads its words, so one sum over all cycles would let the CTAs
// ahead stand in for one behind, and its words would be overwritten.  No CTA
// arrives for cycle c + 4 before every CTA has arrived for c.
//
// Hint.  With many CTAs the polls of those that wait slow down the words the
// others publish, so above PLAN_HINT_ITEMS items a stage a CTA first waits
// (one thread, relaxed, no fence: the words' own numbers decide) until all but
// hint_slack - 1 of the items of the stages before are done.  2M-gate SoC,
// 128 items a stage, per major stage: 4.76 us without, 4.33 / 4.21 / 4.14
// with slack 1 / 4 / 16; 48 items: 2.50 us without, 2.72 with, so those run
// without.  A grid barrier with a release fence instead took 4.39 and 3.33 us.
template <bool X, bool PAIRS>
__global__ void __launch_bounds__(EB, 1) plan_flow_kernel(const __grid_constant__ PlanParams P) {
  extern __shared__ __align__(128) uint8_t dyn[];
  __shared__ uint64_t bar[2];
  uint32_t *const buf0 = reinterpret_cast<uint32_t *>(dyn);
  uint8_t *const slots = dyn + 4 * (size_t)P.nbuf * P.blob_cap;
  uint2 *const words = reinterpret_cast<uint2 *>(slots + P.slot_bytes);
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t rank = blockIdx.x, G = gridDim.x, nms = P.num_major_stages;
  if (t == 0) {
    for (int b = 0; b < 2; ++b)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(plan_smem(&bar[b])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    slots[0] = 0;  // the constant
  }
  __syncthreads();
  PlanFetch F(P, buf0, bar, rank, G);
  const bool two = P.nbuf == 2;
  if (t == PT) F.issue();
  uint32_t n_run = 0;  // items run so far
  for (size_t c = 0; c < P.num_cycles; ++c) {
    const uint32_t *in = P.states + c * P.state_size;
    uint32_t *out = P.states + (c + 1) * P.state_size;
    bool opened = false;
    for (unsigned ms = 0; ms < nms; ++ms) {
      const uint32_t i1 = P.stage_item[ms + 1];
      for (uint32_t it = P.stage_item[ms] + rank; it < i1; it += G) {
        const uint32_t *B = buf0 + (size_t)F.buf_of(n_run) * P.blob_cap;
        // the blob of this item (copied while the last one ran)
        bool ok = plan_mbar_wait(&bar[F.buf_of(n_run)], F.par_of(n_run));
        if (!opened && t == 0 && c >= 3) {
          const unsigned long long target = (unsigned long long)P.active * ((c - 3) / 4 + 1);
          const uint64_t t0 = clock64();
          for (;;) {
            unsigned long long v;
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];"
                         : "=l"(v)
                         : "l"(&g_plan_count[P.slot][(c - 3) & 3])
                         : "memory");
            if (v >= target) break;
            if (*((volatile int *)&g_status[P.slot]) != 0 ||
                (uint64_t)(clock64() - t0) > P.timeout) {
              ok = false;
              break;
            }
          }
        }
        if (P.hint_slack) {
          if (t == 0) {
            const unsigned long long target =
                (unsigned long long)P.stage_item[32] * c + P.stage_item[ms];
            const uint64_t t0 = clock64();
            for (;;) {
              unsigned long long v;
              asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];"
                           : "=l"(v)
                           : "l"(&g_plan_hint[P.slot])
                           : "memory");
              if (v + P.hint_slack > target || (uint64_t)(clock64() - t0) > P.timeout) break;
            }
          }
          __syncthreads();
        }
        const uint32_t ngw = B[PH_NGW], ngr = B[PH_NGR], nw = B[PH_NW];
        const uint32_t io = B[PH_IO];
        const bool isx = X && B[PH_ISX] != 0;
        // ---- state words, and the old words of writeouts that may keep them:
        // lane k of warp w commits writeout word w + 16 k of the item in every
        // cycle, so it reads what it wrote itself, in its own program order
        const uint32_t my_j = warp + (EB / 32) * lane;
        uint2 old = make_uint2(0, 0);
        if (ok) {
          const uint32_t *gw = B + B[PH_OGW];
          constexpr int K = 4;  // words in flight per thread
          for (uint32_t i0 = t; i0 < ngw && ok; i0 += K * EB) {
            uint32_t missing = 0, v[K], x[K];
            size_t at[K];
            uint32_t snap[K];
#pragma unroll
            for (int k = 0; k < K; ++k) {
              const uint32_t i = i0 + k * EB;
              if (i >= ngw) break;
              const uint32_t w = gw[i], o = w & (PLAN_DIRECT - 1);
              const size_t sn = c + (w >> 31);
              snap[k] = (uint32_t)sn;
              if ((w & PLAN_DIRECT) || sn == 0) {
                const uint32_t *s = P.states + sn * P.state_size + o;
                v[k] = ldcg(s);
                x[k] = isx ? ldcg(s + P.xoff) : 0u;
              } else {
                at[k] = (size_t)(sn & 3) * P.rio + o;
                missing |= 1u << k;
              }
            }
            uint64_t t0 = 0;
            for (uint32_t n = 0; missing; ++n) {
              uint4 q[K];
#pragma unroll
              for (int k = 0; k < K; ++k)
                if ((missing >> k) & 1u) {
                  if (X) {
                    q[k] = plan_poll(reinterpret_cast<const uint4 *>(P.exchange) + at[k]);
                  } else {
                    const uint2 r = plan_poll(reinterpret_cast<const uint2 *>(P.exchange) + at[k]);
                    q[k] = make_uint4(r.x, r.y, 0u, r.y);
                  }
                }
#pragma unroll
              for (int k = 0; k < K; ++k)
                if (((missing >> k) & 1u) && q[k].y == snap[k] && q[k].w == snap[k]) {
                  v[k] = q[k].x;
                  x[k] = q[k].z;
                  missing &= ~(1u << k);
                }
              if (n == 0) t0 = clock64();
              if ((n & 255u) == 255u && (*((volatile int *)&g_status[P.slot]) != 0 ||
                                         (uint64_t)(clock64() - t0) > P.timeout)) {
                ok = false;
                break;
              }
            }
#pragma unroll
            for (int k = 0; k < K; ++k)
              if (i0 + k * EB < ngw) words[i0 + k * EB] = make_uint2(v[k], x[k]);
          }
          if (my_j < nw && B[B[PH_OKEEP] + my_j])
            old = make_uint2(ldcg(in + io + my_j), isx ? ldcg(in + (size_t)P.xoff + io + my_j) : 0u);
        }
        // a wait that ran out ends the launch with its status set
        if (__syncthreads_or(!ok)) {
          if (t == 0) atomicCAS(&g_status[P.slot], 0, JQ_ERR_BARRIER_TIMEOUT);
          if (t == PT) F.drain(n_run);
          return;
        }
        if (!opened && t == 0 && c)  // done with the loads of cycle c - 1
          asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(
                           &g_plan_count[P.slot][(c - 1) & 3])
                       : "memory");
        opened = true;
        if (two && t == PT) F.issue();  // into the other buffer: its readers passed this barrier
        // ---- needed bits to bytes
        {
          const uint32_t *ex = B + B[PH_OEXP];
          for (uint32_t i = t; i < ngr; i += EB) {
            const uint32_t e = ex[i];
            const uint2 w = words[e >> 5];
            slots[1 + i] = (uint8_t)(((w.x >> (e & 31)) & 1u) | (isx ? ((w.y >> (e & 31)) & 1u) << 1 : 0u));
          }
        }
        plan_gates<X, PAIRS>(B, slots, ngr);
        plan_srams(P, B, slots, isx);
        // ---- commit: a warp per writeout word
        {
          const uint32_t *com = B + B[PH_OCOM];
          for (uint32_t j = warp; j < nw; j += EB / 32) {
            const PlanWord w = plan_word(com, slots, j, isx);
            if (my_j == j) {
              const size_t o = (size_t)io + j;
              const size_t at = (size_t)((c + 1) & 3) * P.rio + o;
              const uint32_t n = (uint32_t)(c + 1);
              const uint32_t nv = (old.x & ~w.cp) | (w.v & w.cp);
              if (X) {
                // a partition without X leaves the snapshot's host-filled X word
                const uint32_t nx = isx ? (old.y & ~w.cp & ~w.cx) | (w.x & w.cp & ~w.cx) | w.cx
                                        : ldcg(out + P.xoff + o);
                asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(
                                 reinterpret_cast<uint4 *>(P.exchange) + at),
                             "l"(((unsigned long long)n << 32) | nv),
                             "l"(((unsigned long long)n << 32) | nx)
                             : "memory");
                if (isx) out[P.xoff + o] = nx;
              } else {
                asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(
                                 reinterpret_cast<uint2 *>(P.exchange) + at),
                             "l"(((unsigned long long)n << 32) | nv)
                             : "memory");
              }
              out[o] = nv;
              if (P.arr_first) plan_timing(P, out, o, w.cp, c);
            }
          }
        }
        ++n_run;
        if (P.hint_slack) {
          __syncthreads();
          if (t == 0)
            asm volatile("red.relaxed.gpu.global.add.u64 [%0], 1;" ::"l"(&g_plan_hint[P.slot])
                         : "memory");
        }
        if (!two) {
          __syncthreads();
          if (t == PT) F.issue();
        }
      }
    }
  }
}

// The plan on one thread-block cluster whose CTAs each keep a mirror of the
// current and the next snapshot in shared memory (uint2 value and X word per
// state word, or one word without X).  A commit sends each word to every
// CTA's mirror with st.async, counted in bytes by that CTA's mbarrier of the
// major stage, so a stage ends when its words have arrived: no barrier, no
// fence for the snapshot's global stores, no load from L2.  Every CTA that
// receives words runs at least one item a cycle.  A CTA waits for all words
// of the stages before an item of its own, so another one can be ahead of it
// by at most the words of that item's stage in the next cycle: a stage has
// two mbarriers, for even and odd cycles, and neither sees the bytes of two
// phases at once.  Words of snapshot c + 2 overwrite those of c only after
// the last item that reads snapshot c has sent its own.
template <bool X, bool PAIRS>
__global__ void __launch_bounds__(EB, 1) plan_mirror_kernel(const __grid_constant__ PlanParams P) {
  extern __shared__ __align__(128) uint8_t dyn[];
  __shared__ uint64_t bar[2], stage_bar[64];  // stage_bar[2 ms + cycle parity]
  constexpr uint32_t WB = X ? 8 : 4;  // bytes of a mirrored word
  uint32_t *const buf0 = reinterpret_cast<uint32_t *>(dyn);
  uint8_t *const slots = dyn + 4 * (size_t)P.nbuf * P.blob_cap;
  uint32_t *const mirror = reinterpret_cast<uint32_t *>(slots + P.slot_bytes);  // [2][rio]
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t rank = blockIdx.x, G = gridDim.x, nms = P.num_major_stages;
  if (t == 0) {
    for (int b = 0; b < 2; ++b)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(plan_smem(&bar[b])) : "memory");
    for (unsigned k = 0; k < 2 * nms; ++k)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(plan_smem(&stage_bar[k]))
                   : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    slots[0] = 0;  // the constant
  }
  __syncthreads();
  auto arm = [&](unsigned k) {  // thread 0: the mbarrier's next phase expects the stage's words
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                     plan_smem(&stage_bar[k])),
                 "r"(WB * P.stage_words[k >> 1])
                 : "memory");
  };
  if (t == 0)
    for (unsigned k = 0; k < 2 * nms; ++k) arm(k);
  // snapshot 0, and the words nobody writes of snapshot 1
  auto put = [&](uint32_t snap, uint32_t w, uint32_t v, uint32_t x) {
    if (X)
      reinterpret_cast<uint2 *>(mirror)[(size_t)snap * P.rio + w] = make_uint2(v, x);
    else
      mirror[(size_t)snap * P.rio + w] = v;
  };
  if (rank < P.active)
  for (uint32_t w = t; w < P.rio; w += EB)
    put(0, w, ldcg(P.states + w), X ? ldcg(P.states + P.xoff + w) : 0u);
  const uint32_t my_uw = t < P.n_unwritten ? P.unwritten[t] : 0u;
  uint32_t uv = 0, ux = 0;  // thread t's unwritten word of the next snapshot
  auto load_uw = [&](size_t snap) {
    if (t < P.n_unwritten && snap <= P.num_cycles) {
      const uint32_t *s = P.states + snap * P.state_size;
      uv = ldcg(s + my_uw);
      if (X) ux = ldcg(s + P.xoff + my_uw);
    }
  };
  load_uw(1);
  // every CTA's mbarriers are armed before any word is sent
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  PlanFetch F(P, buf0, bar, rank, G);
  const bool two = P.nbuf == 2;
  if (t == PT) F.issue();
  uint32_t n_run = 0;
  bool failed = false;
  // lane k sends to CTA k
  const uint32_t dst_cta = lane < P.active ? lane : 0;
  uint32_t r_mirror, r_bar;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r_mirror) : "r"(plan_smem(mirror)), "r"(dst_cta));
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r_bar) : "r"(plan_smem(stage_bar)), "r"(dst_cta));
  for (size_t c = 0; c < P.num_cycles && !failed && rank < P.active; ++c) {
    uint32_t *out = P.states + (c + 1) * P.state_size;
    const uint32_t si = (uint32_t)(c & 1), so = si ^ 1u;
    for (unsigned ms = 0; ms < nms; ++ms) {
      // the previous stage's words (its phase: one per cycle)
      bool ok = true;
      const size_t pc = ms ? c : c - 1;  // its cycle
      const unsigned pk = 2 * (ms ? ms - 1 : nms - 1) + (uint32_t)(pc & 1);
      if (c || ms) ok = plan_mbar_wait_cluster(&stage_bar[pk], (uint32_t)(pc >> 1) & 1u);
      if (ms == 0) {  // words nobody writes: host-filled in every snapshot
        if (t < P.n_unwritten) put(so, my_uw, uv, ux);
        for (uint32_t i = EB + t; i < P.n_unwritten; i += EB) {
          const uint32_t w = P.unwritten[i];
          put(so, w, ldcg(out + w), X ? ldcg(out + P.xoff + w) : 0u);
        }
        load_uw(c + 2);
      }
      const uint32_t i1 = P.stage_item[ms + 1];
      bool synced = false;
      for (uint32_t it = P.stage_item[ms] + rank; it < i1 || !synced; it += G) {
        const bool have = it < i1;
        const uint32_t *B = buf0 + (size_t)F.buf_of(n_run) * P.blob_cap;
        if (have) ok = plan_mbar_wait(&bar[F.buf_of(n_run)], F.par_of(n_run)) && ok;
        // also: the last item's commit is done with the slots
        if (__syncthreads_or(!ok)) {
          failed = true;
          break;
        }
        // every thread has seen the previous stage's phase
        if (!synced && (c || ms) && t == 0) arm(pk);
        synced = true;
        if (!have) break;
        if (two && t == PT) F.issue();
        const uint32_t ngr = B[PH_NGR], nw = B[PH_NW], io = B[PH_IO];
        const bool isx = X && B[PH_ISX] != 0;
        // ---- needed bits to bytes
        {
          const uint32_t *ex = B + B[PH_OEXP];
          for (uint32_t i = t; i < ngr; i += EB) {
            const uint32_t e = ex[i];
            const uint32_t w = (e >> 6) + ((e & 32u) ? so : si) * P.rio;
            if (X) {
              const uint2 v = reinterpret_cast<const uint2 *>(mirror)[w];
              const uint32_t x = isx ? v.y : 0u;
              slots[1 + i] = (uint8_t)(((v.x >> (e & 31)) & 1u) | (((x >> (e & 31)) & 1u) << 1));
            } else {
              slots[1 + i] = (uint8_t)((mirror[w] >> (e & 31)) & 1u);
            }
          }
        }
        plan_gates<X, PAIRS>(B, slots, ngr);
        plan_srams(P, B, slots, isx);
        // ---- commit: a warp per writeout word, to the snapshot and to every
        // CTA's mirror
        {
          const uint32_t *com = B + B[PH_OCOM];
          for (uint32_t j = warp; j < nw; j += EB / 32) {
            const PlanWord w = plan_word(com, slots, j, isx);
            const size_t o = (size_t)io + j;
            uint32_t ov = 0, ox = 0;
            if (w.cp != 0xffffffffu) {
              if (X) {
                const uint2 p = reinterpret_cast<const uint2 *>(mirror)[(size_t)si * P.rio + o];
                ov = p.x;
                ox = p.y;
              } else {
                ov = mirror[(size_t)si * P.rio + o];
              }
            }
            const uint32_t nv = (ov & ~w.cp) | (w.v & w.cp);
            // a partition without X leaves the snapshot's host-filled X word
            uint32_t nx = 0;
            if (X)
              nx = isx ? (ox & ~w.cp & ~w.cx) | (w.x & w.cp & ~w.cx) | w.cx
                       : ldcg(out + P.xoff + o);
            if (lane < P.active) {
              const uint32_t a = r_mirror + ((uint32_t)so * P.rio + (uint32_t)o) * WB;
              const uint32_t mb = r_bar + 8 * (2 * ms + si);
              if (X)
                asm volatile(
                    "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::
                        "r"(a),
                    "r"(nv), "r"(nx), "r"(mb)
                    : "memory");
              else
                asm volatile(
                    "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::
                        "r"(a),
                    "r"(nv), "r"(mb)
                    : "memory");
            }
            if (lane == 0) {
              out[o] = nv;
              if (isx) out[P.xoff + o] = nx;
              if (P.arr_first) plan_timing(P, out, o, w.cp, c);
            }
          }
        }
        ++n_run;
        if (!two) {
          __syncthreads();
          if (t == PT) F.issue();
        }
      }
      if (failed) break;
    }
  }
  if (failed && t == 0) atomicCAS(&g_status[P.slot], 0, JQ_ERR_BARRIER_TIMEOUT);
  if (t == PT) F.drain(n_run);
  // no CTA leaves while another may still send it words (on failure the
  // others' bounded waits end too), nor before the last stage's words have
  // arrived: the barrier below orders the sends, not their arrival
  if (t == 0 && !failed && P.num_cycles && rank < P.active) {
    const size_t lc = P.num_cycles - 1;
    if (!plan_mbar_wait_cluster(&stage_bar[2 * (nms - 1) + (uint32_t)(lc & 1)],
                                (uint32_t)(lc >> 1) & 1u))
      atomicCAS(&g_status[P.slot], 0, JQ_ERR_BARRIER_TIMEOUT);
  }
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

}  // namespace jqk
