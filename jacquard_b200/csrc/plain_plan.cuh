// Gate-list form of the one-stream interpreter (sm_100a).
//
// The script's boomerang form (shuffle, 8192 -> 1 AND tree, hooks) costs a
// partition about 16 bit gathers per thread, 2 to 6 CTA barriers and the
// serial deep levels per stage, however few of its 8191 positions anything
// reads.  The plan build (plan_build_kernel, once per script, on the device)
// resolves a partition to what its writeouts depend on: the state words it
// reads, the bits of them it needs, its live AND gates by logic level
// (pass-throughs, constants and dead positions folded away), and per
// writeout bit the reference of its value and of its clock enable.  The
// executor (plan_run_kernel) then runs, per item and cycle: one load per
// state word, one byte per needed bit, two byte reads and one byte write per
// gate with one CTA barrier per logic level, and ballots that pack the
// writeouts.  Values are bytes (bit 0 value, bit 1 X) in shared memory,
// named by 15-bit slots with an inversion bit.
//
// What bounds it: latency.  A major stage of one stream is a chain of
// barrier, state load, a few gate levels and the commit; its script data
// (about 25 KB per partition) is copied by TMA one item ahead.
#pragma once
#include "sim_common.cuh"

namespace jqk {

constexpr int PB = 1024;                 // threads of the build kernel
// Threads of the run kernels.  A logic level has 50 to 500 gates of a split
// partition, so more threads only add warps that issue the loop and the
// barrier; 1024 (64 registers, spills) measured 1.1 to 1.4 times slower on
// every design, 256 within 1% on the small design and 8% slower on the 2M-gate one.
constexpr int EB = 512;
constexpr uint32_t PT = EB - 32;         // the thread that issues the blob copies
constexpr uint32_t PLAN_MAX_NS = 64;     // boomerang stages of a partition
constexpr uint32_t PLAN_MAX_LEVELS = 896;
constexpr uint32_t PLAN_MAX_SLOTS = 32768;
constexpr uint32_t PLAN_DIRECT = 1u << 30;  // state word that no partition writes

// Item header (words of the item's blob; section offsets in words, 16-byte
// aligned).
enum PlanHdr : uint32_t {
  PH_WORDS, PH_NGW, PH_NGR, PH_NLEV, PH_NW, PH_IO, PH_NSR, PH_SRAM_OFF, PH_ISX, PH_XOFF,
  PH_OGW, PH_OEXP, PH_OLEV, PH_OGATE, PH_OSRAM, PH_OCOM, PH_OKEEP, PH_SRSLOT, PH_SIZE = 20
};

// Build result: unsupported flag (bit 0: the plan, bit 1: its mirrored form),
// blob words used, the largest blob, slot count and state-word count of any
// item, the words up to the last written one, X use (bit 0: a partition
// without, bit 1: with X) and its offset (min and ~max), the words each major
// stage writes, and the words below `rio` that no partition writes.
struct PlanResult {
  uint32_t unsupported, x_use;
  unsigned long long used;
  uint32_t max_blob, max_slots, max_gw, rio;
  uint32_t xoff_max, xoff_inv_max, n_unwritten, pad;
  uint32_t stage_words[32];
};

struct PlanBuildParams {
  const uint32_t *script;
  const unsigned long long *part_off;  // script word offset of each partition
  const uint32_t *part_ms;             // its major stage
  const uint32_t *items;               // per item: partition, sub | nsub << 16
  const uint32_t *writer;              // per state word: major stage + 1 that writes it, or 0
  uint32_t writer_words;
  uint32_t direct;                     // expansion entries name state words (mirrored form)
  uint32_t *blob;
  unsigned long long blob_cap;
  unsigned long long *item_off;        // per item: blob word offset
  uint32_t *item_words;                // and size
  PlanResult *res;
};

struct PlanShared {
  uint32_t chunk[STAGE_WORDS];
  uint32_t live[PLAN_MAX_NS][256];
  uint8_t lv[8192];
  uint32_t ref_a[8192], ref_b[8192];
  uint16_t woref[8192];
  uint32_t need[256], wneed[256], ext[256];
  uint32_t lev[PLAN_MAX_LEVELS], lev_base[PLAN_MAX_LEVELS];
  uint32_t warp_sum[32];
  int bad;
  uint32_t max_lev, n_gates;
  unsigned long long off;
};

__device__ __forceinline__ uint32_t plan_perm(const uint32_t *chunk, uint32_t q) {
  const uint32_t T = q >> 5, k = q & 31;
  const uint32_t w = chunk[(k >> 3) * 1024 + T * 4 + ((k >> 1) & 3)];
  return ((k & 1) ? (w >> 16) : (w & 0xffffu)) & 8191u;
}
__device__ __forceinline__ uint32_t plan_flag(const uint32_t *chunk, uint32_t q, int f) {
  return (chunk[4096 + 4 * (q >> 5) + f] >> (q & 31)) & 1u;
}
__device__ __forceinline__ void plan_load_chunk(uint32_t *dst, const uint32_t *src) {
  for (uint32_t i = threadIdx.x; i < STAGE_WORDS / 4; i += PB)
    reinterpret_cast<uint4 *>(dst)[i] = ldg4(src + 4 * i);
  __syncthreads();
}
// Exclusive prefix sum over the CTA; every thread calls it.
__device__ uint32_t plan_scan(uint32_t v, uint32_t *warp_sum, uint32_t *total) {
  const uint32_t t = threadIdx.x;
  uint32_t incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t o = __shfl_up_sync(0xffffffffu, incl, d);
    if ((t & 31) >= (uint32_t)d) incl += o;
  }
  __syncthreads();
  if ((t & 31) == 31) warp_sum[t >> 5] = incl;
  __syncthreads();
  uint32_t base = incl - v, n = 0;
  for (uint32_t w = 0; w < PB / 32; ++w) {
    if (w < (t >> 5)) base += warp_sum[w];
    n += warp_sum[w];
  }
  *total = n;
  return base;
}

// Reference of a value while an item is built: logic level << 16 | slot << 1
// | inversion; slot 0 is the constant 0.
// AND of two references: a new gate (returns true), or what it folds to.  An
// ob-forced b input, or a constant 1 on either side, passes the other side on
// with its X bit (X rule with that side 1 and known: the other's X); a known
// 0 gives a known 0.
__device__ __forceinline__ bool plan_and(uint32_t a, uint32_t b, uint32_t xa, uint32_t xb,
                                         uint32_t ob, uint32_t &r, uint32_t &ra, uint32_t &rb) {
  ra = a ^ xa;
  rb = b ^ xb;
  if (ob) {
    r = ra;
    return false;
  }
  if (((rb >> 1) & 0x7fffu) == 0) {
    r = (rb & 1u) ? ra : 0u;
    return false;
  }
  if (((ra >> 1) & 0x7fffu) == 0) {
    r = (ra & 1u) ? rb : 0u;
    return false;
  }
  const uint32_t la = ra >> 16, lb = rb >> 16;
  r = (la > lb ? la : lb) + 1u;  // its level
  return true;
}

// One CTA builds one item: partition `items[2i]`, writeout slots
// [nio * sub / nsub, nio * (sub + 1) / nsub) (partitions with SRAMs have one
// item).  The result's `unsupported` flag is set for what the plan does not
// represent -- a writeout slot that no hook, SRAM or duplicate writes, or a
// permutation that reads one an earlier partition left (both observe the
// per-block arrays of the script kernel), a partition that reads what the
// same major stage writes, or sizes past the limits above -- and the script
// then runs in its own form.
__global__ void __launch_bounds__(PB, 1) plan_build_kernel(PlanBuildParams P, uint32_t n_items) {
  extern __shared__ __align__(16) uint8_t plan_dyn[];
  PlanShared &ps = *reinterpret_cast<PlanShared *>(plan_dyn);
  const uint32_t t = threadIdx.x, item = blockIdx.x;
  if (item >= n_items) return;
  const uint32_t pid = P.items[2 * item], sub = P.items[2 * item + 1] & 0xffffu,
                 nsub = P.items[2 * item + 1] >> 16;
  const uint32_t *m = P.script + P.part_off[pid];
  const uint32_t ns = m[0], nio = m[2], io_off = m[3], nsr = m[4], sram_off = m[5], R = m[6],
                 ndup = m[7], isx = m[8], xoff = m[9];
  const uint32_t my_ms = P.part_ms[pid];
  bool bad = ns > PLAN_MAX_NS || nio > 256 || nsr * 4 + ndup > 256 || nsr + ndup > nio ||
             (nsr && nsub > 1) || R > 32;
  if (bad) {  // uniform
    if (t == 0) atomicOr(&P.res->unsupported, 1u);
    return;
  }
  const uint32_t *gr = m + 256, *ch = gr + 512 * (size_t)R;
  const uint32_t j0 = nio * sub / nsub, j1 = nio * (sub + 1) / nsub;
  const uint32_t hooked = nio - nsr - ndup;  // slots below are hooked
  if (t == 0) ps.bad = 0;
  if (t < 256) {
    ps.wneed[t] = t >= j0 && t < j1 ? 0xffffffffu : 0u;
    ps.need[t] = 0;
  }
  __syncthreads();
  // ---- writeout bits the item needs: its own, their clock enables, and what
  // its SRAMs and needed duplicates stage
  plan_load_chunk(ps.chunk, ch + STAGE_WORDS * (size_t)(ns + 1));
  for (uint32_t q = 32 * j0 + t; q < 32 * j1; q += PB)
    if (!plan_flag(ps.chunk, q, 1)) {
      const uint32_t p = plan_perm(ps.chunk, q);
      if ((p >> 5) >= nio) bad = true;
      else atomicOr(&ps.wneed[p >> 5], 1u << (p & 31));
    }
  __syncthreads();
  plan_load_chunk(ps.chunk, ch + STAGE_WORDS * (size_t)ns);
  for (uint32_t q = t; q < (nsr * 4 + ndup) * 32; q += PB) {
    bool use;
    if (q < nsr * 128) {
      use = (q & 127u) < 96u;
    } else {
      const uint32_t k = (q >> 5) - nsr * 4;  // duplicate k, slot hooked + k
      use = (ps.wneed[hooked + k] >> (q & 31)) & 1u;
    }
    if (use && !plan_flag(ps.chunk, q, 1)) {
      const uint32_t p = plan_perm(ps.chunk, q);
      if ((p >> 5) >= hooked) bad = true;  // (reads no SRAM or duplicate slot: wneed of
      else atomicOr(&ps.wneed[p >> 5], 1u << (p & 31));  // those is complete)
    }
  }
  __syncthreads();
  for (uint32_t j = t; j < hooked; j += PB) {
    const uint32_t hw = m[128 + j / 2], h = (j & 1) ? hw >> 16 : hw & 0xffffu;
    if (ps.wneed[j] && (h >> 8) >= ns) bad = true;
  }
  if (__syncthreads_or(bad)) {
    if (t == 0) atomicOr(&P.res->unsupported, 1u);
    return;
  }
  // ---- liveness, last stage to first (see jq_plain_depth_kernel; an
  // ob-forced b input is not needed at any level)
  for (int ci = (int)ns - 1; ci >= 0; --ci) {
    plan_load_chunk(ps.chunk, ch + STAGE_WORDS * (size_t)ci);
    if (t < 256) ps.ext[t] = ps.need[t];
    __syncthreads();
    for (uint32_t j = t; j < hooked; j += PB) {
      const uint32_t hw = m[128 + j / 2], h = (j & 1) ? hw >> 16 : hw & 0xffffu;
      if ((h >> 8) == (uint32_t)ci && ps.wneed[j]) atomicOr(&ps.ext[h & 255u], ps.wneed[j]);
    }
    __syncthreads();
    if (t == 0) ps.lv[0] = 0;
    for (uint32_t M = 1; M <= 4096; M <<= 1) {
      for (uint32_t c = M + t; c < 2 * M; c += PB) {
        uint8_t l = (uint8_t)((ps.ext[c >> 5] >> (c & 31)) & 1u);
        if (M > 1) {
          const uint32_t h = M >> 1;
          const bool is_b = c >= M + h;
          const uint32_t par = is_b ? c - M : c - h;
          if (ps.lv[par] && !(is_b && plan_flag(ps.chunk, par, 2))) l = 1;
        }
        ps.lv[c] = l;
      }
      __syncthreads();
    }
    if (t < 256) ps.need[t] = 0;
    for (uint32_t c = t; c < 8192; c += PB) {
      const uint32_t w = __ballot_sync(0xffffffffu, ps.lv[c] != 0);
      if ((t & 31) == 0) ps.live[ci][c >> 5] = w;
    }
    __syncthreads();
    for (uint32_t p = 4096 + t; p < 8192; p += PB)
      if (ps.lv[p]) {
        const uint32_t sa = plan_perm(ps.chunk, p - 4096);
        atomicOr(&ps.need[sa >> 5], 1u << (sa & 31));
        if (!plan_flag(ps.chunk, p, 2)) {
          const uint32_t sb = plan_perm(ps.chunk, p);
          atomicOr(&ps.need[sb >> 5], 1u << (sb & 31));
        }
      }
    __syncthreads();
  }
  // ---- global read.  Thread t < 256 appends its masked bits round by round,
  // lowest first; the first appended bit ends up most significant, i.e. at
  // position 32t + total - 1, bits pushed past 31 are lost
  // (csrc/kernel_v1_impl.cuh:87-154).  Needed positions take slots 1, 2, ...
  uint32_t total = 0, n_ent = 0, n_bit = 0;
  const uint32_t nd = t < 256 ? ps.need[t] : 0u;
  if (t < 256) {
    for (uint32_t r = 0; r < R; ++r) total += __popc(__ldg(gr + 512 * r + 2 * t + 1));
    uint32_t i = 0;
    for (uint32_t r = 0; r < R; ++r) {
      const uint2 im = ldg2(gr + 512 * r + 2 * t);
      uint32_t hit = 0;
      for (uint32_t k = im.y; k; k &= k - 1, ++i) {
        const uint32_t pos = total - 1 - i;
        if (pos < 32 && ((nd >> pos) & 1u)) ++hit;
      }
      n_ent += hit != 0;
      n_bit += hit;
      const uint32_t w = im.x & 0x7fffffffu;
      // staged reads: only words that earlier major stages (or nobody) write
      if (hit && (im.x >> 31)) {
        if (w < P.writer_words && P.writer[w] > my_ms) bad = true;
      }
      if (hit && w >= P.writer_words) bad = true;
    }
  }
  uint32_t n_gw = 0, n_gr = 0;
  const uint32_t ent0 = plan_scan(n_ent, ps.warp_sum, &n_gw);
  const uint32_t bit0 = plan_scan(n_bit, ps.warp_sum, &n_gr);
  auto gr_refs = [&]() {
    for (uint32_t p = t; p < 8192; p += PB) ps.ref_a[p] = 0;
    __syncthreads();
    if (t < 256) {
      uint32_t s = 1 + bit0;
      // slots in descending position, the order the emission below walks
      for (int pos = (int)(total < 32 ? total : 32) - 1; pos >= 0; --pos)
        if ((nd >> pos) & 1u) ps.ref_a[32 * t + pos] = s++ << 1;
    }
    __syncthreads();
  };
  // ---- forward over the stages: reference of every live position; with
  // `gates` the gates are written, else counted per level
  auto forward = [&](uint32_t *gates, uint32_t gate0) {
    uint32_t *prev = ps.ref_a, *cur = ps.ref_b;
    for (uint32_t ci = 0; ci < ns; ++ci) {
      plan_load_chunk(ps.chunk, ch + STAGE_WORDS * (size_t)ci);
      auto place = [&](uint32_t p, uint32_t a, uint32_t b) {
        uint32_t r, ra, rb;
        if (plan_and(a, b, plan_flag(ps.chunk, p, 0), plan_flag(ps.chunk, p, 1),
                     plan_flag(ps.chunk, p, 2), r, ra, rb)) {
          const uint32_t l = r < PLAN_MAX_LEVELS ? r : PLAN_MAX_LEVELS - 1;
          const uint32_t k = atomicAdd(&ps.lev[l], 1u);
          if (gates) {
            const uint32_t g = ps.lev_base[l] + k;
            gates[g] = (ra & 0xffffu) | (rb << 16);
            r = (l << 16) | ((gate0 + g) << 1);
          } else {
            r = (l << 16) | (1u << 1);
          }
        }
        cur[p] = r;
      };
      if (t == 0) cur[0] = 0;
      for (uint32_t p = 4096 + t; p < 8192; p += PB) {
        if ((ps.live[ci][p >> 5] >> (p & 31)) & 1u)
          place(p, prev[plan_perm(ps.chunk, p - 4096)], prev[plan_perm(ps.chunk, p)]);
        else
          cur[p] = 0;
      }
      for (uint32_t L = 2048; L; L >>= 1) {
        __syncthreads();
        for (uint32_t p = L + t; p < 2 * L; p += PB) {
          if ((ps.live[ci][p >> 5] >> (p & 31)) & 1u)
            place(p, cur[p + L], cur[p + 2 * L]);
          else
            cur[p] = 0;
        }
      }
      __syncthreads();
      for (uint32_t q = t; q < hooked * 32; q += PB) {
        const uint32_t j = q >> 5;
        const uint32_t hw = m[128 + j / 2], h = (j & 1) ? hw >> 16 : hw & 0xffffu;
        if ((h >> 8) == ci) ps.woref[q] = (uint16_t)cur[32 * (h & 255u) + (q & 31)];
      }
      __syncthreads();
      uint32_t *x = prev;
      prev = cur;
      cur = x;
    }
  };
  gr_refs();
  for (uint32_t l = t; l < PLAN_MAX_LEVELS; l += PB) ps.lev[l] = 0;
  __syncthreads();
  forward(nullptr, 0);
  if (t == 0) {
    uint32_t n = 0, top = 0;
    for (uint32_t l = 1; l < PLAN_MAX_LEVELS; ++l) {
      ps.lev_base[l] = n;
      n += ps.lev[l];
      if (ps.lev[l]) top = l;
    }
    ps.n_gates = n;
    ps.max_lev = top;
    if (ps.lev[PLAN_MAX_LEVELS - 1]) ps.bad = 1;  // deeper levels share the last count
  }
  __syncthreads();
  const uint32_t n_gates = ps.n_gates, n_lev = ps.max_lev, nw = j1 - j0;
  const uint32_t gate0 = 1 + n_gr, sr_slot = gate0 + n_gates, n_slots = sr_slot + 32 * nsr;
  auto al = [](uint32_t w) { return (w + 3u) & ~3u; };
  const uint32_t o_gw = PH_SIZE, o_exp = o_gw + (P.direct ? 0u : al(n_gw)), o_lev = o_exp + al(n_gr),
                 o_gate = o_lev + al(n_lev), o_sram = o_gate + al(n_gates),
                 o_com = o_sram + 96 * nsr, o_keep = o_com + 32 * nw, words = o_keep + al(nw);
  if (n_slots > PLAN_MAX_SLOTS) bad = true;
  if (__syncthreads_or(bad || ps.bad)) {
    if (t == 0) atomicOr(&P.res->unsupported, 1u);
    return;
  }
  if (t == 0) {
    ps.off = atomicAdd(&P.res->used, (unsigned long long)words);
    if (ps.off + words > P.blob_cap) {
      ps.bad = 1;
      atomicOr(&P.res->unsupported, 1u);
    } else {
      P.item_off[item] = ps.off;
      P.item_words[item] = words;
      atomicMax(&P.res->max_blob, words);
      atomicMax(&P.res->max_slots, n_slots);
      atomicMax(&P.res->max_gw, n_gw);
    }
  }
  __syncthreads();
  if (ps.bad) return;
  uint32_t *B = P.blob + ps.off;
  // ---- state words in address order, so the executor's loads coalesce
  // (bitonic sort of (word, entry)); expansion entries name the sorted word,
  // or in the mirrored form the state word itself
  {
    uint32_t *key = ps.ref_b;
    uint16_t *idx = ps.woref;                                    // sorted -> entry
    uint16_t *inv = reinterpret_cast<uint16_t *>(ps.chunk);      // entry -> sorted
    uint32_t n2 = 1;
    while (n2 < n_gw && !P.direct) n2 <<= 1;
    for (uint32_t i = t; i < n2; i += PB) {
      key[i] = 0xffffffffu;
      idx[i] = (uint16_t)i;
    }
    __syncthreads();
    auto walk = [&](auto &&entry) {  // entry(e, word, needed positions of it in order)
      uint32_t e = ent0, i = 0;
      for (uint32_t r = 0; r < R; ++r) {
        const uint2 im = ldg2(gr + 512 * r + 2 * t);
        uint32_t s = 0;
        for (uint32_t k = im.y; k; k &= k - 1, ++i) {
          const uint32_t pos = total - 1 - i;
          if (pos < 32 && ((nd >> pos) & 1u)) {
            entry(e, im.x | (P.writer[im.x & 0x7fffffffu] ? 0u : PLAN_DIRECT), (uint32_t)__ffs(k) - 1);
            ++s;
          }
        }
        e += s != 0;
      }
    };
    if (t < 256 && !P.direct) walk([&](uint32_t e, uint32_t w, uint32_t) { key[e] = w; });
    __syncthreads();
    for (uint32_t size = 2; size <= n2; size <<= 1)
      for (uint32_t stride = size >> 1; stride; stride >>= 1) {
        for (uint32_t i = t; i < n2; i += PB) {
          const uint32_t o = i ^ stride;
          if (o > i) {
            const bool up = !(i & size);
            const uint32_t ki = key[i], ko = key[o];
            if ((ki > ko) == up && ki != ko) {
              key[i] = ko;
              key[o] = ki;
              const uint16_t x = idx[i];
              idx[i] = idx[o];
              idx[o] = x;
            }
          }
        }
        __syncthreads();
      }
    // entries past n_gw hold the largest key; a word index below it never
    // ties with them
    for (uint32_t i = t; i < n_gw && !P.direct; i += PB) {
      B[o_gw + i] = key[i];
      inv[idx[i]] = (uint16_t)i;
    }
    __syncthreads();
    if (t < 256) {
      uint32_t s = bit0;
      if (P.direct)  // word << 6 | staged << 5 | bit
        walk([&](uint32_t, uint32_t w, uint32_t k) {
          const uint32_t i = w & (PLAN_DIRECT - 1);
          if (i >= P.res->rio) atomicOr(&P.res->unsupported, 2u);
          B[o_exp + s++] = (i << 6) | ((w >> 31) << 5) | k;
        });
      else  // sorted word << 5 | bit
        walk([&](uint32_t e, uint32_t, uint32_t k) { B[o_exp + s++] = ((uint32_t)inv[e] << 5) | k; });
    }
    __syncthreads();
  }
  gr_refs();
  for (uint32_t l = t; l < PLAN_MAX_LEVELS; l += PB) ps.lev[l] = 0;
  __syncthreads();
  forward(B + o_gate, gate0);
  for (uint32_t l = t; l < n_lev; l += PB) B[o_lev + l] = ps.lev_base[1 + l] + ps.lev[1 + l];
  // ---- SRAM ports, then the commit: references of the staged words and of
  // each own writeout bit and its clock enable
  plan_load_chunk(ps.chunk, ch + STAGE_WORDS * (size_t)ns);
  auto staged = [&](uint32_t q) -> uint32_t {
    const uint32_t inv = plan_flag(ps.chunk, q, 0);
    return plan_flag(ps.chunk, q, 1) ? inv : ps.woref[plan_perm(ps.chunk, q)] ^ inv;
  };
  for (uint32_t i = t; i < 96 * nsr; i += PB) B[o_sram + i] = staged(128 * (i / 96) + i % 96);
  // duplicate and SRAM slots get their references too
  for (uint32_t q = t; q < 32 * ndup; q += PB)
    if ((ps.wneed[hooked + (q >> 5)] >> (q & 31)) & 1u)
      ps.woref[32 * hooked + q] = (uint16_t)staged(nsr * 128 + q);
  for (uint32_t q = t; q < 32 * nsr; q += PB)
    ps.woref[32 * (hooked + ndup) + q] = (uint16_t)((sr_slot + q) << 1);
  __syncthreads();
  plan_load_chunk(ps.chunk, ch + STAGE_WORDS * (size_t)(ns + 1));
  for (uint32_t i = t; i < 32 * nw; i += PB) {  // a warp per writeout slot
    const uint32_t q = 32 * j0 + i;
    const uint32_t inv = plan_flag(ps.chunk, q, 0);
    const uint32_t cp = plan_flag(ps.chunk, q, 1) ? inv : ps.woref[plan_perm(ps.chunk, q)] ^ inv;
    const uint32_t v = ps.woref[q] ^ plan_flag(ps.chunk, q, 2);
    B[o_com + i] = v | (cp << 16);
    const bool keep = __any_sync(0xffffffffu, cp != 1u);  // not the constant 1
    if ((i & 31) == 0) B[o_keep + (i >> 5)] = keep;
  }
  if (t == 0) {
    B[PH_WORDS] = words;
    B[PH_NGW] = n_gw;
    B[PH_NGR] = n_gr;
    B[PH_NLEV] = n_lev;
    B[PH_NW] = nw;
    B[PH_IO] = io_off + j0;
    B[PH_NSR] = nsr;
    B[PH_SRAM_OFF] = sram_off;
    B[PH_ISX] = isx != 0;
    B[PH_XOFF] = xoff;
    B[PH_OGW] = o_gw;
    B[PH_OEXP] = o_exp;
    B[PH_OLEV] = o_lev;
    B[PH_OGATE] = o_gate;
    B[PH_OSRAM] = o_sram;
    B[PH_OCOM] = o_com;
    B[PH_OKEEP] = o_keep;
    B[PH_SRSLOT] = sr_slot;
  }
}

// Partition offsets and major stages of every entry, and the major stage
// that writes each state word (writer, zeroed; two writers of one word make
// the plan unsupported: their order within a block matters).
__global__ void plan_list_kernel(const size_t *blocks_start, const uint32_t *script,
                                 const uint32_t *part_base, unsigned entries, unsigned num_blocks,
                                 unsigned long long *part_off, uint32_t *part_ms, uint32_t *writer,
                                 uint32_t writer_words, PlanResult *res) {
  const unsigned e = blockIdx.x;
  if (e >= entries) return;
  size_t off = blocks_start[e];
  uint32_t pid = part_base[e];
  const uint32_t ms = e / num_blocks;
  for (;;) {
    const uint32_t ns = script[off];
    if (!ns) break;
    const uint32_t nio = script[off + 2], io = script[off + 3];
    if (threadIdx.x == 0) {
      part_off[pid] = off;
      part_ms[pid] = ms;
      atomicMax(&res->rio, io + nio);
      atomicAdd(&res->stage_words[ms], nio);
      atomicOr(&res->x_use, script[off + 8] ? 2u : 1u);
      if (script[off + 8]) {
        atomicMax(&res->xoff_max, script[off + 9]);
        atomicMax(&res->xoff_inv_max, ~script[off + 9]);
      }
    }
    for (uint32_t j = threadIdx.x; j < nio; j += blockDim.x) {
      if (io + j >= writer_words || io + j < io || atomicExch(&writer[io + j], ms + 1) != 0)
        atomicOr(&res->unsupported, 1u);
    }
    if (script[off + 1]) break;
    off += 256 + 512 * (size_t)script[off + 6] + STAGE_WORDS * ((size_t)ns + 2);
    ++pid;
  }
}

// The words below res->rio that no partition writes (inputs), any order.
__global__ void plan_unwritten_kernel(const uint32_t *writer, uint32_t writer_words,
                                      uint32_t *list, uint32_t cap, PlanResult *res) {
  for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < res->rio && w < writer_words;
       w += gridDim.x * blockDim.x)
    if (!writer[w]) {
      const uint32_t k = atomicAdd(&res->n_unwritten, 1u);
      if (k < cap) list[k] = w;
    }
}

__global__ void plan_count_kernel(const size_t *blocks_start, const uint32_t *script,
                                  uint32_t *counts, unsigned entries) {
  const unsigned e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= entries) return;
  size_t off = blocks_start[e];
  uint32_t n = 0, sram = 0;
  for (;;) {
    const uint32_t ns = script[off];
    if (!ns) break;
    ++n;
    sram |= script[off + 4] != 0;
    if (script[off + 1]) break;
    off += 256 + 512 * (size_t)script[off + 6] + STAGE_WORDS * ((size_t)ns + 2);
  }
  counts[e] = n | (sram << 31);
}

// ------------------------------------------------------------------ executor

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

static __device__ unsigned long long g_plan_count[BAR_SLOTS], g_plan_hint[BAR_SLOTS];

__device__ __forceinline__ uint32_t plan_smem(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ bool plan_mbar_wait(uint64_t *bar, uint32_t parity) {
  uint32_t done = 0;
  const uint64_t t0 = clock64();
  for (;;) {
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(plan_smem(bar)), "r"(parity)
        : "memory");
    if (done) return true;
    if ((uint64_t)(clock64() - t0) > DEFAULT_BARRIER_TIMEOUT) return false;
  }
}

// The same for words other CTAs of the cluster sent.
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

// Gates of an item, one level per CTA barrier; ends with one.  A thread's
// first gate of a level is loaded before the barrier that opens the level.
__device__ __forceinline__ void plan_gates(const uint32_t *B, uint8_t *slots, uint32_t ngr,
                                           bool isx) {
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
      uint32_t r = a & b & 1u;
      if (isx) r |= (a | b) & (a << 1 | a) & (b << 1 | b) & 2u;
      dst[g] = (uint8_t)r;
      g += EB;
      if (g < g1) e = gates[g];
    }
    g = g1 + threadIdx.x;
    g1 = g2;
    if (g < g1) e = gates[g];
    __syncthreads();
  }
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
// every CTA is done with the loads of cycle c - 3.
//
// Hint.  With many CTAs the polls of those that wait slow down the words the
// others publish, so above PLAN_HINT_ITEMS items a stage a CTA first waits
// (one thread, relaxed, no fence: the words' own numbers decide) until all but
// hint_slack - 1 of the items of the stages before are done.  2M-gate SoC,
// 128 items a stage, per major stage: 4.76 us without, 4.33 / 4.21 / 4.14
// with slack 1 / 4 / 16; 48 items: 2.50 us without, 2.72 with, so those run
// without.  A grid barrier with a release fence instead took 4.39 and 3.33 us.
template <bool X>
__global__ void __launch_bounds__(EB, 1) plan_flow_kernel(const __grid_constant__ PlanParams P) {
  extern __shared__ __align__(128) uint8_t dyn[];
  __shared__ uint64_t bar[2];
  uint32_t *const buf0 = reinterpret_cast<uint32_t *>(dyn);
  uint8_t *const slots = dyn + 4 * (size_t)P.nbuf * P.blob_cap;
  uint2 *const words = reinterpret_cast<uint2 *>(slots + P.slot_bytes);
  uint2 *const old0 = words + P.gw_cap;  // [2][256]
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
        uint2 *const old = old0 + 256 * (n_run & 1u);
        // the blob of this item (copied while the last one ran)
        bool ok = plan_mbar_wait(&bar[F.buf_of(n_run)], F.par_of(n_run));
        if (!opened && t == 0 && c >= 3) {
          const unsigned long long target = (unsigned long long)P.active * (c - 2);
          const uint64_t t0 = clock64();
          for (;;) {
            unsigned long long v;
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];"
                         : "=l"(v)
                         : "l"(&g_plan_count[P.slot])
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
        // ---- state words, and the old words of writeouts that may keep them
        // (this CTA wrote those)
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
          const uint32_t j = EB - 1 - t;
          if (j < nw && B[B[PH_OKEEP] + j])
            old[j] = make_uint2(ldcg(in + io + j), isx ? ldcg(in + (size_t)P.xoff + io + j) : 0u);
        }
        // a wait that ran out ends the launch with its status set
        if (__syncthreads_or(!ok)) {
          if (t == 0) atomicCAS(&g_status[P.slot], 0, JQ_ERR_BARRIER_TIMEOUT);
          if (t == PT) F.drain(n_run);
          return;
        }
        if (!opened && t == 0 && c)  // done with the loads of cycle c - 1
          asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(&g_plan_count[P.slot])
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
        plan_gates(B, slots, ngr, isx);
        plan_srams(P, B, slots, isx);
        // ---- commit: a warp per writeout word
        {
          const uint32_t *com = B + B[PH_OCOM], *kp = B + B[PH_OKEEP];
          for (uint32_t j = warp; j < nw; j += EB / 32) {
            const PlanWord w = plan_word(com, slots, j, isx);
            if (lane == 0) {
              const uint2 ow = kp[j] ? old[j] : make_uint2(0, 0);
              const size_t o = (size_t)io + j;
              const size_t at = (size_t)((c + 1) & 3) * P.rio + o;
              const uint32_t n = (uint32_t)(c + 1);
              const uint32_t nv = (ow.x & ~w.cp) | (w.v & w.cp);
              if (X) {
                // a partition without X leaves the snapshot's host-filled X word
                const uint32_t nx = isx ? (ow.y & ~w.cp & ~w.cx) | (w.x & w.cp & ~w.cx) | w.cx
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
template <bool X>
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
        plan_gates(B, slots, ngr, isx);
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
  // others' bounded waits end too)
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

}  // namespace jqk
