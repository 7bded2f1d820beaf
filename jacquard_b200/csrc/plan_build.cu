// Build of the gate-list plan (plan_build.cuh).
#include "plan_build.cuh"

#include <algorithm>
#include <exception>

namespace jqk {

constexpr int PB = 1024;  // threads of the build kernel

struct PlanBuildParams {
  const uint32_t *script;
  const unsigned long long *part_off;  // script word offset of each partition
  const uint32_t *items;               // per item: partition, sub | nsub << 16
  const uint32_t *writer;              // per state word: major stage + 1 that writes it, or 0
  uint32_t read_end;                   // words below it are values (X words lie above)
  uint32_t mode;                       // PlanMode
  uint32_t pair_gates;                 // gates a level up to which levels go in pairs
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
  uint32_t top[PLAN_MAX_NS];  // lowest position of a stage read from outside, below 4096
  uint32_t lev[PLAN_MAX_LEVELS], lev_base[PLAN_MAX_LEVELS];
  uint32_t warp_sum[32];
  int bad;
  uint32_t max_lev, n_gates, pair;
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
// [nio * sub / nsub, nio * (sub + 1) / nsub); of a partition with SRAMs the
// last item has the ports, the duplicate and the SRAM slots, the others share
// the hooked slots (flag bit 2 when one of them reads an SRAM's output).  The
// result's `unsupported` flag is set for what the plan does not
// represent -- a permutation that reads a writeout slot an earlier partition
// left (the per-block arrays of the script kernel), X words read as values, or
// sizes past the limits above; the kernels below find the rest -- and the
// script then runs in its own form.
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
  bool bad = false;
  // another item found the script to be one without a plan
  auto given_up = [&]() {
    return __syncthreads_or(t == 0 && (*(volatile uint32_t *)&P.res->unsupported & 1u));
  };
  if (given_up()) return;
  const uint32_t *gr = m + 256, *ch = gr + 512 * (size_t)R;
  const uint32_t hooked = nio - nsr - ndup;  // slots below are hooked
  uint32_t j0 = nio * sub / nsub, j1 = nio * (sub + 1) / nsub;
  uint32_t ports = nsr;  // SRAM ports of this item: of a split partition's last item
  if (nsr && nsub > 1) {
    const bool last = sub + 1 == nsub;
    j0 = last ? hooked : hooked * sub / (nsub - 1);
    j1 = last ? nio : hooked * (sub + 1) / (nsub - 1);
    ports = last ? nsr : 0;
  }
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
  // an item without the ports cannot read what they read
  bool no_port = false;
  for (uint32_t j = hooked + ndup + t; j < nio; j += PB) no_port |= !ports && ps.wneed[j] != 0;
  if (__syncthreads_or(no_port)) {
    if (t == 0) atomicOr(&P.res->unsupported, 4u);
    return;
  }
  plan_load_chunk(ps.chunk, ch + STAGE_WORDS * (size_t)ns);
  for (uint32_t q = t; q < (nsr * 4 + ndup) * 32; q += PB) {
    bool use;
    if (q < nsr * 128) {
      use = ports && (q & 127u) < 96u;
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
  if (__syncthreads_or(bad)) {
    if (t == 0) atomicOr(&P.res->unsupported, 1u);
    return;
  }
  // ---- liveness, last stage to first (see jq_plain_depth_kernel; an
  // ob-forced b input is not needed at any level)
  for (int ci = (int)ns - 1; ci >= 0; --ci) {
    plan_load_chunk(ps.chunk, ch + STAGE_WORDS * (size_t)ci);
    if (t < 256) ps.ext[t] = ps.need[t];
    if (t == 0) ps.top[ci] = 8191;
    __syncthreads();
    for (uint32_t j = t; j < hooked; j += PB) {
      const uint32_t hw = m[128 + j / 2], h = (j & 1) ? hw >> 16 : hw & 0xffffu;
      if ((h >> 8) == (uint32_t)ci && ps.wneed[j]) atomicOr(&ps.ext[h & 255u], ps.wneed[j]);
    }
    __syncthreads();
    // the shallowest tree level with a position read from outside: the levels
    // above it have nothing live (a flat stage has only level 1)
    if (t < 128 && ps.ext[t]) atomicMin(&ps.top[ci], 32 * t + __ffs(ps.ext[t]) - 1);
    __syncthreads();
    uint32_t M0 = 4096;
    while (M0 > 1 && ps.top[ci] < M0) M0 >>= 1;
    for (uint32_t c = t; c < M0; c += PB) ps.lv[c] = 0;
    for (uint32_t M = M0; M <= 4096; M <<= 1) {
      for (uint32_t c = M + t; c < 2 * M; c += PB) {
        uint8_t l = (uint8_t)((ps.ext[c >> 5] >> (c & 31)) & 1u);
        if (M > M0) {
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
      if (hit && w >= P.read_end) bad = true;
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
  if (__syncthreads_or(bad)) {
    if (t == 0) atomicOr(&P.res->unsupported, 1u);
    return;
  }
  if (given_up()) return;
  // ---- forward over the stages: reference of every live position; with
  // `gates` the gates are written, else counted per level
  auto forward = [&](uint32_t *gates, uint32_t gate0, bool pair) {
    uint32_t *prev = ps.ref_a, *cur = ps.ref_b;
    for (uint32_t ci = 0; ci < ns; ++ci) {
      plan_load_chunk(ps.chunk, ch + STAGE_WORDS * (size_t)ci);
      auto place = [&](uint32_t p, uint32_t a, uint32_t b) {
        uint32_t r, ra, rb;
        if (plan_and(a, b, plan_flag(ps.chunk, p, 0), plan_flag(ps.chunk, p, 1),
                     plan_flag(ps.chunk, p, 2), r, ra, rb)) {
          const uint32_t l = r < PLAN_MAX_LEVELS ? r : PLAN_MAX_LEVELS - 1;
          const uint32_t ph = pair && gates ? (l + 1) / 2 : l;  // its phase
          const uint32_t k = atomicAdd(&ps.lev[ph], 1u);
          if (gates) {
            const uint32_t g = ps.lev_base[ph] + k;
            if (!pair) {
              gates[g] = (ra & 0xffffu) | (rb << 16);
            } else {
              // an operand of an even level: a gate of the odd level before it
              // by its own operands, anything else as (it AND 1)
              auto half = [&](uint32_t o) -> uint32_t {
                if (!(l & 1) && (o >> 16) == l - 1)
                  return gates[2 * (((o >> 1) & 0x7fffu) - gate0)] | ((o & 1u) << 30);
                return (o & 0x7fffu) | (1u << 15);
              };
              const bool odd = l & 1;
              const uint32_t x = odd ? (ra & 0x7fffu) | ((rb & 0x7fffu) << 15) : half(ra);
              const uint32_t y = odd ? 1u | (1u << 15) : half(rb);
              gates[2 * g] = x;
              gates[2 * g + 1] = y;
            }
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
      for (uint32_t L = 2048; L && 2 * L > ps.top[ci]; L >>= 1) {
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
  forward(nullptr, 0, false);
  if (t == 0) {
    uint32_t n = 0, top = 0;
    for (uint32_t l = 1; l < PLAN_MAX_LEVELS; ++l) {
      n += ps.lev[l];
      if (ps.lev[l]) top = l;
    }
    ps.n_gates = n;
    if (ps.lev[PLAN_MAX_LEVELS - 1]) ps.bad = 1;  // deeper levels share the last count
    // pairs of levels where levels are small
    ps.pair = n <= (uint64_t)P.pair_gates * top &&
              1 + n_gr + n + 32 * ports <= PLAN_MAX_SLOTS / 2;
    if (top) atomicMax(&P.res->max_level, (n + top - 1) / top);
    if (!ps.pair) atomicOr(&P.res->unpaired, 1u);
    if (ps.pair) {
      top = (top + 1) / 2;
      for (uint32_t l = 1; l <= top; ++l) ps.lev[l] = ps.lev[2 * l - 1] + ps.lev[2 * l];
    }
    ps.max_lev = top;
    n = 0;
    for (uint32_t l = 1; l <= top; ++l) {
      ps.lev_base[l] = n;
      n += ps.lev[l];
    }
  }
  __syncthreads();
  const bool pair = ps.pair;
  const uint32_t n_gates = ps.n_gates, n_lev = ps.max_lev, nw = j1 - j0;
  const uint32_t gate0 = 1 + n_gr, sr_slot = gate0 + n_gates, n_slots = sr_slot + 32 * ports;
  auto al = [](uint32_t w) { return (w + 3u) & ~3u; };
  const uint32_t o_gw = PH_SIZE, o_exp = o_gw + (P.mode == PLAN_WORDS ? al(n_gw) : 0u), o_lev = o_exp + al(n_gr),
                 o_gate = o_lev + al(n_lev),
                 o_sram = o_gate + al(pair ? 2 * n_gates : n_gates),
                 o_com = o_sram + 96 * ports, o_keep = o_com + 32 * nw, words = o_keep + al(nw);
  if (n_slots > PLAN_MAX_SLOTS) bad = true;
  if (__syncthreads_or(bad || ps.bad)) {
    if (t == 0) atomicOr(&P.res->unsupported, 1u);
    return;
  }
  if (t == 0) {
    ps.off = atomicAdd(&P.res->used, (unsigned long long)words);
    if (ps.off + words > P.blob_cap) {
      ps.bad = 1;
      atomicOr(&P.res->unsupported, 8u);
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
    while (n2 < n_gw && P.mode == PLAN_WORDS) n2 <<= 1;
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
    if (t < 256 && P.mode == PLAN_WORDS) walk([&](uint32_t e, uint32_t w, uint32_t) { key[e] = w; });
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
    for (uint32_t i = t; i < n_gw && P.mode == PLAN_WORDS; i += PB) {
      B[o_gw + i] = key[i];
      inv[idx[i]] = (uint16_t)i;
    }
    __syncthreads();
    if (t < 256) {
      uint32_t s = bit0;
      if (P.mode == PLAN_SIGNALS)  // staged << 31 | word * 32 + bit
        walk([&](uint32_t, uint32_t w, uint32_t k) {
          const uint32_t i = w & (PLAN_DIRECT - 1);
          if (i >= PLAN_DIRECT / 32) atomicOr(&P.res->unsupported, 2u);
          B[o_exp + s++] = (w & 0x80000000u) | (32 * i + k);
        });
      else if (P.mode == PLAN_MIRROR)  // word << 6 | staged << 5 | bit
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
  forward(B + o_gate, gate0, pair);
  for (uint32_t l = t; l < n_lev; l += PB) B[o_lev + l] = ps.lev_base[1 + l] + ps.lev[1 + l];
  // ---- SRAM ports, then the commit: references of the staged words and of
  // each own writeout bit and its clock enable
  plan_load_chunk(ps.chunk, ch + STAGE_WORDS * (size_t)ns);
  auto staged = [&](uint32_t q) -> uint32_t {
    const uint32_t inv = plan_flag(ps.chunk, q, 0);
    return plan_flag(ps.chunk, q, 1) ? inv : ps.woref[plan_perm(ps.chunk, q)] ^ inv;
  };
  for (uint32_t i = t; i < 96 * ports; i += PB) B[o_sram + i] = staged(128 * (i / 96) + i % 96);
  // duplicate and SRAM slots get their references too
  for (uint32_t q = t; q < 32 * ndup; q += PB)
    if ((ps.wneed[hooked + (q >> 5)] >> (q & 31)) & 1u)
      ps.woref[32 * hooked + q] = (uint16_t)staged(nsr * 128 + q);
  for (uint32_t q = t; q < 32 * ports; q += PB)
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
    B[PH_NSR] = ports;
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
    B[PH_PART] = pid;
    B[PH_PAIR] = pair;
  }
}

// Partition offsets and major stages of every entry, and the major stage
// that writes each state word (writer, zeroed; two writers of one word make
// the plan unsupported: their order within a block matters; so do partitions
// past the limits of the build and writeout slots without a hook, here, so
// that the build is spared).  srams: (first
// word, SRAMs) of the partitions with SRAMs, any order.
__global__ void plan_list_kernel(const size_t *blocks_start, const uint32_t *script,
                                 const uint32_t *part_base, unsigned entries, unsigned num_blocks,
                                 unsigned long long *part_off, uint32_t *part_ms, uint32_t *writer,
                                 uint32_t writer_words, uint2 *srams, PlanResult *res) {
  const unsigned e = blockIdx.x;
  if (e >= entries) return;
  size_t off = blocks_start[e];
  uint32_t pid = part_base[e];
  const uint32_t ms = e / num_blocks;
  for (;;) {
    const uint32_t ns = script[off];
    if (!ns) break;
    const uint32_t nio = script[off + 2], io = script[off + 3], nsr = script[off + 4],
                   ndup = script[off + 7];
    bool bad = ns > PLAN_MAX_NS || nio > 256 || nsr * 4 + ndup > 256 || nsr + ndup > nio ||
               script[off + 6] > 32;
    if (!bad)
      for (uint32_t j = threadIdx.x; j < nio - nsr - ndup; j += blockDim.x) {
        const uint32_t hw = script[off + 128 + j / 2], h = (j & 1) ? hw >> 16 : hw & 0xffffu;
        bad |= (h >> 8) >= ns;
      }
    if (bad) atomicOr(&res->unsupported, 1u);
    if (threadIdx.x == 0) {
      part_off[pid] = off;
      part_ms[pid] = ms;
      atomicMax(&res->rio, io + nio);
      atomicAdd(&res->stage_words[ms], nio);
      atomicOr(&res->x_use, script[off + 8] ? 2u : 1u);
      if (script[off + 4])
        srams[atomicAdd(&res->n_sram_parts, 1u)] = make_uint2(script[off + 5], script[off + 4]);
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

// The words below res->rio that no partition writes (inputs), any order; and
// the plan unsupported when two partitions share an SRAM (their order within
// a block, or their major stages, decide what they read) or a partition reads
// what its own major stage writes.
__global__ void plan_unwritten_kernel(const uint32_t *writer, uint32_t writer_words,
                                      uint32_t *list, uint32_t cap, const uint2 *srams,
                                      const uint32_t *script, const unsigned long long *part_off,
                                      const uint32_t *part_ms, uint32_t parts, PlanResult *res) {
  for (uint32_t pid = blockIdx.x; pid < parts; pid += gridDim.x) {
    const uint32_t *m = script + part_off[pid];
    const uint32_t ms = part_ms[pid], entries = 256 * m[6];
    bool bad = false;
    for (uint32_t i = threadIdx.x; i < entries; i += blockDim.x) {
      const uint2 im = ldg2(m + 256 + 2 * i);
      const uint32_t w = im.x & 0x7fffffffu;
      bad |= im.y && (im.x >> 31) && w < writer_words && writer[w] > ms;
    }
    if (bad) atomicOr(&res->unsupported, 1u);
  }
  const uint32_t n = res->n_sram_parts;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint2 a = srams[i];
    const unsigned long long a1 = a.x + (unsigned long long)a.y * SRAM_WORDS;
    for (uint32_t j = 0; j < i; ++j) {
      const uint2 b = srams[j];
      if (b.x < a1 && a.x < b.x + (unsigned long long)b.y * SRAM_WORDS)
        atomicOr(&res->unsupported, 1u);
    }
  }
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

namespace {

// Layout of the plan build's workspace (words; the blobs take the rest).
struct PlanLayout {
  size_t part_base, part_ms, part_off, srams, writer, unwritten, items, item_words, item_off, blob;
  PlanLayout(size_t entries, size_t parts, size_t n_items, size_t writer_words) {
    size_t w = (sizeof(PlanResult) / 4 + 3) & ~(size_t)3;
    auto take = [&](size_t n) {
      const size_t at = w;
      w += (n + 3) & ~(size_t)3;
      return at;
    };
    part_base = take(entries);
    part_ms = take(parts);
    part_off = take(2 * parts);
    srams = take(2 * parts);
    writer = take(writer_words);
    unwritten = take(writer_words);
    items = take(2 * n_items);
    item_words = take(n_items);
    item_off = take(2 * n_items);
    blob = w;
  }
};
constexpr size_t PLAN_MIN_PART = 256 + 3 * (size_t)STAGE_WORDS;  // words of the smallest partition
constexpr size_t PLAN_SPARE_ITEMS = 148;  // items of a stage beyond its partitions

}  // namespace

size_t plan_workspace_words(size_t blocks_data_len, size_t num_blocks, size_t nms,
                            size_t state_words) {
  const size_t entries = num_blocks * nms;
  const size_t parts = blocks_data_len / PLAN_MIN_PART + 1;
  return PlanLayout(entries, parts, parts + nms * PLAN_SPARE_ITEMS, state_words).blob +
         blocks_data_len + nms * PLAN_SPARE_ITEMS * 1024 + 4096;
}

size_t plan_workspace_first(size_t blocks_data_len, size_t num_blocks, size_t nms,
                            size_t state_words) {
  const size_t all = plan_workspace_words(blocks_data_len, num_blocks, nms, state_words);
  return all - blocks_data_len / 2;
}

size_t plan_smem_limit(const void *fn) {
  int dev = 0, optin = 0;
  cudaFuncAttributes fa;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
      cudaFuncGetAttributes(&fa, fn) != cudaSuccess || (size_t)optin < fa.sharedSizeBytes)
    return 0;
  return (size_t)optin - fa.sharedSizeBytes;
}

bool plan_smem_allow(const void *fn) {
  const size_t lim = plan_smem_limit(fn);
  return lim && cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lim) ==
                    cudaSuccess;
}

const uint32_t *PlanBuilder::unwritten() const {
  return ws + PlanLayout(num_blocks * nms, parts, 0, state_words).unwritten;
}

int PlanBuilder::scan_lists(bool *ok) {
  *ok = false;
  const size_t entries = num_blocks * nms;
  const PlanLayout l0(entries, 0, 0, 0);
  if (ws_words < l0.blob) return JQ_ERR_INVALID_ARG;
  entry.resize(entries);
  per_stage.assign(nms, 0);
  std::vector<uint32_t> base(entries);
  plan_count_kernel<<<(unsigned)((entries + 255) / 256), 256, 0, st>>>(
      blocks_start, blocks_data, ws + l0.part_base, (unsigned)entries);
  if (cudaGetLastError() != cudaSuccess) return JQ_ERR_LAUNCH;
  if (cudaMemcpyAsync(entry.data(), ws + l0.part_base, entries * 4, cudaMemcpyDeviceToHost, st) !=
          cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return JQ_ERR_CUDA;
  for (size_t ms = 0; ms < nms; ++ms) {
    for (size_t b = 0; b < num_blocks; ++b) {
      base[ms * num_blocks + b] = (uint32_t)(parts + per_stage[ms]);
      per_stage[ms] += entry[ms * num_blocks + b] & 0x7fffffffu;
    }
    parts += per_stage[ms];
    most = per_stage[ms] > most ? per_stage[ms] : most;
  }
  const PlanLayout l1(entries, parts, 0, state_words);
  if (parts == 0 || ws_words < l1.blob) return JQ_OK;
  PlanResult *res = reinterpret_cast<PlanResult *>(ws);
  if (cudaMemsetAsync(res, 0, sizeof(PlanResult), st) != cudaSuccess ||
      cudaMemsetAsync(ws + l1.writer, 0, state_words * 4, st) != cudaSuccess ||
      cudaMemcpyAsync(ws + l1.part_base, base.data(), entries * 4, cudaMemcpyHostToDevice, st) !=
          cudaSuccess)
    return JQ_ERR_CUDA;
  plan_list_kernel<<<(unsigned)entries, 64, 0, st>>>(
      blocks_start, blocks_data, ws + l1.part_base, (unsigned)entries, (unsigned)num_blocks,
      reinterpret_cast<unsigned long long *>(ws + l1.part_off), ws + l1.part_ms, ws + l1.writer,
      (uint32_t)state_words, reinterpret_cast<uint2 *>(ws + l1.srams), res);
  plan_unwritten_kernel<<<256, 256, 0, st>>>(
      ws + l1.writer, (uint32_t)state_words, ws + l1.unwritten, (uint32_t)state_words,
      reinterpret_cast<const uint2 *>(ws + l1.srams), blocks_data,
      reinterpret_cast<const unsigned long long *>(ws + l1.part_off), ws + l1.part_ms,
      (uint32_t)parts, res);
  if (cudaGetLastError() != cudaSuccess) return JQ_ERR_LAUNCH;
  if (cudaMemcpyAsync(&r, res, sizeof r, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return JQ_ERR_CUDA;
  // one X offset for every partition with X, above the value words
  const bool one_xoff =
      !(r.x_use & 2u) || (r.xoff_max == ~r.xoff_inv_max && r.xoff_max > 0 && r.rio <= r.xoff_max);
  *ok = !r.unsupported && one_xoff;
  return JQ_OK;
}

int PlanBuilder::build_items(PlanMode mode, size_t want, size_t round, uint32_t pair_gates,
                             bool *ok) {
  *ok = false;
  const size_t entries = num_blocks * nms;
  std::vector<uint32_t> items;
  widest = 1;
  size_t pid = 0;
  for (size_t ms = 0; ms < nms; ++ms) {
    size_t nsub = per_stage[ms] ? want / per_stage[ms] : 1;
    nsub = nsub < 1 ? 1 : nsub > PLAN_MAX_NSUB ? PLAN_MAX_NSUB : nsub;
    stage_item[ms] = (uint32_t)(items.size() / 2);
    for (size_t b = 0; b < num_blocks; ++b) {
      const uint32_t c = entry[ms * num_blocks + b];
      const uint32_t ks = (c >> 31) && !split_srams ? 1u : (uint32_t)nsub;
      for (uint32_t k = 0; k < (c & 0x7fffffffu); ++k, ++pid)
        for (uint32_t s = 0; s < ks; ++s) {
          items.push_back((uint32_t)pid);
          items.push_back(s | ks << 16);
        }
    }
    const uint32_t n = (uint32_t)(items.size() / 2) - stage_item[ms];
    widest = n > widest ? n : widest;
  }
  const size_t n_items = items.size() / 2;
  for (size_t ms = nms; ms <= 32; ++ms) stage_item[ms] = (uint32_t)n_items;
  const PlanLayout lay(entries, parts, n_items, state_words);
  if (ws_words < lay.blob + 4) return JQ_OK;
  PlanResult *res = reinterpret_cast<PlanResult *>(ws);
  r.unsupported = 0;
  r.used = 0;
  r.max_blob = r.max_slots = r.max_gw = r.max_level = r.unpaired = 0;
  if (cudaMemcpyAsync(res, &r, sizeof r, cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(ws + lay.items, items.data(), items.size() * 4, cudaMemcpyHostToDevice,
                      st) != cudaSuccess)
    return JQ_ERR_CUDA;
  PlanBuildParams B;
  B.script = blocks_data;
  B.part_off = reinterpret_cast<unsigned long long *>(ws + lay.part_off);
  B.items = ws + lay.items;
  B.writer = ws + lay.writer;
  B.read_end = (uint32_t)state_words;
  if ((r.x_use & 2u) && r.xoff_max < state_words) B.read_end = r.xoff_max;
  B.mode = mode;
  B.pair_gates = pair_gates;
  B.blob = ws + lay.blob;
  B.blob_cap = ws_words - lay.blob;
  B.item_off = reinterpret_cast<unsigned long long *>(ws + lay.item_off);
  B.item_words = ws + lay.item_words;
  B.res = res;
  const int smem = (int)sizeof(PlanShared);
  if (cudaFuncSetAttribute(plan_build_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
      cudaSuccess)
    return JQ_ERR_LAUNCH;
  plan_build_kernel<<<(unsigned)n_items, PB, smem, st>>>(B, (uint32_t)n_items);
  if (cudaGetLastError() != cudaSuccess) return JQ_ERR_LAUNCH;
  if (cudaMemcpyAsync(&r, res, sizeof r, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return JQ_ERR_CUDA;
  used_words = lay.blob + (size_t)r.used;
  blob = ws + lay.blob;
  item_off = B.item_off;
  item_words = B.item_words;
  if ((r.unsupported & 4u) && split_srams) {  // once more without splitting those
    split_srams = false;
    return build_items(mode, want, round, pair_gates, ok);
  }
  *ok = !r.unsupported;
  overflow = r.unsupported == 8u;
  if (*ok && round) {
    std::vector<uint32_t> words(n_items), w2(n_items);
    std::vector<unsigned long long> off(n_items), o2(n_items);
    if (cudaMemcpyAsync(words.data(), item_words, n_items * 4, cudaMemcpyDeviceToHost, st) !=
            cudaSuccess ||
        cudaMemcpyAsync(off.data(), item_off, n_items * 8, cudaMemcpyDeviceToHost, st) !=
            cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      return JQ_ERR_CUDA;
    std::vector<uint32_t> idx(n_items);
    for (size_t i = 0; i < n_items; ++i) idx[i] = (uint32_t)i;
    for (size_t ms = 0; ms < nms; ++ms)
      std::stable_sort(idx.begin() + stage_item[ms], idx.begin() + stage_item[ms + 1],
                       [&](uint32_t x, uint32_t y) { return words[x] > words[y]; });
    // the CTA with the largest item of a round takes the smallest of the next
    for (size_t ms = 0; ms < nms; ++ms)
      for (size_t lo = stage_item[ms] + round; lo < stage_item[ms + 1]; lo += 2 * round)
        std::reverse(idx.begin() + lo,
                     idx.begin() + std::min<size_t>(lo + round, stage_item[ms + 1]));
    for (size_t i = 0; i < n_items; ++i) {
      w2[i] = words[idx[i]];
      o2[i] = off[idx[i]];
    }
    if (cudaMemcpyAsync(B.item_words, w2.data(), n_items * 4, cudaMemcpyHostToDevice, st) !=
            cudaSuccess ||
        cudaMemcpyAsync(B.item_off, o2.data(), n_items * 8, cudaMemcpyHostToDevice, st) !=
            cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      return JQ_ERR_CUDA;
  }
  return JQ_OK;
}

// The lists above are the only host allocations: a caller of the C interface
// gets a status when there is no memory for them.
int PlanBuilder::scan(bool *ok) {
  try {
    return scan_lists(ok);
  } catch (const std::exception &) {
    return JQ_ERR_INVALID_ARG;
  }
}

int PlanBuilder::build(PlanMode mode, size_t want, size_t round, uint32_t pair_gates, bool *ok) {
  try {
    return build_items(mode, want, round, pair_gates, ok);
  } catch (const std::exception &) {
    return JQ_ERR_INVALID_ARG;
  }
}

}  // namespace jqk
