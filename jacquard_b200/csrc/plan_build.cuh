// Gate-list plan of a script: what the one-stream executors (plain_plan.cuh)
// and the batched one (batched_plan.cuh) run, built on the device by
// plan_build.cu.
//
// The script's boomerang form (shuffle, 8192 -> 1 AND tree, hooks) costs a
// partition its whole trees, however few of their 8191 positions anything
// reads.  The build resolves an item -- a partition, or a range of its
// writeout slots -- to what its writeouts depend on: the state words (or
// signals) it reads, its live AND gates by logic level (pass-throughs,
// constants and dead positions folded away), its SRAM ports, and per writeout
// bit the references of its value and its clock enable.  A reference is a
// 15-bit slot and an inversion bit; slot 0 is the constant 0.
#pragma once
#include <vector>

#include "sim_common.cuh"

namespace jqk {

constexpr uint32_t PLAN_MAX_NS = 64;     // boomerang stages of a partition
constexpr uint32_t PLAN_MAX_LEVELS = 896;
constexpr uint32_t PLAN_MAX_SLOTS = 32768;
constexpr uint32_t PLAN_DIRECT = 1u << 30;  // state word that no partition writes
constexpr size_t PLAN_MAX_NSUB = 16;

// What an item's blob names its inputs by.
enum PlanMode : uint32_t {
  PLAN_WORDS,    // sorted state words, and (word, bit) per slot
  PLAN_MIRROR,   // (state word, bit) per slot
  PLAN_SIGNALS,  // a signal per slot (batched form)
};
// Gates: one word per gate, its operand references, by logic level; or, in
// items of small levels (PH_PAIR; the caller of the build sets how small), two
// words per gate by pair of levels (a phase).  There each half is an operand
// as the AND of two references x | y << 15 (14-bit slots), inverted by bit 30:
// a gate of an even level names the operands of the odd level before it
// instead of its slot, so a phase needs no barrier inside.

// Item header (words of the item's blob; section offsets in words, 16-byte
// aligned).
enum PlanHdr : uint32_t {
  PH_WORDS, PH_NGW, PH_NGR, PH_NLEV, PH_NW, PH_IO, PH_NSR, PH_SRAM_OFF, PH_ISX, PH_XOFF,
  PH_OGW, PH_OEXP, PH_OLEV, PH_OGATE, PH_OSRAM, PH_OCOM, PH_OKEEP, PH_SRSLOT, PH_PART, PH_PAIR, PH_SIZE = 20
};

// Build result: unsupported flag (bit 0: the plan, bit 1: its mirrored form, bit
// 2: splitting partitions with SRAMs, bit 3: the workspace was too small),
// blob words used, the largest blob, slot count and state-word count of any
// item, the words up to the last written one, X use (bit 0: a partition
// without, bit 1: with X) and its offset (min and ~max), the words each major
// stage writes, and the words below `rio` that no partition writes.
struct PlanResult {
  uint32_t unsupported, x_use;
  unsigned long long used;
  uint32_t max_blob, max_slots, max_gw, rio;
  uint32_t xoff_max, xoff_inv_max, n_unwritten;
  uint32_t max_level;     // most gates per level of any item, on average
  uint32_t unpaired;  // an item lists its gates by level
  uint32_t n_sram_parts;  // partitions with SRAMs
  uint32_t stage_words[32];
};

// Host side of a build: the script's partitions, then one build per choice of
// items, in a caller-owned device workspace.
struct PlanBuilder {
  const size_t *blocks_start;
  const uint32_t *blocks_data;
  size_t num_blocks, nms, state_words;
  uint32_t *ws;
  size_t ws_words;
  cudaStream_t st;
  std::vector<uint32_t> entry;      // partitions per entry, bit 31: one has SRAMs
  std::vector<size_t> per_stage;    // partitions per major stage
  size_t parts = 0, most = 0;       // in all, and of the widest stage
  bool split_srams = true;          // partitions with SRAMs may be split
  PlanResult r;                     // of scan(), then of the last build()
  // of the last build()
  uint32_t stage_item[33];
  uint32_t widest;
  size_t used_words;  // (what it takes, when `overflow`)
  bool overflow = false;  // only the workspace's size stood in its way
  const uint32_t *blob, *item_words;
  const unsigned long long *item_off;

  // Partition lists, writers and unwritten words; *ok false when the script
  // has no plan.
  int scan(bool *ok);
  const uint32_t *unwritten() const;
  // Items: every partition of stage ms split towards want / per_stage[ms]
  // ways.  With `round` (items a stage runs at a time) a stage's items are put
  // by decreasing size, every second round reversed.  Items whose levels
  // average at most pair_gates gates list them by pair of levels.
  int build(PlanMode mode, size_t want, size_t round, uint32_t pair_gates, bool *ok);

  // the work of the two; they throw when host memory runs out
  int scan_lists(bool *ok);
  int build_items(PlanMode mode, size_t want, size_t round, uint32_t pair_gates, bool *ok);
};

// Words of workspace a build of any script of this size fits in.
size_t plan_workspace_words(size_t blocks_data_len, size_t num_blocks, size_t nms,
                            size_t state_words);

// The same with item blobs of at most half of the script.
size_t plan_workspace_first(size_t blocks_data_len, size_t num_blocks, size_t nms,
                            size_t state_words);

// Opt-in shared memory per CTA left for the dynamic part of fn.
size_t plan_smem_limit(const void *fn);
// Lets fn have all of it.  The attribute is the function's, not the launch's:
// set to what one plan needs, a launch of a larger plan by another thread
// would be refused.
bool plan_smem_allow(const void *fn);

// mbarrier wait with a bound of about a second.
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

}  // namespace jqk
