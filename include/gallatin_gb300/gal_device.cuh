// gal_device.cuh — device side of the GB300-native Gallatin-compatible allocator.
//
// Header-inline because device malloc/free run inside the caller's kernels.
// The host side (construction, teardown, stats, state export) is the C ABI in
// include/gallatin_gb300.h; the drop-in C++ API is include/gallatin/allocators/.
//
// Algorithm: the reference allocator (chillenzer/gallatin,
// include/gallatin/allocators/gallatin.cuh and friends), restated so a serial
// trace returns the reference's offsets byte for byte.  Layout and
// synchronisation are this library's own:
//   * all metadata in one device region addressed from one state struct
//     (no pointer chasing through per-structure objects);
//   * blocks, queue entries and pinned slots are 32-bit block ids, not Block*;
//   * the malloc word of a block is 64-bit: (tree << 32) | count, so stale
//     claims can never carry a count into the tree field (the reference packs
//     tree << 20 | count into 32 bits, block.cuh:53);
//   * a block's malloc and free counters share one 32-byte record (one L2
//     sector per block, gal_config.block_layout), so the pinned blocks that
//     different SMs claim from never share a sector; the dense layout (all
//     malloc words, then all free counters) remains selectable;
//   * each segment's count of blocks left carries the segment's class and a
//     set-up generation, so one word tells a reservation whose segment it is
//     and it never has to give back into a later owner's count;
//   * every class lock sits in a 32-byte sector of its own;
//   * every spin-wait is bounded by state::spin_limit and reports through the
//     error word instead of trapping (the reference traps, gallatin.cuh:87), and
//     so is every loop that other threads' changes can send round again;
//   * a vEB remove re-checks the emptied child word after clearing its
//     summary bit, with acquire-release fences ordering each thread's word
//     and summary accesses, closing the race that hides a non-empty word;
//   * a failed contiguous-run search does not roll back bits it never took
//     (the reference's exit rollback, veb.cuh:447);
//   * a multi-segment free resets the segment's tree id before returning its
//     bits, so a concurrent claim never meets a stale id (gallatin.cuh:1283-1302
//     returns the bits first).
#pragma once

#include <stdint.h>

#include "../gallatin_gb300.h"

#ifndef GAL_DEVICE_INLINE
#define GAL_DEVICE_INLINE __device__ __forceinline__
#endif
// cold paths stay out of line (register pressure of the hot path); static so
// the header can be included by several translation units
#define GAL_DEVICE_COLD static __device__ __noinline__

namespace gal {

static constexpr uint32_t NOBLK = 0xFFFFFFFFu;
static constexpr uint64_t FAIL = ~0ULL;
static constexpr uint16_t FREE_TREE = 0xFFFF;
static constexpr uint32_t SLICES_PER_BLOCK = 4096;

// retry caps of the reference (gallatin.cuh:108-112, veb.cuh:59)
static constexpr int SLICE_ATTEMPTS = 500 * 10;
static constexpr int VEB_ATTEMPTS = 15;
static constexpr uint32_t VEB_LOSSES = 1024;  // items of one word lost to other threads before a search goes on
static constexpr int GATHER_RETRIES = 8;
static constexpr int BLOCK_ATTEMPTS = 8;
static constexpr int SEGMENT_ATTEMPTS = 8;
static constexpr int SLOT_PROBE_LIMIT = 30;  // SHARED_BLOCK_COUNTER_CUTOFF

struct veb_shape {
  uint32_t layers;
  uint32_t words;                        // words of one tree, all layers
  uint32_t off[GAL_MAX_VEB_LAYERS];      // word offset of each layer (0 = top)
  uint32_t nwords[GAL_MAX_VEB_LAYERS];
  uint64_t items[GAL_MAX_VEB_LAYERS];    // universe of each layer
};

// Everything a kernel needs; lives in device memory (the object a
// Gallatin<>* points to).  A copy of it, passed by value as a kernel parameter
// or kept in shared, local or constant memory, stands for that object: the
// device calls take either (see resident).
struct state {
  char *memory;
  uint64_t num_segments;
  uint64_t seed;
  uint32_t seg_shift;   // log2 bytes_per_segment
  uint32_t min_shift;   // log2 min_size
  uint32_t bps_shift;   // log2 table blocks per segment
  uint32_t num_trees;
  uint32_t policy;
  int32_t smid_override;
  uint32_t spin_limit;
  uint32_t total_slots;
  uint32_t gather_unlocked_below;  // see gal_config
  uint32_t gather_ahead;           // see gal_config
  uint32_t team_width;             // see gal_config (1..32, a power of two)
  uint32_t use_spares;             // see gal_config.spare_blocks
  uint32_t zero_fill;              // see gal_config.zero_fill
  uint32_t slot_base[GAL_MAX_TREES];
  uint32_t slot_count[GAL_MAX_TREES];
  veb_shape veb;
  uint64_t *seg_tree;            // [veb.words]
  uint64_t *sub_trees;           // [num_trees * veb.words]
  uint16_t *tree_ids;            // [S]
  uint32_t *qc;                  // [S] hand-out position
  uint32_t *qfc;                 // [S] return position
  uint32_t *fqfc;                // [S] finalised return position
  unsigned long long *act;       // [S] generation, class and blocks left (see act_word)
  unsigned long long *mwords;    // per block (tree << 32) | count, every mstride-th word
  uint32_t *fctr;                // per block frees counted, every fstride-th word
  uint32_t mstride;              // 4 with fstride 8: one 32-byte record per block
  uint32_t fstride;              // 1 with fstride 1: dense arrays (gal_config.block_layout)
  uint32_t *queues;              // [S << bps_shift] recycle ring (block ids)
  uint32_t *slots;               // [total_slots] pinned blocks
  uint32_t *spares;              // [total_slots] next block per slot, prepared ahead
                                 // (gal_config.spare_blocks; NOBLK: none)
  uint32_t *locks;               // lock word of tree t at t * LOCK_STRIDE; runs at num_trees
  uint32_t *error;               // GAL_DEV_ERR_* bits
  const state *resident;         // the state in device memory that this is (a copy of)
};

// A field of the state (or of its tree shape), which lives in global memory, on
// the device: constant while a kernel runs, so it is read through the read-only path, whose cached lines
// outlive fences.  Ordinary loads miss L1 after every fence or acquire (345
// cycles each, several in a row on the block-request path).
template <class T>
GAL_DEVICE_INLINE __host__ T cfield(const T &f) {
#ifdef __CUDA_ARCH__
  static_assert(sizeof(T) == 8 || sizeof(T) == 4, "a word or a pointer");
  if constexpr (sizeof(T) == 8) {
    const unsigned long long v = __ldg((const unsigned long long *)&f);
    return (T)v;
  } else {
    return (T)__ldg((const unsigned int *)&f);
  }
#else
  return f;
#endif
}
// cfield reads global memory; a copy of the state elsewhere names the one there.
// (A kernel's parameters lie in a window of the global address space.)
GAL_DEVICE_INLINE const state *resident(const state *s) {
  return __isGlobal(s) && !__isGridConstant(s) ? s : s->resident;
}

// ------------------------------------------------------------------ layout
static constexpr uint32_t BLOCK_RECORD_BYTES = 32;  // block_layout 1: one sector per block
static constexpr uint32_t LOCK_STRIDE = 8;          // u32 words between lock words (32 B)
GAL_DEVICE_INLINE __host__ unsigned long long *mword_ptr(const state *s, uint32_t blk) {
  return cfield(s->mwords) + (uint64_t)blk * cfield(s->mstride);
}
GAL_DEVICE_INLINE __host__ uint32_t *fctr_ptr(const state *s, uint32_t blk) {
  return cfield(s->fctr) + (uint64_t)blk * cfield(s->fstride);
}
// A segment's count word: in the low half the reference's active count (blocks
// left to hand out minus one; -1 when none is left or the segment is free) plus
// ACT_BIAS, so adding or subtracting one never carries into the high half,
// which holds the class that owns the segment (ACT_FREE: none) in its low byte
// and the set-up generation in the rest.  The atomic that reserves a block
// thus also says whose segment it was taken from, with no second word to read.
static constexpr uint32_t NOSEG = 0xFFFFFFFFu;  // no segment
static constexpr uint32_t ACT_BIAS = 0x80000000u;
static constexpr uint32_t ACT_FREE = 0xFFu;
GAL_DEVICE_INLINE __host__ int32_t act_unbias(uint32_t low) { return (int32_t)(low - ACT_BIAS); }
GAL_DEVICE_INLINE __host__ int32_t act_count(unsigned long long w) { return act_unbias((uint32_t)w); }
GAL_DEVICE_INLINE __host__ uint32_t act_class(unsigned long long w) { return (uint32_t)(w >> 32) & 0xFFu; }
GAL_DEVICE_INLINE __host__ uint32_t act_gen(unsigned long long w) { return (uint32_t)(w >> 40); }
GAL_DEVICE_INLINE __host__ unsigned long long act_word(uint32_t gen, uint32_t cls, int32_t count) {
  return ((unsigned long long)((gen << 8) | cls) << 32) | (uint32_t)((uint32_t)count + ACT_BIAS);
}

// ------------------------------------------------------------------ helpers
GAL_DEVICE_INLINE uint32_t lane_id() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%laneid;" : "=r"(r));
  return r;
}
// Mask of the lanes executing here.  Read through volatile asm: the
// __activemask() builtin may be re-evaluated by the compiler at a later,
// divergent use site, which splits a warp team across convergence groups.
GAL_DEVICE_INLINE uint32_t active_lanes() {
  uint32_t m;
  asm volatile("activemask.b32 %0;" : "=r"(m));
  return m;
}
GAL_DEVICE_INLINE uint32_t lanemask_lt() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(r));
  return r;
}
// The lanes this lane may aggregate with: the whole warp (team_width 32, the
// reference's coalesced team) or its aligned group of team_width lanes.
GAL_DEVICE_INLINE uint32_t team_group(const state *s) {
  const uint32_t w = cfield(s->team_width);
  if (w >= 32) return 0xFFFFFFFFu;
  return ((1u << w) - 1u) << (lane_id() & ~(w - 1u));
}
GAL_DEVICE_INLINE uint32_t sm_id() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(r));
  return r;
}
GAL_DEVICE_INLINE uint64_t ld_rlx(const uint64_t *p) {
  uint64_t v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
GAL_DEVICE_INLINE uint32_t ld_rlx(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
GAL_DEVICE_INLINE int32_t ld_rlx(const int32_t *p) {
  return (int32_t)ld_rlx((const uint32_t *)p);
}
GAL_DEVICE_INLINE unsigned long long ld_rlx(const unsigned long long *p) {
  return (unsigned long long)ld_rlx((const uint64_t *)p);
}
GAL_DEVICE_INLINE uint16_t ld_rlx(const uint16_t *p) {
  uint16_t v;
  asm volatile("ld.relaxed.gpu.global.u16 %0, [%1];" : "=h"(v) : "l"(p) : "memory");
  return v;
}
// acquire-release fence at device scope: orders this thread's earlier and
// later memory accesses.  It costs a round trip of its own (some 800 cycles
// with nothing outstanding, as much as an atomic), as __threadfence does.
GAL_DEVICE_INLINE void fence_acq_rel() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
GAL_DEVICE_INLINE uint64_t amo_or(uint64_t *p, uint64_t v) {
  return atomicOr((unsigned long long *)p, (unsigned long long)v);
}
GAL_DEVICE_INLINE uint64_t amo_and(uint64_t *p, uint64_t v) {
  return atomicAnd((unsigned long long *)p, (unsigned long long)v);
}
// ... whose later accesses by this thread stay after them; a set that also stays
// after its earlier ones
GAL_DEVICE_INLINE uint64_t and_acquire(uint64_t *p, uint64_t v) {
  uint64_t r;
  asm volatile("atom.acquire.gpu.global.and.b64 %0, [%1], %2;" : "=l"(r) : "l"(p), "l"(v) : "memory");
  return r;
}
GAL_DEVICE_INLINE uint64_t or_acq_rel(uint64_t *p, uint64_t v) {
  uint64_t r;
  asm volatile("atom.acq_rel.gpu.global.or.b64 %0, [%1], %2;" : "=l"(r) : "l"(p), "l"(v) : "memory");
  return r;
}
// atomicAdd whose later accesses by this thread stay after it
GAL_DEVICE_INLINE unsigned long long add_acquire(unsigned long long *p, unsigned long long v) {
  unsigned long long r;
  asm volatile("atom.acquire.gpu.global.add.u64 %0, [%1], %2;" : "=l"(r) : "l"(p), "l"(v) : "memory");
  return r;
}
GAL_DEVICE_INLINE void st_rlx(unsigned long long *p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
GAL_DEVICE_INLINE void st_rlx(uint32_t *p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
GAL_DEVICE_INLINE void st_rlx(uint16_t *p, uint16_t v) {
  asm volatile("st.relaxed.gpu.global.u16 [%0], %1;" ::"l"(p), "h"(v) : "memory");
}
// a store after everything this thread has done and seen so far ...
GAL_DEVICE_INLINE void st_release(uint32_t *p, uint32_t v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// ... and an exchange that takes all of that over with the value it finds
GAL_DEVICE_INLINE uint32_t exch_acquire(uint32_t *p, uint32_t v) {
  uint32_t r;
  asm volatile("atom.acquire.gpu.global.exch.b32 %0, [%1], %2;" : "=r"(r) : "l"(p), "r"(v) : "memory");
  return r;
}
GAL_DEVICE_INLINE uint16_t cas16(uint16_t *p, uint16_t cmp, uint16_t val) {
  return (uint16_t)atomicCAS((unsigned short *)p, (unsigned short)cmp, (unsigned short)val);
}
GAL_DEVICE_INLINE void set_error(const state *s, uint32_t bits) { atomicOr(cfield(s->error), bits); }
// error word plus the first error's site and two values (error[2..9] as 4 u64:
// site, a, b, taken) for gal_error_info
GAL_DEVICE_COLD void set_error_info(const state *s, uint32_t bits, uint64_t site, uint64_t a,
                                    uint64_t b) {
  atomicOr(cfield(s->error), bits);
  unsigned long long *info = (unsigned long long *)(cfield(s->error) + 2);
  if (atomicCAS(&info[3], 0ull, 1ull) == 0ull) {
    info[0] = site;
    info[1] = a;
    info[2] = b;
    __threadfence();
  }
}
enum : uint64_t {
  SITE_RETURN_BAD_TREE = 1,
  SITE_FREE_OVERFLOW = 2,
  SITE_FREE_OUTSIDE = 3,
  SITE_FREE_FREE_SEGMENT = 4,
  SITE_FREE_RUN_TWICE = 5,
  SITE_REQUEST_LOCK = 6,   // request_block: the class lock stayed taken (a: class, b: spins)
  SITE_REQUEST_RETRY = 7,  // request_block: listed segments kept refusing a block (a: class, b: last segment)
  SITE_RUN_LOCK = 8,       // malloc_segment_run: the run lock stayed taken (a: segments wanted)
  SITE_LISTING = 9,        // settle_listing: the segment kept changing (a: class, b: segment)
};
GAL_DEVICE_INLINE void backoff(uint32_t i) { __nanosleep(i < 8 ? 32u << i : 4096u); }

// ceil(log2(x)) for x > 0, 0 for x == 0 (alloc_utils.cuh:382-398)
GAL_DEVICE_INLINE int ceil_log2(uint64_t x) {
  return 63 - __clzll((long long)x) + (__popcll(x) != 1);
}

// MurmurHash64A (Austin Appleby, public domain) of one 8-byte key
GAL_DEVICE_INLINE uint64_t murmur64a_u64(uint64_t key, uint64_t seed) {
  const uint64_t m = 0xc6a4a7935bd1e995ULL;
  uint64_t h = seed ^ (8ULL * m);
  uint64_t k = key * m;
  k ^= k >> 47;
  k *= m;
  h ^= k;
  h *= m;
  h ^= h >> 47;
  h *= m;
  h ^= h >> 47;
  return h;
}

GAL_DEVICE_INLINE uint64_t bitmask(int n) { return n >= 64 ? ~0ULL : ((1ULL << n) - 1ULL); }
GAL_DEVICE_INLINE uint32_t blocks_in_segment(const state *s, uint32_t tree) {
  return 1u << (cfield(s->bps_shift) - tree);
}
GAL_DEVICE_INLINE uint64_t thread_linear_id() {
  return (uint64_t)(threadIdx.x + blockIdx.x * blockDim.x);  // 32-bit as veb.cuh:948
}

// ------------------------------------------------------------------ vEB
// Word layout of one tree: layer 0 (top) first; bit i of layer l word w is
// item 64*w + i of that layer (veb.cuh:109-526, 528-1228).
struct veb_ref {
  uint64_t *w;
  const veb_shape *sh;
  uint64_t seed;
  GAL_DEVICE_INLINE uint64_t *word(int layer, uint64_t high) const { return w + cfield(sh->off[layer]) + high; }
};

GAL_DEVICE_INLINE int veb_find_next(const veb_ref &v, int layer, uint64_t high, int low) {
  if (high >= cfield(v.sh->items[layer])) return -1;  // layer::find_next, veb.cuh:250-275
  uint64_t b = ld_rlx(v.word(layer, high));
  if (low == -1) return __ffsll((long long)b) - 1;
  return __ffsll((long long)(b & ~bitmask(low + 1))) - 1;
}

GAL_DEVICE_INLINE bool veb_query(const veb_ref &v, uint64_t x) {
  return (ld_rlx(v.word(cfield(v.sh->layers) - 1, x >> 6)) >> (x & 63)) & 1ULL;
}

// Takes a word this thread emptied off the summaries above it.
GAL_DEVICE_COLD void veb_unlist(uint64_t *w, const veb_shape *sh, uint32_t word) {
  const veb_ref v{w, sh, 0};
  int layer = (int)cfield(sh->layers) - 1;
  uint64_t high = word;
  while (layer > 0) {
    uint64_t *child = v.word(layer, high);
    layer -= 1;
    const int low = (int)(high & 63);
    high >>= 6;
    fence_acq_rel();
    const uint64_t old = amo_and(v.word(layer, high), ~(1ULL << low));
    fence_acq_rel();
    if (ld_rlx(child) != 0) {  // an insert raced in: keep the summary bit
      amo_or(v.word(layer, high), 1ULL << low);
      return;
    }
    if (__popcll(old) != 1) return;
  }
}

// veb_tree::remove (veb.cuh:737-755) plus the child re-check.  A remove that
// empties a word clears the word's summary bit, then reads the word again: an
// insert that refilled it meanwhile set the word's bit before the summary's,
// and acquire-release fences on both sides order the two accesses of each
// thread (the insert's set of the summary publishes its set of the word), so
// either the insert's summary set lands after this clear or this re-read sees
// the refilled word.  Without them a clear could land after the insert's set
// while the re-read still saw the empty word, leaving a non-empty word behind
// a clear summary bit, where top-down searches never find its items.
// `left` receives the other items the bottom word held.
// ACQUIRE: with all that the item's insert came after (see veb_insert).
template <bool ACQUIRE = false>
GAL_DEVICE_INLINE bool veb_remove(const veb_ref &v, uint64_t x, uint64_t &left) {
  const int layer = (int)cfield(v.sh->layers) - 1;
  const uint64_t high = x >> 6;
  const int low = (int)(x & 63);
  const uint64_t keep = ~(1ULL << low);
  const uint64_t old = ACQUIRE ? and_acquire(v.word(layer, high), keep) : amo_and(v.word(layer, high), keep);
  left = old & ~(1ULL << low);
  if (!(old & (1ULL << low))) return false;
  if (left == 0) veb_unlist(v.w, v.sh, (uint32_t)high);
  return true;
}

template <bool ACQUIRE = false>
GAL_DEVICE_INLINE bool veb_remove(const veb_ref &v, uint64_t x) {
  uint64_t left;
  return veb_remove<ACQUIRE>(v, x, left);
}

// Lists a bottom word this thread found empty in the summaries above it.
GAL_DEVICE_COLD void veb_list_above(uint64_t *w, const veb_shape *sh, uint32_t word) {
  const veb_ref v{w, sh, 0};
  uint64_t high = word, old = 0;
  for (int layer = (int)cfield(sh->layers) - 2; layer >= 0 && old == 0; layer--) {
    fence_acq_rel();
    old = amo_or(v.word(layer, high >> 6), 1ULL << (high & 63));
    high >>= 6;
  }
}

// veb_tree::insert_force_update (veb.cuh:775-798); the fence orders each
// word's set before its summary's (see veb_remove).  ORDERED: the item is there after
// all that this thread has done and seen, and before all that it does next.
template <bool ORDERED = false>
GAL_DEVICE_INLINE bool veb_insert(const veb_ref &v, uint64_t x) {
  const int layer = (int)cfield(v.sh->layers) - 1;
  const uint64_t high = x >> 6;
  const uint64_t bit = 1ULL << (x & 63);
  const uint64_t old = ORDERED ? or_acq_rel(v.word(layer, high), bit) : amo_or(v.word(layer, high), bit);
  if (old == 0) veb_list_above(v.w, v.sh, (uint32_t)high);
  return !((old >> (x & 63)) & 1ULL);
}

// veb_tree::successor_thorough (veb.cuh:878-916): smallest item > q
GAL_DEVICE_COLD uint64_t veb_successor(const veb_ref &v, uint64_t q) {
  const int bottom = (int)cfield(v.sh->layers) - 1;
  uint64_t high = q >> 6;
  int low = (int)(q & 63);
  int layer = bottom;
  for (;;) {
    for (;;) {
      if (veb_find_next(v, layer, high, low) != -1) break;
      if (layer == 0) return FAIL;
      layer -= 1;
      low = (int)(high & 63);
      high >>= 6;
    }
    while (layer != bottom) {
      low = veb_find_next(v, layer, high, low);
      if (low == -1) break;
      layer += 1;
      high = (high << 6) + (uint64_t)low;
      low = -1;
    }
    low = veb_find_next(v, layer, high, low);
    // only a bottom-layer hit is an item; a summary word refilled by a racing
    // insert is searched again from the top of the loop
    if (low != -1 && layer == bottom) return (high << 6) + (uint64_t)low;
  }
}

// veb_tree::lock_offset (veb.cuh:918-937)
GAL_DEVICE_INLINE uint64_t veb_lock_offset(const veb_ref &v, uint64_t start) {
  if (veb_query(v, start) && veb_remove(v, start)) return start;
  for (;;) {
    start = veb_successor(v, start);
    if (start == FAIL) return FAIL;
    if (veb_remove(v, start)) return start;
  }
}

// Trees of up to 64 bottom words (4,096 segments) are searched top-down from
// the one summary word above them: `top` has the bottom words that are not
// empty (a one-layer tree is its only bottom word).  Bottom word 0 is loaded
// along with it, and segments are taken lowest first, so a search costs one or
// two dependent loads (an L2 load of a word another SM has just changed takes
// ~700 cycles); climbing from a start word and coming down again for every
// start tried took eight to ten of them.
struct veb_low {
  uint64_t top, word0;
};
GAL_DEVICE_INLINE bool veb_shallow(const veb_ref &v) {
  return cfield(v.sh->nwords[cfield(v.sh->layers) - 1]) <= 64;
}
GAL_DEVICE_INLINE uint64_t *veb_bottom(const veb_ref &v) {
  return v.w + cfield(v.sh->off[cfield(v.sh->layers) - 1]);
}
GAL_DEVICE_INLINE veb_low veb_load_low(const veb_ref &v, const uint64_t *bottom) {
  const uint32_t layers = cfield(v.sh->layers);
  veb_low l;
  l.top = layers > 1 ? ld_rlx(v.w + cfield(v.sh->off[layers - 2])) : 1ull;
  l.word0 = ld_rlx(bottom);
  return l;
}
GAL_DEVICE_INLINE uint64_t veb_low_word(const veb_low &l, const uint64_t *bottom, uint64_t high) {
  return high ? ld_rlx(bottom + high) : l.word0;
}

// veb_tree::malloc_first (veb.cuh:979-991): takes the smallest item.  Threads
// that lose it to one another would all go for the next smallest together, one
// winner per round trip; each loser goes on from the word as its own attempt
// left it, at a place of its own, so k contenders are served in a few round
// trips.  One thread alone never loses and always gets the smallest.
// `l` is the start of the search, loaded by the caller.
GAL_DEVICE_COLD uint64_t veb_malloc_first_deep(uint64_t *w, const veb_shape *sh) {
  const veb_ref v{w, sh, 0};
  for (int a = 0; a < VEB_ATTEMPTS; a++) {
    uint64_t o = veb_lock_offset(v, 0);
    if (o != FAIL) return o;
  }
  return FAIL;
}
GAL_DEVICE_INLINE uint64_t veb_malloc_first(const veb_ref &v, veb_low l) {
  if (!veb_shallow(v)) return veb_malloc_first_deep(v.w, v.sh);
  uint64_t *bottom = veb_bottom(v);
  const uint32_t spread = (uint32_t)(thread_linear_id() * 0x9E3779B1u) >> 26;
  for (int a = 0; a < VEB_ATTEMPTS; a++, l = veb_load_low(v, bottom)) {
    for (uint64_t top = l.top; top; top &= top - 1ull) {
      const uint64_t high = (uint64_t)(__ffsll((long long)top) - 1);
      uint64_t word = veb_low_word(l, bottom, high);
      for (uint32_t turn = 0, lost = 0; word && lost < VEB_LOSSES; turn = spread, lost++) {
        const uint64_t turned = (word >> turn) | (turn ? word << (64u - turn) : 0ull);
        const uint64_t low = ((uint64_t)(__ffsll((long long)turned) - 1) + turn) & 63u;
        if (veb_remove(v, (high << 6) + low, word)) return (high << 6) + low;
      }
    }
  }
  return FAIL;
}

GAL_DEVICE_COLD uint64_t veb_find_random_deep(uint64_t *w, const veb_shape *sh, uint64_t seed, uint64_t tid) {
  const veb_ref v{w, sh, seed};
  const uint64_t U = cfield(sh->items[cfield(sh->layers) - 1]);
  const uint64_t h1 = murmur64a_u64(tid, seed);
  const uint64_t h2 = murmur64a_u64(tid, h1);
  uint64_t empty_from = U;  // no item in [empty_from, U)
  for (uint64_t a = 0; a < (uint64_t)VEB_ATTEMPTS; a++) {
    uint64_t start = (h1 + a * h2) % U;
    if (start >= empty_from) continue;
    if (veb_query(v, start)) return start;
    uint64_t idx = veb_successor(v, start);
    if (idx != FAIL) return idx;
    empty_from = start;
  }
  return veb_successor(v, 0);
}

// veb_tree::find_random_valid_index (veb.cuh:946-977): of 15 hashed starts the
// first with a listed item at or above it gives the smallest such item; if none
// has one, the smallest item above 0.  A start has one exactly when it does not
// exceed the largest listed item, so the starts are tried in registers once
// that is known, and a tree that lists one item other than 0 needs none (the
// hashes took 1,200 cycles).  A deeper tree is searched from each start; one
// that found nothing shows that no item lies in [start, U), and later starts at
// or above the lowest such start are skipped.
GAL_DEVICE_INLINE uint64_t veb_find_random(const veb_ref &v, uint64_t tid) {
  const uint64_t U = cfield(v.sh->items[cfield(v.sh->layers) - 1]);
  if (!veb_shallow(v)) return veb_find_random_deep(v.w, v.sh, v.seed, tid);
  const uint64_t *bottom = veb_bottom(v);
  const veb_low l = veb_load_low(v, bottom);
  uint64_t top = l.top, last = 0, last_word = 0;  // the highest word with an item
  while (top) {
    last = 63u - (uint64_t)__clzll((long long)top);
    last_word = veb_low_word(l, bottom, last);
    if (last_word) break;
    top &= ~(1ull << last);  // emptied since its summary was read
  }
  if (!last_word) return FAIL;
  const uint64_t largest = (last << 6) + 63u - (uint64_t)__clzll((long long)last_word);
  uint64_t start = 1;
  if ((top & (top - 1ull)) != 0 || (last_word & (last_word - 1ull)) != 0 || largest == 0) {
    const uint64_t h1 = murmur64a_u64(tid, v.seed);
    const uint64_t h2 = murmur64a_u64(tid, h1);
    if ((U & (U - 1ull)) == 0) {  // only the low bits of the starts count
      const uint32_t mask = (uint32_t)U - 1u;
      uint32_t at = (uint32_t)h1;
#pragma unroll 5
      for (int a = 0; a < VEB_ATTEMPTS; a++, at += (uint32_t)h2)
        if ((at & mask) <= largest) {
          start = at & mask;
          break;
        }
    } else {
      for (uint64_t a = 0; a < (uint64_t)VEB_ATTEMPTS; a++) {
        const uint64_t at = (h1 + a * h2) % U;
        if (at <= largest) {
          start = at;
          break;
        }
      }
    }
    if (start > largest) return FAIL;  // item 0 alone, and no start found it
  }
  // the smallest item at or above start
  uint64_t high = start >> 6;
  uint64_t word = (high == last ? last_word : veb_low_word(l, bottom, high)) & ~bitmask((int)(start & 63u));
  while (!word) {  // reaches `last` at the latest, whose remembered word holds an item above start
    const uint64_t above = top & ~bitmask((int)high + 1);
    high = above ? (uint64_t)(__ffsll((long long)above) - 1) : last;
    word = high >= last ? last_word : veb_low_word(l, bottom, high);
  }
  return (high << 6) + (uint64_t)(__ffsll((long long)word) - 1);
}

// Any listed item, a different one for different `spread`s (FAIL: none): for a
// thread that another has beaten to the item the rule above gives, which
// threads that search together mostly agree on.
GAL_DEVICE_INLINE uint64_t veb_find_any(const veb_ref &v, uint32_t spread) {
  if (!veb_shallow(v)) return veb_find_random(v, spread);
  const uint64_t *bottom = veb_bottom(v);
  const veb_low l = veb_load_low(v, bottom);
  uint64_t top = l.top;
  for (uint32_t k = top ? spread % (uint32_t)__popcll(top) : 0; k; k--) top = top & (top - 1ull);
  for (; top; top &= top - 1ull) {
    const uint64_t high = (uint64_t)(__ffsll((long long)top) - 1);
    uint64_t word = veb_low_word(l, bottom, high);
    if (!word) continue;
    for (uint32_t k = (spread >> 8) % (uint32_t)__popcll(word); k; k--) word &= word - 1ull;
    return (high << 6) + (uint64_t)(__ffsll((long long)word) - 1);
  }
  return FAIL;
}

// veb_tree::find_first_valid_index (veb.cuh:940-944): smallest listed id
GAL_DEVICE_INLINE uint64_t veb_find_first(const veb_ref &v) {
  if (veb_shallow(v)) {
    const uint64_t *bottom = veb_bottom(v);
    const veb_low l = veb_load_low(v, bottom);
    for (uint64_t top = l.top; top; top &= top - 1ull) {
      const uint64_t high = (uint64_t)(__ffsll((long long)top) - 1);
      const uint64_t word = veb_low_word(l, bottom, high);
      if (word) return (high << 6) + (uint64_t)(__ffsll((long long)word) - 1);
    }
    return FAIL;
  }
  if (veb_query(v, 0)) return 0;
  return veb_successor(v, 0);
}

GAL_DEVICE_INLINE int cfc64(uint64_t b) {  // alloc_utils.cuh:440-453
  int p = __popcll(b);
  if (p == 0 || p == 64) return p;
  return __ffsll((long long)~b) - 1;
}

GAL_DEVICE_INLINE void veb_rollback(const veb_ref &v, uint64_t start_block, uint64_t nbits) {
  const int bottom = (int)cfield(v.sh->layers) - 1;  // layer::rollback, veb.cuh:305-321
  while (nbits > 64) {
    amo_or(v.word(bottom, start_block), ~0ULL);
    nbits -= 64;
    start_block++;
  }
  amo_or(v.word(bottom, start_block), bitmask((int)nbits));
}

// layer::gather_multiple (veb.cuh:323-452) on the bottom layer: claims a run
// ending in the trailing ones of a word, scanning words from the top down.
GAL_DEVICE_COLD uint64_t veb_gather_run(const veb_ref &v, uint64_t needed) {
  const int bottom = (int)cfield(v.sh->layers) - 1;
  uint64_t sb = cfield(v.sh->nwords[bottom]) - 1;
  // every pass either moves down a word or retries one that changed under it;
  // bound the retries so heavy interference ends in a clean failure
  uint64_t budget = 8ull * cfield(v.sh->nwords[bottom]) + 1024;
  while (sb != 0) {
    if (budget-- == 0) return FAIL;
    uint64_t n = needed;
    uint64_t *w = v.word(bottom, sb);
    int c = cfc64(ld_rlx(w));
    if (c == 0) {
      sb -= 1;
      continue;
    }
    if ((uint64_t)c >= n) {
      uint64_t acq = bitmask((int)n) << (c - (int)n);
      uint64_t got = amo_and(w, ~acq);
      if ((uint64_t)__popcll(got & acq) == n) return sb * 64 + (uint64_t)(c - (int)n);
      amo_or(w, acq & got);
      continue;
    }
    uint64_t got = amo_and(w, ~bitmask(c));
    if (__popcll(got & bitmask(c)) != c) {
      amo_or(w, got & bitmask(c));
      continue;
    }
    n -= (uint64_t)c;
    bool ok = true;
    while (n > 64) {
      if (sb == 0) {  // run would leave the arena (the reference indexes word -1):
        veb_rollback(v, sb, needed - n);  // give back words 0 .. the first one
        return FAIL;
      }
      sb--;
      uint64_t full = amo_and(v.word(bottom, sb), 0ULL);
      if (__popcll(full) != 64) {
        amo_or(v.word(bottom, sb), full);
        veb_rollback(v, sb + 1, needed - n);
        ok = false;
        break;
      }
      n -= 64;
    }
    if (!ok) continue;
    if (sb == 0) {  // the same: the words taken start at word 0
      veb_rollback(v, sb, needed - n);
      return FAIL;
    }
    sb--;
    uint64_t fmask = bitmask((int)n) << (64 - n);
    uint64_t fb = amo_and(v.word(bottom, sb), ~fmask);
    if ((uint64_t)__popcll(fb & fmask) == n) return sb * 64 + 64 - n;
    amo_or(v.word(bottom, sb), fmask & fb);
    veb_rollback(v, sb + 1, needed - n);
  }
  return FAIL;
}

// A run of n segments (at most 64) for a thread that met another one searching:
// taken from the trailing ones of one word with a compare-and-swap, as
// veb_gather_run takes it but from any of the topmost RUN_CHOICES words that
// have room, each thread starting at one of its own.  Nothing is held by a
// failed try, so the threads need no lock among themselves.  FAIL: no single
// word has room (a run across words needs the locked search).
static constexpr int RUN_CHOICES = 16;
GAL_DEVICE_COLD uint64_t veb_gather_in_word(const veb_ref &v, uint64_t n) {
  const int bottom = (int)cfield(v.sh->layers) - 1;
  uint64_t *const words = v.word(bottom, 0);
  uint32_t pick[RUN_CHOICES];
  int choices = 0;
  // eight loads in flight: the words below a full top cost one round trip per eight
  for (int64_t hi = (int64_t)cfield(v.sh->nwords[bottom]) - 1; hi >= 0 && choices < RUN_CHOICES; hi -= 8) {
    uint64_t w[8];
#pragma unroll
    for (int k = 0; k < 8; k++) w[k] = hi - k >= 0 ? ld_rlx(words + (hi - k)) : 0ull;
#pragma unroll
    for (int k = 0; k < 8; k++)
      if ((uint64_t)cfc64(w[k]) >= n && choices < RUN_CHOICES) pick[choices++] = (uint32_t)(hi - k);
  }
  if (choices == 0) return FAIL;
  int at = (int)(((uint32_t)(thread_linear_id() * 0x9E3779B1u) >> 16) % (uint32_t)choices);
  for (int tries = 0; tries < choices; tries++) {
    uint64_t *word = words + pick[at];
    uint64_t seen = ld_rlx(word);
    uint32_t lost = 0;
    for (int c; (uint64_t)(c = cfc64(seen)) >= n && lost < VEB_LOSSES; lost++) {
      const uint64_t acq = bitmask((int)n) << (c - (int)n);
      const uint64_t got = atomicCAS((unsigned long long *)word, (unsigned long long)seen,
                                     (unsigned long long)(seen & ~acq));
      if (got == seen) {
        if ((seen & ~acq) == 0) veb_unlist(v.w, v.sh, pick[at]);
        return (uint64_t)pick[at] * 64u + (uint64_t)(c - (int)n);
      }
      seen = got;
    }
    if (++at == choices) at = 0;
  }
  return FAIL;
}

// veb_tree::gather_multiple (veb.cuh:1160-1196)
GAL_DEVICE_COLD uint64_t veb_gather_multiple(const veb_ref &v, uint64_t n) {
  uint64_t found = veb_gather_run(v, n);
  if (found == FAIL) return FAIL;
  uint64_t lo = found;
  for (int i = (int)cfield(v.sh->layers) - 2; i >= 0; i--) {
    uint64_t hi = (lo + n - 1) / 64 + 1;
    lo = lo / 64;
    n = hi - lo;
    for (uint64_t wb = lo; wb < lo + n; wb++) {
      if (ld_rlx(v.word(i + 1, wb)) != 0) continue;
      amo_and(v.word(i, wb / 64), ~(1ULL << (wb % 64)));
      fence_acq_rel();
      // an insert that refilled the word between the load and the clear found
      // the summary bit still set and left it: put it back, as veb_remove does
      if (ld_rlx(v.word(i + 1, wb)) != 0) amo_or(v.word(i, wb / 64), 1ULL << (wb % 64));
    }
  }
  return found;
}

// veb_tree::return_multiple (veb.cuh:1198-1218, layer form veb.cuh:495-523)
GAL_DEVICE_COLD void veb_return_multiple(const veb_ref &v, uint64_t start, uint64_t n) {
  const int bottom = (int)cfield(v.sh->layers) - 1;
  uint64_t bi = start / 64;
  int bs = (int)(start % 64);
  uint64_t left = n;
  while (left + (uint64_t)bs > 64) {
    int add = 64 - bs;
    amo_or(v.word(bottom, bi), bitmask(add) << bs);
    bs = 0;
    bi++;
    left -= (uint64_t)add;
  }
  amo_or(v.word(bottom, bi), bitmask((int)left) << bs);
  // maybe_return_layer_bits (veb.cuh:1128-1154) lists a word only when it is
  // full; an edge word that the claim emptied comes back partly filled and
  // would stay unlisted (its segments unreachable by every single-item
  // search).  Every non-empty word is listed here; a listed word that a
  // racing remove empties again is skipped by veb_successor.
  uint64_t lo = start;
  for (int i = bottom - 1; i >= 0; i--) {
    uint64_t hi = (lo + n - 1) / 64 + 1;
    lo = lo / 64;
    n = hi - lo;
    fence_acq_rel();  // the words below are set before their summaries (see veb_remove)
    for (uint64_t wb = lo; wb < lo + n; wb++)
      if (ld_rlx(v.word(i + 1, wb)) != 0) amo_or(v.word(i, wb / 64), 1ULL << (wb % 64));
  }
}

GAL_DEVICE_INLINE veb_ref seg_tree(const state *s) { return veb_ref{cfield(s->seg_tree), &s->veb, cfield(s->seed)}; }
GAL_DEVICE_INLINE veb_ref sub_tree(const state *s, uint32_t t) {
  return veb_ref{cfield(s->sub_trees) + (uint64_t)t * cfield(s->veb.words), &s->veb, cfield(s->seed) + t};
}

// ------------------------------------------------------------------ locks
// one lock word per class (and one for runs) in a 32-byte sector of its own;
// the reference keeps them as bits of one word (gallatin.cuh:1513-1519)
GAL_DEVICE_INLINE bool try_lock(const state *s, uint32_t bit) {
  return atomicExch(cfield(s->locks) + bit * LOCK_STRIDE, 1u) == 0u;
}
// What the locks keep apart is set by atomics one by one; a thread that sees a
// lock open before the last of them only searches or gathers once more.
GAL_DEVICE_INLINE void unlock(const state *s, uint32_t bit) {
  st_rlx(cfield(s->locks) + bit * LOCK_STRIDE, 0u);
}

// ------------------------------------------------------------------ table
// alloc_table::setup_segment (memory_table.cuh:746-818) in two steps, the second
// after a fence.  The segment was taken from the segment tree and is this
// thread's alone; `taken` of its blocks (0 or 1) are handed out with the set-up.
GAL_DEVICE_INLINE bool setup_begin(const state *s, uint64_t seg, uint32_t tree, uint32_t taken) {
  if (ld_rlx(&cfield(s->tree_ids)[seg]) != FREE_TREE) return false;
  st_rlx(&cfield(s->tree_ids)[seg], (uint16_t)tree);
  const uint32_t nb = blocks_in_segment(s, tree);
  uint32_t *q = cfield(s->queues) + (seg << cfield(s->bps_shift));
  if (nb >= 4) {
    for (uint32_t i = 0; i < nb; i += 4) *(uint4 *)(q + i) = make_uint4(NOBLK, NOBLK, NOBLK, NOBLK);
  } else {
    for (uint32_t i = 0; i < nb; i++) q[i] = NOBLK;
  }
  st_rlx(&cfield(s->qc)[seg], taken);
  st_rlx(&cfield(s->qfc)[seg], 0u);
  st_rlx(&cfield(s->fqfc)[seg], 0u);
  return true;
}
// count -1 -> nb - 1 - taken, class ACT_FREE -> tree, the next generation, by
// addition: a reservation attempt still in flight from before the segment's
// release gives its one back into this count, as it took it from the count it
// found, and the word need not be read (its high half changes only here and
// in the release: (gen << 8 | ACT_FREE) + tree + 1 is (gen + 1) << 8 | tree).
// Returns the word it found, so that the count is open before the caller lists
// the segment: a thread that found it refusing would take it off again for good.
GAL_DEVICE_INLINE unsigned long long setup_open(const state *s, uint64_t seg, uint32_t tree, uint32_t taken) {
  static_assert(ACT_FREE == 0xFFu, "one more than ACT_FREE carries into the generation");
  return atomicAdd(&cfield(s->act)[seg],
                   ((unsigned long long)(tree + 1u) << 32) + blocks_in_segment(s, tree) - taken);
}

// Gallatin::gather_new_segment (gallatin.cuh:1465-1510): the smallest free
// segment becomes the class's (-1: none).  With `take` its first block (pos 0)
// is the caller's: it is counted out before the segment is listed, and a segment
// of one block is not listed at all, as it would be taken off again by the same
// thread.  `l`: the segment tree's first words, which the caller loads while it
// waits for the class lock.  `more`: further segments wanted, for threads that
// wait for the lock; as many as the same word of the segment tree has are
// gathered along, their set-ups side by side, so that they cost little more
// than the one (16 segments one after another took 110 us of a call that
// wanted 256 blocks).
GAL_DEVICE_INLINE veb_low free_segments_low(const state *s) {
  const veb_ref v = seg_tree(s);
  return veb_load_low(v, veb_bottom(v));
}
GAL_DEVICE_COLD int64_t gather_new_segment(const state *s, uint32_t tree, bool take, veb_low l, uint32_t more = 0) {
  const veb_ref free_segs = seg_tree(s);
  const uint64_t seg = veb_malloc_first(free_segs, l);
  if (seg == FAIL) return -1;
  const uint64_t base = seg & ~63ull;
  uint64_t extra = 0;
  if (more && veb_shallow(free_segs)) {
    uint64_t *const word = veb_bottom(free_segs) + (seg >> 6);
    uint64_t seen = ld_rlx(word);
    for (uint32_t k = 0; k < more && seen; k++, seen &= seen - 1ull) extra |= seen & (0ull - seen);
    if (extra) {
      const uint64_t old = amo_and(word, ~extra);
      extra &= old;
      if (extra && (old & ~extra) == 0) veb_unlist(free_segs.w, free_segs.sh, (uint32_t)(seg >> 6));
    }
  }
  bool ok = setup_begin(s, seg, tree, take ? 1u : 0u);
  if (!ok) {
    set_error(s, GAL_DEV_ERR_SEGMENT_SETUP);
    if (!extra) return -1;
  }
  for (uint64_t b = extra; b; b &= b - 1ull) {
    const uint64_t g = base + (uint64_t)__ffsll((long long)b) - 1u;
    if (!setup_begin(s, g, tree, 0)) {
      set_error(s, GAL_DEV_ERR_SEGMENT_SETUP);
      extra &= ~(b & (0ull - b));
    }
  }
  fence_acq_rel();
  unsigned long long closed = act_word(0, ACT_FREE, 0);
  if (ok) closed &= setup_open(s, seg, tree, take ? 1u : 0u);
  for (uint64_t b = extra; b; b &= b - 1ull)
    closed &= setup_open(s, base + (uint64_t)__ffsll((long long)b) - 1u, tree, 0);
  // (the counts are open before the listings below: their atomics have answered)
  if (act_class(closed) != ACT_FREE) set_error(s, GAL_DEV_ERR_SEGMENT_SETUP);
  const veb_ref sub = sub_tree(s, tree);
  if (ok && (!take || blocks_in_segment(s, tree) > 1)) veb_insert(sub, seg);
  for (uint64_t b = extra; b; b &= b - 1ull) veb_insert(sub, base + (uint64_t)__ffsll((long long)b) - 1u);
  return ok ? (int64_t)seg : -1;
}

// A class's tree lists the segments that have a block to give, as far as its
// atomics let it: whoever raises a count lists the segment after that, and who
// finds a listed segment without one takes it off again.  A segment counts as
// serving while its word has the class and a count that is not negative.
GAL_DEVICE_INLINE bool serves(const state *s, uint32_t tree, uint64_t seg) {
  const unsigned long long w = ld_rlx(&cfield(s->act)[seg]);
  return act_class(w) == tree && act_count(w) >= 0;
}

// The two steps of a listing; true: it agrees with the count.
GAL_DEVICE_COLD bool listing_on(const state *s, uint32_t tree, uint32_t seg) {
  veb_insert<true>(sub_tree(s, tree), seg);
  return serves(s, tree, seg);
}
GAL_DEVICE_COLD bool listing_off(const state *s, uint32_t tree, uint32_t seg) {
  return !veb_remove<true>(sub_tree(s, tree), seg) || !serves(s, tree, seg);
}
// Makes the listing of a segment in the tree of class `tree` agree with its count.
//   listed: it is, but has no block to give (or is another class's by now).  It is
//     taken off by the thread that took its last block, or by any that finds it
//     meanwhile, so that nobody waits for the former.  Blocks may have come home
//     since, and then it is listed again (who raised the count and listed the
//     segment before this removal is seen here, who lists it after it undoes
//     the removal).
//   not listed: this thread has raised its count.  Raised first: a search that
//     found the segment listed and its count still negative would take it off,
//     and the next listing is a lap of the ring away.  The segment may have been
//     emptied, or released and set up for another class, in between: then it
//     does not stay listed.
// The release of a segment closes its count word before it unlists it, so a
// listing made here and still valid when the word is read again is either right
// or taken off by the release.  One thread alone never has to undo a step.
// (The steps are functions of their own, and whoever returns blocks calls this
// after return_block, not inside it: the registers of a chain of calls add up in
// every kernel that frees.)
GAL_DEVICE_COLD void settle_listing(const state *s, uint32_t tree, uint32_t seg, bool listed) {
  for (uint32_t tries = 0; tries < cfield(s->spin_limit); tries++) {
    if (!listed && listing_on(s, tree, seg)) return;
    if (listing_off(s, tree, seg)) return;
    listed = false;
  }
  if (!listing_on(s, tree, seg))  // left listed: the next search meets it again
    set_error_info(s, GAL_DEV_ERR_TIMEOUT, SITE_LISTING, tree, seg);
}
GAL_DEVICE_INLINE void unlist_refusing(const state *s, uint32_t tree, uint64_t seg) {
  settle_listing(s, tree, (uint32_t)seg, true);
}
GAL_DEVICE_INLINE void list_serving(const state *s, uint32_t tree, uint64_t seg) {
  settle_listing(s, tree, (uint32_t)seg, false);
}

// Releases segment `seg` of class `tree` when its count word still reads
// `gen` with every block home (nb - 1): removes it from the class's tree,
// frees its class and lists it in the segment tree (the release steps of
// Gallatin::return_block, gallatin.cuh:1663-1722, finish_freeing_block,
// memory_table.cuh:1226-1241).  NOSEG, or `list` when the segment has moved on.
GAL_DEVICE_COLD uint32_t release_segment(const state *s, uint64_t seg, uint32_t tree, uint32_t gen, uint32_t nb,
                                         uint32_t list) {
  const unsigned long long home = act_word(gen, tree, (int32_t)nb - 1);
  if (atomicCAS(&cfield(s->act)[seg], home, act_word(gen, ACT_FREE, -1)) != home) return list;
  fence_acq_rel();  // closed before it is taken off (see settle_listing)
  veb_remove(sub_tree(s, tree), seg);
  // closed and unlisted, the segment is this thread's alone
  if (ld_rlx(&cfield(s->tree_ids)[seg]) != (uint16_t)tree) set_error(s, GAL_DEV_ERR_SEGMENT_SETUP);
  st_rlx(&cfield(s->tree_ids)[seg], FREE_TREE);
  veb_insert<true>(seg_tree(s), seg);
  return NOSEG;
}

// Gives back a reservation taken from segment `seg` that no block came of.
// While it was held the count stayed below every-block-home, so no release
// could run; if giving it back brings the count there and blocks were handed
// out in this generation (every one of them has come home, the last return
// having found the count one short), the segment is released here.  While it
// was held the count may also have read negative with a block there to give,
// and a search that met the segment then has taken it off its tree: it is
// listed again.
GAL_DEVICE_COLD void give_back_reservation(const state *s, uint64_t seg) {
  const unsigned long long old = add_acquire(&cfield(s->act)[seg], 1ull);
  const uint32_t tree = act_class(old);
  if (tree >= cfield(s->num_trees) || act_count(old) + 1 < 0) return;
  const uint32_t nb = blocks_in_segment(s, tree);
  if (act_count(old) + 1 == (int32_t)nb - 1 && ld_rlx(&cfield(s->qc)[seg]) != 0 &&
      release_segment(s, seg, tree, act_gen(old), nb, 0) == NOSEG)
    return;
  list_serving(s, tree, seg);
}

// alloc_table::get_block (memory_table.cuh:915-993)
// The reference subtracts one from the segment's count and adds it back when
// the count went negative or the segment belongs to another class
// (memory_table.cuh:923-929, get_slot_in_segment / return_slot_to_segment).
// An add-back that lands after the segment was released and set up again
// raises the new owner's count above its blocks, and one that lands after the
// segment's last return leaves it unreleased.  Here the count word carries the
// class: a word of another class or a count already negative is not touched,
// and the subtraction carries into a new set-up (see setup_open), so the
// only give-backs left are the rare ones of a race between the load and the
// subtraction, which give_back_reservation settles.  The new block's malloc
// word is stored, not yet published: whoever installs the block fences first.
GAL_DEVICE_COLD uint32_t get_block(const state *s, uint64_t seg, uint32_t tree, bool &last) {
  last = false;
  const unsigned long long seen = ld_rlx(&cfield(s->act)[seg]);
  if (act_class(seen) != tree || act_count(seen) < 0) return NOBLK;  // another class's, or nothing left
  const unsigned long long old = add_acquire(&cfield(s->act)[seg], ~0ull);  // minus one
  if (act_count(old) < 0 || act_class(old) != tree) {
    // the last block went to another thread meanwhile, or the segment was
    // released and set up for another class
    give_back_reservation(s, seg);
    return NOBLK;
  }
  uint32_t nb = blocks_in_segment(s, tree);
  uint32_t pos = atomicAdd(&cfield(s->qc)[seg], 1u);
  uint32_t blk;
  if (pos < nb) {
    blk = (uint32_t)(seg << cfield(s->bps_shift)) + pos;
  } else {
    uint32_t *e = cfield(s->queues) + (seg << cfield(s->bps_shift)) + (pos & (nb - 1u));
    blk = exch_acquire(e, NOBLK);
    for (uint32_t i = 0; blk == NOBLK && i < cfield(s->spin_limit); i++) {  // a return still in flight
      backoff(i);
      blk = exch_acquire(e, NOBLK);
    }
    if (blk == NOBLK) {
      set_error(s, GAL_DEV_ERR_NULL_QUEUE);
      return NOBLK;
    }
  }
  st_rlx(mword_ptr(s, blk), (unsigned long long)tree << 32);  // Block::init_malloc
  last = act_count(old) == 0;
  return blk;
}

// Waits between attempts at a segment another thread is working on: a gather
// takes a few microseconds, so the first waits are short; a wait that lasts
// grows to backoff's.  (Growing after 24 tries left the last of 152 threads
// that asked one class together waiting up to 290 us.)
GAL_DEVICE_INLINE void backoff_gather(uint32_t i) { __nanosleep(i < 64 ? 100u : i < 1024 ? 400u : 4096u); }

// Threads that wait for the lock of class `tree` to gather a segment, counted
// beside the lock, and the segments wanted for them besides the one that is
// gathered anyway.  A thread that never waited leaves the count at 0.
static constexpr uint32_t MORE_SEGMENTS = 7;
GAL_DEVICE_INLINE uint32_t *waiters_of(const state *s, uint32_t tree) {
  return cfield(s->locks) + tree * LOCK_STRIDE + 1;
}
GAL_DEVICE_INLINE uint32_t more_segments(const state *s, uint32_t tree, uint32_t waiting) {
  return min(MORE_SEGMENTS, waiting / blocks_in_segment(s, tree));
}

// The rest of a block request that took the last block of a segment
// (gallatin.cuh:1598-1612): with gather_ahead the class's next segment is
// gathered, and the emptied one leaves its class's tree.  Split from
// request_block so that a claim's block can be installed first: the teams
// waiting for it do not wait for the gather, and one thread alone leaves the
// same state either way.  The next segment is listed before the emptied one is
// taken off, so the class's word does not empty and its summaries stay as they
// are.
// Only one thread of a class gathers ahead at a time, whatever its lock policy
// (alone, a thread always finds the lock free): each would add a segment to a
// class that needs one, and threads that take a class's last blocks together
// would leave it holding hundreds.
static constexpr uint32_t SEG_UNLISTED = 0x80000000u;  // with a segment: it was never listed
GAL_DEVICE_COLD void finish_emptied(const state *s, uint32_t tree, uint32_t emptied) {
  if (cfield(s->gather_ahead)) {
    const veb_low l = free_segments_low(s);
    const uint32_t waiting = ld_rlx(waiters_of(s, tree));
    if (try_lock(s, tree)) {
      gather_new_segment(s, tree, false, l, more_segments(s, tree, waiting));
      unlock(s, tree);
    }
  }
  if (!(emptied & SEG_UNLISTED)) unlist_refusing(s, tree, emptied);
}
// The steps of a block request are functions of their own with few arguments:
// what a caller keeps across a call stays in registers at every level of the
// chain, and the chain's depth is what a kernel that calls malloc is compiled
// for (as one function with its helpers inlined: 26 more registers).
// A listed segment of the class (FAIL: none); after a wait any of them.
GAL_DEVICE_COLD uint64_t find_segment(const state *s, uint32_t tree, uint32_t tid, uint32_t waited) {
  const veb_ref sub = sub_tree(s, tree);
  if (cfield(s->policy) == GAL_POLICY_LOWEST) return veb_find_first(sub);
  if (waited) return veb_find_any(sub, (tid + waited) * 0x9E3779B1u >> 8);
  return veb_find_random(sub, tid);
}
// A new segment for a request that found none listed (first block taken);
// -1: none is free, -2: another thread of the class is gathering one.
// Classes with few blocks per segment need a segment per few requests: the
// class lock only serialises them (serially the lock is always free).
GAL_DEVICE_COLD int64_t gather_on_demand(const state *s, uint32_t tree) {
  const veb_low l = free_segments_low(s);
  if (blocks_in_segment(s, tree) < cfield(s->gather_unlocked_below)) return gather_new_segment(s, tree, true, l);
  const uint32_t waiting = ld_rlx(waiters_of(s, tree));
  if (ld_rlx(cfield(s->locks) + tree * LOCK_STRIDE) != 0u || !try_lock(s, tree)) return -2;
  const int64_t got = gather_new_segment(s, tree, true, l, more_segments(s, tree, waiting));
  unlock(s, tree);
  return got;
}

// Gallatin::request_new_block_from_tree (gallatin.cuh:1525-1631): the block in
// the low half (NOBLK: none), and in the high half, for request_done, the
// segment whose last block it was, else NOSEG.
GAL_DEVICE_INLINE uint32_t requested_block(uint64_t r) { return (uint32_t)r; }
GAL_DEVICE_COLD uint64_t request_block_begin(const state *s, uint32_t tree, uint32_t tid) {
  uint32_t waited = 0, blk = NOBLK, emptied = NOSEG;
  uint32_t gather_fails = 0, counted = 0;  // counted: among the waiters
  for (;;) {
    const uint64_t seg = find_segment(s, tree, tid, waited);
    if (seg == FAIL) {
      const int64_t got = gather_on_demand(s, tree);
      if (got >= 0) {
        blk = (uint32_t)got << cfield(s->bps_shift);
        st_rlx(mword_ptr(s, blk), (unsigned long long)tree << 32);
        if (blocks_in_segment(s, tree) == 1) emptied = (uint32_t)got | SEG_UNLISTED;
        break;
      }
      if (got == -1) {
        // segment tree empty: nothing a retry by this thread alone changes
        if (++gather_fails >= (uint32_t)GATHER_RETRIES) break;
        backoff(gather_fails);
        continue;
      }
      if (!counted) atomicAdd(waiters_of(s, tree), 1u);
      counted = 1;
    } else {
      bool last = false;
      blk = get_block(s, seg, tree, last);
      if (last) emptied = (uint32_t)seg;
      if (blk != NOBLK) break;
      if (last) finish_emptied(s, tree, (uint32_t)seg);  // counted out, but its block never came
      else unlist_refusing(s, tree, seg);
      emptied = NOSEG;
    }
    if (++waited > cfield(s->spin_limit)) {
      set_error_info(s, GAL_DEV_ERR_TIMEOUT, seg == FAIL ? SITE_REQUEST_LOCK : SITE_REQUEST_RETRY, tree,
                     seg == FAIL ? (uint64_t)waited : seg);
      break;
    }
    backoff_gather(waited);
  }
  if (counted) atomicSub(waiters_of(s, tree), 1u);
  return ((uint64_t)emptied << 32) | blk;
}
GAL_DEVICE_INLINE void request_done(const state *s, uint32_t tree, uint64_t r) {
  if ((uint32_t)(r >> 32) != NOSEG) finish_emptied(s, tree, (uint32_t)(r >> 32));
}
GAL_DEVICE_INLINE uint32_t request_block(const state *s, uint32_t tree, uint32_t tid) {
  const uint64_t r = request_block_begin(s, tree, tid);
  request_done(s, tree, r);
  return requested_block(r);
}

// Gallatin::return_block (gallatin.cuh:1637-1726) with reserve_segment_slot,
// finalize_free_queue and finish_freeing_block (memory_table.cuh:906-910,1158-1241)
// Returns what is to be listed after it (see block_returned; NOSEG: nothing).
GAL_DEVICE_COLD uint32_t return_block(const state *s, uint32_t blk) {
  uint64_t seg = blk >> cfield(s->bps_shift);
  uint16_t tree = ld_rlx(&cfield(s->tree_ids)[seg]);
  if (tree >= cfield(s->num_trees)) {
    set_error_info(s, GAL_DEV_ERR_BAD_FREE, SITE_RETURN_BAD_TREE, blk, tree);
    return NOSEG;
  }
  uint32_t nb = blocks_in_segment(s, tree);
  uint32_t pos = atomicAdd(&cfield(s->qfc)[seg], 1u);
  uint32_t live = pos & (nb - 1u);
  // with the block's free counter at 0: counts are interchangeable, so whoever
  // takes the entry may have been let in by another block's return
  st_release(cfield(s->queues) + (seg << cfield(s->bps_shift)) + live, blk);
  // The reference finalises returns in position order with a CAS spin
  // (memory_table.cuh:906-910) so a hand-out never meets an empty ring entry;
  // get_block here waits (bounded) for an entry still in flight instead, so a
  // return only counts itself, leaving the same counter value.
  atomicAdd(&cfield(s->fqfc)[seg], 1u);
  // re-register at the 10% crossing (gallatin.cuh:1646): live/nb >= 0.1 and
  // (live-1)/nb < 0.1 in doubles; for the power-of-two nb used here that is
  // 10*live > nb >= 10*(live-1) with live-1 taken as unsigned (live 0 never).
  const bool crossing = live != 0 && 10ull * live > nb && 10ull * (live - 1) < nb;
  const uint32_t list = crossing ? (uint32_t)seg << 8 | tree : NOSEG;
  fence_acq_rel();  // the ring entry before the count that lets it be handed out
  const unsigned long long old = add_acquire(&cfield(s->act)[seg], 1ull);
  if ((uint32_t)(act_count(old) + 2) == nb)  // all_blocks_free: the count was nb - 2
    return release_segment(s, seg, tree, act_gen(old), nb, list);
  return list;
}
GAL_DEVICE_INLINE void block_returned(const state *s, uint32_t list) {
  if (list != NOSEG) list_serving(s, list & 0xFFu, list >> 8);
}

// Block::block_free_multiple + reset_free + free_block (block.cuh:87-98,200-212,
// gallatin.cuh:1732-1766)
GAL_DEVICE_INLINE void credit_done(const state *s, uint32_t blk, uint32_t old, uint32_t n);
GAL_DEVICE_INLINE void credit_frees(const state *s, uint32_t blk, uint32_t n) {
  credit_done(s, blk, atomicAdd(fctr_ptr(s, blk), n), n);
}
// the block's free counter was `old` before this thread added n
GAL_DEVICE_INLINE void credit_done(const state *s, uint32_t blk, uint32_t old, uint32_t n) {
  if (old + n == SLICES_PER_BLOCK) {
    st_rlx(fctr_ptr(s, blk), 0u);  // published with the block's ring entry
    block_returned(s, return_block(s, blk));
  } else if (old + n > SLICES_PER_BLOCK) {
    set_error_info(s, GAL_DEV_ERR_BAD_FREE, SITE_FREE_OVERFLOW, blk,
                   ((uint64_t)old << 32) | n);
  }
}

// Gives back a block this thread took for a slot or a spare and could not
// install: closes it to further claims (its count goes past the end) and
// credits the slices nobody claimed, so it returns to its segment now, or
// once the slices a claim did take (one that read the block in an earlier
// life and landed after its hand-out) are freed.  Crediting all 4,096 would
// return it under those live slices.
GAL_DEVICE_COLD void retire_block(const state *s, uint32_t blk) {
  const unsigned long long old = atomicAdd(mword_ptr(s, blk), (unsigned long long)SLICES_PER_BLOCK);
  const uint32_t handed_out = (uint32_t)old;
  if (handed_out < SLICES_PER_BLOCK) credit_frees(s, blk, SLICES_PER_BLOCK - handed_out);
}

// Gallatin::free_offset (gallatin.cuh:1774-1827): team by block, one atomic
GAL_DEVICE_INLINE void free_block_slices(const state *s, uint32_t blk) {
  uint32_t active = active_lanes();
  uint32_t team = __match_any_sync(active, blk) & team_group(s);
  if ((int)lane_id() == __ffs(team) - 1) credit_frees(s, blk, (uint32_t)__popc(team));
}

// ------------------------------------------------------------------ pinned slots
// per_size_pinned_blocks::get_valid_block_index (shared_block_storage.cuh:119-134)
// Returns the slot index; `blk` receives the block read from it (one read per
// probed slot, the last one doubling as the reference's get_my_block read).
GAL_DEVICE_INLINE uint32_t pick_slot(const state *s, uint32_t tree, uint32_t &blk) {
  const uint32_t n = cfield(s->slot_count[tree]);
  const uint32_t *slots = cfield(s->slots) + cfield(s->slot_base[tree]);
  uint32_t smid = cfield(s->smid_override) >= 0 ? (uint32_t)cfield(s->smid_override) : sm_id();
  int my = (int)(smid < n ? smid : (n & (n - 1u)) == 0 ? smid & (n - 1u) : smid % n);
  int original = my;
  int counter = 0;
  uint32_t v = ld_rlx(&slots[my]);
  while (v == NOBLK && my != original - 1) {
    my = (my + 1) % (int)n;
    v = ld_rlx(&slots[my]);
    if (++counter >= SLOT_PROBE_LIMIT) break;
  }
  blk = v;
  return (uint32_t)my;
}

// Requests a block for the empty slot or spare word `at`.
GAL_DEVICE_COLD bool request_into(const state *s, uint32_t tree, uint32_t *at, uint32_t tid, bool slot) {
  const uint64_t r = request_block_begin(s, tree, tid);
  bool ok = false;
  if (requested_block(r) != NOBLK) {
    fence_acq_rel();
    ok = atomicCAS(at, NOBLK, requested_block(r)) == NOBLK;
    if (!ok) {
      if (slot) set_error(s, GAL_DEV_ERR_SLOT_SWAP);
      retire_block(s, requested_block(r));  // hand the block back
    }
  }
  request_done(s, tree, r);  // after the waiting teams have their block
  return ok;
}

// Gallatin::replace_block (gallatin.cuh:1083-1138)
GAL_DEVICE_INLINE bool replace_block(const state *s, uint32_t tree, uint32_t slot, uint32_t blk, uint32_t tid) {
  uint32_t *sp = cfield(s->slots) + cfield(s->slot_base[tree]) + slot;
  if (atomicCAS(sp, blk, NOBLK) != blk) return true;
  return request_into(s, tree, sp, tid, true);
}

// Spare blocks (gal_config.spare_blocks): the slot's prepared next block is
// swapped in with one CAS, so other warps see a fresh block at once instead of
// an empty slot for the length of a segment search; the search then refills
// the spare.  swap_spare returns whether the caller should refill (it falls
// back to replace_block when no spare was ready).
GAL_DEVICE_INLINE bool swap_spare(const state *s, uint32_t tree, uint32_t slot, uint32_t blk, uint32_t tid) {
  const uint32_t si = cfield(s->slot_base[tree]) + slot;
  const uint32_t nx = atomicExch(cfield(s->spares) + si, NOBLK);
  if (nx == NOBLK) {
    replace_block(s, tree, slot, blk, tid);
  } else if (atomicCAS(cfield(s->slots) + si, blk, nx) != blk) {
    retire_block(s, nx);  // the slot moved on: give the spare back
    return false;
  }
  return true;
}
GAL_DEVICE_INLINE void refill_spare(const state *s, uint32_t tree, uint32_t slot, uint32_t tid) {
  uint32_t *at = cfield(s->spares) + cfield(s->slot_base[tree]) + slot;
  if (ld_rlx(at) == NOBLK) request_into(s, tree, at, tid, false);
}

// Gallatin::boot_block (gallatin.cuh:726-787)
GAL_DEVICE_COLD bool boot_block(const state *s, uint32_t tree, uint32_t slot, uint32_t tid) {
  if (slot >= cfield(s->slot_count[tree])) return false;
  uint32_t blk = request_block(s, tree, tid);
  if (blk == NOBLK) return false;
  if (ld_rlx(&cfield(s->tree_ids)[blk >> cfield(s->bps_shift)]) != tree) return false;
  fence_acq_rel();
  return atomicCAS(cfield(s->slots) + cfield(s->slot_base[tree]) + slot, NOBLK, blk) == NOBLK;
}

// ------------------------------------------------------------------ addresses
GAL_DEVICE_INLINE char *slice_ptr(const state *s, uint32_t blk, uint64_t idx, uint32_t tree) {
  uint64_t seg = blk >> cfield(s->bps_shift);
  uint64_t q = blk & ((1u << cfield(s->bps_shift)) - 1u);
  return cfield(s->memory) + (seg << cfield(s->seg_shift)) + (((q << 12) + idx) << (cfield(s->min_shift) + tree));
}

// ------------------------------------------------------------------ malloc tiers
// Gallatin::malloc_slice_allocation (gallatin.cuh:865-1078): warp team per
// size class, one atomicAdd on the pinned block per team.  Two ways to know
// the team: as the reference does, the lanes executing each attempt together
// (NAMED = false: every attempt re-forms the teams from the active lanes, and
// a lane leaves the loop as soon as it has its slice); or named by the caller
// (NAMED = true: `pending`, the lanes that called together and ask for
// slices, shrinks as lanes get their slices, and every warp-wide step of an
// attempt names it, so a team holds every caller of its class even when the
// callers' earlier branches left them in separate groups).
// A CTA's copy of its SM's pinned blocks, in shared memory (gal::malloc_cached):
// per class the block last read from the class's pinned slot and that slot.
// A copy that has gone stale (its block exhausted or replaced) shows up in the
// claim itself -- the count comes back at or past the block's end, or with
// another class -- and is dropped, so the next team reads the slot again.
struct slot_cache {
  uint32_t blk[GAL_MAX_TREES];
  uint32_t slot[GAL_MAX_TREES];
};

// every thread of the CTA, followed by a __syncthreads()
GAL_DEVICE_INLINE void slot_cache_init(slot_cache &c) {
  if (threadIdx.x < GAL_MAX_TREES) {
    c.blk[threadIdx.x] = NOBLK;
    c.slot[threadIdx.x] = 0;
  }
}

// The rare part of a claim, out of line so the claim's common path keeps few
// values live across calls: credits the slices this lane gives back and, for
// the team's leader when the block must be replaced, swaps in the slot's spare
// (or replaces the block).  Returns the slot when its spare wants a refill,
// else NOBLK.
GAL_DEVICE_COLD uint32_t claim_slow_path(const state *s, uint32_t tree, uint32_t slot, uint32_t blk, uint32_t credit,
                                         bool lead) {
  if (credit) credit_frees(s, blk, credit);
  if (!lead) return NOBLK;
  const uint32_t tid = (uint32_t)thread_linear_id();
  if (cfield(s->use_spares)) return swap_spare(s, tree, slot, blk, tid) ? slot : NOBLK;
  replace_block(s, tree, slot, blk, tid);
  return NOBLK;
}

// A block is exhausted by exactly one claim -- the one that crosses slice
// 4095 -- and that claim's team replaces it in its pinned slot.  A team that
// claimed from a block it read some time before (a CTA's slot_cache, or a
// slow team) may cross a block that has since been recycled into another
// slot or a spare; its replace then finds its own slot holding something else
// and does nothing, and the slot that does hold the block keeps it exhausted.
// Every failed claim still adds to the block's count, so a block left
// exhausted in a slot soon reads far past its end: a team that reads its
// slot's block more than STUCK_MARGIN slices past the end, has tried
// STUCK_ATTEMPTS times and still finds the block in the slot replaces it itself
// (a compare-and-swap on the slot, so at most one replacement happens).  The
// rightful crosser swaps its block within a few round trips of the end; where
// many SMs share a slot their failed claims pass the margin in that time, and
// without the attempts (some 20 us of them) they took the swap from the crosser
// and requested blocks that had to be handed back.  One thread alone never
// meets an exhausted block in its slot, so serial offsets are unchanged.
static constexpr uint32_t STUCK_MARGIN = 1u << 12;
static constexpr int STUCK_ATTEMPTS = 16;
// What an attempt needs after a call off its common path.  Kept in memory across
// the call (volatile), not in registers: the compiler stacks the registers of a
// caller and of the whole chain it calls, so what is held here while a block is
// requested would be held by every kernel that calls malloc.
struct parked {
  volatile uint64_t state, result;
  volatile uint32_t tree, count, live;
  volatile int attempt;
};
template <bool NAMED>
GAL_DEVICE_INLINE void *malloc_slices(const state *s, uint32_t tree, uint32_t count, uint32_t pending,
                                      slot_cache *cache = nullptr) {
  parked keep;
  for (int attempt = 0; attempt < SLICE_ATTEMPTS; attempt++) {
    const uint32_t lane = lane_id();
    const uint32_t active = NAMED ? pending : active_lanes();
    const uint32_t team = __match_any_sync(active, tree) & team_group(s);
    const int leader = __ffs(team) - 1;
    const int last = 31 - __clz(team);
    const uint32_t lt = lanemask_lt();
    // every lane of a team reads the same slot words in the same instruction
    // (one broadcast transaction), so the team needs no leader branch here
    uint32_t seen = NOBLK, slot = 0;
    if (cache) {
      seen = *(volatile uint32_t *)&cache->blk[tree];
      slot = *(volatile uint32_t *)&cache->slot[tree];
    }
    const bool fresh = seen == NOBLK;  // read from the pinned slot this attempt
    if (fresh) {
      slot = pick_slot(s, tree, seen);
      if (cache && seen != NOBLK) {  // every lane of the team writes the same values
        *(volatile uint32_t *)&cache->slot[tree] = slot;
        *(volatile uint32_t *)&cache->blk[tree] = seen;
      }
    }
    const uint32_t blk = __shfl_sync(active, seen, leader);
    // teams whose slot was empty retry; the rest carry on with mask `live`
    const uint32_t live = __ballot_sync(active, blk != NOBLK);
    if (!NAMED && blk == NOBLK) continue;
    void *result = nullptr;
    bool refill = false;
    if (blk != NOBLK) {
      uint32_t prefix, total;
      if (__all_sync(live, count == 1)) {
        prefix = (uint32_t)__popc(team & lt);
        total = (uint32_t)__popc(team);
      } else {  // big slices: counts are powers of two up to one block
        prefix = 0;
        total = 0;
        for (uint32_t c = 1; c <= SLICES_PER_BLOCK; c <<= 1) {
          uint32_t b = __ballot_sync(live, count == c) & team;
          prefix += c * (uint32_t)__popc(b & lt);
          total += c * (uint32_t)__popc(b);
        }
      }
      unsigned long long old = 0;
      if ((int)lane == last) old = atomicAdd(mword_ptr(s, blk), (unsigned long long)total);
      old = __shfl_sync(live, old, last);
      // (counts past 2^24 are as exhausted as any: sums below stay in 32 bits)
      const uint32_t cnt = min((uint32_t)old, 1u << 24);
      const bool foreign = (uint32_t)(old >> 32) != tree;
      uint32_t credit = 0;
      bool lead = false;
      if (!foreign && count == 1 && cnt + total < SLICES_PER_BLOCK) {  // all but one claim in hundreds
        result = slice_ptr(s, blk, cnt + prefix, tree);
      } else {
        const uint32_t alloc = cnt + prefix;
        const bool start_valid = alloc <= SLICES_PER_BLOCK - 1;
        const bool end_valid = alloc + count <= SLICES_PER_BLOCK;
        const bool valid = start_valid && end_valid;
        if (valid && !foreign) result = slice_ptr(s, blk, alloc, tree);
        // slices this lane gives back: the rest of a run, or the part of it past
        // the block's end (block_correct_frees), and a claimed slice of a block
        // that serves another class now (Block::check_valid failed)
        credit = (start_valid ? (end_valid ? count - 1 : SLICES_PER_BLOCK - alloc) : 0u) + (valid && foreign ? 1u : 0u);
        // the team's lanes take consecutive slices: one of them holds slice 4095
        // exactly when the claim crosses it
        bool replace = cnt < SLICES_PER_BLOCK && cnt + total >= SLICES_PER_BLOCK;
        const bool exhausted = !foreign && cnt >= SLICES_PER_BLOCK;
        if (cache) {  // exhausted, replaced or foreign: the next team reads the slot again
          if ((replace || exhausted || foreign) && (int)lane == leader) atomicCAS(&cache->blk[tree], blk, NOBLK);
        }
        if (exhausted && fresh && attempt >= STUCK_ATTEMPTS && cnt >= SLICES_PER_BLOCK + STUCK_MARGIN &&
            ld_rlx(cfield(s->slots) + cfield(s->slot_base[tree]) + slot) == blk)
          replace = true;  // the slot has held an exhausted block for a while: replace it here
        lead = replace && (int)lane == leader;
      }
      uint32_t group = live;
      if (credit || lead) {
        keep.state = (uint64_t)s;
        keep.result = (uint64_t)result;
        keep.tree = tree;
        keep.count = count;
        keep.live = live;
        keep.attempt = attempt;
        const uint32_t r = claim_slow_path(s, tree, slot, blk, credit, lead);
        refill = r != NOBLK;
        slot = r;
        s = (const state *)keep.state;
        result = (void *)keep.result;
        tree = keep.tree;
        count = keep.count;
        group = keep.live;
        attempt = keep.attempt;
      }
      __syncwarp(group);
    }
    if (NAMED) pending = __ballot_sync(active, result == nullptr);
    if (refill) {  // the team's other lanes go on
      keep.state = (uint64_t)s;
      keep.result = (uint64_t)result;
      keep.tree = tree;
      keep.count = count;
      keep.attempt = attempt;
      refill_spare(s, tree, slot, (uint32_t)thread_linear_id());
      s = (const state *)keep.state;
      result = (void *)keep.result;
      tree = keep.tree;
      count = keep.count;
      attempt = keep.attempt;
    }
    if (result) return result;
  }
  return nullptr;
}

// Gallatin::malloc_block_allocation (gallatin.cuh:828-861), Block::malloc_fill_block
GAL_DEVICE_INLINE void *malloc_whole_block(const state *s, uint32_t tree) {
  volatile uint32_t kept = tree, attempts = BLOCK_ATTEMPTS;  // see `parked`
  while (attempts) {
    attempts = attempts - 1u;
    const uint32_t blk = request_block(s, kept, (uint32_t)thread_linear_id());
    if (blk == NOBLK) return nullptr;
    unsigned long long old = atomicAdd(mword_ptr(s, blk), (unsigned long long)SLICES_PER_BLOCK);
    uint32_t old_count = (uint32_t)old;
    if ((uint32_t)(old >> 32) != kept) set_error(s, GAL_DEV_ERR_BLOCK_TREE);
    atomicAdd(fctr_ptr(s, blk), (SLICES_PER_BLOCK - 1) - old_count);
    if (old_count == 0) return slice_ptr(s, blk, 0, kept);
    credit_frees(s, blk, 1);
  }
  return nullptr;
}

// marks the run of `count` segments from idx, taken by this thread
GAL_DEVICE_INLINE void own_run(const state *s, uint64_t idx, uint32_t count) {
  if (ld_rlx(&cfield(s->tree_ids)[idx]) != FREE_TREE) set_error(s, GAL_DEV_ERR_SEGMENT_SETUP);
  else st_rlx(&cfield(s->tree_ids)[idx], (uint16_t)(cfield(s->num_trees) + 1 + count));
}

// Gallatin::malloc_segment_allocation (gallatin.cuh:790-826).  The reference
// queues every request on one lock; 85 runs asked for together then took 8 us
// each, one after another.  A request that finds the lock taken looks for its
// run inside one word by itself first and waits only if there is none.
GAL_DEVICE_COLD void *malloc_segment_run(const state *s, uint32_t count) {
  for (int a = 0; a < SEGMENT_ATTEMPTS; a++) {
    uint32_t spins = 0;
    while (!try_lock(s, cfield(s->num_trees))) {
      if (spins == 0 && count <= 64) {
        const uint64_t idx = veb_gather_in_word(seg_tree(s), count);
        if (idx != FAIL) {
          own_run(s, idx, count);
          return cfield(s->memory) + (idx << cfield(s->seg_shift));
        }
      }
      if (++spins > cfield(s->spin_limit)) {
        set_error_info(s, GAL_DEV_ERR_TIMEOUT, SITE_RUN_LOCK, count, spins);
        return nullptr;
      }
      backoff(spins);
    }
    uint64_t idx = veb_gather_multiple(seg_tree(s), count);
    if (idx != FAIL) {
      own_run(s, idx, count);
      unlock(s, cfield(s->num_trees));
      return cfield(s->memory) + (idx << cfield(s->seg_shift));
    }
    unlock(s, cfield(s->num_trees));
  }
  return nullptr;
}

// calloc mode (gal_config.zero_fill): the requested bytes, rounded up to 16,
// are cleared by the allocating thread.  Every allocation starts on a 16-byte
// boundary and covers at least its request rounded up to 16 (slices are at
// least 16 B), so the stores stay inside it.
GAL_DEVICE_COLD void zero_fill(void *p, uint64_t size) {
  uint4 *q = (uint4 *)p;
  const uint64_t n = size ? (size + 15) >> 4 : 1;
  for (uint64_t i = 0; i < n; i++) q[i] = make_uint4(0u, 0u, 0u, 0u);
}
GAL_DEVICE_INLINE void *handed_out(const state *s, void *p, uint64_t size) {
  if (p && cfield(s->zero_fill)) zero_fill(p, size);
  return p;
}

// the block and segment tiers of Gallatin::malloc (gallatin.cuh:1203-1258)
GAL_DEVICE_COLD void *malloc_large(const state *s, uint64_t size, int block_tree) {
  if (block_tree < (int)cfield(s->num_trees)) return malloc_whole_block(s, (uint32_t)block_tree);
  const uint64_t count = ((size - 1) >> cfield(s->seg_shift)) + 1;  // (may not fit 32 bits)
  return count <= cfield(s->num_segments) ? malloc_segment_run(s, (uint32_t)count) : nullptr;
}

// Gallatin::malloc (gallatin.cuh:1186-1276) called by the lanes in `callers`
// together.  Those that ask for slices reach malloc_slices on one path (the
// class and run length are selects, not branches), so single slices and runs
// of the same class share a team.
template <bool NAMED>
GAL_DEVICE_INLINE void *malloc_from(const state *s, uint64_t size, uint32_t callers, slot_cache *cache = nullptr) {
  const int T = (int)cfield(s->num_trees), min_shift = (int)cfield(s->min_shift);
  const int bits = size > 1 ? 64 - __clzll((long long)(size - 1)) : 0;  // ceil(log2)
  const int t = max(bits - min_shift, 0);
  const int block_tree = bits - (min_shift + 12);
  const bool slices = t < T || block_tree < 0;
  const uint32_t members = __ballot_sync(callers, slices);
  if (!slices) {
    const volatile uint64_t kept = size;  // see `parked`
    void *p = malloc_large(s, size, block_tree);
    return handed_out(s, p, kept);
  }
  // big slices (4 KiB < size <= 32 KiB by default): runs of the last class
  const bool big = t >= T;
  const uint32_t count = 1u << (big ? t - (T - 1) : 0);
  const uint32_t tree = (uint32_t)(big ? T - 1 : t);
  return handed_out(s, malloc_slices<NAMED>(s, tree, count, members, cache), size);
}

// Gallatin::malloc as the reference calls it: each attempt's team is the lanes
// executing it together (its coalesced_threads(), gallatin.cuh:883).
GAL_DEVICE_INLINE void *malloc(const state *s, uint64_t size) {
  return malloc_from<false>(resident(s), size, active_lanes());
}

// malloc for kernels whose CTAs serve many requests (persistent loops): the
// teams take the pinned block from the CTA's slot_cache in shared memory and
// read the pinned slot in global memory only when the copy has gone stale, so
// a team's claim costs one L2 round trip instead of two.  Same results
// contract as malloc.
GAL_DEVICE_INLINE void *malloc_cached(const state *s, uint64_t size, slot_cache &cache) {
  return malloc_from<false>(resident(s), size, active_lanes(), &cache);
}

// malloc with the calling lanes named: every lane of `callers` calls with the
// same mask (the contract of the *_sync warp intrinsics), and the lanes asking
// for slices of one class form one team whatever grouping of diverged lanes
// the scheduler chose.
GAL_DEVICE_INLINE void *malloc_team(const state *s, uint64_t size, uint32_t callers) {
  return malloc_from<true>(resident(s), size, callers);
}

// multi-segment free (gallatin.cuh:1394-1417, 1283-1302), id reset first
GAL_DEVICE_COLD void free_segment_run(const state *s, uint64_t seg, uint16_t tree) {
  uint32_t count = (uint32_t)tree - cfield(s->num_trees) - 1;
  if (cas16(&cfield(s->tree_ids)[seg], tree, FREE_TREE) != tree) {
    set_error_info(s, GAL_DEV_ERR_BAD_FREE, SITE_FREE_RUN_TWICE, seg, tree);
    return;
  }
  __threadfence();
  veb_return_multiple(seg_tree(s), seg, count);
}

// Gallatin::free (gallatin.cuh:1378-1461)
GAL_DEVICE_INLINE void free(const state *s, void *ptr) {
  s = resident(s);
  uint64_t off = (uint64_t)((char *)ptr - cfield(s->memory));
  uint64_t seg = off >> cfield(s->seg_shift);
  if (seg >= cfield(s->num_segments)) {
    set_error_info(s, GAL_DEV_ERR_BAD_FREE, SITE_FREE_OUTSIDE, off, 0);
    return;
  }
  uint16_t tree = ld_rlx(&cfield(s->tree_ids)[seg]);
  if (tree >= cfield(s->num_trees)) {
    if (tree == FREE_TREE || tree == cfield(s->num_trees)) {
      set_error_info(s, GAL_DEV_ERR_BAD_FREE, SITE_FREE_FREE_SEGMENT, off, tree);
      return;
    }
    free_segment_run(s, seg, tree);
    return;
  }
  uint64_t in_seg = off & ((1ull << cfield(s->seg_shift)) - 1ull);
  uint32_t blk = (uint32_t)(seg << cfield(s->bps_shift)) + (uint32_t)(in_seg >> (cfield(s->min_shift) + tree + 12));
  free_block_slices(s, blk);
}

// free of a live pointer whose request size the caller knows: a slice's class
// follows from the size, so the pointer's segment need not be looked up (the
// first of free's two dependent round trips).
GAL_DEVICE_INLINE void free_sized(const state *s, void *ptr, uint64_t size) {
  s = resident(s);
  const int T = (int)cfield(s->num_trees), min_shift = (int)cfield(s->min_shift);
  const int bits = size > 1 ? 64 - __clzll((long long)(size - 1)) : 0;
  const int t = max(bits - min_shift, 0);
  if (t >= T && bits >= min_shift + 12) {  // a block or segments
    gal::free(s, ptr);
    return;
  }
  const uint64_t off = (uint64_t)((char *)ptr - cfield(s->memory));
  const uint64_t in_seg = off & ((1ull << cfield(s->seg_shift)) - 1ull);
  free_block_slices(s, (uint32_t)((off >> cfield(s->seg_shift)) << cfield(s->bps_shift)) +
                           (uint32_t)(in_seg >> (min_shift + min(t, T - 1) + 12)));
}

// block id of a live pointer (slice or whole block), NOBLK for a segment run
GAL_DEVICE_INLINE uint32_t block_of(const state *s, const void *ptr, uint16_t &tree_out) {
  s = resident(s);
  uint64_t off = (uint64_t)((const char *)ptr - cfield(s->memory));
  uint64_t seg = off >> cfield(s->seg_shift);
  uint16_t tree = seg < cfield(s->num_segments) ? ld_rlx(&cfield(s->tree_ids)[seg]) : FREE_TREE;
  tree_out = tree;
  if (tree >= cfield(s->num_trees)) return NOBLK;
  uint64_t in_seg = off & ((1ull << cfield(s->seg_shift)) - 1ull);
  return (uint32_t)(seg << cfield(s->bps_shift)) + (uint32_t)(in_seg >> (cfield(s->min_shift) + tree + 12));
}

// Frees the pointers p[k] with go[k] set, as N calls of free() would, but
// with their table lookups and their free-counter atomics each issued back to
// back so the round trips overlap.  Warp teams form per k, as in free().
// `classes`, when given, is a copy of tree_ids taken after every pointer
// passed was allocated (see stage_classes); a live pointer's segment keeps
// its class, so the copy answers the lookup without a trip to L2.
template <int N>
GAL_DEVICE_INLINE void free_n(const state *s, void *const (&p)[N], const bool (&go)[N],
                              const uint16_t *classes = nullptr) {
  s = resident(s);
  uint16_t tree[N];
  uint64_t off[N];
#pragma unroll
  for (int k = 0; k < N; k++) {
    tree[k] = FREE_TREE;
    off[k] = go[k] ? (uint64_t)((char *)p[k] - cfield(s->memory)) : 0;
    if (go[k] && (off[k] >> cfield(s->seg_shift)) < cfield(s->num_segments))
      tree[k] = classes ? classes[off[k] >> cfield(s->seg_shift)] : ld_rlx(&cfield(s->tree_ids)[off[k] >> cfield(s->seg_shift)]);
  }
  uint32_t blk[N], old[N], cnt[N];
  bool lead[N];
#pragma unroll
  for (int k = 0; k < N; k++) {
    lead[k] = false;
    blk[k] = NOBLK;
    if (!go[k]) continue;
    if (tree[k] >= cfield(s->num_trees)) {  // segment runs and bad pointers: the scalar path
      gal::free(s, p[k]);
      continue;
    }
    uint64_t in_seg = off[k] & ((1ull << cfield(s->seg_shift)) - 1ull);
    blk[k] = (uint32_t)((off[k] >> cfield(s->seg_shift)) << cfield(s->bps_shift)) +
             (uint32_t)(in_seg >> (cfield(s->min_shift) + tree[k] + 12));
  }
#pragma unroll
  for (int k = 0; k < N; k++) {
    if (blk[k] == NOBLK) continue;
    const uint32_t active = active_lanes();
    const uint32_t team = __match_any_sync(active, blk[k]) & team_group(s);
    lead[k] = (int)lane_id() == __ffs(team) - 1;
    cnt[k] = (uint32_t)__popc(team);
    if (lead[k]) old[k] = atomicAdd(fctr_ptr(s, blk[k]), cnt[k]);
  }
#pragma unroll
  for (int k = 0; k < N; k++)
    if (lead[k]) credit_done(s, blk[k], old[k], cnt[k]);
}

// Segments whose classes fit in CLASS_STAGE_BYTES of shared memory can be
// staged for free_n: every thread of the CTA calls stage_classes, then
// __syncthreads().  Returns false (nothing staged) for larger arenas.
static constexpr uint32_t CLASS_STAGE_BYTES = 32768;
GAL_DEVICE_INLINE bool stage_classes(const state *s, uint16_t *smem) {
  s = resident(s);
  if (cfield(s->num_segments) * 2 > CLASS_STAGE_BYTES) return false;
  for (uint64_t g = threadIdx.x; g < cfield(s->num_segments); g += blockDim.x) smem[g] = ld_rlx(&cfield(s->tree_ids)[g]);
  return true;
}

// a block's malloc word in the reference packing, (tree << 20) + count (block.cuh:53,220)
GAL_DEVICE_INLINE uint32_t export_mword(const state *s, uint32_t blk) {
  const unsigned long long w = *mword_ptr(s, blk);
  return (uint32_t)(((w >> 32) << 20) + (w & 0xFFFFFFFFull));
}

// bytes a request of `size` occupies (Gallatin::get_allocated_size, gallatin.cuh:1152-1183)
GAL_DEVICE_INLINE uint64_t allocated_size(const state *s, uint64_t size) {
  s = resident(s);
  if (size < 16) size = 16;
  int bits = ceil_log2(size);
  int tree = bits - (int)cfield(s->min_shift);
  if (tree > (int)cfield(s->num_trees)) {
    int block_tree = bits - (int)(cfield(s->min_shift) + 12);
    if (block_tree > (int)cfield(s->num_trees)) return (((size - 1) >> cfield(s->seg_shift)) + 1) << cfield(s->seg_shift);
  }
  return 1ull << bits;
}

GAL_DEVICE_INLINE bool owns(const state *s, const void *p) {
  s = resident(s);
  return (uint64_t)((const char *)p - cfield(s->memory)) < (cfield(s->num_segments) << cfield(s->seg_shift));
}

}  // namespace gal
