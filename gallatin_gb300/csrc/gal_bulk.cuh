// gal_bulk.cuh — the batched kernels: a CTA serves a chunk of requests with one
// claim per size class, and frees a chunk of pointers with one atomic per block.
//
// One thread per request with warp teams (gal::malloc) makes a slot read and a
// claim atomic per class and warp, a dependent chain of round trips that every
// warp repeats and that every block replacement on its SM holds up.  Here a CTA
// ranks its requests per class in shared memory, one warp per class claims all
// of the class's slices, and every thread computes its pointers: one chain per
// chunk.  Whole blocks are taken directly for every 4,096 slices a class needs;
// only the rest goes through the pinned slot.  A claim that crosses the end of
// the pinned block takes its missing slices from the next block before that
// block is installed.  Bound by the block requests of the claims that cross
// (two to five round trips of 700-800 cycles each, more where many CTAs ask one
// class together) and by the refills of the spares behind them: of the 31 us of
// 1 Mi mixed requests 6 load and rank, 8 claim and store, the rest waits for
// refills.  4 Mi mixed requests: 98 -> 67 us against one request per thread.
#pragma once

#include "../../include/gallatin_gb300/gal_device.cuh"

namespace gal {

static constexpr int BULK_THREADS = 512;  // a warp for each of GAL_MAX_TREES classes
static constexpr int BULK_RUNS = 24;      // block runs a class may use per chunk
static constexpr int BULK_ATTEMPTS = 64;
static_assert(BULK_THREADS / 32 >= GAL_MAX_TREES, "one warp claims for each class");

struct bulk_smem {
  uint32_t want[GAL_MAX_TREES];  // slices asked for, by class
  uint32_t nruns[GAL_MAX_TREES];
  char *at[GAL_MAX_TREES][BULK_RUNS];  // first slice of the run
  uint32_t len[GAL_MAX_TREES][BULK_RUNS];
  uint32_t last_blk[BULK_RUNS];  // the last class's blocks
  uint32_t credit[BULK_RUNS];    // frees owed to the last class's runs (multi-slice requests)
};

// One thread claims `want` slices of class `tree` and records the runs it got
// (they may add up to less: no block to be had, or too many runs).  Returns the
// slot whose spare is to be refilled once the slices are in use (NOBLK: none).
GAL_DEVICE_COLD uint32_t bulk_claim(const state *s, uint32_t tree, uint32_t want, bulk_smem &sm) {
  const uint32_t tid = (uint32_t)thread_linear_id();
  uint32_t n = 0, refill = NOBLK;
  // takes up to `need` slices of a block, installed or not; false: none of them
  // are this class's to use.  A block read in an earlier life may be claimed
  // from by a slow team at any time, so every take is an atomic on its count.
  // crossed: nothing is left of the block and this thread is to replace it.
  uint32_t crossed = 0, rest = want;
  auto take = [&](uint32_t blk, uint32_t need) {
    const unsigned long long old = atomicAdd(mword_ptr(s, blk), (unsigned long long)need);
    const uint32_t cnt = (uint32_t)old;
    crossed = 0;
    if (cnt >= SLICES_PER_BLOCK) return false;
    const uint32_t got = min(need, SLICES_PER_BLOCK - cnt);
    if ((uint32_t)(old >> 32) != tree) {  // recycled for another class since it was read
      credit_frees(s, blk, got);
      return false;
    }
    crossed = cnt + need > SLICES_PER_BLOCK - 1;
    sm.at[tree][n] = slice_ptr(s, blk, cnt, tree);
    if (tree == s->num_trees - 1) sm.last_blk[n] = blk;
    sm.len[tree][n] = got;
    n++;
    rest -= got;
    return true;
  };
  for (int attempt = 0; attempt < BULK_ATTEMPTS && rest >= SLICES_PER_BLOCK && n < (uint32_t)BULK_RUNS; attempt++) {
    const uint32_t blk = request_block(s, tree, tid);
    if (blk == NOBLK) break;
    take(blk, SLICES_PER_BLOCK);  // all that is left of it: it never enters a slot
  }
  uint32_t refused = NOBLK, refusals = 0;  // the exhausted block last met, and how often in a row
  for (int attempt = 0; attempt < BULK_ATTEMPTS && rest && rest < SLICES_PER_BLOCK && n < (uint32_t)BULK_RUNS;
       attempt++) {
    uint32_t blk;
    const uint32_t slot = pick_slot(s, tree, blk);
    if (blk == NOBLK || blk == refused || !take(blk, rest)) {
      // empty or exhausted: its crosser is installing the next block.  (A block
      // met again is only looked at, as every take adds to its count.)
      refusals = blk != NOBLK && blk == refused ? refusals + 1u : 0u;
      refused = blk;
      if (refusals < (uint32_t)STUCK_ATTEMPTS || (uint32_t)ld_rlx(mword_ptr(s, blk)) < SLICES_PER_BLOCK) {
        if (refusals >= (uint32_t)STUCK_ATTEMPTS) refused = NOBLK;  // it is a block to claim from again
        __nanosleep(blk == NOBLK ? 200u : 100u);
        continue;
      }
      refused = NOBLK;  // nobody replaces it (see STUCK_ATTEMPTS): done here
    } else {
      refused = NOBLK;
      if (!crossed) continue;
    }
    const uint32_t at = s->slot_base[tree] + slot;
    uint32_t next = s->use_spares ? atomicExch(s->spares + at, NOBLK) : NOBLK;
    if (s->use_spares) {
      if (refill != NOBLK && refill != slot) refill_spare(s, tree, refill, tid);  // of a slot crossed before
      refill = slot;
    }
    const uint32_t found = next != NOBLK ? blk : NOBLK;  // what the slot holds until the next block is in
    if (next == NOBLK && atomicCAS(s->slots + at, blk, NOBLK) != blk) continue;
    uint64_t asked = ~0ull;  // nothing to finish
    for (int tries = 0; tries < BLOCK_ATTEMPTS; tries++) {
      if (next == NOBLK) {
        asked = request_block_begin(s, tree, tid);
        next = requested_block(asked);
        if (next == NOBLK) break;
      }
      if (!rest || n >= (uint32_t)BULK_RUNS || (take(next, rest) && !crossed)) break;
      // slow teams and this claim have used it up: not a block for the slot
      request_done(s, tree, asked);
      asked = ~0ull;
      next = NOBLK;
    }
    if (next == NOBLK) {  // no block to be had: the slot is left empty
      if (found != NOBLK) atomicCAS(s->slots + at, found, NOBLK);
      break;
    }
    fence_acq_rel();
    if (atomicCAS(s->slots + at, found, next) != found) {  // the slot moved on
      if (found == NOBLK) set_error(s, GAL_DEV_ERR_SLOT_SWAP);
      retire_block(s, next);
    }
    request_done(s, tree, asked);
  }
  sm.nruns[tree] = n;
  return refill;
}

// Requests the claims do not serve, out of line.
GAL_DEVICE_COLD void *bulk_fallback(const state *s, uint64_t size) { return gal::malloc(s, size); }

// out[i] = malloc(sizes[i]) for the CTA's K x BULK_THREADS requests from
// `base` on (fewer at the end of the list).  ZERO: calloc mode.  `out` may be
// `sizes`: a size is read again only before its pointer is written.
template <int K, bool ZERO>
__device__ __forceinline__ void bulk_malloc(const state *s, const uint64_t *sizes, uint64_t n, uint64_t base,
                                            void **out, bulk_smem &sm) {
  const int T = (int)cfield(s->num_trees), min_shift = (int)cfield(s->min_shift);
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5, lt = lanemask_lt();
  if (threadIdx.x < GAL_MAX_TREES) sm.want[threadIdx.x] = 0;
  if (threadIdx.x < BULK_RUNS) sm.credit[threadIdx.x] = 0;
  const uint64_t i0 = base + threadIdx.x;
  // each request's class and, for the last class, log2 of its slices
  uint64_t size[K];
#pragma unroll
  for (int k = 0; k < K; k++) {
    const uint64_t i = i0 + (uint64_t)k * BULK_THREADS;
    size[k] = sizes[i < n ? i : base];  // no branch: the loads go out together
  }
  uint32_t pos[K];
  uint32_t cls[K], lg[K];
  constexpr uint32_t NONE = 0x1F, OTHER = 0x1E;  // no request; a block or segments
#pragma unroll
  for (int k = 0; k < K; k++) {
    const int bits = size[k] > 1 ? 64 - __clzll((long long)(size[k] - 1)) : 0;  // ceil(log2)
    const int t = max(bits - min_shift, 0);
    const bool mine = i0 + (uint64_t)k * BULK_THREADS < n, slices = t < T || bits < min_shift + 12;
    cls[k] = !mine ? NONE : slices ? (uint32_t)min(t, T - 1) : OTHER;
    lg[k] = mine && slices && t >= T ? (uint32_t)(t - (T - 1)) : 0u;
  }
  __syncthreads();
  bool multi = false;
#pragma unroll
  for (int k = 0; k < K; k++) {
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, cls[k]);
    uint32_t before = (uint32_t)__popc(peers & lt), all = (uint32_t)__popc(peers);
    if (__any_sync(0xFFFFFFFFu, lg[k] != 0)) {  // runs of slices: sums in place of counts
      multi = true;
      const uint32_t mine = cls[k] == (uint32_t)(T - 1) ? 1u << lg[k] : 0u;
      uint32_t upto = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, upto, o);
        if ((int)lane >= o) upto += v;
      }
      const uint32_t sum = __shfl_sync(0xFFFFFFFFu, upto, 31);
      if (mine) {
        before = upto - mine;
        all = sum;
      }
    }
    const int leader = __ffs(peers) - 1;
    uint32_t at = 0;
    if ((int)lane == leader && cls[k] < GAL_MAX_TREES) at = atomicAdd(&sm.want[cls[k]], all);
    pos[k] = __shfl_sync(0xFFFFFFFFu, at, leader) + before;
  }
  __syncthreads();
  uint32_t refill = NOBLK;
  const uint32_t want = (int)warp < T ? sm.want[warp] : 0u;
  if (want && lane == 0) refill = bulk_claim(s, warp, want, sm);
  __syncthreads();
  uint32_t unserved = 0;  // requests k left to the per-thread path
#pragma unroll
  for (int k = 0; k < K; k++) {
    if (cls[k] == NONE) continue;
    void *p = nullptr;
    if (cls[k] != OTHER) {
      const uint32_t t = cls[k], c = 1u << lg[k];
      const uint32_t runs = sm.nruns[t];
      uint32_t r = pos[k], j = 0;
      while (j < runs && r >= sm.len[t][j]) r -= sm.len[t][j++];
      if (j < runs && r + c <= sm.len[t][j]) {
        p = sm.at[t][j] + ((uint64_t)r << (min_shift + t));
        if (c > 1) atomicAdd(&sm.credit[j], c - 1u);  // one free comes back for the whole run
      } else if (c > 1) {
        // its slices are spread over runs: each part goes back where it came from
        for (uint32_t left = c; left && j < runs; j++, r = 0) {
          const uint32_t part = min(left, sm.len[t][j] - r);
          atomicAdd(&sm.credit[j], part);
          left -= part;
        }
      }
    }
    if (!p) {
      unserved |= 1u << k;
      continue;
    }
    const uint64_t i = i0 + (uint64_t)k * BULK_THREADS;
    if (ZERO) zero_fill(p, sizes[i]);
    out[i] = p;
  }
  // before the fallback, whose waits must not hold up what others wait for
  if (refill != NOBLK) refill_spare(s, warp, refill, (uint32_t)thread_linear_id());
  for (; unserved; unserved &= unserved - 1u) {
    const uint64_t i = i0 + (uint64_t)(__ffs(unserved) - 1) * BULK_THREADS;
    out[i] = bulk_fallback(s, sizes[i]);  // clears its own bytes in calloc mode
  }
  if (__syncthreads_or(multi) && (int)warp == T - 1 && lane < sm.nruns[warp] && sm.credit[lane])
    credit_frees(s, sm.last_blk[lane], sm.credit[lane]);
}

// ------------------------------------------------------------------ frees
// Warp teams per block (gal::free_n) made eight atomics for the 32 neighbours of
// a mixed list and left the blocks that completed to a few lanes, one five-step
// return after the other: the SMs were busy for 41 % of the kernel's time.  A CTA
// counts its pointers by block in shared memory instead, and the blocks are
// credited by different warps.  Bound by the returns of the last blocks (4 Mi
// mixed pointers: 63 -> 33 us, of which reading the list takes 5).
static constexpr int BULK_FREE_THREADS = 256;

// A CTA's chunk of pointers (K per thread) by block: a hash table of (block,
// frees), half full at most, and the list of its used places.
template <int K>
struct bulk_free_smem {
  static constexpr uint32_t CHUNK = BULK_FREE_THREADS * K, SLOTS = 2 * CHUNK;
  uint32_t blk[SLOTS];
  uint32_t frees[SLOTS];
  uint16_t used[CHUNK];
  uint32_t nused;
};

template <int K>
__device__ __forceinline__ void bulk_free_init(bulk_free_smem<K> &sm) {
  for (uint32_t i = threadIdx.x; i < sm.SLOTS; i += BULK_FREE_THREADS) {
    sm.blk[i] = NOBLK;
    sm.frees[i] = 0;
  }
  if (threadIdx.x == 0) sm.nused = 0;
}

// Frees the chunk of ptrs[0, n) at `base` (nullptr: nothing), one free-counter
// atomic per block it touches; `classes`: a copy of tree_ids (stage_classes) or
// nullptr.  Called by the whole CTA, the table empty before and after.
template <int K>
__device__ __forceinline__ void bulk_free(const state *s, void *const *ptrs, uint64_t n, uint64_t base,
                                          const uint16_t *classes, bulk_free_smem<K> &sm) {
  constexpr uint32_t SLOTS = bulk_free_smem<K>::SLOTS;
  const uint64_t i0 = base + threadIdx.x;
  const uint64_t segments = cfield(s->num_segments);
  const uint32_t T = cfield(s->num_trees), seg_shift = cfield(s->seg_shift), bps_shift = cfield(s->bps_shift);
  const uint32_t to_block = cfield(s->min_shift) + 12u;
  char *const memory = cfield(s->memory);
  char *p[K];
#pragma unroll
  for (int k = 0; k < K; k++) {
    const uint64_t i = i0 + (uint64_t)k * BULK_FREE_THREADS;
    p[k] = i < n ? (char *)ptrs[i] : nullptr;
  }
  uint32_t scalar = 0;  // pointers k that are no slices or blocks
#pragma unroll
  for (int k = 0; k < K; k++) {
    if (!p[k]) continue;
    const uint64_t off = (uint64_t)(p[k] - memory), seg = off >> seg_shift;
    uint32_t tree = FREE_TREE;
    if (seg < segments) tree = classes ? classes[seg] : ld_rlx(&cfield(s->tree_ids)[seg]);
    if (tree >= T) {
      scalar |= 1u << k;
      continue;
    }
    const uint64_t in_seg = off & ((1ull << seg_shift) - 1ull);
    const uint32_t blk = ((uint32_t)seg << bps_shift) + (uint32_t)(in_seg >> (to_block + tree));
    uint32_t h = (blk * 2654435761u) >> 7 & (SLOTS - 1u);
    for (;;) {  // the table holds at most one block per pointer: half its places
      uint32_t found = *(volatile uint32_t *)&sm.blk[h];
      if (found == NOBLK) {
        found = atomicCAS(&sm.blk[h], NOBLK, blk);
        if (found == NOBLK) {
          sm.used[atomicAdd(&sm.nused, 1u)] = (uint16_t)h;
          found = blk;
        }
      }
      if (found == blk) break;
      h = (h + 1u) & (SLOTS - 1u);
    }
    atomicAdd(&sm.frees[h], 1u);
  }
  __syncthreads();
  // the used places, neighbours to different warps: a block that completes is
  // returned (five round trips) beside the others, not after them
  const uint32_t nused = sm.nused;
  constexpr uint32_t WARPS = BULK_FREE_THREADS / 32;
  for (uint32_t e = (threadIdx.x & 31u) * WARPS + (threadIdx.x >> 5); e < nused; e += BULK_FREE_THREADS) {
    const uint32_t h = sm.used[e], blk = sm.blk[h], c = sm.frees[h];
    sm.blk[h] = NOBLK;
    sm.frees[h] = 0;
    credit_frees(s, blk, c);
  }
  for (; scalar; scalar &= scalar - 1u)  // segment runs and bad pointers
    gal::free(s, ptrs[i0 + (uint64_t)(__ffs(scalar) - 1) * BULK_FREE_THREADS]);
  __syncthreads();
  if (threadIdx.x == 0) sm.nused = 0;
  __syncthreads();
}

}  // namespace gal
