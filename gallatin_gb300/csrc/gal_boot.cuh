// gal_boot.cuh — booting and retiring the pinned slots with one CTA.
//
// The reference boots its slots one after another with one thread
// (boot_shared_block_container_one_thread, gallatin.cuh:196-221), and that
// order fixes which block every slot gets.  With one slot per SM in nine
// classes it is 1,368 block requests in a chain: 11.9 ms for a trim at one slot
// per SM (21.3 ms before the requests themselves were made cheaper).  Here the
// same end state is computed in parallel by 1,024 threads in 42 us; bound by
// the thirty dependent round trips of its phases (retiring 14, releases 10,
// booting 18).
//
//   * Blocks of one segment must come home in slot order (their ring entries);
//     blocks of different segments have nothing in common but bits of the
//     trees, whose end state does not depend on the order.  So spares and slots
//     are retired 3,072 at a time, each thread finding how many earlier blocks
//     of the same segment come home with its own.
//   * A class whose tree lists no segment boots from fresh segments only: slot
//     i gets block i mod nb of the class's (i / nb)-th gathered segment, and the
//     segments gathered, class by class, are the smallest free ids in order.
//     (Segment 0 gives its class one block only when the hashed search never
//     starts at 0: listed alone, it is then not found.)  Such classes are
//     booted together.  A class that still lists segments
//     (live allocations hold some of their blocks), whose lock is held, or
//     that needs more segments than are free takes the one-thread loop, which
//     stays the definition of the order.
#pragma once

#include "../../include/gallatin_gb300/gal_device.cuh"

namespace gal {

static constexpr int BOOT_THREADS = 1024;
static constexpr int BOOT_WARPS = BOOT_THREADS / 32;

static constexpr int RETIRE = 3;  // spares and slots a thread retires at a time

struct boot_smem {
  // retire: (row, segment, blocks), one per segment a warp completed blocks of
  unsigned long long done[RETIRE * BOOT_THREADS];
  uint16_t before[RETIRE * BOOT_THREADS];  // of an entry's segment in earlier rows ...
  uint16_t all[RETIRE * BOOT_THREADS];     // ... and in all
  uint32_t ndone, nclose;
  uint32_t scan[BOOT_WARPS];
  uint16_t list[BOOT_THREADS];     // boot: the gathered segments of a tile
  uint32_t fast[GAL_MAX_TREES];    // the class lists no segment and its lock is free
  uint32_t first[GAL_MAX_TREES + 1];
  uint32_t lone[GAL_MAX_TREES];    // the class would lose segment 0 (finds_lone_zero)
};

// Whether veb_find_random finds segment 0 when its tree lists nothing else: it
// is at or above no start but 0, and the search after the starts is above 0.
static __device__ bool finds_lone_zero(const state *s, uint32_t t) {
  if (s->policy == GAL_POLICY_LOWEST) return true;
  const uint64_t U = s->num_segments;
  const bool pow2 = (U & (U - 1)) == 0;
  const uint64_t h1 = murmur64a_u64(0, s->seed + t);
  const uint64_t h2 = murmur64a_u64(0, h1);
  for (uint64_t a = 0; a < (uint64_t)VEB_ATTEMPTS; a++)
    if ((pow2 ? (h1 + a * h2) & (U - 1) : (h1 + a * h2) % U) == 0) return true;
  return false;
}
// Segments that n blocks of class t take, `lone` of them from segment 0
static __device__ uint32_t boot_segments(const state *s, uint32_t t, uint32_t n, uint32_t lone) {
  const uint32_t nb = blocks_in_segment(s, t);
  const uint32_t shift = (uint32_t)__ffs(nb) - 1u;
  n -= lone;
  if (lone && n == 0) return 1;
  return lone + (s->gather_ahead ? (n >> shift) + 1u : (n + nb - 1u) >> shift);
}

// blk[k] of thread i is the (k * BOOT_THREADS + i)-th block of a tile, in the
// order in which one thread would retire them (NOBLK: none): what as many
// retire_block calls do.
static __device__ void retire_tile(const state *s, const uint32_t (&blk)[RETIRE], boot_smem &sm) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, lt = lanemask_lt();
  uint32_t handed_out[RETIRE], freed[RETIRE], seg[RETIRE], returned[RETIRE], same[RETIRE];
  uint32_t entry[RETIRE];
  uint16_t tree[RETIRE];
  bool home[RETIRE];
  if (threadIdx.x == 0) sm.ndone = 0;
#pragma unroll
  for (int k = 0; k < RETIRE; k++)
    handed_out[k] = blk[k] == NOBLK
                        ? SLICES_PER_BLOCK
                        : (uint32_t)atomicAdd(mword_ptr(s, blk[k]), (unsigned long long)SLICES_PER_BLOCK);
#pragma unroll
  for (int k = 0; k < RETIRE; k++)
    freed[k] = handed_out[k] < SLICES_PER_BLOCK ? atomicAdd(fctr_ptr(s, blk[k]), SLICES_PER_BLOCK - handed_out[k]) : 0u;
#pragma unroll
  for (int k = 0; k < RETIRE; k++) {
    const uint32_t n = SLICES_PER_BLOCK - min(handed_out[k], SLICES_PER_BLOCK);
    home[k] = n && freed[k] + n == SLICES_PER_BLOCK;
    seg[k] = home[k] ? blk[k] >> s->bps_shift : 0u;
    tree[k] = home[k] ? ld_rlx(&s->tree_ids[seg[k]]) : FREE_TREE;
    returned[k] = home[k] ? ld_rlx(&s->qfc[seg[k]]) : 0u;
    if (n && freed[k] + n > SLICES_PER_BLOCK)
      set_error_info(s, GAL_DEV_ERR_BAD_FREE, SITE_FREE_OVERFLOW, blk[k], ((uint64_t)freed[k] << 32) | n);
  }
  __syncthreads();  // ndone
#pragma unroll
  for (int k = 0; k < RETIRE; k++) {
    if (home[k]) st_rlx(fctr_ptr(s, blk[k]), 0u);
    if (home[k] && tree[k] >= s->num_trees) {
      set_error_info(s, GAL_DEV_ERR_BAD_FREE, SITE_RETURN_BAD_TREE, blk[k], tree[k]);
      home[k] = false;
    }
    // a warp's blocks by segment; the first lane of each segment speaks for it
    same[k] = __match_any_sync(0xFFFFFFFFu, home[k] ? seg[k] : 0xFFFFFFFFu);
    entry[k] = ~0u;
    if (home[k] && (int)lane == __ffs(same[k]) - 1) {
      entry[k] = atomicAdd(&sm.ndone, 1u);
      sm.done[entry[k]] = (unsigned long long)(k * BOOT_WARPS + warp) << 32 | seg[k] << 16 | (uint32_t)__popc(same[k]);
    }
  }
  __syncthreads();  // also: every thread has read its segments' return positions
  // a thread per entry, not per lane that made one: a hundred entries keep four
  // warps at this, where every warp at its own took 15 us
  const uint32_t ndone = sm.ndone;
  for (uint32_t i = threadIdx.x; i < ndone; i += BOOT_THREADS) {
    const unsigned long long own = sm.done[i];
    uint32_t before = 0, all = 0;
#pragma unroll 4
    for (uint32_t e = 0; e < ndone; e++) {
      const unsigned long long d = sm.done[e];
      const uint32_t n = ((uint32_t)(d ^ own) >> 16) == 0 ? (uint32_t)d & 0xFFFFu : 0u;
      all += n;
      if ((d >> 32) < (own >> 32)) before += n;
    }
    sm.before[i] = (uint16_t)before;
    sm.all[i] = (uint16_t)all;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < RETIRE; k++) {
    const uint32_t before = entry[k] != ~0u ? sm.before[entry[k]] : 0u;
    const uint32_t rank = __shfl_sync(0xFFFFFFFFu, before, __ffs(same[k]) - 1) + (uint32_t)__popc(same[k] & lt);
    if (home[k]) {
      const uint32_t nb = blocks_in_segment(s, tree[k]);
      const uint32_t live = (returned[k] + rank) & (nb - 1u);
      st_rlx(s->queues + ((uint64_t)seg[k] << s->bps_shift) + live, blk[k]);
      if (live != 0 && 10ull * live > nb && 10ull * (live - 1) < nb) veb_insert(sub_tree(s, tree[k]), seg[k]);
    }
  }
  if (threadIdx.x == 0) sm.nclose = 0;
  fence_acq_rel();
  __syncthreads();  // also: done is read
  // the first of a segment settles its counters: listed, so that every thread
  // has one (a release is a chain of some ten round trips)
#pragma unroll
  for (int k = 0; k < RETIRE; k++)
    if (entry[k] != ~0u && sm.before[entry[k]] == 0)
      sm.done[atomicAdd(&sm.nclose, 1u)] = (unsigned long long)tree[k] << 32 | seg[k] << 16 | sm.all[entry[k]];
  __syncthreads();
  for (uint32_t e = threadIdx.x; e < sm.nclose; e += BOOT_THREADS) {
    const unsigned long long d = sm.done[e];
    const uint32_t t = (uint32_t)(d >> 32), g = (uint32_t)d >> 16, n = (uint32_t)d & 0xFFFFu;
    const uint32_t nb = blocks_in_segment(s, t);
    atomicAdd(&s->qfc[g], n);
    atomicAdd(&s->fqfc[g], n);
    const unsigned long long old = atomicAdd(&s->act[g], (unsigned long long)n);
    if (act_count(old) + (int32_t)n == (int32_t)nb - 1) release_segment(s, g, t, act_gen(old), nb, NOSEG);
  }
  __syncthreads();
}

// every spare and pinned block, spares first; the words are left empty
static __device__ void retire_all(const state *s, boot_smem &sm) {
  const uint32_t n = s->total_slots;
  for (uint32_t base = 0; base < 2 * n; base += RETIRE * BOOT_THREADS) {
    uint32_t blk[RETIRE];
#pragma unroll
    for (int k = 0; k < RETIRE; k++) {
      const uint32_t i = base + k * BOOT_THREADS + threadIdx.x;
      blk[k] = i < n ? atomicExch(s->spares + i, NOBLK) : i < 2 * n ? atomicExch(s->slots + (i - n), NOBLK) : NOBLK;
    }
    retire_tile(s, blk, sm);
  }
}

// A fresh segment of class t, its first `taken` blocks given to the slots from
// `slot` on: what setup_begin, setup_open and `taken` get_block calls leave, in two steps
// with a fence between them (full warp; false: listed free, yet owned).
static __device__ bool boot_segment(const state *s, uint32_t seg, uint32_t t, uint32_t slot, uint32_t taken) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t nb = blocks_in_segment(s, t);
  if (ld_rlx(&s->tree_ids[seg]) != FREE_TREE) {
    if (lane == 0) {
      set_error(s, GAL_DEV_ERR_SEGMENT_SETUP);
      if (taken) set_error(s, GAL_DEV_ERR_BOOT);
    }
    return false;
  }
  const uint32_t blk0 = seg << s->bps_shift;
  for (uint32_t i = lane; i < nb; i += 32) st_rlx(s->queues + blk0 + i, NOBLK);
  for (uint32_t i = lane; i < taken; i += 32) {
    st_rlx(mword_ptr(s, blk0 + i), (unsigned long long)t << 32);
    st_rlx(s->slots + s->slot_base[t] + slot + i, blk0 + i);
  }
  if (lane == 0) {
    st_rlx(&s->tree_ids[seg], (uint16_t)t);
    st_rlx(&s->qc[seg], taken);
    st_rlx(&s->qfc[seg], 0u);
    st_rlx(&s->fqfc[seg], 0u);
  }
  return true;
}
static __device__ void boot_open(const state *s, uint32_t seg, uint32_t t, uint32_t taken) {
  atomicAdd(&s->act[seg], ((unsigned long long)(t + 1u) << 32) + blocks_in_segment(s, t) - taken);  // see setup_open
  if (taken < blocks_in_segment(s, t)) veb_insert(sub_tree(s, t), seg);
}

// Boots every slot (all empty) in the one-thread order.  One CTA of
// BOOT_THREADS, no device malloc or free in flight.
static __device__ void boot_all(const state *s, boot_smem &sm) {
  const uint32_t T = s->num_trees, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const veb_ref segs = seg_tree(s);
  const uint32_t nwords = s->veb.nwords[s->veb.layers - 1];  // at most 1,024: 65,532 segments
  uint64_t *bottom = veb_bottom(segs);
  if (threadIdx.x >= 32 && threadIdx.x < 32 + T) {
    const uint32_t t = threadIdx.x - 32;
    sm.lone[t] = blocks_in_segment(s, t) > 1 && !finds_lone_zero(s, t);
  }
  if (threadIdx.x < T)
    sm.fast[threadIdx.x] = ld_rlx(sub_tree(s, threadIdx.x).w) == 0 && ld_rlx(s->locks + threadIdx.x * LOCK_STRIDE) == 0;
  __syncthreads();
  for (uint32_t t0 = 0; t0 < T;) {
    uint32_t t1 = t0;  // classes [t0, t1) are booted together
    while (t1 < T && sm.fast[t1]) t1++;
    // free segments below this thread's word
    const uint64_t word = t1 > t0 && threadIdx.x < nwords ? ld_rlx(bottom + threadIdx.x) : 0ull;
    if (warp == 0) {  // the classes' first gathered segments: lane t's class, summed in order
      const bool mine = lane >= t0 && lane < t1;
      const uint32_t lone0 = (uint32_t)(__shfl_sync(0xFFFFFFFFu, word, 0) & 1ull) && t1 > t0 ? sm.lone[t0] : 0u;
      const uint32_t n = mine ? boot_segments(s, lane, s->slot_count[lane], lane == t0 ? lone0 : 0u) : 0u;
      uint32_t upto = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, upto, o);
        if ((int)lane >= o) upto += v;
      }
      if (mine) sm.first[lane] = upto - n;
      if (mine && lane == t1 - 1) sm.first[t1] = upto;
      if (lane == 0) sm.lone[t0] = lone0;
    }
    uint32_t below = (uint32_t)__popcll(word);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, below, o);
      if ((int)lane >= o) below += v;
    }
    if (lane == 31) sm.scan[warp] = below;
    __syncthreads();
    uint32_t sum = 0, free_segments = 0;
    for (uint32_t w = 0; w < (uint32_t)BOOT_WARPS; w++) {
      if (w < warp) sum += sm.scan[w];
      free_segments += sm.scan[w];
    }
    below += sum - (uint32_t)__popcll(word);
    const uint32_t total = t1 > t0 ? sm.first[t1] : 0;
    if (t1 == t0 || total > free_segments) {
      const uint32_t end = t1 > t0 ? t1 : t0 + 1;
      if (threadIdx.x == 0)
        for (uint32_t t = t0; t < end; t++)
          for (uint32_t i = 0; i < s->slot_count[t]; i++)
            if (!boot_block(s, t, i, 0)) set_error(s, GAL_DEV_ERR_BOOT);
      t0 = end;
      __syncthreads();
      continue;
    }
    uint64_t taken = word;  // the bits of `word` among the first `total` free segments
    if (below >= total) {
      taken = 0;
    } else if (below + (uint32_t)__popcll(word) > total) {  // its lowest total - below
      uint32_t end = 0;  // the most bits [0, end) that hold no more
#pragma unroll
      for (uint32_t step = 32; step; step >>= 1)
        if ((uint32_t)__popcll(word & bitmask((int)(end + step))) <= total - below) end += step;
      taken = word & bitmask((int)end);
    }
    if (taken) {
      amo_and(bottom + threadIdx.x, ~taken);
      if (taken == word) {  // emptied: off the summaries, as veb_remove does
        uint64_t high = threadIdx.x;
        for (int layer = (int)s->veb.layers - 2; layer >= 0; layer--) {
          const uint64_t bit = 1ull << (high & 63u);
          high >>= 6;
          if (amo_and(segs.word(layer, high), ~bit) != bit) break;
        }
      }
    }
    for (uint32_t base = 0; base < total; base += BOOT_THREADS) {
      uint32_t r = below;
      for (uint64_t b = taken; b; b &= b - 1ull, r++)
        if (r >= base && r - base < (uint32_t)BOOT_THREADS)
          sm.list[r - base] = (uint16_t)(threadIdx.x * 64u + (uint32_t)__ffsll((long long)b) - 1u);
      __syncthreads();
      // entry e of the tile: its class, its blocks, the first of its slots
      auto entry = [&](uint32_t e, uint32_t &t, uint32_t &slot) {
        t = t0;
        while (base + e >= sm.first[t + 1]) t++;
        const uint32_t n = s->slot_count[t], j = base + e - sm.first[t];
        const uint32_t lone = t == t0 ? sm.lone[t0] : 0u;
        // blocks of the class's segments before this one, and of this one
        slot = lone && j ? ((j - 1u) << (s->bps_shift - t)) + 1u : j << (s->bps_shift - t);
        const uint32_t most = lone && !j ? 1u : blocks_in_segment(s, t);
        return min(most, n - min(n, slot));
      };
      uint32_t mine = 0;  // the warp's entries that were set up
      for (uint32_t e = warp, k = 0; e < (uint32_t)BOOT_THREADS && base + e < total; e += BOOT_WARPS, k++) {
        uint32_t t, slot;
        const uint32_t taken = entry(e, t, slot);
        if (boot_segment(s, sm.list[e], t, slot, taken)) mine |= 1u << k;
      }
      fence_acq_rel();
      __syncwarp();
      if ((mine >> lane) & 1u) {  // lane k opens the warp's k-th
        const uint32_t e = warp + lane * BOOT_WARPS;
        uint32_t t, slot;
        const uint32_t taken = entry(e, t, slot);
        boot_open(s, sm.list[e], t, taken);
      }
      __syncthreads();
    }
    t0 = t1;
  }
}

}  // namespace gal
