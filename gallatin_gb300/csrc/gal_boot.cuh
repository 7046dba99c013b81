// gal_boot.cuh — booting and retiring the pinned slots with one CTA.
//
// The reference boots its slots one after another with one thread
// (boot_shared_block_container_one_thread, gallatin.cuh:196-221), and that
// order fixes which block every slot gets.  With one slot per SM in nine
// classes it is 1,368 block requests in a chain: 11.9 ms for a trim at one slot
// per SM (21.3 ms before the requests themselves were made cheaper).  Here the
// same end state is computed in parallel by 1,024 threads; bound by the dozen
// dependent round trips of its phases.
//
//   * Blocks of one segment must come home in slot order (their ring entries);
//     blocks of different segments have nothing in common but bits of the
//     trees, whose end state does not depend on the order.  So the slots are
//     retired 1,024 at a time, each thread finding how many earlier blocks of
//     the same segment come home with its own.
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

struct boot_smem {
  uint16_t key[BOOT_WARPS][32];    // retire: segments completed by a warp ...
  uint16_t count[BOOT_WARPS][32];  // ... and how many blocks of each
  uint32_t nkeys[BOOT_WARPS];
  uint32_t scan[BOOT_WARPS];
  uint32_t total_free;
  uint16_t list[BOOT_THREADS];     // boot: the gathered segments of a tile
  uint32_t fast[GAL_MAX_TREES];    // the class lists no segment and its lock is free
  uint32_t first[GAL_MAX_TREES + 1];
  uint32_t lone0;                  // class t0 takes segment 0 and finds it no more
};

// Whether veb_find_random finds segment 0 when its tree lists nothing else: it
// is at or above no start but 0, and the search after the starts is above 0.
static __device__ bool finds_lone_zero(const state *s, uint32_t t) {
  if (s->policy == GAL_POLICY_LOWEST) return true;
  const uint64_t U = s->num_segments;
  const uint64_t h1 = murmur64a_u64(0, s->seed + t);
  const uint64_t h2 = murmur64a_u64(0, h1);
  for (uint64_t a = 0; a < (uint64_t)VEB_ATTEMPTS; a++)
    if ((h1 + a * h2) % U == 0) return true;
  return false;
}
// Segments that n blocks of class t take, `lone` of them from segment 0
static __device__ uint32_t boot_segments(const state *s, uint32_t t, uint32_t n, uint32_t lone) {
  const uint32_t nb = blocks_in_segment(s, t);
  n -= lone;
  if (lone && n == 0) return 1;
  return lone + (s->gather_ahead ? n / nb + 1u : (n + nb - 1u) / nb);
}

// Threads i of a tile hold a block taken from a slot or spare (NOBLK: none), in
// slot order: what k retire_block calls in that order do.
static __device__ void retire_tile(const state *s, uint32_t blk, boot_smem &sm) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  bool home = false;
  uint32_t seg = 0, nb = 1;
  uint16_t tree = 0;
  if (blk != NOBLK) {
    const unsigned long long old = atomicAdd(mword_ptr(s, blk), (unsigned long long)SLICES_PER_BLOCK);
    const uint32_t handed_out = (uint32_t)old;
    if (handed_out < SLICES_PER_BLOCK) {
      const uint32_t n = SLICES_PER_BLOCK - handed_out;
      const uint32_t freed = atomicAdd(fctr_ptr(s, blk), n);
      if (freed + n == SLICES_PER_BLOCK) {
        st_rlx(fctr_ptr(s, blk), 0u);
        seg = blk >> s->bps_shift;
        tree = ld_rlx(&s->tree_ids[seg]);
        home = tree < s->num_trees;
        if (home) nb = blocks_in_segment(s, tree);
        else set_error_info(s, GAL_DEV_ERR_BAD_FREE, SITE_RETURN_BAD_TREE, blk, tree);
      } else if (freed + n > SLICES_PER_BLOCK) {
        set_error_info(s, GAL_DEV_ERR_BAD_FREE, SITE_FREE_OVERFLOW, blk, ((uint64_t)freed << 32) | n);
      }
    }
  }
  const uint32_t returned = home ? ld_rlx(&s->qfc[seg]) : 0u;
  // a warp's blocks by segment; the first lane of each segment speaks for it
  const uint32_t same = __match_any_sync(0xFFFFFFFFu, home ? seg : 0xFFFFFFFFu);
  const bool speaks = home && (int)lane == __ffs(same) - 1;
  const uint32_t speakers = __ballot_sync(0xFFFFFFFFu, speaks);
  if (speaks) {
    const uint32_t at = (uint32_t)__popc(speakers & lanemask_lt());
    sm.key[warp][at] = (uint16_t)seg;
    sm.count[warp][at] = (uint16_t)__popc(same);
  }
  if (lane == 0) sm.nkeys[warp] = (uint32_t)__popc(speakers);
  __syncthreads();  // also: every thread has read its segment's return position
  uint32_t before = 0, all = 0;
  if (speaks)
    for (uint32_t w = 0; w < (uint32_t)BOOT_WARPS; w++)
      for (uint32_t k = 0; k < sm.nkeys[w]; k++)
        if (sm.key[w][k] == seg) {
          all += sm.count[w][k];
          if (w < warp) before += sm.count[w][k];
        }
  const bool closes = speaks && before == 0;  // the first warp of a segment settles its counters
  before = __shfl_sync(0xFFFFFFFFu, before, __ffs(same) - 1);
  if (home) {
    const uint32_t live = (returned + before + (uint32_t)__popc(same & lanemask_lt())) & (nb - 1u);
    st_rlx(s->queues + ((uint64_t)seg << s->bps_shift) + live, blk);
    if (live != 0 && 10ull * live > nb && 10ull * (live - 1) < nb) veb_insert(sub_tree(s, tree), seg);
  }
  fence_acq_rel();
  __syncthreads();
  if (closes) {
    atomicAdd(&s->qfc[seg], all);
    atomicAdd(&s->fqfc[seg], all);
    const unsigned long long old = atomicAdd(&s->act[seg], (unsigned long long)all);
    if (act_count(old) + (int32_t)all == (int32_t)nb - 1) release_segment(s, seg, tree, act_gen(old), nb);
  }
  __syncthreads();
}

// every block in the n words at `from`, which are left empty
static __device__ void retire_all(const state *s, uint32_t *from, uint32_t n, boot_smem &sm) {
  for (uint32_t base = 0; base < n; base += BOOT_THREADS) {
    const uint32_t i = base + threadIdx.x;
    retire_tile(s, i < n ? atomicExch(from + i, NOBLK) : NOBLK, sm);
  }
}

// one fresh segment of class t, its first `taken` blocks given to the slots
// from `slot` on: what setup_segment and `taken` get_block calls leave (full warp)
static __device__ void boot_segment(const state *s, uint32_t seg, uint32_t t, uint32_t slot, uint32_t taken) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t nb = blocks_in_segment(s, t);
  if (ld_rlx(&s->tree_ids[seg]) != FREE_TREE) {  // listed free, yet owned
    if (lane == 0) {
      set_error(s, GAL_DEV_ERR_SEGMENT_SETUP);
      if (taken) set_error(s, GAL_DEV_ERR_BOOT);
    }
    return;
  }
  const uint32_t blk0 = seg << s->bps_shift;
  for (uint32_t i = lane; i < nb; i += 32) st_rlx(s->queues + blk0 + i, NOBLK);
  for (uint32_t i = lane; i < taken; i += 32) {
    st_rlx(mword_ptr(s, blk0 + i), (unsigned long long)t << 32);
    st_rlx(s->slots + s->slot_base[t] + slot + i, blk0 + i);
  }
  __syncwarp();
  if (lane == 0) {
    const uint32_t high = (uint32_t)(ld_rlx(&s->act[seg]) >> 32);
    const uint32_t next = (((high >> 8) + 1u) << 8) | t;
    s->tree_ids[seg] = (uint16_t)t;
    st_rlx(&s->qc[seg], taken);
    st_rlx(&s->qfc[seg], 0u);
    st_rlx(&s->fqfc[seg], 0u);
    fence_acq_rel();
    atomicAdd(&s->act[seg], ((unsigned long long)(next - high) << 32) + nb - taken);
    if (taken < nb) veb_insert(sub_tree(s, t), seg);
  }
}

// Boots every slot (all empty) in the one-thread order.  One CTA of
// BOOT_THREADS, no device malloc or free in flight.
static __device__ void boot_all(const state *s, boot_smem &sm) {
  const uint32_t T = s->num_trees, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const veb_ref segs = seg_tree(s);
  const uint32_t nwords = s->veb.nwords[s->veb.layers - 1];  // at most 1,024: 65,532 segments
  uint64_t *bottom = veb_bottom(segs);
  if (threadIdx.x < T)
    sm.fast[threadIdx.x] = ld_rlx(sub_tree(s, threadIdx.x).w) == 0 && ld_rlx(s->locks + threadIdx.x * LOCK_STRIDE) == 0;
  __syncthreads();
  for (uint32_t t0 = 0; t0 < T;) {
    uint32_t t1 = t0;  // classes [t0, t1) are booted together
    while (t1 < T && sm.fast[t1]) t1++;
    if (threadIdx.x == 0) {
      uint32_t at = 0;
      sm.lone0 = (ld_rlx(bottom) & 1ull) && blocks_in_segment(s, t0) > 1 && !finds_lone_zero(s, t0);
      for (uint32_t t = t0; t < t1; t++) {
        sm.first[t] = at;
        at += boot_segments(s, t, s->slot_count[t], t == t0 ? sm.lone0 : 0u);
      }
      sm.first[t1] = at;
    }
    // free segments below this thread's word
    const uint64_t word = t1 > t0 && threadIdx.x < nwords ? ld_rlx(bottom + threadIdx.x) : 0ull;
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
    if (below >= total) taken = 0;
    else
      for (uint32_t n = below + (uint32_t)__popcll(word); n > total; n--)
        taken &= ~(1ull << (63 - __clzll((long long)taken)));
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
      for (uint32_t e = warp; e < (uint32_t)BOOT_THREADS && base + e < total; e += BOOT_WARPS) {
        uint32_t t = t0;
        while (base + e >= sm.first[t + 1]) t++;
        const uint32_t n = s->slot_count[t], j = base + e - sm.first[t];
        const uint32_t lone = t == t0 ? sm.lone0 : 0u;
        // blocks of the class's segments before this one, and of this one
        const uint32_t slot = lone && j ? ((j - 1u) << (s->bps_shift - t)) + 1u : j << (s->bps_shift - t);
        const uint32_t most = lone && !j ? 1u : blocks_in_segment(s, t);
        boot_segment(s, sm.list[e], t, slot, min(most, n - min(n, slot)));
      }
      __syncthreads();
    }
    t0 = t1;
  }
}

}  // namespace gal
