// Kernels of a user's own that allocate through gal::malloc and gal::free, and
// single steps of the allocator run in a chosen order.  Compiled by build() and
// driven by tests/test_gpu_device.py; `s` is the allocator's device state.
#include <cuda_runtime.h>
#include <stdint.h>

#include <gallatin_gb300/gal_device.cuh>

#include "../../gallatin_gb300/csrc/gal_bulk.cuh"

namespace {

__device__ __forceinline__ uint64_t mix(uint64_t z) {
  z ^= z >> 30;
  z *= 0xBF58476D1CE4E5B9ull;
  z ^= z >> 27;
  z *= 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// whole blocks of `size` bytes asked for and freed by every thread, at most `keep`
// (up to 4) held at a time; kept[4 * thread ..] is what it holds (null: nothing)
__global__ void k_blocks(const gal::state *s, uint64_t size, uint32_t turns, uint32_t keep, uint64_t seed,
                         void **kept, unsigned long long *failed) {
  const uint64_t me = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  void *held[4] = {};
  uint32_t n = 0;
  for (uint32_t j = 0; j < 4; j++)
    if (kept[4 * me + j]) held[n++] = kept[4 * me + j];
  for (uint32_t k = 0; k < turns; k++) {
    const uint64_t r = mix(seed + me * turns + k);
    if (n < keep && (n == 0 || (r & 1u))) {
      void *p = gal::malloc(s, size);
      if (!p) atomicAdd(failed, 1ull);
      else held[n++] = p;
    } else {
      const uint32_t j = (uint32_t)(r >> 8) % n;
      gal::free(s, held[j]);
      held[j] = held[--n];
    }
  }
  for (uint32_t j = 0; j < 4; j++) kept[4 * me + j] = j < n ? held[j] : nullptr;
}

// Every thread asks for `turns` sizes, log-uniform over [16, hi], stamps each
// allocation at both ends and frees it `keep` (at most 4) of its own requests
// later, its stamps checked.  form 0: malloc and free; 1: malloc and free_sized;
// 2: malloc_cached and free_sized.  out: failed, wrong stamps.
__global__ void k_churn(const gal::state *s, uint32_t turns, uint32_t hi_bits, uint32_t keep, int form, uint64_t seed,
                        unsigned long long *out) {
  __shared__ gal::slot_cache cache;
  gal::slot_cache_init(cache);
  __syncthreads();
  const uint64_t me = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  uint64_t *held[5] = {}, len[5] = {}, id[5] = {};
  uint32_t n = 0, bad = 0, failed = 0;
  auto drop = [&]() {  // the oldest
    bad += held[0][0] != id[0] || held[0][len[0] / 8 - 1] != id[0];
    if (form == 0) gal::free(s, held[0]);
    else gal::free_sized(s, held[0], len[0]);
    n--;
    for (uint32_t j = 0; j < n; j++) {
      held[j] = held[j + 1];
      len[j] = len[j + 1];
      id[j] = id[j + 1];
    }
  };
  for (uint32_t k = 0; k < turns; k++) {
    const uint64_t r = mix(seed + me * turns + k), bits = 4 + r % (hi_bits - 3);
    const uint64_t size = min((1ull << bits) + ((r >> 16) & ((1ull << bits) - 1)), 1ull << hi_bits);
    uint64_t *p = (uint64_t *)(form == 2 ? gal::malloc_cached(s, size, cache) : gal::malloc(s, size));
    if (!p) {
      failed++;
    } else {
      held[n] = p;
      len[n] = size;
      id[n] = me << 32 | k;
      p[0] = p[size / 8 - 1] = id[n];
      n++;
    }
    if (n > keep) drop();
  }
  while (n) drop();
  if (failed) atomicAdd(&out[0], (unsigned long long)failed);
  if (bad) atomicAdd(&out[1], (unsigned long long)bad);
}

// out[i] = malloc(size) from every thread, one per thread
__global__ void k_fill(const gal::state *s, uint64_t size, uint64_t n, void **out) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = gal::malloc(s, size);
}

// Every device call once through `s`, wherever that state is kept.  out: failed,
// wrong answers, in the way of k_churn's stamps.
__device__ void every_call(const gal::state *s, uint64_t seed, gal::slot_cache &cache, unsigned long long *out) {
  const uint64_t me = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int k = 0; k < 6; k++) {
    const uint64_t size = 16 + mix(seed + 8 * me + k) % 9000;
    uint64_t *p = (uint64_t *)(k % 3 == 0 ? gal::malloc(s, size)
                               : k % 3 == 1 ? gal::malloc_cached(s, size, cache)
                                            : gal::malloc_team(s, size, 0xFFFFFFFFu));
    bool ok = p != nullptr;
    if (ok) {
      p[0] = p[size / 8 - 1] = me;
      uint16_t tree;
      const uint64_t held = gal::allocated_size(s, size);
      ok = gal::owns(s, p) && held >= size && held < 2 * size && gal::block_of(s, p, tree) != gal::NOBLK;
    }
    __syncwarp();
    ok = ok && p[0] == me && p[size / 8 - 1] == me;
    if (!ok) atomicAdd(&out[p ? 1 : 0], 1ull);
    if (p && k == 0) {
      gal::free(s, p);
    } else if (p && k == 1) {
      gal::free_sized(s, p, size);
    } else if (p) {
      void *const list[1] = {p};
      const bool go[1] = {true};
      gal::free_n<1>(s, list, go);
    }
    __syncwarp();
  }
}
__constant__ gal::state constant_state;
__global__ void k_state_pointer(const gal::state *s, int form, uint64_t seed, unsigned long long *out) {
  __shared__ gal::slot_cache cache;
  __shared__ gal::state copy;
  gal::slot_cache_init(cache);
  if (threadIdx.x == 0) copy = *s;
  __syncthreads();
  gal::state local = *s;
  if (form == 0) every_call(s, seed, cache, out);
  if (form == 1) every_call(&copy, seed, cache, out);
  if (form == 2) every_call(&local, seed, cache, out);
  if (form == 3) every_call(&constant_state, seed, cache, out);
}
__global__ void k_state_value(const gal::state s, uint64_t seed, unsigned long long *out) {
  __shared__ gal::slot_cache cache;
  gal::slot_cache_init(cache);
  __syncthreads();
  every_call(&s, seed, cache, out);
}
__global__ void k_state_grid_constant(const __grid_constant__ gal::state s, uint64_t seed, unsigned long long *out) {
  __shared__ gal::slot_cache cache;
  gal::slot_cache_init(cache);
  __syncthreads();
  every_call(&s, seed, cache, out);
}

// Of block `blk` all slices but `left` handed out; the number that were not yet.
__device__ uint32_t use_up(const gal::state *s, uint32_t blk, uint32_t left) {
  const uint32_t count = (uint32_t)gal::ld_rlx(gal::mword_ptr(s, blk)), to = gal::SLICES_PER_BLOCK - left;
  if (count >= to) return 0;
  atomicAdd(gal::mword_ptr(s, blk), (unsigned long long)(to - count));
  return to - count;
}

// One thread's chunk claim of `want` slices of class `tree` when every pinned
// block has `slot_left` slices left and every spare `spare_left`, as after claims
// of slow teams.  out: slices claimed, runs, slices left in the slot's block,
// blocks that could not be read.  Everything is given back.
__global__ void k_chunk_claim(const gal::state *s, uint32_t tree, uint32_t want, uint32_t slot_left,
                              uint32_t spare_left, unsigned long long *out) {
  __shared__ gal::bulk_smem sm;
  constexpr uint32_t MOST = 64;
  uint32_t blks[2 * MOST], used[2 * MOST], n = 0;
  const uint32_t slots = s->slot_count[tree], base = s->slot_base[tree];
  if (slots > MOST) return;
  for (uint32_t i = 0; i < slots; i++) {
    if (s->use_spares) gal::refill_spare(s, tree, i, 0);
    for (uint32_t spare = 0; spare <= (s->use_spares ? 1u : 0u); spare++) {
      const uint32_t blk = gal::ld_rlx((spare ? s->spares : s->slots) + base + i);
      if (blk == gal::NOBLK) {
        out[3]++;
        continue;
      }
      used[n] = use_up(s, blk, spare ? spare_left : slot_left);
      blks[n++] = blk;
    }
  }
  const uint32_t refill = gal::bulk_claim(s, tree, want, sm);
  for (uint32_t j = 0; j < sm.nruns[tree]; j++) out[0] += sm.len[tree][j];
  out[1] = sm.nruns[tree];
  uint32_t blk;
  gal::pick_slot(s, tree, blk);
  const uint32_t count = blk == gal::NOBLK ? gal::SLICES_PER_BLOCK : (uint32_t)gal::ld_rlx(gal::mword_ptr(s, blk));
  out[2] = count < gal::SLICES_PER_BLOCK ? gal::SLICES_PER_BLOCK - count : 0;
  if (refill != gal::NOBLK) gal::refill_spare(s, tree, refill, 0);
  for (uint32_t j = 0; j < sm.nruns[tree]; j++) {
    uint16_t t;
    gal::credit_frees(s, gal::block_of(s, sm.at[tree][j], t), sm.len[tree][j]);
  }
  for (uint32_t k = 0; k < n; k++)
    if (used[k]) gal::credit_frees(s, blks[k], used[k]);
}

// One thread: a segment of class `tree` with one block left to give, whose count
// a reservation meant for an earlier owner takes below zero; a request that
// meets it then; the reservation given back.  `fresh`: a segment gathered ahead,
// none of its blocks handed out (classes of one block per segment).  out:
// listed at first, the request got a block, listed after it, listed at the end.
__global__ void k_give_back(const gal::state *s, uint32_t tree, int fresh, unsigned long long *out) {
  const int64_t got = gal::gather_new_segment(s, tree, !fresh, gal::free_segments_low(s));
  if (got < 0) return;
  const uint64_t seg = (uint64_t)got;
  const uint32_t first = (uint32_t)seg << s->bps_shift, nb = gal::blocks_in_segment(s, tree);
  bool last;
  if (!fresh) {
    *gal::mword_ptr(s, first) = (unsigned long long)tree << 32;
    for (uint32_t k = 0; k + 2 < nb; k++) gal::get_block(s, seg, tree, last);
  }
  out[0] = gal::veb_query(gal::sub_tree(s, tree), seg);
  atomicAdd(&s->act[seg], ~0ull);
  out[1] = gal::get_block(s, seg, tree, last) != gal::NOBLK;
  gal::unlist_refusing(s, tree, seg);
  out[2] = gal::veb_query(gal::sub_tree(s, tree), seg);
  gal::give_back_reservation(s, seg);
  out[3] = gal::veb_query(gal::sub_tree(s, tree), seg);
  if (!fresh)
    for (uint32_t k = 0; k + 1 < nb; k++) gal::retire_block(s, first + k);
}

}  // namespace

#define RUN(...)                                                   \
  __VA_ARGS__;                                                     \
  if (cudaGetLastError() != cudaSuccess) return 1;                 \
  return cudaDeviceSynchronize() == cudaSuccess ? 0 : 2

extern "C" {

int dev_blocks(const gal::state *s, uint64_t size, uint32_t ctas, uint32_t threads, uint32_t turns, uint32_t keep,
               uint64_t seed, void **kept, unsigned long long *failed) {
  RUN(k_blocks<<<ctas, threads>>>(s, size, turns, keep, seed, kept, failed));
}

int dev_churn(const gal::state *s, uint32_t ctas, uint32_t threads, uint32_t turns, uint32_t hi_bits, uint32_t keep,
              int form, uint64_t seed, unsigned long long *out) {
  RUN(k_churn<<<ctas, threads>>>(s, turns, hi_bits, keep, form, seed, out));
}

int dev_fill(const gal::state *s, uint64_t size, uint64_t n, void **out) {
  RUN(k_fill<<<(unsigned)((n + 255) / 256), 256>>>(s, size, n, out));
}

// form: the state in global (0), shared (1), local (2) or constant memory (3), a
// kernel's parameter (4) or one whose address is taken (5)
int dev_state_copy(const gal::state *s, int form, uint64_t seed, unsigned long long *out) {
  gal::state value;
  if (cudaMemcpy(&value, s, sizeof(value), cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
  if (cudaMemcpyToSymbol(constant_state, &value, sizeof(value)) != cudaSuccess) return 4;
  if (form < 4) {
    RUN(k_state_pointer<<<32, 128>>>(s, form, seed, out));
  } else if (form == 4) {
    RUN(k_state_value<<<32, 128>>>(value, seed, out));
  } else {
    RUN(k_state_grid_constant<<<32, 128>>>(value, seed, out));
  }
}

int dev_chunk_claim(const gal::state *s, uint32_t tree, uint32_t want, uint32_t slot_left, uint32_t spare_left,
                    unsigned long long *out) {
  RUN(k_chunk_claim<<<1, 1>>>(s, tree, want, slot_left, spare_left, out));
}

int dev_give_back(const gal::state *s, uint32_t tree, int fresh, unsigned long long *out) {
  RUN(k_give_back<<<1, 1>>>(s, tree, fresh, out));
}

}  // extern "C"
