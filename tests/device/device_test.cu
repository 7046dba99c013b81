// Kernels of a user's own that allocate through gal::malloc and gal::free, and
// single steps of the allocator run in a chosen order.  Compiled by build() and
// driven by tests/test_gpu_device.py; `s` is the allocator's device state.
#include <cuda_runtime.h>
#include <stdint.h>

#include <gallatin_gb300/gal_device.cuh>

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
  void *held[4];
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

int dev_give_back(const gal::state *s, uint32_t tree, int fresh, unsigned long long *out) {
  RUN(k_give_back<<<1, 1>>>(s, tree, fresh, out));
}

}  // extern "C"
