// Kernels of a user's own that allocate through gal::malloc and gal::free, and
// single steps of the allocator run in a chosen order.  Compiled by build() and
// driven by tests/test_gpu_device.py; `s` is the allocator's device state.
#include <cuda_runtime.h>
#include <stdint.h>

#include <gallatin_gb300/gal_device.cuh>

namespace {

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

int dev_give_back(const gal::state *s, uint32_t tree, int fresh, unsigned long long *out) {
  RUN(k_give_back<<<1, 1>>>(s, tree, fresh, out));
}

}  // extern "C"
