// gal_serve.cu — device jobs of the served request loop (gallatin_gb300/serve.py).
//
// Two job kinds, each a grid of gal_job_ctas(kind, n) CTAs allocating through
// the device allocator while other jobs run on other streams:
//   * vector: n uint32 values pushed back into device vectors whose capacity
//     starts at 1,024 elements and doubles through malloc / copy / free (the
//     growth of the reference's data_structs/single_vector.cuh:86-143); CTA b
//     of G grows its own vector over elements [b n / G, (b + 1) n / G), so a
//     large job crosses 4 KiB slices, 8-32 KiB slice runs, whole blocks and
//     multi-segment runs;
//   * queue (QUEUE_THREADS threads per gal_job_ctas CTA): n enqueue/dequeue
//     operations on per-thread FIFO queues of 32 B nodes (malloc on enqueue,
//     free on dequeue), drained at the end.
// result[0] = checksum (sum of the vector's values / of every dequeued value),
// which depends only on the job's id and size; result[1] = mallocs + frees;
// result[2] = failed mallocs.  hist (optional) receives the latency of every
// malloc and free the job makes, in SM cycles (clock64 around the call),
// binned by lat_bin: each CTA counts in shared memory (one shared atomic per
// call) and adds its non-zero bins to hist at the end.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/gallatin_gb300.h"
#include "../../include/gallatin_gb300/gal_device.cuh"

namespace {

constexpr int JOB_THREADS = 1024;
constexpr int BINS = GAL_JOB_LAT_BINS;

__device__ __forceinline__ uint32_t job_value(uint64_t job, uint64_t j) {
  uint64_t x = job * 0x9E3779B97F4A7C15ull + j * 0xBF58476D1CE4E5B9ull + 0x94D049BB133111EBull;
  x ^= x >> 31;
  x *= 0xD6E8FEB86659FD93ull;
  return (uint32_t)(x >> 32);
}

// c for c < 4, else 4 floor(log2 c) + the two bits below the leading one:
// four bins per power of two (bin edges within 19% of each other)
__device__ __forceinline__ uint32_t lat_bin(long long cycles) {
  const uint64_t c = cycles > 0 ? (uint64_t)cycles : 0;
  if (c < 4) return (uint32_t)c;
  const uint32_t e = 63u - (uint32_t)__clzll((long long)c);
  const uint32_t b = 4u * e + (uint32_t)((c >> (e - 2)) & 3u);
  return b < (uint32_t)BINS ? b : (uint32_t)BINS - 1u;
}

struct job_hist {
  uint32_t n[2 * BINS];  // mallocs, then frees
};

__device__ __forceinline__ void hist_init(job_hist &h) {
  for (int i = threadIdx.x; i < 2 * BINS; i += blockDim.x) h.n[i] = 0;
}
__device__ __forceinline__ void hist_add(job_hist &h, int which, long long cycles) {
  atomicAdd(&h.n[which * BINS + lat_bin(cycles)], 1u);
}
__device__ __forceinline__ void hist_flush(const job_hist &h, unsigned long long *out) {
  if (!out) return;
  for (int i = threadIdx.x; i < 2 * BINS; i += blockDim.x)
    if (h.n[i]) atomicAdd(&out[i], (unsigned long long)h.n[i]);
}

// `n` elements from `from` to `to` (16-byte aligned), a CTA's threads in turn:
// four 16-byte loads in flight each
__device__ __forceinline__ void copy_elements(uint32_t *to, const uint32_t *from, uint64_t n) {
  constexpr int F = 4;
  const uint64_t quads = n / 4;
  for (uint64_t q0 = threadIdx.x; q0 < quads; q0 += (uint64_t)JOB_THREADS * F) {
    uint4 v[F];
#pragma unroll
    for (int k = 0; k < F; k++)
      if (q0 + (uint64_t)k * JOB_THREADS < quads) v[k] = ((const uint4 *)from)[q0 + (uint64_t)k * JOB_THREADS];
#pragma unroll
    for (int k = 0; k < F; k++)
      if (q0 + (uint64_t)k * JOB_THREADS < quads) ((uint4 *)to)[q0 + (uint64_t)k * JOB_THREADS] = v[k];
  }
  for (uint64_t j = quads * 4 + threadIdx.x; j < n; j += JOB_THREADS) to[j] = from[j];
}

// Bound by what one SM moves: a CTA fills a buffer, doubles it and copies what
// is there, 16 bytes a thread at a time between one malloc/free pair and the
// next.  Pushing, copying and summing one element per thread and turn took
// 1.57 ms for 1 Mi elements (256 threads); now 0.36.
__global__ void __launch_bounds__(JOB_THREADS)
    k_job_vector(const gal::state *s, uint64_t job, uint64_t n, unsigned long long *result,
                 unsigned long long *hist) {
  __shared__ uint32_t *buf;
  __shared__ uint32_t *next;
  __shared__ job_hist lh;
  const int t = threadIdx.x;
  // this CTA's share of the job's elements
  const uint64_t lo = n * blockIdx.x / gridDim.x, hi = n * (blockIdx.x + 1) / gridDim.x;
  const uint64_t m = hi - lo;
  hist_init(lh);
  __syncthreads();
  if (t == 0) {
    long long c0 = clock64();
    buf = (uint32_t *)gal::malloc(s, 1024 * sizeof(uint32_t));
    hist_add(lh, 0, clock64() - c0);
  }
  __syncthreads();
  unsigned long long ops = 1;
  bool failed = buf == nullptr;
  uint64_t cap = 1024, size = 0;
  while (!failed) {
    // push up to the capacity
    const uint64_t end = min(m, cap);
    for (uint64_t j = size + 4ull * t; j < end; j += 4ull * JOB_THREADS) {  // size: 0 or the last capacity
      uint4 v;
      v.x = job_value(job, lo + j);
      v.y = job_value(job, lo + j + 1);
      v.z = job_value(job, lo + j + 2);
      v.w = job_value(job, lo + j + 3);
      if (j + 4 <= end) {
        *(uint4 *)(buf + j) = v;
      } else {
        buf[j] = v.x;
        if (j + 1 < end) buf[j + 1] = v.y;
        if (j + 2 < end) buf[j + 2] = v.z;
      }
    }
    size = end;
    if (m <= cap) break;
    // grow: malloc 2x, copy, free the old buffer
    if (t == 0) {
      long long c0 = clock64();
      next = (uint32_t *)gal::malloc(s, 2 * cap * sizeof(uint32_t));
      hist_add(lh, 0, clock64() - c0);
    }
    __syncthreads();  // also: every element is pushed
    ops++;
    failed = next == nullptr;
    if (failed) break;
    copy_elements(next, buf, size);
    __syncthreads();
    if (t == 0) {
      long long c0 = clock64();
      gal::free(s, buf);
      hist_add(lh, 1, clock64() - c0);
      buf = next;
    }
    ops++;
    cap *= 2;
    __syncthreads();
  }
  __syncthreads();
  unsigned long long sum = 0;
  if (!failed) {
    constexpr int F = 4;
    const uint64_t quads = m / 4;
    for (uint64_t q0 = t; q0 < quads; q0 += (uint64_t)JOB_THREADS * F) {
      uint4 v[F] = {};
#pragma unroll
      for (int k = 0; k < F; k++)
        if (q0 + (uint64_t)k * JOB_THREADS < quads) v[k] = ((const uint4 *)buf)[q0 + (uint64_t)k * JOB_THREADS];
#pragma unroll
      for (int k = 0; k < F; k++) sum += (unsigned long long)v[k].x + v[k].y + v[k].z + v[k].w;
    }
    for (uint64_t j = quads * 4 + t; j < m; j += JOB_THREADS) sum += buf[j];
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
  if ((t & 31) == 0 && sum) atomicAdd(&result[0], sum);  // 64-bit partial sums: no carry is lost
  __syncthreads();
  if (t == 0) {
    if (buf) {
      long long c0 = clock64();
      gal::free(s, buf);
      hist_add(lh, 1, clock64() - c0);
      ops++;
    }
    atomicAdd(&result[1], ops);
    atomicAdd(&result[2], (unsigned long long)failed);
  }
  __syncthreads();
  hist_flush(lh, hist);
}

struct qnode {
  qnode *next;
  uint64_t value;
  uint64_t pad[2];  // a 32 B node
};

constexpr int QUEUE_THREADS = 1024;  // threads a job has per gal_job_ctas CTA
constexpr int QUEUE_BLOCK = 64;      // ... launched in CTAs of

// Bound by the latency of its calls, one after another in every thread (a third
// of a malloc's claim and half of a free's atomic are round trips of 800
// cycles).  A job's threads are spread over sixteen times as many CTAs, so that
// fewer warps of an SM claim from its one pinned block at a time; the block is
// kept in shared memory (gal::malloc_cached), a free's class follows from the
// node's size, and a node's link and value are loaded when it becomes the
// head, while the calls before its dequeue run.  512 Ki operations: 3.13 ms with
// CTAs of 1,024 threads and none of this; now 1.74, 1.56, 1.54, 1.46 ms in CTAs of
// 256, 128, 64, 32 (forty jobs at once: 2.79, 2.54, 2.41, 2.54 ms).
__global__ void __launch_bounds__(QUEUE_BLOCK, 8)
    k_job_queue(const gal::state *s, uint64_t job, uint64_t n, uint64_t nt, unsigned long long *result,
                unsigned long long *hist) {
  __shared__ job_hist lh;
  __shared__ gal::slot_cache cache;
  hist_init(lh);
  gal::slot_cache_init(cache);
  __syncthreads();
  // thread t of the job's nt runs its share of the n operations
  const uint64_t t = (uint64_t)blockIdx.x * QUEUE_BLOCK + threadIdx.x;
  const uint64_t mine = n / nt + (t < n % nt ? 1 : 0);
  qnode *head = nullptr, *tail = nullptr;
  ulonglong2 first = make_ulonglong2(0, 0);  // the head's link and value
  unsigned long long sum = 0, ops = 0, failed = 0;
  auto dequeue = [&]() {
    qnode *q = head;
    head = (qnode *)first.x;
    sum += first.y;
    if (head) first = *(const ulonglong2 *)head;
    else tail = nullptr;
    long long c0 = clock64();
    gal::free_sized(s, q, sizeof(qnode));
    hist_add(lh, 1, clock64() - c0);
    ops++;
  };
  for (uint64_t o = 0; o < mine; o++) {
    uint64_t key = (t << 40) ^ o;
    uint32_t h = job_value(job, key);
    if (head == nullptr || h % 10 < 6) {  // enqueue
      long long c0 = clock64();
      qnode *q = (qnode *)gal::malloc_cached(s, sizeof(qnode), cache);
      hist_add(lh, 0, clock64() - c0);
      ops++;
      if (!q) {
        failed++;
        continue;
      }
      *(ulonglong2 *)q = make_ulonglong2(0, h);
      if (tail) {
        tail->next = q;
        if (tail == head) first.x = (unsigned long long)q;
      } else {
        head = q;
        first = make_ulonglong2(0, h);
      }
      tail = q;
    } else {
      dequeue();
    }
  }
  while (head) dequeue();  // drain
  atomicAdd(&result[0], sum);
  atomicAdd(&result[1], ops);
  if (failed) atomicAdd(&result[2], failed);
  __syncthreads();
  hist_flush(lh, hist);
}

}  // namespace

extern "C" uint32_t gal_job_ctas(uint32_t kind, uint64_t n) {
  const uint64_t g = kind == GAL_JOB_VECTOR ? n >> 20 : n >> 18;
  return g < 1 ? 1u : g > 8 ? 8u : (uint32_t)g;
}

extern "C" int gal_job_launch(gal_handle *h, uint32_t kind, uint64_t job_id, uint64_t n,
                              unsigned long long *result, unsigned long long *hist, void *stream) {
  if (!h || !result || kind > GAL_JOB_QUEUE) return GAL_ERR_ARGS;
  const gal::state *d = (const gal::state *)gal_device_state(h);
  cudaStream_t st = (cudaStream_t)stream;
  const unsigned g = gal_job_ctas(kind, n);
  if (kind == GAL_JOB_VECTOR)
    k_job_vector<<<g, JOB_THREADS, 0, st>>>(d, job_id, n, result, hist);
  else
    k_job_queue<<<g * (QUEUE_THREADS / QUEUE_BLOCK), QUEUE_BLOCK, 0, st>>>(
        d, job_id, n, (uint64_t)g * QUEUE_THREADS, result, hist);
  return cudaGetLastError() == cudaSuccess ? GAL_OK : GAL_ERR_CUDA;
}
