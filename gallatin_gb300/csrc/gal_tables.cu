// gal_tables.cu — batched uneven instances: many chained hash tables served by
// the device allocator in one launch per phase (the workload of the reference's
// data_structs/chaining_table.cuh:114-327, which has no delete; the table here
// is this library's own).
//
// Table t holds n_t pairs of 64-bit keys and values.  Its bucket array (one
// 64-bit head word per bucket, bit 0 the bucket's lock) and every 128-byte
// node come from the allocator.  A node: next pointer, a 7-bit used mask, one
// tag byte (eight hash bits) and a key/value pair for each of seven places
// (8 + 1 + 7 + 7 x 16 = 128 B, the 128 B class).
//
// Phases, each a kernel of its own over all tables (ops flattened, table by
// binary search over the offsets held in shared memory):
//   insert every key; delete the keys whose coin is set (a node left empty is
//   unlinked and freed); look up every key (deleted ones must be absent);
//   reinsert the deleted keys; look up every key (all present, right value);
//   count the live pairs of every table; free every node and bucket array.
// Node allocation inside an insert: per thread under the bucket lock (plain
// form; the CTA keeps a copy of its pinned block, which spares the claim a round
// trip), or CTA-aggregated (batched form: every thread holds a node ready, and
// the threads that used theirs ask for the next together through
// gal::cta_malloc).  The nodes held ready must not be what the arena is short of:
// a thread takes its own along from one insert phase to the next, and once one
// lacks a node the others put theirs into a queue for those that lack one, and
// only a thread whose bucket is full asks.  (Freed, they would leave gaps in
// blocks that come back only when all of their slices are free.)  What is left
// is freed with the tables.
//
// Bound by latency: an op is a chain of scattered round trips (lock 800 cycles,
// a node 700-1,000 from L2, more from DRAM, a release 800-1,600).  What kept the
// phases from overlapping them was divergence: lanes that held a lock waited for
// the warp's others to get theirs, so an instruction ran for 6 to 8 lanes, each
// group paid fences and claims of its own, and a node was searched one key at a
// time.  Now a lane tries its lock once per turn; the lanes that got theirs
// search, allocate, change and release together and fetch their next op, the
// others (one in twenty, so most warps have one) keep theirs for the next turn.
// What bounds an insert now is its three or four scattered 32-byte sectors, which
// it writes to L2: keeping the lock to the next turn, so that one fence serves
// the release and the next acquire, gave nothing (0.46 and 0.47 ms).
// 8.6 M pairs in 128 tables, one slot per SM, in ms, before and now: insert 2.22,
// 0.46; delete 1.47, 0.22; lookups 0.43 + 0.71, 0.15 + 0.16; reinsert 1.70, 0.27;
// teardown 0.81, 0.11.
//
// Keys: a bijective 64-bit mix of (table << 32 | index) so the keys of a table
// are distinct and uniform; value = another mix of the key; coin = bit 0 of a
// third mix.  gallatin_gb300/tables.py restates them on the host.
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>

#include "../../include/gallatin_gb300.h"
#include "../../include/gallatin_gb300/gal_device.cuh"
#include "gal_batch.cuh"

extern "C" {
/* Result of gal_bench_tables (mirrored in gallatin_gb300/_abi.py). */
typedef struct gal_tables_result {
  float ms[6];                 /* insert, delete, lookup-after-delete, reinsert, lookup, teardown */
  uint64_t total_pairs;
  uint64_t inserted;           /* inserts that added a pair (phases 0 and 3) */
  uint64_t deleted;
  uint64_t nodes_allocated;
  uint64_t nodes_freed;        /* by deletes and teardown */
  uint64_t spare_nodes_freed;  /* batched form: claimed, then not needed */
  uint64_t malloc_failed;
  uint64_t lock_timeouts;
  uint64_t missing;            /* keys absent that should be present */
  uint64_t unexpected;         /* deleted keys still present */
  uint64_t wrong_value;
  uint64_t count_mismatch;     /* tables whose live pairs != expected */
  uint64_t error_word;
  uint64_t setup_failed;       /* bucket arrays the allocator refused */
} gal_tables_result;
}

namespace {

constexpr int TBT = 256;          // CTA size of the table kernels
constexpr int MAX_TABLES = 4096;  // offsets held in shared memory
constexpr uint32_t SLOTS = 7;
constexpr uint32_t FULL = (1u << SLOTS) - 1u;

struct node {
  unsigned long long next;
  unsigned long long meta;  // byte 0: used mask; byte 1 + k: tag of place k
  ulonglong2 pair[SLOTS];   // key, value: one 16-byte load or store
};
static_assert(sizeof(node) == 128, "one 128 B slice per node");

struct alignas(16) table_desc {
  unsigned long long *heads;
  uint64_t nbuckets;  // a power of two
};

enum : int { S_INSERTED, S_DELETED, S_NODES, S_NODES_FREED, S_SPARE, S_MFAIL, S_LOCK, S_MISSING,
             S_UNEXPECTED, S_WRONG, S_COUNT_MISMATCH, S_SETUP_FAILED, S_N };

__host__ __device__ __forceinline__ uint64_t mix64(uint64_t z) {  // splitmix64 finaliser (a bijection)
  z ^= z >> 30;
  z *= 0xBF58476D1CE4E5B9ull;
  z ^= z >> 27;
  z *= 0x94D049BB133111EBull;
  z ^= z >> 31;
  return z;
}
__device__ __forceinline__ uint64_t table_key(uint32_t t, uint64_t i, uint64_t seed) {
  return mix64((((uint64_t)t << 32) | i) + seed * 0x9E3779B97F4A7C15ull);
}
__device__ __forceinline__ uint64_t table_val(uint64_t key) { return mix64(key ^ 0x5851F42D4C957F2Dull); }
__device__ __forceinline__ bool table_coin(uint64_t key) { return mix64(key + 0x2545F4914F6CDD1Dull) & 1u; }
__device__ __forceinline__ uint64_t table_hash(uint64_t key) { return mix64(key ^ 0x9E3779B97F4A7C15ull); }
__device__ __forceinline__ uint64_t bucket_of(uint64_t hash, uint64_t nb) { return hash & (nb - 1u); }
__device__ __forceinline__ uint32_t tag_of(uint64_t hash) { return (uint32_t)(hash >> 56); }

// per-thread counters, summed per warp once at the end of a phase kernel
struct counters {
  uint32_t c[S_N];
};
__device__ __forceinline__ void count(counters &lc, int which, uint32_t n = 1) { lc.c[which] += n; }
__device__ __forceinline__ void count_global(unsigned long long *stats, int which, uint32_t n = 1) {
  if (n) atomicAdd(&stats[which], (unsigned long long)n);
}
// full warp
__device__ __forceinline__ void flush(unsigned long long *stats, const counters &lc) {
#pragma unroll
  for (int k = 0; k < S_N; k++) {
    uint32_t v = __reduce_add_sync(0xFFFFFFFFu, lc.c[k]);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&stats[k], (unsigned long long)v);
  }
}

// Turns that a lane tries a lock without a pause.  A lock is held for a few turns;
// one that is held longer waits for a malloc that finds nothing, in an arena that
// is full, and the limit on the turns is to be a limit of time (some 0.4 s).
constexpr uint32_t WAITS_BRIEFLY = 64;
// Bucket lock: bit 0 of the head word.  One try (a round trip whether or not
// somebody holds it); true: `head` is the list, this thread's until it unlocks.
__device__ __forceinline__ bool try_lock_bucket(unsigned long long *hp, unsigned long long &head) {
  asm volatile("atom.acquire.gpu.global.or.b64 %0, [%1], 1;" : "=l"(head) : "l"(hp) : "memory");
  return !(head & 1ull);
}
__device__ __forceinline__ void unlock_bucket(unsigned long long *hp, unsigned long long head) {
  asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(hp), "l"(head) : "memory");
}

// the table of flattened op i
__device__ __forceinline__ uint32_t table_of(const uint64_t *off, uint32_t ntab, uint64_t i) {
  uint32_t lo = 0, hi = ntab;  // off[lo] <= i < off[hi]
  while (hi - lo > 1) {
    uint32_t mid = (lo + hi) >> 1;
    if (off[mid] <= i) lo = mid;
    else hi = mid;
  }
  return lo;
}

// The used places of a node whose tag is `tag`.
__device__ __forceinline__ uint32_t tagged(unsigned long long meta, uint32_t tag) {
  const uint32_t all = tag * 0x01010101u;
  const uint32_t lo = __vcmpeq4((uint32_t)(meta >> 8), all) & 0x01010101u;
  const uint32_t hi = __vcmpeq4((uint32_t)(meta >> 40), all) & 0x00010101u;
  // one bit per byte, gathered by the product's bits 24-27
  return (((lo * 0x01020408u) >> 24) | ((hi * 0x01020408u) >> 24) << 4) & (uint32_t)meta & FULL;
}
__device__ __forceinline__ unsigned long long with_place(unsigned long long meta, uint32_t k, uint32_t tag) {
  return (meta & ~(0xFFull << (8 + 8 * k))) | (unsigned long long)tag << (8 + 8 * k) | 1ull << k;
}

// Under the lock: the key's place (found: n, slot, meta, val, prev: its
// predecessor or 0 for the head, next), else a node with room (n, slot, meta), or n == 0.
// Node words are read past L1: another SM may have written them under the same
// bucket lock since this SM last cached the line.  One 16-byte load answers for
// a node unless a tag matches (the key's own, or one time in 256): loading all
// seven keys took five loads a node, each a scattered line per lane, and bound
// the lookups by L1 (84 % of its throughput).
struct probe {
  node *n;
  uint32_t slot;
  bool found;
  unsigned long long meta;
  node *prev;
  unsigned long long next;
  unsigned long long val;
};
// A node's link and meta; its whole line comes to L2 with them, as one of its
// pairs is read or written next (4 % of a delete, 6 % of a reinsert).
__device__ __forceinline__ ulonglong2 ld_node(const node *n) {
  ulonglong2 v;
  asm volatile("ld.global.cg.L2::128B.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(n) : "memory");
  return v;
}
__device__ __forceinline__ probe find(unsigned long long head, uint64_t key, uint32_t tag) {
  probe r{};
  node *prev = nullptr;
  for (node *n = (node *)(head & ~1ull); n;) {
    const ulonglong2 w = ld_node(n);
    for (uint32_t m = tagged(w.y, tag); m; m &= m - 1u) {
      const uint32_t k = (uint32_t)__ffs(m) - 1u;
      const ulonglong2 kv = __ldcg(&n->pair[k]);
      if (kv.x == key) return probe{n, k, true, w.y, prev, w.x, kv.y};
    }
    if (!r.n && ((uint32_t)w.y & FULL) != FULL) {
      r.n = n;
      r.slot = (uint32_t)__ffs(~(uint32_t)w.y & FULL) - 1u;
      r.meta = w.y;
    }
    prev = n;
    n = (node *)w.x;
  }
  return r;
}

// A thread's op between its turns and across a turn's malloc, and its counts,
// in shared memory and read back where they are wanted: held in registers they
// were spilled, and a spill is written through to L2 (some 20 M of the 47 M write
// requests of 8.6 M inserts; 260 bytes of spills a thread, now 42).  With the
// descriptors read as constants and the CTA's copy of its pinned block: insert
// 0.71 -> 0.46 ms, reinsert 0.48 -> 0.37, aggregated form 0.70 -> 0.54.
// Where the coin selects half of the ops a warp looks through 32 at a time and
// keeps those of the phase in a ring from which its free lanes serve themselves:
// each lane looking for itself (up to three ops a turn, for the few lanes that
// were free) was 8,400 of a delete's 20,600 cycles a turn.  Delete 0.34 -> 0.22,
// reinsert 0.37 -> 0.27.  Where every op is the phase's a lane takes its own
// (insert 0.46 ms, 0.50 through a ring).
template <bool RING>
struct pending {
  volatile uint64_t key[TBT], hp[TBT], head[TBT];
  volatile uint32_t tag[TBT], waited[TBT];
  volatile uint32_t pairs[TBT], nodes[TBT];  // inserted and allocated, or deleted and freed
  volatile uint64_t i[RING ? 1 : TBT];               // the lane's next op, or
  volatile uint32_t ready[RING ? 2 * TBT : 1], ready_table[RING ? 2 * TBT : 1];  // the ops that no lane has
  // taken yet, a ring of 64 for each warp: index in the table, table
};
// Whether an insert phase is short of nodes: a word for all CTAs, which each looks
// at once in LOOK_TURNS turns (the look holds the CTA up for a round trip).
enum : uint32_t { NODES_ENOUGH = 0, NODES_SHORT = 1, NODES_GONE = 2 };
constexpr uint32_t LOOK_TURNS = 8;
// Turns in which a lacked node may come from another CTA: that one may be in a
// request that the allocator is about to refuse, which takes up to 100 ms, so
// after the first the turns are slow.
constexpr uint32_t LACK_TURNS = 240, LACK_SLOWLY = 4 * LOOK_TURNS;
// The nodes that threads held ready: between the insert phases (one place for
// each thread of a grid), and those for threads that lack one.
struct node_pool {
  unsigned long long *kept, *queue;  // [cap] each, 0: none
  unsigned long long *ends;          // taken, put
  uint32_t cap;
};
__device__ __forceinline__ bool put_node(const node_pool &p, node *n) {
  const unsigned long long at = atomicAdd(&p.ends[1], 1ull);
  if (at >= p.cap) return false;
  asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p.queue + at), "l"(n) : "memory");
  return true;
}
__device__ __noinline__ node *take_node(const gal::state *s, const node_pool &p) {
  for (int tries = 0; tries < 16; tries++) {
    const unsigned long long at = gal::ld_rlx(&p.ends[0]);
    if (at >= min(gal::ld_rlx(&p.ends[1]), (unsigned long long)p.cap)) break;
    if (atomicCAS(&p.ends[0], at, at + 1) != at) continue;
    for (uint32_t i = 0; i < gal::cfield(s->spin_limit); i++) {  // its place is taken, it follows at once
      unsigned long long n;
      asm volatile("atom.acquire.gpu.global.exch.b64 %0, [%1], 0;" : "=l"(n) : "l"(p.queue + at) : "memory");
      if (n) return (node *)n;
      gal::backoff(i);
    }
    break;
  }
  return nullptr;
}
struct node_state {
  unsigned long long *left;  // the word for all
  volatile uint32_t seen;    // ... as last seen
  volatile uint32_t turns;
  volatile uint8_t lacked[TBT];  // turns that the thread's op has stayed for want of a node
};
// A thread found its bucket full and has no node for it: true while its op stays.
__device__ __forceinline__ bool lacks_node(node_state &nodes, uint32_t me) {
  const uint32_t turns = nodes.lacked[me];
  const bool stays = nodes.seen != NODES_GONE && turns < LACK_TURNS;
  const uint32_t now = stays ? NODES_SHORT : NODES_GONE;
  atomicMax(nodes.left, (unsigned long long)now);
  nodes.seen = now;
  nodes.lacked[me] = turns + 1u;
  return stays;
}
// One turn of an insert, by a whole warp together: true when the op is done.
// A bucket without room takes `spare`, when there is one (null afterwards);
// MALLOC: else a node from the allocator under the lock.  Without either the op
// stays for LACK_TURNS more turns, then it fails.  The warp meets before
// the malloc, whose teams are the lanes that call together: lanes that left the
// search one by one claimed one by one.  The others have written their pairs by
// then, and the release at the end finds those writes done.
template <bool MALLOC, bool RING>
__device__ __forceinline__ bool insert_turn(const gal::state *s, pending<RING> &op, bool go, node *&spare,
                                            gal::slot_cache &cache, unsigned long long *stats, node_state &nodes) {
  const uint32_t me = threadIdx.x;
  bool mine = false, full = false;
  if (go) {
    unsigned long long head;
    mine = try_lock_bucket((unsigned long long *)op.hp[me], head);
    if (mine) {
      op.head[me] = head;
      const uint64_t key = op.key[me];
      const uint32_t tag = op.tag[me];
      const probe p = find(head, key, tag);
      full = !p.n;
      if (p.n) {
        p.n->pair[p.slot] = make_ulonglong2(key, table_val(key));
        if (!p.found) {
          p.n->meta = with_place(p.meta, p.slot, tag);
          op.pairs[me] += 1u;
        }
      }
    }
  }
  __syncwarp();
  if (full) {
    node *n = spare;
    if (MALLOC) n = (node *)gal::malloc_cached(s, sizeof(node), cache);
    spare = nullptr;
    if (n) {
      const uint64_t key = op.key[me];
      *(ulonglong2 *)n = make_ulonglong2(op.head[me], with_place(0, 0, op.tag[me]));
      n->pair[0] = make_ulonglong2(key, table_val(key));
      op.head[me] = (uint64_t)n;
      op.pairs[me] += 1u;
      if (MALLOC) op.nodes[me] += 1u;
    } else {
      if constexpr (!MALLOC) full = lacks_node(nodes, me);
      if (MALLOC || !full) count_global(stats, S_MFAIL);
    }
    if constexpr (!MALLOC) full = full && !n;
  }
  __syncwarp();
  if (mine) unlock_bucket((unsigned long long *)op.hp[me], op.head[me]);
  if constexpr (MALLOC) {
    return mine;
  } else {
    if (mine && !full) nodes.lacked[me] = 0;
    return mine && !full;
  }
}

template <bool RING>
__device__ __forceinline__ bool delete_turn(const gal::state *s, pending<RING> &op, bool go) {
  const uint32_t me = threadIdx.x;
  unsigned long long head = 0;
  const bool mine = go && try_lock_bucket((unsigned long long *)op.hp[me], head);
  probe p{};
  if (mine) p = find(head, op.key[me], op.tag[me]);
  __syncwarp();
  node *dead = nullptr;
  if (mine) {
    if (p.found) {
      const unsigned long long meta = p.meta & ~(1ull << p.slot);
      op.pairs[me] += 1u;
      if ((uint32_t)meta & FULL) {
        p.n->meta = meta;
      } else {  // unlink and free the empty node
        if (p.prev) p.prev->next = p.next;
        else head = p.next;
        dead = p.n;
      }
    }
    unlock_bucket((unsigned long long *)op.hp[me], head);
  }
  __syncwarp();
  if (dead) {
    gal::free_sized(s, dead, sizeof(node));
    op.nodes[me] += 1u;
  }
  return mine;
}

__device__ __forceinline__ void lookup_op(const unsigned long long *hp, uint64_t key, uint32_t tag, bool expect,
                                          counters &lc) {
  const probe p = find(__ldcg(hp), key, tag);
  if (expect && !p.found) count(lc, S_MISSING);
  if (!expect && p.found) count(lc, S_UNEXPECTED);
  if (expect && p.found && p.val != table_val(key)) count(lc, S_WRONG);
}

// phase ops
enum : int { PH_INSERT = 0, PH_DELETE = 1, PH_CHECK_DELETED = 2, PH_REINSERT = 3, PH_CHECK_ALL = 4 };

// One phase; BATCHED: nodes of an insert phase come from gal::cta_malloc.
// Registers for five CTAs per SM where the phase allocates, although the
// allocator's rare paths then spill (insert at 4, 5 and 6 CTAs: 0.49, 0.46 and
// 0.45 ms with a slot per SM, 0.17, 0.17 and 0.20 for 1.7 M pairs with shared
// slots), and for six where it only frees or reads.
template <int PHASE, bool BATCHED>
__global__ void __launch_bounds__(TBT, PHASE == PH_INSERT || PHASE == PH_REINSERT ? 5 : 6)
    k_tables_phase(const gal::state *s, uint32_t ntab, const uint64_t *offsets, const table_desc *desc, uint64_t seed,
                   unsigned long long *stats, const __grid_constant__ node_pool pool) {
  constexpr bool INSERTS = PHASE == PH_INSERT || PHASE == PH_REINSERT;
  constexpr bool LOCKS = INSERTS || PHASE == PH_DELETE;
  extern __shared__ uint64_t off[];  // [ntab + 1]
  __shared__ gal::cta_claim_smem cm;
  __shared__ gal::slot_cache cache;
  constexpr bool RING = PHASE == PH_DELETE || PHASE == PH_REINSERT;
  __shared__ pending<RING> op;
  __shared__ node_state nodes;
  if constexpr (INSERTS && BATCHED) {
    nodes.lacked[threadIdx.x] = 0;
    if (threadIdx.x == 0) {
      nodes.left = stats + S_N + 1 + (PHASE == PH_REINSERT);
      nodes.seen = NODES_ENOUGH;
      nodes.turns = 0;
    }
  }
  for (uint32_t i = threadIdx.x; i <= ntab; i += blockDim.x) off[i] = offsets[i];
  if (INSERTS && BATCHED) gal::cta_claim_init(cm);
  if (INSERTS && !BATCHED) gal::slot_cache_init(cache);
  __syncthreads();
  counters lc = {};
  const uint64_t total = off[ntab];
  const uint32_t me = threadIdx.x;
  auto place = [&](uint32_t t, uint64_t key, uint32_t &tag) {
    const ulonglong2 w = __ldg((const ulonglong2 *)desc + t);  // (in lines that an acquire leaves in L1)
    const uint64_t hash = table_hash(key);
    tag = tag_of(hash);
    return (unsigned long long *)w.x + bucket_of(hash, w.y);
  };
  if (LOCKS) {
    const uint32_t lane = me & 31u, warp = me / 32u, lt = gal::lanemask_lt();
    // RING: 32 ops at a time for the warp, the next at `at`.  Else one for the lane.
    uint64_t at = ((uint64_t)blockIdx.x * TBT + me) - (RING ? lane : 0u);
    if (!RING) op.i[me] = at;
    uint32_t first = 0, have = 0;  // of the warp's ring
    op.pairs[me] = 0;
    op.nodes[me] = 0;
    bool go = false;
    node *spare = nullptr;
    if constexpr (PHASE == PH_REINSERT && BATCHED) spare = (node *)pool.kept[(uint64_t)blockIdx.x * TBT + me];
    for (;;) {
      uint32_t t = 0, index = 0;
      bool mine = false, more = go;  // takes op `index` of table t up; is not through yet
      if (RING) {
        const uint32_t idle = __ballot_sync(0xFFFFFFFFu, !go), want = (uint32_t)__popc(idle);
        while (have < want && at < total) {
          const uint64_t i = at + lane;
          bool sel = i < total;
          if (sel) {
            t = table_of(off, ntab, i);
            index = (uint32_t)(i - off[t]);
            sel = table_coin(table_key(t, index, seed)) && __ldg((const uint64_t *)(desc + t));
          }
          const uint32_t selected = __ballot_sync(0xFFFFFFFFu, sel);
          if (sel) {
            const uint32_t k = warp * 64u + ((first + have + (uint32_t)__popc(selected & lt)) & 63u);
            op.ready[k] = index;
            op.ready_table[k] = t;
          }
          have += (uint32_t)__popc(selected);
          at += (uint64_t)gridDim.x * TBT;
        }
        __syncwarp();
        const uint32_t r = (uint32_t)__popc(idle & lt);
        mine = !go && r < have;
        if (mine) {
          const uint32_t k = warp * 64u + ((first + r) & 63u);
          index = op.ready[k];
          t = op.ready_table[k];
        }
        const uint32_t taken = min(want, have);
        first += taken;
        have -= taken;
      } else {
        const uint64_t i = op.i[me];
        if (!go && i < total) {
          t = table_of(off, ntab, i);
          index = (uint32_t)(i - off[t]);
          mine = __ldg((const uint64_t *)(desc + t));  // (a table without buckets has no ops)
          op.i[me] = i + (uint64_t)gridDim.x * TBT;
          more = true;
        }
      }
      if (mine) {
        const uint64_t key = table_key(t, index, seed);
        uint32_t tag;
        op.hp[me] = (uint64_t)place(t, key, tag);
        op.key[me] = key;
        op.tag[me] = tag;
        op.waited[me] = 0;
        if constexpr (INSERTS && BATCHED) nodes.lacked[me] = 0;
        go = more = true;
      }
      if (INSERTS && BATCHED) {
        if (me == 0) {
          const uint32_t turn = nodes.turns + 1u;
          nodes.turns = turn;
          if (turn % LOOK_TURNS == 0) nodes.seen = (uint32_t)gal::ld_rlx(nodes.left);
        }
        if (!__syncthreads_or(more)) break;
        bool asks = !spare;
        if (nodes.seen != NODES_ENOUGH && !nodes.lacked[me]) {
          asks = false;
          if (spare && put_node(pool, spare)) spare = nullptr;
        } else if (asks && go && nodes.seen != NODES_ENOUGH) {
          spare = take_node(s, pool);
          const uint32_t turn = nodes.lacked[me];
          asks = !spare && turn == 1;  // (nothing else is freed meanwhile)
          if (!spare && turn > LACK_SLOWLY) __nanosleep(1000000);
        }
        node *n = (node *)gal::cta_malloc(s, sizeof(node), go && asks, cm);
        if (n) {
          spare = n;
          op.nodes[me] += 1u;
        }
      } else if (!__any_sync(0xFFFFFFFFu, more)) {
        break;
      }
      const bool done = INSERTS ? insert_turn<!BATCHED>(s, op, go, spare, cache, stats, nodes)
                                : delete_turn(s, op, go);
      if (done) go = false;
      if (go) {
        const uint32_t w = op.waited[me] + 1u;
        op.waited[me] = w;
        if (w > gal::cfield(s->spin_limit)) {
          count_global(stats, S_LOCK);
          go = false;
        } else if (w >= WAITS_BRIEFLY) {
          gal::backoff(w);
        }
      }
      __syncwarp();
    }
    if constexpr (INSERTS && BATCHED) {  // held ready to the end
      if (spare && nodes.seen != NODES_ENOUGH && put_node(pool, spare)) spare = nullptr;
      pool.kept[(uint64_t)blockIdx.x * TBT + me] = (unsigned long long)spare;
    }
    count(lc, INSERTS ? S_INSERTED : S_DELETED, op.pairs[me]);
    count(lc, INSERTS ? S_NODES : S_NODES_FREED, op.nodes[me]);
    __syncwarp();
  } else {
    for (uint64_t i = (uint64_t)blockIdx.x * TBT + me; i < total; i += (uint64_t)gridDim.x * TBT) {
      const uint32_t t = table_of(off, ntab, i);
      const uint64_t key = table_key(t, i - off[t], seed);
      uint32_t tag;
      const unsigned long long *hp = place(t, key, tag);
      if (__ldg((const uint64_t *)(desc + t))) lookup_op(hp, key, tag, PHASE == PH_CHECK_ALL || !table_coin(key), lc);
    }
    __syncwarp();
  }
  flush(stats, lc);  // whole warps
}

// one CTA per table: its bucket array from the allocator, zeroed
__global__ void __launch_bounds__(TBT)
    k_tables_setup(const gal::state *s, const uint64_t *offsets, table_desc *desc,
                   unsigned long long *stats) {
  __shared__ unsigned long long *heads;
  const uint32_t t = blockIdx.x;
  const uint64_t n = offsets[t + 1] - offsets[t];
  uint64_t nb = 16;
  while (nb * 4 < n) nb <<= 1;  // ~4 pairs per bucket
  if (threadIdx.x == 0) {
    heads = (unsigned long long *)gal::malloc(s, nb * sizeof(unsigned long long));
    desc[t].heads = heads;
    desc[t].nbuckets = nb;
    if (!heads) count_global(stats, S_SETUP_FAILED);
  }
  __syncthreads();
  if (!heads) return;
  for (uint64_t b = threadIdx.x; b < nb / 2; b += blockDim.x) ((ulonglong2 *)heads)[b] = make_ulonglong2(0, 0);
}

// The kernels below walk every bucket: TABLE_CTAS CTAs per table, as one per
// table left the chip to the largest (128 tables of 4 Ki-256 Ki pairs: count
// 404, dump 3,101, teardown 805 us).
constexpr int TABLE_CTAS = 32;
#define EACH_BUCKET(b, d)                                                                               \
  for (uint64_t b = (uint64_t)blockIdx.y * TBT + threadIdx.x; b < (d).nbuckets; b += (uint64_t)gridDim.y * TBT)

// live pairs of every table
__global__ void __launch_bounds__(TBT) k_tables_count(const table_desc *desc, unsigned long long *live) {
  const table_desc d = desc[blockIdx.x];
  if (!d.heads) return;
  uint32_t mine = 0;
  EACH_BUCKET(b, d)
    for (node *n = (node *)(__ldcg(&d.heads[b]) & ~1ull); n;) {
      const ulonglong2 w = __ldcg((const ulonglong2 *)n);
      mine += (uint32_t)__popc((uint32_t)w.y & FULL);
      n = (node *)w.x;
    }
  mine = __reduce_add_sync(0xFFFFFFFFu, mine);
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(&live[blockIdx.x], (unsigned long long)mine);
}
// ... compared with the expected counts
__global__ void __launch_bounds__(TBT)
    k_tables_compare(uint32_t ntab, const uint64_t *offsets, const table_desc *desc, const unsigned long long *live,
                     unsigned long long *stats) {
  const uint32_t t = blockIdx.x * TBT + threadIdx.x;
  if (t < ntab && desc[t].heads && live[t] != offsets[t + 1] - offsets[t]) count_global(stats, S_COUNT_MISMATCH);
}

// (key, value) pairs of table `which` appended to out, a warp's pairs of one
// turn with one reservation
__global__ void __launch_bounds__(TBT)
    k_tables_dump(const table_desc *desc, uint32_t which, unsigned long long *keys, unsigned long long *vals,
                  uint64_t cap, unsigned long long *n_out) {
  const table_desc d = desc[which];
  if (!d.heads) return;
  const uint32_t lane = threadIdx.x & 31u;
  for (uint64_t b0 = (uint64_t)blockIdx.y * TBT; b0 < d.nbuckets; b0 += (uint64_t)gridDim.y * TBT) {
    const uint64_t b = b0 + threadIdx.x;
    node *n = b < d.nbuckets ? (node *)(__ldcg(&d.heads[b]) & ~1ull) : nullptr;
    while (__any_sync(0xFFFFFFFFu, n != nullptr)) {
      ulonglong2 w[8] = {};
#pragma unroll
      for (int k = 0; k < 8; k++)
        if (n) w[k] = __ldcg((const ulonglong2 *)n + k);
      const unsigned long long *words = (const unsigned long long *)w;  // link, meta, pairs
      const uint32_t used = n ? (uint32_t)w[0].y & FULL : 0u, mine = (uint32_t)__popc(used);
      uint32_t upto = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, upto, o);
        if (lane >= (uint32_t)o) upto += v;
      }
      unsigned long long at = 0;
      if (lane == 31 && upto) at = atomicAdd(n_out, (unsigned long long)upto);
      at = __shfl_sync(0xFFFFFFFFu, at, 31) + upto - mine;
#pragma unroll
      for (int k = 0; k < (int)SLOTS; k++)
        if ((used >> k) & 1u) {
          if (at < cap) {
            keys[at] = words[2 + 2 * k];
            vals[at] = words[3 + 2 * k];
          }
          at++;
        }
      n = n ? (node *)w[0].x : nullptr;
    }
  }
}

// every node back to the allocator, then (k_tables_drop) every bucket array
__global__ void __launch_bounds__(TBT)
    k_tables_destroy(const gal::state *s, const table_desc *desc, unsigned long long *stats) {
  const table_desc d = desc[blockIdx.x];
  if (!d.heads) return;
  uint32_t freed = 0;
  EACH_BUCKET(b, d) {
    node *n = (node *)(__ldcg(&d.heads[b]) & ~1ull);
    while (n) {
      node *nx = (node *)__ldcg(&n->next);
      gal::free_sized(s, n, sizeof(node));
      freed++;
      n = nx;
    }
  }
  freed = __reduce_add_sync(0xFFFFFFFFu, freed);
  if ((threadIdx.x & 31) == 0) count_global(stats, S_NODES_FREED, freed);
}
// the nodes that were held ready and not needed
__global__ void __launch_bounds__(TBT) k_tables_spares(const gal::state *s, node_pool pool, unsigned long long *stats) {
  const uint32_t i = blockIdx.x * TBT + threadIdx.x;
  uint32_t freed = 0;
  if (i < 2u * pool.cap) {  // (the queue follows the places)
    const unsigned long long n = pool.kept[i];
    if (n) {
      gal::free_sized(s, (void *)n, sizeof(node));
      freed = 1;
    }
  }
  freed = __reduce_add_sync(0xFFFFFFFFu, freed);
  if ((threadIdx.x & 31) == 0) count_global(stats, S_SPARE, freed);
}
__global__ void __launch_bounds__(TBT) k_tables_drop(const gal::state *s, uint32_t ntab, const table_desc *desc) {
  const uint32_t t = blockIdx.x * TBT + threadIdx.x;
  if (t < ntab && desc[t].heads) gal::free(s, desc[t].heads);
}

}  // namespace

extern "C" {

/* The table workload on an allocator: n_tables tables, table t holding
 * offsets[t+1] - offsets[t] pairs (host array of n_tables + 1 prefix sums),
 * keys from `seed`; batched selects the CTA-aggregated node allocation.
 * Phases and checks as described at the top of this file.  When dump_keys is
 * not null, the pairs of table dump_table after the last lookup are copied
 * there (at most dump_cap; *dump_n receives the count). */
int gal_bench_tables(gal_handle *h, uint32_t n_tables, const uint64_t *offsets, uint64_t seed,
                     int batched, gal_tables_result *res, uint32_t dump_table, uint64_t *dump_keys,
                     uint64_t *dump_vals, uint64_t dump_cap, uint64_t *dump_n) {
  if (!h || !res || !offsets || n_tables == 0 || n_tables > MAX_TABLES) return GAL_ERR_ARGS;
  for (uint32_t t = 0; t < n_tables; t++)
    if (offsets[t + 1] < offsets[t] || offsets[t + 1] - offsets[t] >= (1ull << 32)) return GAL_ERR_ARGS;
  memset(res, 0, sizeof(*res));
  const gal::state *d = (const gal::state *)gal_device_state(h);
  int rc = GAL_OK;
  // one device buffer: offsets, descriptors, per-table counts, counters, and
  // the dumped pairs with their number
  const bool dump = dump_keys && dump_vals && dump_n && dump_table < n_tables && dump_cap;
  // (the pairs on 256-byte boundaries: a copy from an odd word ran at 4 GB/s)
  // (after the pairs' number, per insert phase whether it is short of nodes)
  const size_t head_words = ((size_t)n_tables * 4 + 1 + S_N + 3 + 31) / 32 * 32;
  const size_t pair_words = dump ? ((size_t)dump_cap + 31) / 32 * 32 : 0;
  size_t pool_words = 0;
  node_pool pool = {};
  static_assert(sizeof(table_desc) == 16, "two words per table");
  uint64_t *buf = nullptr;
  cudaEvent_t ev[8] = {};  // phase boundaries 0-5, teardown 6-7
  unsigned long long hs[S_N];
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const uint64_t total = offsets[n_tables];
  const uint64_t need_ctas = (total + TBT - 1) / TBT;
  const size_t smem = (n_tables + 1) * sizeof(uint64_t);
  const dim3 all_buckets(n_tables, TABLE_CTAS);
#define TK(x)                        \
  do {                               \
    if ((x) != cudaSuccess) {        \
      rc = GAL_ERR_CUDA;             \
      goto done;                     \
    }                                \
  } while (0)
  if (batched) {
    int most = 0, per_sm = 0;  // the larger of the two insert grids
    TK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&most, k_tables_phase<PH_INSERT, true>, TBT, smem));
    TK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tables_phase<PH_REINSERT, true>, TBT, smem));
    const uint64_t fit = (uint64_t)sms * std::max(std::max(most, per_sm), 1);
    pool.cap = (uint32_t)std::min<uint64_t>(need_ctas ? need_ctas : 1, fit) * TBT;
    pool_words = 2 * (size_t)pool.cap + 2;
  }
  TK(cudaMalloc(&buf, (head_words + 2 * pair_words + pool_words) * sizeof(uint64_t)));
  {
  table_desc *d_desc = (table_desc *)buf;
  uint64_t *d_off = buf + 2 * (size_t)n_tables;
  unsigned long long *live = (unsigned long long *)(d_off + n_tables + 1), *stats = live + n_tables;
  unsigned long long *d_n = stats + S_N, *d_keys = (unsigned long long *)buf + head_words, *d_vals = d_keys + pair_words;
  TK(cudaMemcpy(d_off, offsets, (n_tables + 1) * sizeof(uint64_t), cudaMemcpyHostToDevice));
  TK(cudaMemset(live, 0, (n_tables + S_N + 3) * sizeof(uint64_t)));
  if (batched) {
    pool.kept = (unsigned long long *)d_vals + pair_words;
    pool.queue = pool.kept + pool.cap;
    pool.ends = pool.queue + pool.cap;
    TK(cudaMemset(pool.kept, 0, pool_words * sizeof(uint64_t)));
  }
  for (auto &e : ev) TK(cudaEventCreate(&e));
  k_tables_setup<<<n_tables, TBT>>>(d, d_off, d_desc, stats);
  TK(cudaGetLastError());
  TK(cudaEventRecord(ev[0]));
  {
    auto phase = [&](auto kern) {
      int per_sm = 0;
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, TBT, smem);
      const uint64_t fit = (uint64_t)sms * (per_sm > 0 ? per_sm : 1);
      kern<<<(unsigned)std::min<uint64_t>(need_ctas ? need_ctas : 1, fit), TBT, smem>>>(d, n_tables, d_off, d_desc,
                                                                                        seed, stats, pool);
      return cudaGetLastError();
    };
    TK(batched ? phase(k_tables_phase<PH_INSERT, true>) : phase(k_tables_phase<PH_INSERT, false>));
    TK(cudaEventRecord(ev[1]));
    TK(phase(k_tables_phase<PH_DELETE, false>));
    TK(cudaEventRecord(ev[2]));
    TK(phase(k_tables_phase<PH_CHECK_DELETED, false>));
    TK(cudaEventRecord(ev[3]));
    TK(batched ? phase(k_tables_phase<PH_REINSERT, true>) : phase(k_tables_phase<PH_REINSERT, false>));
    TK(cudaEventRecord(ev[4]));
    TK(phase(k_tables_phase<PH_CHECK_ALL, false>));
    TK(cudaEventRecord(ev[5]));
  }
  k_tables_count<<<all_buckets, TBT>>>(d_desc, live);
  TK(cudaGetLastError());
  k_tables_compare<<<(n_tables + TBT - 1) / TBT, TBT>>>(n_tables, d_off, d_desc, live, stats);
  TK(cudaGetLastError());
  if (dump) {
    k_tables_dump<<<dim3(1, TABLE_CTAS * 8), TBT>>>(d_desc, dump_table, d_keys, d_vals, dump_cap, d_n);
    TK(cudaGetLastError());
    TK(cudaMemcpy(dump_n, d_n, 8, cudaMemcpyDeviceToHost));
    uint64_t got = *dump_n < dump_cap ? *dump_n : dump_cap;
    TK(cudaMemcpy(dump_keys, d_keys, got * 8, cudaMemcpyDeviceToHost));
    TK(cudaMemcpy(dump_vals, d_vals, got * 8, cudaMemcpyDeviceToHost));
  }
  TK(cudaEventRecord(ev[6]));
  k_tables_destroy<<<all_buckets, TBT>>>(d, d_desc, stats);
  TK(cudaGetLastError());
  k_tables_drop<<<(n_tables + TBT - 1) / TBT, TBT>>>(d, n_tables, d_desc);
  TK(cudaGetLastError());
  if (batched) {
    k_tables_spares<<<(2 * pool.cap + TBT - 1) / TBT, TBT>>>(d, pool, stats);
    TK(cudaGetLastError());
  }
  TK(cudaEventRecord(ev[7]));
  TK(cudaEventSynchronize(ev[7]));
  TK(cudaEventElapsedTime(&res->ms[5], ev[6], ev[7]));
  for (int k = 0; k < 5; k++) TK(cudaEventElapsedTime(&res->ms[k], ev[k], ev[k + 1]));
  TK(cudaMemcpy(hs, stats, sizeof(hs), cudaMemcpyDeviceToHost));
  }
  res->total_pairs = total;
  res->inserted = hs[S_INSERTED];
  res->deleted = hs[S_DELETED];
  res->nodes_allocated = hs[S_NODES];
  res->nodes_freed = hs[S_NODES_FREED];
  res->spare_nodes_freed = hs[S_SPARE];
  res->malloc_failed = hs[S_MFAIL];
  res->lock_timeouts = hs[S_LOCK];
  res->missing = hs[S_MISSING];
  res->unexpected = hs[S_UNEXPECTED];
  res->wrong_value = hs[S_WRONG];
  res->count_mismatch = hs[S_COUNT_MISMATCH];
  res->setup_failed = hs[S_SETUP_FAILED];
  {
    uint32_t w = 0;
    gal_last_error(h, &w);
    res->error_word = w;
  }
#undef TK
done:
  for (auto &e : ev)
    if (e) cudaEventDestroy(e);
  if (buf) cudaFree(buf);
  return rc;
}

}  // extern "C"
