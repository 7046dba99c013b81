"""The work that programs on this allocator do, as cases to be measured.

A case is a dict of plain values; `kind` says which program it stands for:

  calls   one malloc call for n requests, a record written into and read back
          from every allocation, one free call (the batched or the per-thread
          entry points)
  large   the same with large, block and multi-segment requests among 64 B ones
  churn   rounds of frees of a random half of what lives and n new requests,
          every record read back when its allocation is freed
  phase   one phase of a longer program: requests, records, frees, then trim and
          a look at the statistics
  tables  many chained hash tables whose nodes a kernel allocates itself
  served  a queue of jobs (growing vectors, linked queues), each a kernel that
          allocates through the device allocator, on several streams

`knobs`: "reference" is the reference's geometry and pinned slots (the default
configuration), "tuned" the throughput settings of the integration notes.
`graph`: the pass is captured once as a CUDA graph and replayed, as a program
does whose step always has the same shape; otherwise it is launched call by call.
"""
import math

import numpy as np
import torch

import gallatin_gb300 as G
from gallatin_gb300 import serve, tables

GIB = 1 << 30
KNOBS = {
    "reference": {},
    "tuned": dict(pinned_slots_first=0, pinned_slots_min=0, gather_unlocked_below=16,
                  bytes_per_segment=64 << 20, spare_blocks=1, l2_fetch_bytes=32),
}


def listed():
    return [
        # the smallest call: a kernel-sized list of equal small objects, launch and latency bound
        dict(name="call-256x64B", kind="calls", api="batched", graph=True, knobs="reference", n=256, lo=64, hi=64, gib=2),
        # an ordinary ragged batch of mixed objects at the default configuration
        dict(name="call-100003-mixed", kind="calls", api="batched", graph=True, knobs="reference", n=100003, lo=17,
             hi=4096, gib=8),
        # the largest: one round of the mixed churn's requests (4 Mi of 16 B-4 KiB)
        dict(name="call-4Mi-mixed", kind="calls", api="batched", graph=True, knobs="tuned", n=4 << 20, lo=17, hi=4096,
             gib=64),
        # the reference's global test: a million threads, each one 16 B allocation
        dict(name="threads-1Mi-16B", kind="calls", api="per_thread", graph=True, knobs="reference", n=1 << 20, lo=16,
             hi=16, gib=4),
        # one request per thread from a user's kernel, mixed sizes, an odd count
        dict(name="threads-1000003-mixed", kind="calls", api="per_thread", graph=True, knobs="tuned", n=1000003, lo=17,
             hi=4096, gib=32),
        # buffers above the largest slice: runs of 2-8 slices
        dict(name="call-30011-runs", kind="calls", api="batched", graph=True, knobs="tuned", n=30011, lo=4097, hi=32768,
             gib=32),
        # whole blocks and contiguous segments of 64 KiB-256 MiB with 20 requests of 64 B for each
        dict(name="large-256", kind="large", knobs="reference", n=256, small=20, gib=48),
        # a long-lived pool: eight rounds, each freeing half of what lives and allocating 256 Ki more
        dict(name="churn-8x256Ki", kind="churn", graph=True, knobs="tuned", n=256 << 10, rounds=8, lo=17, hi=4096, gib=32),
        # between two phases of a program: everything freed, trimmed, statistics read
        dict(name="phase-200003-trim", kind="phase", knobs="tuned", n=200003, lo=17, hi=4096, gib=32),
        # hash tables of uneven sizes, nodes allocated one by one under the bucket lock
        dict(name="tables-128", kind="tables", knobs="tuned", batched=False, n=128, lo=12, hi=18, gib=32),
        # the same at the default configuration, nodes allocated per thread block
        dict(name="tables-96-grouped", kind="tables", knobs="reference", batched=True, n=96, lo=10, hi=16, gib=8),
        # forty jobs of 1 Ki-1 Mi elements or operations through the request loop
        dict(name="served-40", kind="served", knobs="reference", n=40, lo=10, hi=20, gib=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["calls"] * 7 + ["large", "churn", "phase", "tables", "served"])
    knobs = rng.choice(["reference", "tuned"])
    if kind == "calls":
        what = rng.choice(["one", "mixed", "mixed", "runs"])
        lo, hi = 17, 4096
        most = 4 << 20 if knobs == "tuned" else 1 << 20
        if what == "one":
            lo = hi = _log_int(rng, 16, 1024)
        elif what == "runs":
            lo, hi, most = 4097, 32768, 60000
        n = _log_int(rng, 64, most)
        return dict(kind=kind, api=rng.choice(["batched", "batched", "per_thread"]), graph=rng.random() < 0.75,
                    knobs=knobs, n=n, lo=lo, hi=hi, gib=64 if knobs == "tuned" else 16)
    if kind == "large":
        return dict(kind=kind, knobs="reference", n=_log_int(rng, 16, 256), small=rng.randint(0, 20), gib=48)
    if kind == "churn":
        return dict(kind=kind, graph=rng.random() < 0.75, knobs="tuned", n=_log_int(rng, 10000, 262144),
                    rounds=rng.randint(3, 8), lo=17, hi=4096, gib=32)
    if kind == "phase":
        return dict(kind=kind, knobs=knobs, n=_log_int(rng, 1000, 200003), lo=17, hi=4096, gib=32)
    if kind == "tables":
        lo = rng.randint(6, 12)
        return dict(kind=kind, knobs=knobs, batched=rng.random() < 0.5, n=rng.randint(16, 96), lo=lo,
                    hi=lo + rng.randint(1, 5), gib=32)
    lo = rng.randint(8, 12)
    return dict(kind="served", knobs="reference", n=rng.randint(8, 40), lo=lo, hi=lo + rng.randint(4, 8), gib=16)


# ---------------------------------------------------------------- inputs
def _rng(case, seed):
    return np.random.default_rng([seed, case["n"]])


def _sizes(case, rng, n):
    """Request sizes: the class log-uniform over [lo, hi], uniform inside it."""
    if case["lo"] == case["hi"]:
        return np.full(n, case["lo"], dtype=np.int64)
    s = 2.0 ** rng.uniform(math.log2(case["lo"]), math.log2(case["hi"]), n)
    return np.clip(np.rint(s).astype(np.int64), case["lo"], case["hi"])


def _keys(rng, n):
    return rng.integers(-(1 << 62), 1 << 62, n, dtype=np.int64)


def _inputs(case, seed):
    """Host inputs of a case: sizes, the records stored, and what is freed when."""
    rng = _rng(case, seed)
    kind, n = case["kind"], case["n"]
    if kind in ("calls", "phase"):
        return dict(sizes=_sizes(case, rng, n), keys=_keys(rng, n))
    if kind == "large":
        large = (2.0 ** rng.uniform(16, 28, n)).astype(np.int64)
        sizes = np.concatenate([large, np.full(n * case["small"], 64, dtype=np.int64)])
        rng.shuffle(sizes)
        return dict(sizes=sizes, keys=_keys(rng, len(sizes)))
    if kind == "churn":
        r = case["rounds"]
        live = np.zeros(0, dtype=np.int64)
        frees = []
        for k in range(r):
            freed = np.zeros(len(live), dtype=bool)
            freed[rng.permutation(len(live))[: len(live) // 2]] = True
            frees.append(live[freed])
            live = np.concatenate([live[~freed], np.arange(k * n, (k + 1) * n, dtype=np.int64)])
        return dict(sizes=_sizes(case, rng, r * n), keys=_keys(rng, r * n), frees=frees[1:] + [live])
    if kind == "tables":
        # the tables' sizes are the case's, their keys the seed's
        sizes = np.floor(2.0 ** np.random.default_rng(n).uniform(case["lo"], case["hi"], n)).astype(np.uint64)
        return dict(table_sizes=sizes, table_seed=int(rng.integers(1, 1 << 31)))
    queue = rng.random(n) < 0.5
    ops = (2.0 ** rng.uniform(case["lo"], case["hi"], n)).astype(np.int64)
    first = int(rng.integers(1, 1 << 20))
    return dict(jobs=[dict(id=first + i, kind=int(serve.JOB_QUEUE if queue[i] else serve.JOB_VECTOR), n=int(ops[i]),
                           arrival=0.0) for i in range(n)])


# ---------------------------------------------------------------- state
class _Arena:
    """The arena's memory as an array of 64-bit words (for the records)."""

    def __init__(self, base, nbytes):
        self.__cuda_array_interface__ = {"shape": (nbytes // 8,), "typestr": "<i8", "data": (base, False),
                                         "version": 2, "strides": None}


class _State:
    """An allocator and one set of inputs; closes the allocator when dropped."""

    def __init__(self, case, seed):
        self.case = case
        self.g = G.Gallatin.generate_on_device(case["gib"] * GIB, 42, zero_arena=0, **KNOBS[case["knobs"]])
        x = _inputs(case, seed)
        for k, v in x.items():
            setattr(self, k, v)
        if "sizes" in x:
            self.base = self.g.arena_base
            self.arena = torch.as_tensor(_Arena(self.base, self.g.arena_bytes), device="cuda")
            self.sizes = torch.from_numpy(self.sizes).cuda()
            self.keys = torch.from_numpy(self.keys).cuda()
            self.ptrs = torch.zeros_like(self.sizes)
            self.words = torch.zeros_like(self.sizes)
            if "frees" in x:
                self.frees = [torch.from_numpy(f).cuda() for f in self.frees]
            if case.get("graph"):
                self._capture()
        elif "jobs" in x:
            self.server = serve.Server(self.g, slots=16)

    def _capture(self):
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _pass(self)  # torch's own first-use work stays out of the capture
        torch.cuda.current_stream().wait_stream(side)
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph):
            self.out = _pass(self)

    def __del__(self):
        self.graph = self.out = self.arena = None
        g = getattr(self, "g", None)
        if g is not None:
            g.close()


def prepare(case, seed):
    return _State(case, seed)


# ---------------------------------------------------------------- one pass
def _word_index(s, ptrs, out):
    """Arena word of each pointer (a refused request reads as word 0)."""
    torch.clamp(ptrs, min=s.base, out=out)
    out -= s.base
    out >>= 3
    return out


def _calls(s, stream):
    """Allocate, store the records, read them back, free."""
    per_thread = s.case.get("api") == "per_thread" or s.case["kind"] == "large"
    (s.g.malloc_per_thread if per_thread else s.g.malloc_batched)(s.sizes, s.ptrs, stream)
    at = _word_index(s, s.ptrs, s.words)
    s.arena.index_put_((at,), s.keys)
    got = s.arena[at]
    (s.g.free_per_thread if per_thread else s.g.free_batched)(s.ptrs, stream)
    return got


def _churn(s, stream):
    n, out = s.case["n"], []
    for r in range(s.case["rounds"]):
        lo, hi = r * n, (r + 1) * n
        s.g.malloc_batched(s.sizes[lo:hi], s.ptrs[lo:hi], stream)
        at = _word_index(s, s.ptrs[lo:hi], s.words[lo:hi])
        s.arena.index_put_((at,), s.keys[lo:hi])
        out.append(s.arena[s.words[s.frees[r]]])
        s.g.free_batched(s.ptrs[s.frees[r]], stream)
    return out


def run(state):
    if state.case.get("graph"):
        state.graph.replay()
        return state.out
    return _pass(state)


def _pass(s):
    stream = torch.cuda.current_stream().cuda_stream
    kind = s.case["kind"]
    if kind in ("calls", "large"):
        return {"records": _calls(s, stream)}
    if kind == "churn":
        return {"records": _churn(s, stream)}
    if kind == "phase":
        got = _calls(s, stream)
        s.g.trim(stream)
        st = s.g.stats()
        return {"records": got, "free_segments": int(st.free_segments), "largest_free_run": int(st.largest_free_run),
                "class_segments": np.array(list(st.tree_segments), dtype=np.int64),
                "class_listed": np.array(list(st.tree_listed), dtype=np.int64),
                "multi_segment_allocs": int(st.multi_segment_allocs), "errors": int(st.error_word)}
    if kind == "tables":
        which = int(np.argmax(s.table_sizes))
        d = tables.run(s.g, s.table_sizes, s.table_seed, s.case["batched"], dump_table=which)
        keys, vals = (torch.from_numpy(x.view(np.int64)).cuda() for x in d["dump"])
        keys, order = keys.sort()  # the largest table's pairs, in whatever order its chains held them
        return {"keys": keys, "values": vals[order],
                "inserted": int(d["inserted"]), "deleted": int(d["deleted"]), "violations": int(d["violations"]),
                "nodes_left": int(d["nodes_allocated"] - d["nodes_freed"] - d["spare_nodes_freed"])}
    d = s.server.run(s.jobs, realtime=False)
    return {"checksums": d["checksums"].view(np.int64), "ops": int(d["ops"]), "failed": int(d["failed_mallocs"]),
            "errors": int(d["error_word"])}


# ---------------------------------------------------------------- what a pass needs
def work(case):
    kind, n = case["kind"], case["n"]
    if kind in ("calls", "phase"):
        return {"bytes": 48 * n, "flops": 0}  # sizes, pointers out and in, records in, through the arena and out
    if kind == "large":
        return {"bytes": 48 * n * (1 + case["small"]), "flops": 0}
    if kind == "churn":
        return {"bytes": 48 * n * case["rounds"], "flops": 0}
    if kind == "tables":
        # expected pairs; each is written by its insert, half are deleted and written again, and two lookups read it
        a, b = case["lo"] * math.log(2), case["hi"] * math.log(2)
        pairs = n * (math.exp(b) - math.exp(a)) / (b - a)
        return {"bytes": 16 * pairs * 4.5, "flops": 0}
    a, b = case["lo"] * math.log(2), case["hi"] * math.log(2)
    each = n / 2 * (math.exp(b) - math.exp(a)) / (b - a)
    # a vector's 4 B elements written and read; a queue's enqueues (at least half of its operations) write and
    # read the link and the value of a node
    return {"bytes": each * 8 + each / 2 * 32, "flops": 0}


def exact(case, seed):
    """The records that went in, in the order in which they come out."""
    if case["kind"] in ("tables", "served"):
        return None
    x = _inputs(case, seed)
    if case["kind"] == "churn":
        return {"records": [x["keys"][f] for f in x["frees"]]}
    if case["kind"] == "phase":
        return {"records": x["keys"], "free_segments": None, "largest_free_run": None, "class_segments": None,
                "class_listed": None, "multi_segment_allocs": None, "errors": None}
    return {"records": x["keys"]}
