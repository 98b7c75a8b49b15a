// Internal declarations shared by the translation units of libxtb200.so.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <string>
#include <unordered_map>

#include "../../include/xtric.h"

namespace xt {

constexpr int kWarp = 32;
// int32 column arrays carry this many spare entries past their end
constexpr size_t kColPad = 8;

// ---- context ---------------------------------------------------------------
// device block read back by the synchronous counts in one copy: the error word
// that kernels set when their input or a bounded wait fails, and a total
constexpr int kErrInput = 3;  // its bits of a build: an id out of range (1), offsets not monotone (2)
constexpr int kErrStageTimeout = 8, kErrCoreTimeout = 16;  // of a count: a staging wait, a wait of the core's gave up
constexpr int kErrWaits = kErrStageTimeout | kErrCoreTimeout;
struct CountOut {
  int err;
  int reserved;
  int64_t total;
  int64_t words[12];  // read_words
};

struct Ctx {
  int device = 0;
  int sm_count = 148;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  cudaStream_t copy_stream = nullptr;  // host-to-device copies that overlap the build (created on first use)
  std::string last_error;
  int64_t fail_alloc_countdown = 0;  // test hook: >0 counts down to a failing allocation
  CountOut *d_out = nullptr;
  int *d_err = nullptr;  // &d_out->err: reused by kernels that check their own inputs
  int64_t launches = 0;  // kernels of this library launched on this context
  // device bytes this context holds (its own allocations) and their high-water mark
  std::unordered_map<void *, size_t> live;
  int64_t bytes_live = 0, bytes_peak = 0;
  // optional totals shared by several contexts (a server's slots): bytes live
  // in all of them together and the high-water mark of that sum
  std::atomic<int64_t> *shared_live = nullptr, *shared_peak = nullptr;
};

// Launch-configuration wrapper that counts the library's own kernel launches.
inline dim3 counted(Ctx *c, dim3 grid) {
  c->launches++;
  return grid;
}

// Stream-ordered device allocation with the context's failure hook.
xt_status dalloc(Ctx *c, void **p, size_t bytes);
void dfree(Ctx *c, void *p);

template <class T>
xt_status dalloc_n(Ctx *c, T **p, size_t n) {
  return dalloc(c, reinterpret_cast<void **>(p), n * sizeof(T));
}

// Waits for the context's stream and brings n words from device addresses to the
// host in one copy (each copy into pageable memory holds the host for 7 us).
xt_status read_words(Ctx *c, int n, const void *const *from, int64_t *to);

// Records a CUDA error (if any) and converts it to a status.
xt_status cuda_status(Ctx *c, cudaError_t e, const char *what);
xt_status set_error(Ctx *c, xt_status s, const std::string &msg);

#define XT_CUDA(ctx, call)                                   \
  do {                                                       \
    cudaError_t xt_e_ = (call);                              \
    if (xt_e_ != cudaSuccess) return xt::cuda_status((ctx), xt_e_, #call); \
  } while (0)

#define XT_TRY(expr)                  \
  do {                                \
    xt_status xt_s_ = (expr);         \
    if (xt_s_ != XT_OK) return xt_s_; \
  } while (0)

// ---- oriented graph on the device ------------------------------------------
struct Plan;  // degree-binned schedule, built once per graph

// Pad value of the padded column array: negative, so below every vertex id
// (no membership test accepts it).
constexpr int32_t kPadSentinel = -2;

// In-record of edge u->v, stored with the head v: the columns of N+(u) that
// rank above v, i.e. the suffix d_colp[s, s+len) after v's own position
// (s indexes the padded column array).
// Every triangle (u,v,w) has its w in exactly this suffix and in N+(v).
// Packed in 8 bytes: pair = s / 8 (the 32-byte pair the suffix starts in)
// and lw = len | (s % 8) << kRecLenBits, so s < 2^35 and len < 2^29. The
// tail u is kept apart (Graph::d_irec_u), built when a per-vertex or
// per-edge count first needs it.
struct __align__(8) InRec {
  uint32_t pair;
  uint32_t lw;
};
constexpr int kRecLenBits = 29;
constexpr int64_t kMaxColp = int64_t(1) << 35;      // padded columns the records can address
constexpr int64_t kMaxRecLen = int64_t(1) << kRecLenBits;
__host__ __device__ inline InRec make_inrec(int64_t s, int64_t len) {
  InRec r;
  r.pair = uint32_t(s >> 3);
  r.lw = uint32_t(len) | (uint32_t(s & 7) << kRecLenBits);
  return r;
}
__host__ __device__ inline int64_t rec_s(InRec r) { return (int64_t(r.pair) << 3) | int64_t(r.lw >> kRecLenBits); }
__host__ __device__ inline int32_t rec_len(InRec r) { return int32_t(r.lw & uint32_t(kMaxRecLen - 1)); }

// The graph's dense core (core.cu): operand tiles and work items of the part
// of the count that runs on the tensor cores. Empty (n_items 0) for graphs
// that gain nothing by it.
struct Core {
  int nb = 0;                 // row blocks of 128, from the highest id down
  int64_t *d_tile0 = nullptr;  // per row block: its first operand tile (nb + 1; one allocation with the next three)
  int32_t *d_jw = nullptr;     // ... its width / 256 (0: none)
  int32_t *d_cut = nullptr;    // ... the first head id whose record from the block is counted here
  int32_t *d_item0 = nullptr;  // ... its items' place in the list
  uint8_t *d_tiles = nullptr;
  uint16_t *d_before = nullptr;  // per tile pair and row: the row's entries at positions before them
  int2 *d_items = nullptr;    // (row block, column step)
  int jtop = 0;               // the widest row block's d_jw
  // per-vertex and per-edge counts, built by their first: the symmetric core, the
  // transposed tiles, the row blocks wider than each step
  uint8_t *d_sym = nullptr, *d_xt = nullptr;
  int32_t *d_list = nullptr;
  int64_t n_tiles = 0, n_items = 0;
  int64_t gain_fs = 0;        // estimated, of a global count
};

struct Graph {
  Ctx *ctx = nullptr;
  int64_t nv = 0;
  int64_t n_input = 0;
  int64_t ne = 0;  // |E+|
  int orient = XT_ORIENT_DEGREE;
  // Vertices are renumbered so that the orientation rank IS the id: under
  // XT_ORIENT_DEGREE, internal id = position in (degree, input id) order;
  // under XT_ORIENT_ID the numbering is the input's. Every edge then points
  // from the lower to the higher internal id and rows ascend by rank.
  int64_t *d_off = nullptr;   // out-CSR offsets, nv+1
  int32_t *d_col = nullptr;   // out-CSR columns N+(u), ne (+kColPad), rows ascending
  int64_t *d_ioff = nullptr;  // in-record offsets per head v, nv+1
  InRec *d_irec = nullptr;    // one record per edge u->v, grouped by v (ne + 2: the last 16 bytes are slack
                              //   for 16-byte aligned bulk prefetches)
  // the first in-record of each head that the count does not stream (no
  // candidates, or the core's): nv
  int64_t *d_iend = nullptr;
  Core core;
  bool no_core = false;         // the batch form counts per graph: no core
  int32_t *d_irec_u = nullptr;  // the tail u of each record, built on first use (per-vertex, per-edge)
  // The columns again, each row starting on an 8-column (32-byte) boundary
  // and padded with kPadSentinel: the count streams suffixes from here in
  // whole 32-byte pairs without masking. d_poff[u] is row u's start.
  int32_t *d_colp = nullptr;
  int64_t *d_poff = nullptr;  // nv+1
  int32_t *d_perm = nullptr;  // internal id -> input id (null when identity)
  int64_t max_degree = 0;
  int64_t max_out_degree = 0;
  int64_t max_in_degree = 0;
  int64_t tune_block_work = 0;  // schedule overrides (0: choose automatically)
  int64_t tune_warp_work = 0;
  int64_t tune_bitmap_bits = 0;
  int prefetch_suffix = 0;      // global count: bulk L2 prefetch of each record's suffix (1) or not (0)
  int lane_merge = 0;            // lane tasks: two-pointer merge (1) or binary search (0) over N+(v)
  int cluster_tier = 0;         // global count: heads over a CTA's member set on thread-block clusters (1) or
                                //   as CTA tasks over parts of their members (0, the default: faster)
  int cuckoo_iters = -1;        // test hook: cuckoo eviction chain limit (-1: the default)
  int claim_block = 0;          // warp tasks taken per atomic on their cursor (0: 4 for a batch, else 1)
  int64_t tier_lane_work = -1;  // tier limits (-1: automatic, 0: tier off)
  int64_t tier_warp_work = -1;
  int32_t *d_group = nullptr;   // internal id -> group (graph of a batch), or null
  int64_t n_groups = 0;
  // a captured count (CUDA graph) writing the total and the per-group
  // counts into d_res[0] and d_res[1..n_groups]
  cudaGraphExec_t exec = nullptr;
  int64_t exec_kernels = 0;  // library kernels inside `exec`, counted per replay
  int64_t *d_res = nullptr;
  int64_t wedge_work = 0;   // sum over oriented (u,v) of d+(v)
  int64_t stream_work = 0;  // sum over u of C(d+(u), 2): the suffix columns the count streams
  int64_t colp_len = 0;     // entries of the padded column array
  Plan *plan = nullptr;
  Plan *shard_plans = nullptr;  // schedules cut for numbers of shards, each built by the first count that
                                //   needs it, the last one first
  int plan_for = 1;             // the shards make_plan cuts for
};

// Optional: the rows still in host memory. build_from_edges then copies
// them into d_src/d_dst (device buffers of ne rows) in chunks on the
// context's copy stream and turns each chunk into keys as soon as it lands,
// so key generation overlaps the copy-in.
struct HostRows {
  const int32_t *src, *dst;
};

// The graphs of a batch (device tables; ng 0: one graph): graph g's rows are
// [eoff[g], eoff[g+1]), its ids, local in those rows, [voff[g], voff[g+1]).
struct BatchTables {
  const int64_t *eoff = nullptr, *voff = nullptr;
  int64_t ng = 0;
};

// Builds the oriented CSR from a device edge list (int32 ids) of ne rows.
// Rows may repeat, be one-directional or self loops.
xt_status build_from_edges(Ctx *c, int64_t nv, int64_t ne, const int32_t *d_src, const int32_t *d_dst,
                           int orient, Graph *g, const HostRows *upload = nullptr, const BatchTables &bt = {});
// Builds from a device CSR (int64 offsets and tails). canonical: rows already
// sorted, deduped, symmetric and loop-free, so no sort is needed. ne_known: the
// entries, where the caller has seen that the offsets start at 0 and end there.
xt_status build_from_csr(Ctx *c, int64_t nv, const int64_t *d_off, const int64_t *d_tails, bool canonical,
                         int orient, Graph *g, int64_t ne_known = -1);
void free_graph_device(Graph *g);
// Reads a vite binary file (8- or 4-byte fields) through pinned staging
// buffers into a device CSR and builds from it (vite.cu).
xt_status build_from_vite(Ctx *c, const char *path, int elem_bytes, bool canonical, int orient, Graph *g);

// Builds the disjoint union of ng graphs (host offset tables, device edge
// rows with graph-local ids) as one graph with a per-vertex group map.
xt_status build_batch(Ctx *c, int64_t ng, const int64_t *h_voff, const int64_t *h_eoff, const int32_t *d_src,
                      const int32_t *d_dst, int orient, Graph *g, const HostRows *upload = nullptr);

// The dense core (core.cu), in the builder's order: widths chosen from the
// unique rows, kept or dropped once their sums are read back, then operands
// and items from the finished graph; its part of a count.
constexpr int kCoreSums = 4;  // words read back: tiles, items, widest row block, gain in fs
xt_status core_plan(Ctx *c, Graph *g, const int64_t *rstart, const uint32_t *cols, int64_t m, int64_t **d_sums);
void core_decide(Ctx *c, Graph *g, const int64_t *sums);
xt_status core_finish(Ctx *c, Graph *g);
xt_status core_count(Graph *g, int64_t *d_global, int64_t *d_pv, unsigned int *d_es, int shard, int nshards);
void core_free(Graph *g);
int64_t core_bytes(const Graph *g);  // what a count reads of it
// test hook: whether the core's kernels that the calling thread launches give up at once
void core_give_up(bool on);

// Builds (or rebuilds) the per-graph schedule and graph statistics.
xt_status make_plan(Graph *g);
void free_plan(Graph *g);

// Launches the count on the graph's context stream. d_global: one int64
// (overwritten); d_pv: nv int64 (nullable, overwritten).
// d_groups: n_groups int64 per-group counts (graphs built as a batch), nullable.
// d_support: ne int64, the triangles on each oriented edge in out-CSR order
// (nullable; not together with d_pv).
// shard / nshards: count only every nshards-th task of the schedule from
// task `shard` on (each tier's list alike); the nshards shards' outputs sum
// to the whole count's.
xt_status count_graph(Graph *g, int64_t *d_global, int64_t *d_pv, int64_t *d_groups = nullptr,
                      int64_t *d_support = nullptr, int shard = 0, int nshards = 1);
// Synchronises the context stream and reports a count whose bounded device
// wait gave up (XT_ERR_TIMEOUT); the synchronous count calls end with it.
// total (nullable) receives the context block's total.
xt_status count_status(Ctx *c, int64_t *total = nullptr);
// tasks of the global count's thread-block cluster tier in the graph's plan (0 without a plan)
int64_t cluster_task_count(const Graph *g);
// lane tasks in the graph's plan (0 without a plan)
int64_t lane_task_count(const Graph *g);

// ---- device helpers ----------------------------------------------------------
// Programmatic dependent launch: the next kernel of the stream, if it was
// launched so, may start now; and that kernel's wait until this one is complete
// and its writes are visible (at once in a kernel launched the plain way).
__device__ __forceinline__ void pdl_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// row holding position e, from a row at or before it: a few steps, then a search
// (a run of empty rows can be long)
__device__ __forceinline__ int64_t row_from(const int64_t *__restrict__ off, int64_t nv, int64_t r, int64_t e) {
  for (int i = 0; i < 8; i++) {
    if (r + 1 >= nv || off[r + 1] > e) return r;
    r++;
  }
  int64_t lo = r, hi = nv;
  while (hi - lo > 1) {
    const int64_t mid = lo + (hi - lo) / 2;
    if (off[mid] <= e) lo = mid;
    else hi = mid;
  }
  return lo;
}
// The same for a whole warp with ascending e and one r: the next 32 starts are
// read at once and searched by shuffles, so the lanes wait for one load
__device__ __forceinline__ int64_t row_near(const int64_t *__restrict__ off, int64_t nv, int64_t r, int64_t e, int lane) {
  const int64_t next = r + 1 + lane < nv ? off[r + 1 + lane] : INT64_MAX;
  int j = 0;
#pragma unroll
  for (int s = 16; s; s >>= 1)
    if (__shfl_sync(0xffffffffu, next, j + s - 1) <= e) j += s;
  if (__shfl_sync(0xffffffffu, next, j) <= e) j++;
  return j < 32 ? r + j : row_from(off, nv, r + 32, e);
}
// the last row of nv starting at or before e, searched by the whole warp (33 ways a step)
__device__ __forceinline__ int64_t row_of(const int64_t *__restrict__ off, int64_t nv, int64_t e, int lane) {
  int64_t lo = 0, hi = nv;
  while (hi - lo > 1) {
    const int64_t w = (hi - lo + 31) / 32, x = lo + lane * w;
    const unsigned m = __ballot_sync(0xffffffffu, x < hi && off[x] <= e);
    if (m) lo += (31 - __clz(int(m))) * w;  // lane 0 fails only where e lies before every row
    hi = lo + w < hi ? lo + w : hi;
  }
  return lo;
}

}  // namespace xt

// The host set-up of the reference's random geometric graph (host_io.cpp):
// radius, each strip rank's first LCG value and its strip [lo, lo + range).
xt_status xt_rgg_setup(int64_t nv, int nprocs, double radius, double *rn, int64_t *x0, double *lo, double *range);

struct xt_ctx {
  xt::Ctx c;
};
struct xt_graph {
  xt::Graph g;
};
