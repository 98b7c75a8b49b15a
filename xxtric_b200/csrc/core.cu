// The dense core of the oriented graph, counted on the tensor cores.
//
// In (degree, id) rank order the columns of a power-law graph crowd the top
// ranks: on R-MAT 2^22, 44% of the candidates the count streams lie in blocks
// of the adjacency matrix that hold an edge in every 10th to 50th place. There
// a contraction does 8,192 multiply-adds per SM and cycle where the streaming
// kernel (count.cu) spends about 15 instructions on a candidate, so those
// blocks leave its schedule and are counted here.
//
// Notation: rank position i of a vertex counts from the top, i = nv - 1 - id,
// so N+(u) are positions below u's. Rows are taken in blocks of 128 positions,
// columns in chunks of 128. Row block b has a width T_b (a multiple of 256,
// at most kCoreWidth; 0: none): the triangles u < v < w (ids) with u in block b
// and v among the top T_b positions (w, above v, is then too) are
//     sum over v of X[u][v] * (sum over w of X[u][w] * X[v][w]),
// X the 0/1 adjacency matrix, the inner sum a product of the rows of block b
// with the rows of the top T_b vertices. Every one of them has its streamed
// candidates in the in-records u->v, which the builder puts last among v's
// records (Graph::d_iend[v] is the first of them) and the schedule leaves out.
// The reference has no counterpart: its kernels intersect sorted lists
// (counting.cu:95-131).
//
// Per vertex and per edge the same blocks give every triangle's other corners
// and edges. With S the symmetric adjacency matrix of the core, D = X S under the
// mask X holds for each edge u->c of the row block its core triangles whose lowest
// corner is u: D's row sums are twice u's, its column sums are those of c as a
// middle or highest corner, and its entries the supports. The third edge v->w
// needs the sum over u of X[u][v] X[u][w], a product along the row blocks (their
// tiles transposed), cut into segments of row blocks.
//
// Operands: one byte per element in 16 KB tiles of 128 rows x 128 columns, laid
// out in memory as a 128-byte-swizzled K-major operand sits in shared memory
// (16-byte piece p of row r at p ^ (r & 7)), so a tile is one bulk copy.
#include <cub/cub.cuh>

#include <algorithm>
#include <numeric>

#include "xt_internal.cuh"

namespace xt {

constexpr int kCoreRows = 128;          // rows of a block, columns of a chunk
constexpr int kCoreTile = kCoreRows * 128;
constexpr int kCoreStep = 256;          // widths are multiples of this: the columns of one work item
constexpr int kCoreMaxJ = 64;           // widths up to 64 * 256
constexpr int kCoreWidth = kCoreMaxJ * kCoreStep;
constexpr int kCoreMinBlk = kCoreWidth / kCoreRows;  // the core's own rows
constexpr int kCoreMaxBlk = 8192;       // row blocks looked at: the top 2^20 vertices
constexpr int kCoreMinRow = 16;         // shorter rows gain less than their share of a step

// The rule of T_b weighs, per block, the streamed candidates it takes away
// against the chunk steps (128 x 256 x 128 multiply-adds) it adds, each at the
// rate the whole GPU runs it: a candidate of these long suffixes 0.4 ps, a
// chunk step 2.2 ns (3.8e15 operations a second), both measured on R-MAT 2^24
// and 2^22 and Chung-Lu 2^22. The optimum is flat: steps taken at 1 or 4 ns
// move those counts by 2%.
constexpr int64_t kCandFs = 400;
constexpr int64_t kStepFs = 2200000;
// below this gain in all (20 us) the second launch is not worth it
constexpr int64_t kCoreMinFs = int64_t(20) * 1000 * 1000 * 1000;
constexpr int64_t kCoreMaxBytes = 16;  // operand bytes per edge, at most

// J = T_b / 256 of row block blockIdx.x: four rows a warp, each lane holding
// the benefit of two widths. A row has C(c, 2) candidates whose v lies in the
// top T positions, c its columns there: its entries from the end on, 128 at a
// time, go into a histogram of 256 positions a bin, whose prefix sum is c.
// (Sixteen rows a warp, or binary searches for every width, took 190 us on
// R-MAT 2^21: chains of misses in the widest rows' blocks.)
__global__ void __launch_bounds__(1024) k_core_pick(int64_t nv, const int64_t *__restrict__ rstart,
                                                    const int64_t *__restrict__ off, const uint32_t *__restrict__ cols,
                                                    int32_t *__restrict__ jw, int32_t *__restrict__ cut,
                                                    unsigned long long *__restrict__ gain) {
  __shared__ unsigned long long s_ben[kCoreMaxJ];
  __shared__ int s_hist[32][kCoreMaxJ];
  __shared__ unsigned s_all;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b = blockIdx.x;
  if (threadIdx.x < kCoreMaxJ) s_ben[threadIdx.x] = 0;
  if (threadIdx.x == 0) s_all = 0;
  __syncthreads();
  unsigned long long ben0 = 0, ben1 = 0;
  // lane l < 4 holds the warp's row l: its end and length
  int64_t end = 0;
  int32_t len = 0;
  {
    const int64_t u = nv - 1 - (int64_t(b) * kCoreRows + warp * 4 + lane);
    if (lane < 4 && u >= 0) {
      len = int32_t(off[u + 1] - off[u]);
      end = rstart[u] + len;
    }
    if (len < kCoreMinRow) len = 0;
    const unsigned all = __reduce_add_sync(0xffffffffu, unsigned(min(int64_t(len) * (len - 1) / 2, int64_t(1) << 20)));
    if (lane == 0 && all) atomicAdd(&s_all, all);
  }
  __syncthreads();
  // all candidates of its rows cannot pay for the narrowest width: no columns read
  // (R-MAT 2^21 107 -> 94 us, a geometric graph of 2^20 vertices 48 -> 31)
  if ((unsigned long long)s_all * kCandFs <= (unsigned long long)(4 * kStepFs)) {
    if (threadIdx.x == 0) {
      jw[b] = 0;
      cut[b] = 0x7fffffff;
    }
    return;
  }
  const uint32_t top = uint32_t(nv - 1);
  for (int q = 0; q < 4; q++) {
    const int32_t n = __shfl_sync(0xffffffffu, len, q);
    if (n == 0) continue;
    const uint32_t *last = cols + __shfl_sync(0xffffffffu, end, q) - 1 - lane;
    s_hist[warp][lane] = 0;
    s_hist[warp][lane + 32] = 0;
    __syncwarp();
    for (int32_t at = 0; at < n; at += 128) {
      uint32_t x[4];
#pragma unroll
      for (int h = 0; h < 4; h++) x[h] = at + 32 * h + lane < n ? top - last[-(at + 32 * h)] : 0xffffffffu;
#pragma unroll
      for (int h = 0; h < 4; h++)
        if (x[h] < uint32_t(kCoreWidth)) atomicAdd(&s_hist[warp][x[h] / kCoreStep], 1);
      if (!__any_sync(0xffffffffu, x[3] < uint32_t(kCoreWidth))) break;
    }
    __syncwarp();
    int c0 = s_hist[warp][lane], c1 = s_hist[warp][lane + 32];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a0 = __shfl_up_sync(0xffffffffu, c0, o), a1 = __shfl_up_sync(0xffffffffu, c1, o);
      if (lane >= o) {
        c0 += a0;
        c1 += a1;
      }
    }
    c1 += __shfl_sync(0xffffffffu, c0, 31);
    ben0 += (unsigned long long)c0 * (unsigned long long)(c0 - (c0 > 0)) / 2;
    ben1 += (unsigned long long)c1 * (unsigned long long)(c1 - (c1 > 0)) / 2;
    __syncwarp();
  }
  if (ben0) atomicAdd(&s_ben[lane], ben0);
  if (ben1) atomicAdd(&s_ben[lane + 32], ben1);
  __syncthreads();
  if (warp != 0) return;
  const int jmax = b / 2 + 1;  // the rows' own positions bound their columns
  long long best = 0;
  int bj = 0;
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int j = lane + 32 * h + 1;
    const unsigned long long ben = s_ben[j - 1];
    // item i of the block runs 2 i + 2 chunk steps; reading its accumulator
    // and building its operand cost about two more
    const long long net = (long long)(ben * kCandFs) - (long long)(int64_t(j) * (j + 3) * kStepFs);
    if (j <= jmax && net > best) {
      best = net;
      bj = j;
    }
  }
  for (int o = 16; o; o >>= 1) {
    const long long ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int oj = __shfl_xor_sync(0xffffffffu, bj, o);
    if (ob > best || (ob == best && oj < bj)) {
      best = ob;
      bj = oj;
    }
  }
  if (lane == 0) {
    jw[b] = bj;
    const int64_t c = nv - int64_t(bj) * kCoreStep;
    cut[b] = bj ? int32_t(c > 0 ? c : 0) : 0x7fffffff;
    if (best > 0) atomicAdd(gain, (unsigned long long)best);
  }
}

// chunks stored for row block b: a core row's own columns (an even number of
// chunks, so that an item reads whole pairs), any other's width
__device__ __forceinline__ int core_chunks(int b, int j, int jtop) { return b < 2 * jtop ? (b | 1) + 1 : 2 * j; }

// Tile and item offsets of the nb row blocks (one CTA, at most 8 blocks a
// thread; tiles and items scanned as the halves of one 64-bit sum).
__global__ void __launch_bounds__(1024) k_core_layout(int nb, const int32_t *__restrict__ jw,
                                                      int64_t *__restrict__ tile0, int32_t *__restrict__ item0,
                                                      int64_t *__restrict__ sums) {
  using Scan = cub::BlockScan<unsigned long long, 1024>;
  __shared__ typename Scan::TempStorage ts;
  __shared__ int s_top;
  constexpr int kPer = kCoreMaxBlk / 1024;
  if (threadIdx.x == 0) s_top = 0;
  __syncthreads();
  int j[kPer], top = 0;
#pragma unroll
  for (int i = 0; i < kPer; i++) {
    const int b = threadIdx.x * kPer + i;
    j[i] = b < nb ? jw[b] : 0;
    top = max(top, j[i]);
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if ((threadIdx.x & 31) == 0 && top) atomicMax(&s_top, top);
  __syncthreads();
  top = s_top;
  unsigned long long own = 0, at, tot;
#pragma unroll
  for (int i = 0; i < kPer; i++) {
    const int b = threadIdx.x * kPer + i;
    if (b < nb) own += (unsigned long long)core_chunks(b, j[i], top) << 32 | (unsigned long long)j[i];
  }
  Scan(ts).ExclusiveSum(own, at, tot);
#pragma unroll
  for (int i = 0; i < kPer; i++) {
    const int b = threadIdx.x * kPer + i;
    if (b >= nb) break;
    tile0[b] = int64_t(at >> 32);
    item0[b] = int32_t(at & 0xffffffffu);
    at += (unsigned long long)core_chunks(b, j[i], top) << 32 | (unsigned long long)j[i];
  }
  if (threadIdx.x == 0) {
    tile0[nb] = int64_t(tot >> 32);
    sums[0] = int64_t(tot >> 32);
    sums[1] = int64_t(tot & 0xffffffffu);
    sums[2] = top;
  }
}

// Work items (row block, column step): groups of 32 row blocks, within one the
// longest items first, so the CTAs that run together share the operand of
// their columns and the last ones are short.
__global__ void k_core_items(int nb, const int32_t *__restrict__ jw, const int32_t *__restrict__ item0,
                             int2 *__restrict__ items) {
  const int lane = threadIdx.x & 31;
  const int b = (blockIdx.x * blockDim.x + threadIdx.x);
  if ((b & ~31) >= nb) return;
  const int j = b < nb ? jw[b] : 0;
  int at = __shfl_sync(0xffffffffu, b < nb ? item0[b] : 0, 0);
  for (int t = kCoreMaxJ - 1; t >= 0; t--) {
    const unsigned m = __ballot_sync(0xffffffffu, j > t);
    if (j > t) items[at + __popc(m & ((1u << lane) - 1u))] = make_int2(b, t);
    at += __popc(m);
  }
}

// The operand tiles, two chunks (32 KB) per CTA, set in shared memory and
// written out whole: two threads a row set the row's bytes from the first of
// its positions in these chunks (the positions ascend from the row's end).
// before: per tile pair and row, the row's entries at positions before them.
__global__ void __launch_bounds__(256) k_core_tiles(int64_t nv, int nb, const int64_t *__restrict__ off,
                                                    const int32_t *__restrict__ col,
                                                    const int64_t *__restrict__ tile0, uint8_t *__restrict__ tiles,
                                                    uint16_t *__restrict__ before) {
  __shared__ __align__(16) uint8_t s_t[2 * kCoreTile];
  const int lane = threadIdx.x & 31, r = threadIdx.x >> 1;
  const int64_t t = 2 * int64_t(blockIdx.x);
  for (int i = threadIdx.x; i < 2 * kCoreTile / 16; i += 256)
    reinterpret_cast<int4 *>(s_t)[i] = make_int4(0, 0, 0, 0);
  int b = 0, end = nb;  // the row block holding tile t, by 32-way steps
  while (end - b > 1) {
    const int w = (end - b + 31) / 32, x = b + lane * w;
    const unsigned m = __ballot_sync(0xffffffffu, x < end && tile0[x] <= t);
    b += (31 - __clz(int(m))) * w;
    end = min(end, b + w);
  }
  const int64_t c0 = (t - tile0[b]) * kCoreRows;  // first position of these columns
  const int64_t u = nv - 1 - (int64_t(b) * kCoreRows + r);
  __syncthreads();
  if (u >= 0) {
    const int64_t e0 = off[u], e1 = off[u + 1];
    int64_t lo = e0, hi = e1;  // entries [e0, lo) lie at positions >= c0
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (nv - 1 - int64_t(col[mid]) >= c0) lo = mid + 1;
      else hi = mid;
    }
    if ((threadIdx.x & 1) == 0) before[t / 2 * kCoreRows + r] = uint16_t(e1 - lo);
    for (int64_t p = lo - 1 - (threadIdx.x & 1); p >= e0; p -= 2) {
      const int64_t c = nv - 1 - int64_t(col[p]) - c0;
      if (c >= kCoreStep) break;
      const int x = int(c) & 127;
      s_t[(int(c) >> 7) * kCoreTile + r * 128 + (((x >> 4) ^ (r & 7)) << 4) + (x & 15)] = 1;
    }
  }
  __syncthreads();
  int4 *out = reinterpret_cast<int4 *>(tiles + t * kCoreTile);
  for (int i = threadIdx.x; i < 2 * kCoreTile / 16; i += 256) out[i] = reinterpret_cast<int4 *>(s_t)[i];
}

// ---- the product --------------------------------------------------------------

constexpr int kCoreStages = 4;
constexpr int kCoreStageBytes = 3 * kCoreTile;  // 128 rows of X, 256 rows of the core
constexpr int kCoreThreads = 192;
constexpr size_t kCoreSmem = size_t(kCoreStages) * kCoreStageBytes + 1024;
constexpr uint32_t kCoreWaitLimit = 1u << 22;

// what a product gives: the total; every vertex's count; every edge's, for the
// edges from the row blocks, and for the edges inside the core
enum CoreKind { kCoreTotal = 0, kCoreVertices = 1, kCoreEdges = 2, kCoreInner = 3 };
constexpr int kCoreSeg = 64;  // kCoreInner: row blocks of one item, at most

struct CoreArgs {
  const uint8_t *tiles;
  const int64_t *tile0;
  const int2 *items;
  int64_t n;       // items of this launch: items[0], items[stride], ...
  int64_t stride;
  unsigned long long *global;
  int *err;
  int give_up;     // as if a wait had given up already (test hook)
  // per vertex and per edge
  const uint8_t *sym;      // S: tile (row block, chunk) at row block * 2 jtop + chunk
  const int32_t *jw;
  int jtop;
  int shard, nshards;      // of the row blocks (kCoreInner: of the items)
  int64_t nv;
  const int64_t *off, *poff;
  const uint16_t *before;
  unsigned long long *rows2;  // twice the count of each row as the lowest corner
  unsigned long long *pv;
  unsigned int *es;
  // kCoreInner
  const uint8_t *xt;       // the transposed tiles
  const int32_t *list;     // level t: first tiles of the row blocks wider than t steps, nb entries each
  const int32_t *count;    // ... how many
  int nb;
};

__device__ __forceinline__ uint32_t core_smem(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void core_bar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(core_smem(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void core_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(core_smem(bar)) : "memory");
}
__device__ __forceinline__ void core_expect(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(core_smem(bar)), "r"(bytes)
               : "memory");
}
// waits for the barrier's phase, at most kCoreWaitLimit tries; gives up early
// once another warp of the CTA has (the limit as a kernel argument cost the products
// 3%, 70 us of a R-MAT 2^24 count)
__device__ __forceinline__ bool core_wait(uint64_t *bar, uint32_t parity, volatile int *fail) {
  for (uint32_t it = 0; it < kCoreWaitLimit; it++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(core_smem(bar)), "r"(parity)
        : "memory");
    if (done) return true;
    if ((it & 255u) == 255u && *fail) return false;
  }
  *fail = 1;
  return false;
}
__device__ __forceinline__ void core_copy(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   core_smem(dst)),
               "l"(src), "r"(bytes), "r"(core_smem(bar))
               : "memory");
}
// 128-byte-swizzled K-major operand at a 1,024-byte aligned shared address:
// 8-row groups 1,024 bytes apart
__device__ __forceinline__ uint64_t core_desc(uint32_t saddr) {
  return uint64_t((saddr & 0x3ffffu) >> 4) | (uint64_t(1) << 16) | (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) |
         (uint64_t(2) << 61);
}
__device__ __forceinline__ void core_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(uint32_t(acc))
      : "memory");
}
__device__ __forceinline__ void core_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(core_smem(bar))
               : "memory");
}
// 32 columns of this warp's 32 accumulator rows
__device__ __forceinline__ void core_ld32(uint32_t taddr, int32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
        "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}

// An item of one kind: its accumulator's rows are row block b, its columns the
// positions 256 j on; `steps` chunk steps.
struct CoreItem {
  int b, j, steps;
  int level, first;  // kCoreInner: the list, and the first of its entries
};
// item i of the launch; false when it is another shard's
template <int KIND>
__device__ __forceinline__ bool core_item(const CoreArgs &a, const int32_t *pfx, int64_t i, CoreItem &it) {
  it.level = it.first = 0;
  if (KIND == kCoreInner) {
    if (a.nshards > 1 && i % a.nshards != a.shard) return false;
    int t = 0;  // the level holding item i
    while (int64_t(pfx[t + 1]) <= i) t++;
    const int segs = (a.count[t] + kCoreSeg - 1) / kCoreSeg, k = int(i - pfx[t]);
    const int cell = k / segs;  // (row block 2t or 2t + 1, column step 0 .. t)
    it.b = 2 * t + (cell > t);
    it.j = cell > t ? cell - t - 1 : cell;
    it.level = t;
    it.first = (k - cell * segs) * kCoreSeg;
    it.steps = min(kCoreSeg, a.count[t] - it.first);
    return true;
  }
  const int2 x = a.items[i * a.stride];
  it.b = x.x;
  it.j = x.y;
  if (KIND == kCoreTotal) {
    it.steps = 2 * x.y + 2;
    return true;
  }
  it.steps = 2 * a.jw[x.x];
  return a.nshards <= 1 || x.x % a.nshards == a.shard;
}

// One persistent CTA per SM. Warp 0 brings in the tiles of each chunk step,
// warp 1 issues the products of unsigned bytes into one of two 256-column
// accumulators (32-bit integers: exact), warps 2 to 5 read the other and add it
// up under its mask (the item's two chunks of X): 3.8e15 operations/s on R-MAT
// 2^24, near the tensor rate; 48 KB are read from L2 a step.
template <int KIND>
__global__ void __launch_bounds__(kCoreThreads, 1) k_core_count(const CoreArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *st = smem_raw + ((1024 - (core_smem(smem_raw) & 1023)) & 1023);
  __shared__ __align__(8) uint64_t s_full[kCoreStages], s_empty[kCoreStages], s_tfull[2], s_tempty[2], s_drain;
  __shared__ uint32_t s_tmem;
  __shared__ int s_fail;
  __shared__ int32_t s_pfx[kCoreMaxJ + 2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_launch_dependents();  // the streaming kernel's CTAs start as this one's leave
  if (threadIdx.x == 0) {
    for (int i = 0; i < kCoreStages; i++) {
      core_bar_init(&s_full[i], 1);
      core_bar_init(&s_empty[i], 1);
    }
    for (int i = 0; i < 2; i++) {
      core_bar_init(&s_tfull[i], 1);
      core_bar_init(&s_tempty[i], 4);
    }
    core_bar_init(&s_drain, 1);
    s_fail = a.give_up;
    if (KIND == kCoreInner) {  // items before each level
      int32_t at = 0;
      for (int t = 0; t < a.jtop; t++) {
        s_pfx[t] = at;
        at += 2 * (t + 1) * ((a.count[t] + kCoreSeg - 1) / kCoreSeg);
      }
      s_pfx[a.jtop] = at;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(core_smem(&s_tmem)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_tmem;
  volatile int *fail = &s_fail;
  const int64_t n = KIND == kCoreInner ? int64_t(s_pfx[a.jtop]) : a.n;
  CoreItem it;

  if (warp == 0) {
    uint32_t k = 0;  // loads issued
    // stage k's buffer once it is free, its barrier expecting the step's bytes
    auto stage = [&]() -> uint8_t * {
      const uint32_t sg = k % kCoreStages;
      if (!core_wait(&s_empty[sg], ((k / kCoreStages) & 1u) ^ 1u, fail)) return nullptr;
      core_expect(&s_full[sg], kCoreStageBytes);
      return st + sg * kCoreStageBytes;
    };
    if (KIND != kCoreInner && lane == 0) {
      bool ok = true;
      for (int64_t i = blockIdx.x; i < n && ok; i += gridDim.x) {
        if (!core_item<KIND>(a, s_pfx, i, it)) continue;
        const uint8_t *x = a.tiles + a.tile0[it.b] * kCoreTile, *y0, *y1;
        if (KIND == kCoreTotal) {
          y0 = a.tiles + a.tile0[2 * it.j] * kCoreTile;
          y1 = a.tiles + a.tile0[2 * it.j + 1] * kCoreTile;
        } else {
          y0 = a.sym + int64_t(2 * it.j) * (2 * a.jtop) * kCoreTile;
          y1 = y0 + int64_t(2 * a.jtop) * kCoreTile;
        }
        for (int c = 0; c < it.steps; c++, k++) {
          uint8_t *d = stage();
          if (!d) {
            ok = false;
            break;
          }
          uint64_t *bar = &s_full[k % kCoreStages];
          core_copy(d, x + int64_t(c) * kCoreTile, kCoreTile, bar);
          core_copy(d + kCoreTile, y0 + int64_t(c) * kCoreTile, kCoreTile, bar);
          core_copy(d + 2 * kCoreTile, y1 + int64_t(c) * kCoreTile, kCoreTile, bar);
        }
      }
    }
    if (KIND == kCoreInner) {  // the whole warp: each lane reads one of 32 row blocks' first tiles
      bool ok = true;
      for (int64_t i = blockIdx.x; i < n && ok; i += gridDim.x) {
        if (!core_item<KIND>(a, s_pfx, i, it)) continue;
        for (int c0 = 0; c0 < it.steps && ok; c0 += 32) {
          const int m = min(32, it.steps - c0);
          const int32_t own = lane < m ? a.list[int64_t(it.level) * a.nb + it.first + c0 + lane] : 0;
          for (int c = 0; c < m && ok; c++) {
            const int64_t t = __shfl_sync(0xffffffffu, own, c);
            if (lane == 0) {
              uint8_t *d = stage();
              ok = d != nullptr;
              if (ok) {
                uint64_t *bar = &s_full[k % kCoreStages];
                core_copy(d, a.xt + (t + it.b) * kCoreTile, kCoreTile, bar);
                core_copy(d + kCoreTile, a.xt + (t + 2 * it.j) * kCoreTile, 2 * kCoreTile, bar);
                k++;
              }
            }
            ok = __shfl_sync(0xffffffffu, int(ok), 0);
          }
        }
      }
    }
    // the copies in flight land before the CTA leaves its shared memory to another:
    // always, as the products may give up after the last copy has been issued
    if (lane == 0)
      for (uint32_t q = k > kCoreStages ? k - kCoreStages : 0; q < k; q++) {
        int quiet = 0;
        core_wait(&s_full[q % kCoreStages], (q / kCoreStages) & 1u, &quiet);
      }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = (2u << 4) | (uint32_t(kCoreStep / 8) << 17) | (uint32_t(kCoreRows / 16) << 24);
      uint32_t k = 0, t = 0;
      for (int64_t i = blockIdx.x; i < n && !*fail; i += gridDim.x) {
        if (!core_item<KIND>(a, s_pfx, i, it)) continue;
        if (!core_wait(&s_tempty[t & 1], ((t >> 1) & 1u) ^ 1u, fail)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d = tmem + (t & 1) * kCoreStep;
        bool ok = true;
        for (int c = 0; c < it.steps; c++, k++) {
          const uint32_t sg = k % kCoreStages;
          if (!core_wait(&s_full[sg], (k / kCoreStages) & 1u, fail)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t sa = core_smem(st + sg * kCoreStageBytes);
          const uint64_t da = core_desc(sa), db = core_desc(sa + kCoreTile);
#pragma unroll
          for (int q = 0; q < 4; q++)  // 32 of the chunk's 128 columns each
            core_mma(d, da + 2 * q, db + 2 * q, idesc, c > 0 || q > 0);
          core_commit(&s_empty[sg]);
        }
        if (!ok) break;
        core_commit(&s_tfull[t & 1]);
        t++;
      }
      core_commit(&s_drain);  // every product issued is done before the accumulators are given back
      int quiet = 0;
      core_wait(&s_drain, 0, &quiet);
    }
    __syncwarp();
  } else {
    const int quad = warp & 3, r = quad * 32 + lane;  // this warp's accumulator rows
    int64_t acc = 0;
    uint32_t t = 0;
    for (int64_t i = blockIdx.x; i < n; i += gridDim.x) {
      if (!core_item<KIND>(a, s_pfx, i, it)) continue;
      const int64_t mt = a.tile0[it.b] + 2 * it.j;  // the mask's first tile
      const uint8_t *x = a.tiles + mt * kCoreTile + r * 128;
      uint4 m[16];  // X of the item's 256 columns
#pragma unroll
      for (int q = 0; q < 16; q++)
        m[q] = __ldg(reinterpret_cast<const uint4 *>(x + (q >> 3) * kCoreTile + (((q & 7) ^ (r & 7)) << 4)));
      const int64_t row = int64_t(it.b) * kCoreRows + r, u = a.nv - 1 - row;
      unsigned int *es = nullptr;  // per edge: the row's entry at the next position
      if ((KIND == kCoreEdges || KIND == kCoreInner) && u >= 0)
        es = a.es + a.poff[u] + (a.off[u + 1] - a.off[u]) - 1 - a.before[mt / 2 * kCoreRows + r];
      if (!__all_sync(0xffffffffu, core_wait(&s_tfull[t & 1], (t >> 1) & 1u, fail))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      int32_t sum = 0;
#pragma unroll
      for (int g = 0; g < kCoreStep / 32; g++) {
        int32_t v[32];
        core_ld32(tmem + (t & 1) * kCoreStep + g * 32 + (uint32_t(quad * 32) << 16), v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        int32_t cs = 0;  // per vertex: column sum of column 32 g + lane over this warp's rows
#pragma unroll
        for (int h = 0; h < 8; h++) {
          const uint4 &q = m[2 * g + (h >> 2)];
          const uint32_t w = (h & 3) == 0 ? q.x : (h & 3) == 1 ? q.y : (h & 3) == 2 ? q.z : q.w;
          if (KIND == kCoreTotal) {
            sum += int32_t(w & 0xffu) * v[4 * h] + int32_t((w >> 8) & 0xffu) * v[4 * h + 1] +
                   int32_t((w >> 16) & 0xffu) * v[4 * h + 2] + int32_t(w >> 24) * v[4 * h + 3];
          } else {
#pragma unroll
            for (int e = 0; e < 4; e++) {
              const bool in = (w >> (8 * e)) & 1u;
              const int32_t d = in ? v[4 * h + e] : 0;
              if (KIND != kCoreInner) sum += d;
              if (KIND == kCoreVertices) {
                const int32_t c = __reduce_add_sync(0xffffffffu, d);
                if (lane == 4 * h + e) cs = c;
              } else {
                if (d) atomicAdd(es, unsigned(d));
                es -= in ? 1 : 0;
              }
            }
          }
        }
        if (KIND == kCoreVertices && cs)
          atomicAdd(&a.pv[a.nv - 1 - (int64_t(it.j) * kCoreStep + g * 32 + lane)], (unsigned long long)cs);
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) core_arrive(&s_tempty[t & 1]);
      t++;
      if (KIND == kCoreTotal) acc += sum;
      else if (KIND != kCoreInner && sum) atomicAdd(&a.rows2[row], (unsigned long long)sum);
    }
    if (KIND == kCoreTotal) {
      for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0 && acc) atomicAdd(a.global, (unsigned long long)acc);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  if (threadIdx.x == 0 && s_fail && a.err) atomicOr(a.err, kErrCoreTimeout);
}

// ---- operands of the per-vertex and per-edge products ------------------------------

// byte (row, column) of a tile
__device__ __forceinline__ int core_at(int row, int col) {
  return row * 128 + (((col >> 4) ^ (row & 7)) << 4) + (col & 15);
}
// 16 columns (piece p) of row r of the transpose of a tile in shared memory
__device__ __forceinline__ uint4 core_transposed(const uint8_t *s, int r, int p) {
  uint32_t w[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    w[q] = 0;
#pragma unroll
    for (int e = 0; e < 4; e++) w[q] |= uint32_t(s[core_at(16 * p + 4 * q + e, r)]) << (8 * e);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// S, tile by tile: the core's own tiles below the diagonal, their transposes
// above it, both on it
__global__ void __launch_bounds__(256) k_core_sym(int width, const int64_t *__restrict__ tile0,
                                                  const uint8_t *__restrict__ tiles, uint8_t *__restrict__ sym) {
  __shared__ __align__(16) uint8_t s_t[kCoreTile];
  const int i = blockIdx.x / width, k = blockIdx.x % width;
  const uint8_t *src = tiles + (i >= k ? tile0[i] + k : tile0[k] + i) * kCoreTile;
  uint4 *out = reinterpret_cast<uint4 *>(sym + int64_t(blockIdx.x) * kCoreTile);
  for (int q = threadIdx.x; q < kCoreTile / 16; q += 256)
    reinterpret_cast<uint4 *>(s_t)[q] = reinterpret_cast<const uint4 *>(src)[q];
  __syncthreads();
  for (int q = threadIdx.x; q < kCoreTile / 16; q += 256) {
    const int r = q >> 3, p = (q & 7) ^ (r & 7);
    uint4 x = i >= k ? reinterpret_cast<uint4 *>(s_t)[q] : make_uint4(0, 0, 0, 0);
    if (i <= k) {
      const uint4 y = core_transposed(s_t, r, p);
      x = make_uint4(x.x | y.x, x.y | y.y, x.z | y.z, x.w | y.w);
    }
    out[q] = x;
  }
}
// every tile's transpose, in its place of a second array
__global__ void __launch_bounds__(256) k_core_turn(const uint8_t *__restrict__ tiles, uint8_t *__restrict__ xt) {
  __shared__ __align__(16) uint8_t s_t[kCoreTile];
  const uint4 *src = reinterpret_cast<const uint4 *>(tiles + int64_t(blockIdx.x) * kCoreTile);
  uint4 *out = reinterpret_cast<uint4 *>(xt + int64_t(blockIdx.x) * kCoreTile);
  for (int q = threadIdx.x; q < kCoreTile / 16; q += 256) reinterpret_cast<uint4 *>(s_t)[q] = src[q];
  __syncthreads();
  for (int q = threadIdx.x; q < kCoreTile / 16; q += 256) {
    const int r = q >> 3;
    out[q] = core_transposed(s_t, r, (q & 7) ^ (r & 7));
  }
}
// level blockIdx.x: the row blocks wider than that many steps, by their first tiles
__global__ void __launch_bounds__(1024) k_core_levels(int nb, const int32_t *__restrict__ jw,
                                                      const int64_t *__restrict__ tile0, int32_t *__restrict__ list,
                                                      int32_t *__restrict__ count) {
  using Scan = cub::BlockScan<int, 1024>;
  __shared__ typename Scan::TempStorage ts;
  int at = 0;
  for (int b0 = 0; b0 < nb; b0 += 1024) {
    const int b = b0 + threadIdx.x, in = b < nb && jw[b] > int(blockIdx.x);
    int pos, tot;
    Scan(ts).ExclusiveSum(in, pos, tot);
    if (in) list[int64_t(blockIdx.x) * nb + at + pos] = int32_t(tile0[b]);
    at += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) count[blockIdx.x] = at;
}
// half of each row's doubled count: to its vertex, and all of them to the total
__global__ void __launch_bounds__(256) k_core_halves(const unsigned long long *__restrict__ rows2, int64_t rows,
                                                     int64_t nv, unsigned long long *__restrict__ total,
                                                     unsigned long long *__restrict__ pv) {
  unsigned long long sum = 0;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < rows; i += int64_t(gridDim.x) * blockDim.x) {
    const unsigned long long h = rows2[i] / 2;
    if (!h) continue;
    sum += h;
    if (pv) atomicAdd(&pv[nv - 1 - i], h);
  }
  using Red = cub::BlockReduce<unsigned long long, 256>;
  __shared__ typename Red::TempStorage ts;
  sum = Red(ts).Sum(sum);
  if (threadIdx.x == 0 && sum) atomicAdd(total, sum);
}

// ---- per vertex and per edge without operands ---------------------------------------

// The credits of the core's records where the operands' memory cannot be had: a
// CTA per head of the core, a warp per record, each candidate looked up among the
// head's columns. No memory of its own; slower than the products (R-MAT 2^20 per
// edge 5.7 ms a count against 1.6, 2^21 per vertex 9.4 against 3.1), so only then.
// Shards take the same shares as the products', whatever path the others are on: a
// record's by its row block, the third edge's by the item of kCoreInner that holds it.
constexpr int kSearchThreads = 512;
constexpr int kSearchSmem = kCoreWidth * int(sizeof(unsigned));  // a counter a position of the core
template <bool EDGES>
__global__ void __launch_bounds__(kSearchThreads)
    k_core_search(const CoreArgs a, const int64_t *__restrict__ ioff, const int64_t *__restrict__ iend,
                  const InRec *__restrict__ rec, const int32_t *__restrict__ colp) {
  using Scan = cub::BlockScan<int, kSearchThreads>;
  using Red = cub::BlockReduce<unsigned long long, kSearchThreads>;
  extern __shared__ unsigned s_hits[];  // by position, of the head's columns, this shard's
  __shared__ uint32_t s_in[kCoreWidth / 32];  // the positions that are the head's columns
  __shared__ union {
    typename Scan::TempStorage scan;
    typename Red::TempStorage red;
  } ts;
  __shared__ int s_wider[kCoreMaxJ + 1];         // row blocks wider than t steps
  __shared__ int64_t s_item0[kCoreMaxJ + 1];     // kCoreInner's items before level t
  __shared__ uint8_t s_seg[kCoreMaxBlk];         // level t: each row block's segment
  constexpr int kPer = kCoreMaxBlk / kSearchThreads;
  static_assert(kCoreMaxBlk / kCoreSeg <= 256, "a segment's index fits a byte");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool split = EDGES && a.nshards > 1;
  if (split) {
    for (int t = threadIdx.x; t <= kCoreMaxJ; t += kSearchThreads) s_wider[t] = 0;
    __syncthreads();
    for (int b = threadIdx.x; b < a.nb; b += kSearchThreads)
      if (a.jw[b] > 0) atomicAdd(&s_wider[a.jw[b] - 1], 1);  // exactly that wide, first
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int t = kCoreMaxJ - 1; t >= 0; t--) s_wider[t] += s_wider[t + 1];
      int64_t at = 0;
      for (int t = 0; t <= kCoreMaxJ; t++) {
        s_item0[t] = at;
        at += 2 * (t + 1) * ((s_wider[t] + kCoreSeg - 1) / kCoreSeg);
      }
    }
    __syncthreads();
  }
  unsigned long long total = 0;
  int level = -1;
  const int64_t heads = min(a.nv, int64_t(a.jtop) * kCoreStep);
  for (int64_t pos = blockIdx.x; pos < heads; pos += gridDim.x) {
    const int64_t v = a.nv - 1 - pos, k0 = iend[v], k1 = ioff[v + 1];
    const int64_t m0 = a.poff[v];
    const int32_t dv = int32_t(a.off[v + 1] - a.off[v]);
    const int t = int(pos / kCoreStep);
    const int segs = split ? (s_wider[t] + kCoreSeg - 1) / kCoreSeg : 1;
    if (split && t != level) {
      level = t;
      int own = 0, at, wide[kPer];
      __syncthreads();
#pragma unroll
      for (int i = 0; i < kPer; i++) {
        const int b = threadIdx.x * kPer + i;
        wide[i] = b < a.nb && a.jw[b] > t;
        own += wide[i];
      }
      Scan(ts.scan).ExclusiveSum(own, at);
#pragma unroll
      for (int i = 0; i < kPer; i++) {
        s_seg[threadIdx.x * kPer + i] = uint8_t(at / kCoreSeg);
        at += wide[i];
      }
      __syncthreads();
    }
    for (int i = threadIdx.x; i < kCoreWidth / 32; i += kSearchThreads) s_in[i] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < dv; i += kSearchThreads) {
      const int x = int(a.nv - 1 - colp[m0 + i]);  // below pos
      atomicOr(&s_in[x >> 5], 1u << (x & 31));
      s_hits[x] = 0;
    }
    __syncthreads();
    unsigned long long hv = 0;
    for (int64_t k = k0 + warp; k < k1; k += kSearchThreads / 32) {
      const InRec r = rec[k];
      const int64_t s = rec_s(r);
      const int32_t len = rec_len(r);
      if (len == 0 || dv == 0) continue;
      const int64_t u = row_of(a.poff, a.nv, s - 1, lane);
      const int b = int((a.nv - 1 - u) / kCoreRows);
      const bool mine = a.nshards <= 1 || b % a.nshards == a.shard;
      if (!mine && !EDGES) continue;
      const int64_t item = split ? s_item0[t] + int64_t((pos / kCoreRows) & 1) * (t + 1) * segs + s_seg[b] : 0;
      unsigned h = 0;
      for (int32_t q = lane; q < len; q += 32) {
        const int x = int(a.nv - 1 - colp[s + q]);  // below pos
        if (!((s_in[x >> 5] >> (x & 31)) & 1u)) continue;
        h++;
        if (EDGES && mine) atomicAdd(&a.es[s + q], 1u);
        if (!split || (item + x / kCoreStep * segs) % a.nshards == a.shard) atomicAdd(&s_hits[x], 1u);
      }
      if (!mine) continue;
      hv += h;
      h = __reduce_add_sync(0xffffffffu, h);
      if (lane == 0 && h) {
        if (EDGES) atomicAdd(&a.es[s - 1], h);
        else atomicAdd(&a.pv[u], (unsigned long long)h);
      }
    }
    total += hv;
    for (int o = 16; o; o >>= 1) hv += __shfl_xor_sync(0xffffffffu, hv, o);
    if (!EDGES && hv && lane == 0) atomicAdd(&a.pv[v], hv);
    __syncthreads();
    for (int i = threadIdx.x; i < dv; i += kSearchThreads) {
      const int32_t w = colp[m0 + i];
      const unsigned h = s_hits[a.nv - 1 - w];
      if (!h) continue;
      if (EDGES) atomicAdd(&a.es[m0 + i], h);
      else atomicAdd(&a.pv[w], (unsigned long long)h);
    }
    __syncthreads();
  }
  __syncthreads();
  total = Red(ts.red).Sum(total);
  if (threadIdx.x == 0 && total) atomicAdd(a.global, total);
}

// ---- host side ------------------------------------------------------------------

static thread_local bool t_give_up = false;  // xt_debug_give_up
void core_give_up(bool on) { t_give_up = on; }

// Widths of the row blocks from the unique rows (row u: cols[rstart[u]] on, as
// many as off says), and their layout; *d_sums has kCoreSums words once the
// stream gets there. Leaves g->core empty (and *d_sums null) for graphs that
// cannot gain, and where the tables' memory cannot be had.
xt_status core_plan(Ctx *c, Graph *g, const int64_t *rstart, const uint32_t *cols, int64_t n, int64_t **d_sums) {
  *d_sums = nullptr;
  Core &k = g->core;
  // by degree, n rows without many repeats have some (2n)^1.5 / 6 candidates at most: below
  // 2^17 rows less than the least gain. By id there is no such bound; small id-ordered graphs
  // go without a core all the same, as their builds are short next to picking one
  if (g->no_core || n < (int64_t(1) << 17)) return XT_OK;
  const int64_t blocks = (g->nv + kCoreRows - 1) / kCoreRows;
  k.nb = int(std::max<int64_t>(kCoreMinBlk, std::min<int64_t>(blocks, kCoreMaxBlk)));
  // one allocation for the row blocks' tables: tile0, then jw, cut, item0
  if (dalloc_n(c, &k.d_tile0, size_t(k.nb + 1) + size_t(3 * k.nb + 1) / 2) != XT_OK ||
      dalloc_n(c, d_sums, kCoreSums) != XT_OK) {
    core_free(g);
    return XT_OK;
  }
  k.d_jw = reinterpret_cast<int32_t *>(k.d_tile0 + k.nb + 1);
  k.d_cut = k.d_jw + k.nb;
  k.d_item0 = k.d_cut + k.nb;
  XT_CUDA(c, cudaMemsetAsync(*d_sums, 0, kCoreSums * sizeof(int64_t), c->stream));
  k_core_pick<<<counted(c, dim3(k.nb)), 1024, 0, c->stream>>>(g->nv, rstart, g->d_off, cols, k.d_jw, k.d_cut,
                                                             reinterpret_cast<unsigned long long *>(*d_sums) + 3);
  k_core_layout<<<counted(c, dim3(1)), 1024, 0, c->stream>>>(k.nb, k.d_jw, k.d_tile0, k.d_item0, *d_sums);
  XT_CUDA(c, cudaGetLastError());
  return XT_OK;
}

// sums read back: keeps the core or drops it
void core_decide(Ctx *c, Graph *g, const int64_t *sums) {
  Core &k = g->core;
  if (k.nb == 0) return;
  // dropped also where the operands would outgrow the edges' own memory (a few
  // dense rows that reach far into a sparse core)
  if (sums[3] < kCoreMinFs || sums[1] == 0 || sums[0] * kCoreTile > kCoreMaxBytes * g->ne) {
    core_free(g);
    return;
  }
  k.n_tiles = sums[0];
  k.n_items = sums[1];
  k.jtop = int(sums[2]);
  k.gain_fs = sums[3];
}

// Operands and work items from the finished out-CSR. Called when the build's
// scratch has been given back (more of it than the operands' 16 bytes an edge, so
// they do not raise the build's peak); where their memory cannot be had the graph
// goes on without a core, all of its records streamed.
xt_status core_finish(Ctx *c, Graph *g) {
  Core &k = g->core;
  if (k.n_items == 0) return XT_OK;
  if (dalloc_n(c, &k.d_tiles, size_t(k.n_tiles) * kCoreTile) != XT_OK ||
      dalloc_n(c, &k.d_before, size_t(k.n_tiles / 2) * kCoreRows) != XT_OK ||
      dalloc_n(c, &k.d_items, size_t(k.n_items)) != XT_OK) {
    core_free(g);
    return cuda_status(c, cudaMemcpyAsync(g->d_iend, g->d_ioff + 1, sizeof(int64_t) * g->nv,
                                          cudaMemcpyDeviceToDevice, c->stream), "records without a core");
  }
  k_core_tiles<<<counted(c, dim3(unsigned(k.n_tiles / 2))), 256, 0, c->stream>>>(g->nv, k.nb, g->d_off, g->d_col,
                                                                                 k.d_tile0, k.d_tiles, k.d_before);
  k_core_items<<<counted(c, dim3(unsigned((k.nb + 255) / 256))), 256, 0, c->stream>>>(k.nb, k.d_jw, k.d_item0,
                                                                                     k.d_items);
  XT_CUDA(c, cudaGetLastError());
  for (auto fn : {k_core_count<kCoreTotal>, k_core_count<kCoreVertices>, k_core_count<kCoreEdges>,
                  k_core_count<kCoreInner>})
    XT_CUDA(c, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kCoreSmem)));
  return XT_OK;
}

// adds the core's triangles to *d_global: of every nshards-th item from
// `shard`, or, with d_pv (internal numbering) or d_es (padded column positions),
// of every nshards-th row block, with each triangle credited to its vertices
// or edges. The operands of the latter are built by their first count and kept;
// a count recorded into a CUDA graph before that builds its own each time, and
// one that cannot have their memory searches instead (k_core_search).
xt_status core_count(Graph *g, int64_t *d_global, int64_t *d_pv, unsigned int *d_es, int shard, int nshards) {
  Ctx *c = g->ctx;
  Core &k = g->core;
  CoreArgs a = {};
  a.tiles = k.d_tiles;
  a.tile0 = k.d_tile0;
  a.items = k.d_items;
  a.n = k.n_items;
  a.stride = 1;
  a.global = reinterpret_cast<unsigned long long *>(d_global);
  a.err = c->d_err;
  a.give_up = t_give_up ? 1 : 0;
  a.nv = g->nv;
  if (!d_pv && !d_es) {
    if (k.n_items <= shard) return XT_OK;
    a.items = k.d_items + shard;
    a.n = (k.n_items - shard + nshards - 1) / nshards;
    a.stride = nshards;
    const unsigned grid = unsigned(std::min<int64_t>(a.n, c->sm_count));
    k_core_count<kCoreTotal><<<counted(c, dim3(grid)), kCoreThreads, kCoreSmem, c->stream>>>(a);
    XT_CUDA(c, cudaGetLastError());
    return XT_OK;
  }
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(c->stream, &cap) != cudaSuccess) cudaGetLastError();
  const bool keep = cap == cudaStreamCaptureStatusNone;
  const int width = 2 * k.jtop;
  uint8_t *sym = k.d_sym, *xt = k.d_xt;
  int32_t *list = k.d_list;
  const int64_t rows = int64_t(k.nb) * kCoreRows;
  unsigned long long *rows2 = nullptr;
  bool have = sym || dalloc_n(c, &sym, size_t(width) * width * kCoreTile) == XT_OK;
  if (have && !k.d_sym) {
    if (keep) k.d_sym = sym;
    k_core_sym<<<counted(c, dim3(unsigned(width * width))), 256, 0, c->stream>>>(width, k.d_tile0, k.d_tiles, sym);
  }
  if (have && d_es && !xt) {
    if (!list) have = dalloc_n(c, &list, size_t(k.jtop) * k.nb + k.jtop) == XT_OK;
    if (keep) k.d_list = list;
    have = have && dalloc_n(c, &xt, size_t(k.n_tiles) * kCoreTile) == XT_OK;
    if (have) {
      if (keep) k.d_xt = xt;
      k_core_turn<<<counted(c, dim3(unsigned(k.n_tiles))), 256, 0, c->stream>>>(k.d_tiles, xt);
      k_core_levels<<<counted(c, dim3(unsigned(k.jtop))), 1024, 0, c->stream>>>(k.nb, k.d_jw, k.d_tile0, list,
                                                                               list + int64_t(k.jtop) * k.nb);
    }
  }
  have = have && dalloc_n(c, &rows2, size_t(rows)) == XT_OK;
  cudaError_t e = have ? cudaMemsetAsync(rows2, 0, sizeof(*rows2) * rows, c->stream) : cudaSuccess;
  a.sym = sym;
  a.jw = k.d_jw;
  a.jtop = k.jtop;
  a.shard = shard;
  a.nshards = nshards;
  a.off = g->d_off;
  a.poff = g->d_poff;
  a.before = k.d_before;
  a.rows2 = rows2;
  a.pv = reinterpret_cast<unsigned long long *>(d_pv);
  a.es = d_es;
  a.xt = xt;
  a.list = list;
  a.count = list ? list + int64_t(k.jtop) * k.nb : nullptr;
  a.nb = k.nb;
  if (!have) {
    const auto search = d_es ? k_core_search<true> : k_core_search<false>;
    const int64_t heads = std::min(g->nv, int64_t(k.jtop) * kCoreStep);
    e = cudaFuncSetAttribute(search, cudaFuncAttributeMaxDynamicSharedMemorySize, kSearchSmem);
    search<<<counted(c, dim3(unsigned(std::min<int64_t>(heads, c->sm_count * 3)))), kSearchThreads, kSearchSmem,
             c->stream>>>(a, g->d_ioff, g->d_iend, g->d_irec, g->d_colp);
    if (e == cudaSuccess) e = cudaGetLastError();
  } else if (e == cudaSuccess) {
    // a shard's items recur every nshards-th in the list, and a CTA takes every grid-th:
    // without a common factor every CTA comes upon some (with 8 shards and 148 CTAs 37 did
    // all the work: an eighth of R-MAT 2^22 per edge 1,899 us, 1,782 with 147; half of 2^20
    // 984 and 925)
    unsigned grid = unsigned(c->sm_count);
    while (grid > 1 && std::gcd(grid, unsigned(nshards)) != 1) grid--;
    if (d_es) {
      k_core_count<kCoreEdges><<<counted(c, dim3(grid)), kCoreThreads, kCoreSmem, c->stream>>>(a);
      k_core_count<kCoreInner><<<counted(c, dim3(grid)), kCoreThreads, kCoreSmem, c->stream>>>(a);
    } else {
      k_core_count<kCoreVertices><<<counted(c, dim3(grid)), kCoreThreads, kCoreSmem, c->stream>>>(a);
    }
    k_core_halves<<<counted(c, dim3(unsigned(std::min<int64_t>(rows / 256 + 1, c->sm_count * 4)))), 256, 0,
                    c->stream>>>(rows2, std::min(rows, g->nv), g->nv, a.global, a.pv);
    e = cudaGetLastError();
  }
  dfree(c, rows2);
  if (sym != k.d_sym) dfree(c, sym);
  if (xt != k.d_xt) dfree(c, xt);
  if (list != k.d_list) dfree(c, list);
  XT_CUDA(c, e);
  return XT_OK;
}

int64_t core_bytes(const Graph *g) {
  const Core &k = g->core;
  if (k.n_items == 0) return 0;
  return k.n_tiles * kCoreTile + k.n_items * int64_t(sizeof(int2)) + int64_t(sizeof(int64_t)) * (k.nb + 1);
}

void core_free(Graph *g) {
  Core &k = g->core;
  for (void *p : {(void *)k.d_tile0, (void *)k.d_tiles, (void *)k.d_before, (void *)k.d_items, (void *)k.d_sym, (void *)k.d_xt,
                  (void *)k.d_list}) dfree(g->ctx, p);
  g->core = Core{};
}

}  // namespace xt
