/* On-device binned-SAH BVH build.
 *
 * The reference builds its binary SAH BVH on one CPU thread (aggregate/native/BvhBuilder.cpp:48-253,
 * four candidate planes per axis, one O(n) pass per candidate) and its OptiX path hands the
 * build to the driver (aggregate/api/optix/host.cpp:440-480).  Here the build runs on the GPU,
 * top-down and breadth-first, with centroid binning:
 *
 *   k_begin          ids, the scene's box and centroid bounds, the root task and its chunks
 *   large nodes (> small_task primitives), three kernels per level:
 *     k_bin          centroid bins per axis in shared memory, merged into the node's global bins
 *     k_split        one CTA per node: SAH over bins*3 candidate planes, node allocation, children; the
 *                    last CTA to finish cuts the next level into chunks
 *     k_partition    primitive ids scattered to the children's ranges of the other id buffer, and the
 *                    children's centroid bounds on the way
 *   nodes of 33 to small_task primitives: k_build_small, one CTA per subtree, one primitive per thread
 *   nodes of <= 32 primitives: k_build_warps, one warp per subtree (exact sweep SAH over sorted
 *     centroids, no barriers)
 *   k_node_hist, k_scan_sums, k_scan_apply, k_permute: leaves sorted, nodes in depth-first order
 *
 * The task, chunk and node counts stay on the device: the host enqueues the levels of a balanced tree
 * and a few more and reads the counts once; only a tree with large nodes left goes on.
 *
 * Leaves list their primitives in a contiguous range of `order`; each leaf's range is finally
 * sorted by primitive index so the layout is deterministic (atomics only reorder primitives
 * inside a node's range, and SAH decisions depend on the set of primitives, not their order).
 * Child boxes are padded outwards by 2^-20 relative so transformed-instance boxes stay
 * conservative.  Below depth kMedianDepth nodes are split at their median position, which bounds
 * the depth (and the traversal stack) for any input.
 */
#include <algorithm>
#include <cfloat>
#include <chrono>

#include "bvh_build.cuh"
#include "traverse.cuh"

namespace nb {
namespace {

constexpr int kMaxBins = 32;
constexpr uint32_t kSmallTaskDefault = 256;
/* Primitives per CTA in the level kernels: 256 to 1024, four CTAs per SM where there are enough.  The
 * tree does not depend on it. */
constexpr uint32_t kMinChunk = 256, kMaxChunk = 1024;
constexpr int kMedianDepth = 40;
constexpr int kBlock = 256;
constexpr int kCtaPrims = 256; /* largest subtree of a CTA: one primitive per thread */
constexpr int kHardLeaf = 16;
constexpr int kSmallStack = 64;

struct Task {
  uint32_t begin, end;
  int32_t parent, slot, depth, buf;
  float lo[3], hi[3];
};

struct Bins {
  unsigned cnt[3][kMaxBins];
  float lo[3][kMaxBins][3];
  float hi[3][kMaxBins][3];
};

struct SplitInfo {
  int axis, bin, median;
  uint32_t mid;
  unsigned left_ptr, right_ptr;
  int child[2]; /* the children's tasks of the next level; -1: built by a CTA or a warp */
  float cmin[3], scale[3];
};

/* One level's counts. */
struct Level {
  unsigned tasks, chunks, done; /* done: CTAs of k_split that have finished */
};
constexpr int kMaxLevels = 96; /* kMedianDepth binned levels and 27 of halving, with room */

/* The build's counters, cleared before it. */
struct Counters {
  unsigned nodes, leaves, errors, small, warps, small_next, warp_next;
  int max_depth;
  unsigned begin_done;
  Level level[kMaxLevels];
};
constexpr int kWarpPrims = 32;

struct Chunk {
  uint32_t task, begin, end;
};

struct Shared {
  const float4 *lo, *hi;
  uint32_t *ids0, *ids1;
  float4 *nodes;
  /* An inner node's index until the last pass is the position its right child begins at, which no other
   * node shares, so nodes and leaves need no counter (93 k of each, by atomics on three words: k_build_warps
   * 147 us, without them 133). */
  uint2 *node_at; /* per position: the first primitive's position and the depth of its node; ~0: none */
  uint2 *leaf_at; /* per position: primitives (0: none) and depth of the leaf that begins there */
  uint32_t *order;
  Counters *n;
  Task *large[2]; /* a level's tasks, by the level's parity; likewise bins, cb and chunks */
  Bins *tbins[2];
  float *cb[2];
  Chunk *chunks[2];
  SplitInfo *splits;
  float *scene; /* box lo, hi, centroid lo, hi */
  Task *tasks;  /* subtrees of 33..small_task primitives from the front, of <= 32 from the back */
  uint32_t max_tasks, max_chunks, chunk;
  int bins, max_leaf, hard_leaf;
  uint32_t small_task;
  float cost_trav;
};

__device__ __forceinline__ uint32_t *ids_of(const Shared &s, int buf) { return buf ? s.ids1 : s.ids0; }

__device__ __forceinline__ void atomic_min_f(float *a, float v) {
  if (v >= 0.f)
    atomicMin(reinterpret_cast<int *>(a), __float_as_int(v));
  else
    atomicMax(reinterpret_cast<unsigned *>(a), __float_as_uint(v));
}
__device__ __forceinline__ void atomic_max_f(float *a, float v) {
  if (v >= 0.f)
    atomicMax(reinterpret_cast<int *>(a), __float_as_int(v));
  else
    atomicMin(reinterpret_cast<unsigned *>(a), __float_as_uint(v));
}

/* Adds each valid lane's primitive (box bl, bh) to bin b of one axis's shared bins.  When every lane
 * of the warp falls in the same bin (neighbouring primitives of a large node often do) the warp
 * reduces first and one lane adds, instead of 32 same-address atomics that execute one after the
 * other.  Counts, minima and maxima are exact, so the bins are the same either way.  All 32 lanes
 * call it. */
__device__ __forceinline__ void bin_add(unsigned *cnt, float (*lo)[3], float (*hi)[3], int b, bool valid,
                                        const float4 &bl, const float4 &bh) {
  const unsigned same = __match_any_sync(0xffffffffu, valid ? b : -1);
  if (same == 0xffffffffu) {
    if (!valid) return; /* uniform: an invalid lane's -1 matches only other invalid lanes */
    float l0 = bl.x, l1 = bl.y, l2 = bl.z, h0 = bh.x, h1 = bh.y, h2 = bh.z;
    for (int o = 16; o > 0; o >>= 1) {
      l0 = fminf(l0, __shfl_xor_sync(0xffffffffu, l0, o)), l1 = fminf(l1, __shfl_xor_sync(0xffffffffu, l1, o));
      l2 = fminf(l2, __shfl_xor_sync(0xffffffffu, l2, o)), h0 = fmaxf(h0, __shfl_xor_sync(0xffffffffu, h0, o));
      h1 = fmaxf(h1, __shfl_xor_sync(0xffffffffu, h1, o)), h2 = fmaxf(h2, __shfl_xor_sync(0xffffffffu, h2, o));
    }
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(&cnt[b], 32u);
      atomic_min_f(&lo[b][0], l0), atomic_min_f(&lo[b][1], l1), atomic_min_f(&lo[b][2], l2);
      atomic_max_f(&hi[b][0], h0), atomic_max_f(&hi[b][1], h1), atomic_max_f(&hi[b][2], h2);
    }
  } else if (valid) {
    atomicAdd(&cnt[b], 1u);
    atomic_min_f(&lo[b][0], bl.x), atomic_min_f(&lo[b][1], bl.y), atomic_min_f(&lo[b][2], bl.z);
    atomic_max_f(&hi[b][0], bh.x), atomic_max_f(&hi[b][1], bh.y), atomic_max_f(&hi[b][2], bh.z);
  }
}

__device__ __forceinline__ float3 centroid(const Shared &s, uint32_t i) {
  float4 a = __ldg(s.lo + i), b = __ldg(s.hi + i);
  return make_float3((a.x + b.x) * 0.5f, (a.y + b.y) * 0.5f, (a.z + b.z) * 0.5f);
}
__device__ __forceinline__ float comp(float3 v, int a) { return a == 0 ? v.x : (a == 1 ? v.y : v.z); }

__device__ __forceinline__ float half_area(const float lo[3], const float hi[3]) {
  float dx = fmaxf(hi[0] - lo[0], 0.f), dy = fmaxf(hi[1] - lo[1], 0.f), dz = fmaxf(hi[2] - lo[2], 0.f);
  return dx * dy + dy * dz + dz * dx;
}

/* Bin mapping shared by binning and partitioning (identical inputs give identical bins). */
__device__ __forceinline__ float bin_scale(float cmin, float cmax, int nb) {
  float ext = cmax - cmin;
  return ext > 0.f ? (float)nb * (1.f - 1e-6f) / ext : 0.f;
}
__device__ __forceinline__ int bin_of(float c, float cmin, float scale, int nb) {
  int b = (int)((c - cmin) * scale);
  return b < 0 ? 0 : (b >= nb ? nb - 1 : b);
}

__device__ __forceinline__ float pad_lo(float x) { return x - (fabsf(x) * 9.5367431640625e-07f + 1e-30f); }
__device__ __forceinline__ float pad_hi(float x) { return x + (fabsf(x) * 9.5367431640625e-07f + 1e-30f); }

__device__ void write_child(float4 *nodes, int node, int slot, const float lo[3], const float hi[3]) {
  float *n = reinterpret_cast<float *>(nodes + 4 * node);
  const float lx = pad_lo(lo[0]), ly = pad_lo(lo[1]), lz = pad_lo(lo[2]);
  const float hx = pad_hi(hi[0]), hy = pad_hi(hi[1]), hz = pad_hi(hi[2]);
  if (slot == 0) {
    n[0] = lx, n[1] = ly, n[2] = hx, n[3] = hy;
    n[8] = lz, n[9] = hz;
  } else {
    n[4] = lx, n[5] = ly, n[6] = hx, n[7] = hy;
    n[10] = lz, n[11] = hz;
  }
}
__device__ void write_ref(float4 *nodes, int node, int slot, int32_t ref) {
  int32_t *n = reinterpret_cast<int32_t *>(nodes + 4 * node);
  n[12 + slot] = ref;
  n[14 + slot] = 0;
}

/* The inner node of task t, split at `mid` (0 for a root that is one leaf). */
__device__ __forceinline__ int new_node(const Shared &s, const Task &t, uint32_t mid) {
  s.node_at[mid] = make_uint2(t.begin, (uint32_t)t.depth);
  return (int)mid;
}

/* Thread 0 only: records a finished leaf (ids already copied into order[begin, end)). */
__device__ void finish_leaf(const Shared &s, const Task &t) {
  const uint32_t n = t.end - t.begin;
  const int32_t ref = leaf_ref(t.begin, n);
  if (t.parent < 0) { /* whole scene in one leaf: root with an empty second child */
    const float elo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, ehi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    const int node = new_node(s, t, 0);
    write_child(s.nodes, node, 0, t.lo, t.hi);
    write_child(s.nodes, node, 1, elo, ehi);
    write_ref(s.nodes, node, 0, ref);
    write_ref(s.nodes, node, 1, ref);
  } else {
    write_ref(s.nodes, t.parent, t.slot, ref);
  }
  s.leaf_at[t.begin] = make_uint2(n, (uint32_t)t.depth);
}

/* Hands a task on: to the next level (its index there is returned), a CTA or a warp (-1). */
__device__ __forceinline__ int push_task(const Shared &s, const Task &t, int next_level) {
  const uint32_t n = t.end - t.begin;
  if (n > s.small_task) {
    const unsigned i = atomicAdd(&s.n->level[next_level].tasks, 1u);
    s.large[next_level & 1][i] = t;
    return (int)i;
  }
  if (n > (uint32_t)kWarpPrims)
    s.tasks[atomicAdd(&s.n->small, 1u)] = t;
  else
    s.tasks[s.max_tasks - 1u - atomicAdd(&s.n->warps, 1u)] = t;
  return -1;
}

/* Every kernel of the build starts with this: the next one may be launched while this one runs, and
 * this one's predecessor has ended with its writes visible (programmatic dependent launch: the build is
 * some sixty short kernels; 163 k triangles 741 -> 681 us). */
__device__ __forceinline__ void chain() {
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
}

/* ------------------------------------------------------------------ large nodes */

/* A task's centroid bounds and bins before its level, by the calling block. */
__device__ void init_task(const Shared &s, int parity, int t) {
  Bins &B = s.tbins[parity][t];
  for (int i = threadIdx.x; i < 3 * s.bins; i += blockDim.x) {
    const int a = i / s.bins, b = i % s.bins;
    B.cnt[a][b] = 0u;
    for (int k = 0; k < 3; k++) B.lo[a][b][k] = FLT_MAX, B.hi[a][b][k] = -FLT_MAX;
  }
  if (threadIdx.x < 6) s.cb[parity][6 * t + threadIdx.x] = threadIdx.x < 3 ? FLT_MAX : -FLT_MAX;
}

/* The chunk list of a level whose tasks are complete: every task's primitives cut into s.chunk pieces,
 * in task order, by one block of kBlock threads: per tile of kBlock tasks a scan of their chunk counts,
 * then the tile's chunks over the threads, each finding its task by bisection. */
__device__ void make_chunks(const Shared &s, int level) {
  __shared__ unsigned warp_sum[kBlock / 32];
  __shared__ unsigned offs[kBlock + 1];
  __shared__ uint32_t begins[kBlock], ends[kBlock];
  const unsigned nt = __ldcg(&s.n->level[level].tasks);
  const Task *tasks = s.large[level & 1];
  Chunk *chunks = s.chunks[level & 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned base = 0;
  for (unsigned t0 = 0; t0 < nt; t0 += kBlock) {
    const unsigned t = t0 + threadIdx.x;
    uint32_t b = 0, e = 0;
    unsigned c = 0;
    if (t < nt) {
      b = __ldcg(&tasks[t].begin);
      e = __ldcg(&tasks[t].end);
      c = (e - b + s.chunk - 1) / s.chunk;
    }
    unsigned x = c; /* inclusive scan within the warp, then over the warps */
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sum[w] = x;
    begins[threadIdx.x] = b;
    ends[threadIdx.x] = e;
    __syncthreads();
    unsigned before = 0, tile = 0;
    for (int j = 0; j < kBlock / 32; j++) {
      if (j < w) before += warp_sum[j];
      tile += warp_sum[j];
    }
    offs[threadIdx.x] = before + x - c;
    if (threadIdx.x == 0) offs[kBlock] = tile;
    __syncthreads();
    for (unsigned k = threadIdx.x; k < tile; k += kBlock) {
      int lo = 0, hi = kBlock; /* the last task whose first chunk is <= k (tasks past nt have none) */
      while (hi - lo > 1) {
        const int m = (lo + hi) >> 1;
        if (offs[m] <= k)
          lo = m;
        else
          hi = m;
      }
      const uint32_t cb = begins[lo] + (k - offs[lo]) * s.chunk;
      if (base + k < s.max_chunks)
        chunks[base + k] = Chunk{t0 + (unsigned)lo, cb, min(ends[lo], cb + s.chunk)};
      else
        atomicAdd(&s.n->errors, 1u); /* cannot happen (the capacity bounds the chunks): a build failure */
    }
    base += tile;
    __syncthreads();
  }
  if (threadIdx.x == 0) s.n->level[level].chunks = base;
}

/* True in every thread of the last of `blocks` CTAs to arrive at *done; what the others wrote before is
 * visible to it. */
__device__ bool last_block(unsigned *done, unsigned blocks) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(done, 1u) == blocks - 1u;
  __syncthreads();
  if (last) __threadfence();
  return last;
}

__device__ __forceinline__ void block_minmax3(float l[3], float h[3], float *sh /* 6 * 32 */) {
  for (int o = 16; o > 0; o >>= 1)
    for (int k = 0; k < 3; k++) {
      l[k] = fminf(l[k], __shfl_xor_sync(0xffffffffu, l[k], o));
      h[k] = fmaxf(h[k], __shfl_xor_sync(0xffffffffu, h[k], o));
    }
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (lane == 0)
    for (int k = 0; k < 3; k++) {
      sh[k * 32 + w] = l[k];
      sh[(3 + k) * 32 + w] = h[k];
    }
  __syncthreads();
  for (int k = 0; k < 3; k++) {
    float a = FLT_MAX, b = -FLT_MAX;
    for (int j = 0; j < nw; j++) {
      a = fminf(a, sh[k * 32 + j]);
      b = fmaxf(b, sh[(3 + k) * 32 + j]);
    }
    l[k] = a;
    h[k] = b;
  }
  __syncthreads();
}

__global__ void k_init(Shared s) {
  uint32_t *c = reinterpret_cast<uint32_t *>(s.n);
  for (uint32_t i = threadIdx.x; i < sizeof(Counters) / 4; i += blockDim.x) c[i] = 0u;
  if (threadIdx.x < 12) s.scene[threadIdx.x] = threadIdx.x / 3 % 2 ? -FLT_MAX : FLT_MAX;
}

/* Primitive ids, and the box and centroid bounds of all primitives (one set of atomics per block); the
 * last block makes the root task. */
__global__ void __launch_bounds__(kBlock) k_begin(Shared s, uint32_t n) {
  chain();
  __shared__ float sh[6 * 32];
  float l[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, h[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
  float cl[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, ch[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4 a = s.lo[i], b = s.hi[i];
    s.ids0[i] = i;
    l[0] = fminf(l[0], a.x), l[1] = fminf(l[1], a.y), l[2] = fminf(l[2], a.z);
    h[0] = fmaxf(h[0], b.x), h[1] = fmaxf(h[1], b.y), h[2] = fmaxf(h[2], b.z);
    const float c[3] = {(a.x + b.x) * 0.5f, (a.y + b.y) * 0.5f, (a.z + b.z) * 0.5f};
    for (int k = 0; k < 3; k++) cl[k] = fminf(cl[k], c[k]), ch[k] = fmaxf(ch[k], c[k]);
  }
  block_minmax3(l, h, sh);
  block_minmax3(cl, ch, sh);
  if (threadIdx.x < 3) {
    atomic_min_f(s.scene + threadIdx.x, l[threadIdx.x]);
    atomic_max_f(s.scene + 3 + threadIdx.x, h[threadIdx.x]);
    atomic_min_f(s.scene + 6 + threadIdx.x, cl[threadIdx.x]);
    atomic_max_f(s.scene + 9 + threadIdx.x, ch[threadIdx.x]);
  }
  if (!last_block(&s.n->begin_done, gridDim.x)) return;
  if (threadIdx.x == 0) {
    Task t{0u, n, -1, 0, 0, 0, {}, {}};
    for (int k = 0; k < 3; k++) t.lo[k] = __ldcg(s.scene + k), t.hi[k] = __ldcg(s.scene + 3 + k);
    push_task(s, t, 0);
  }
  __threadfence();
  __syncthreads();
  if (n <= s.small_task) return;
  init_task(s, 0, 0);
  __syncthreads();
  if (threadIdx.x < 6) s.cb[0][threadIdx.x] = __ldcg(s.scene + 6 + threadIdx.x);
  make_chunks(s, 0);
}

__global__ void __launch_bounds__(kBlock) k_bin(Shared s, int level) {
  chain();
  if (blockIdx.x >= s.n->level[level].chunks) return;
  const Task *tasks = s.large[level & 1];
  const Chunk *chunks = s.chunks[level & 1];
  const float *cb = s.cb[level & 1];
  Bins *bins = s.tbins[level & 1];
  __shared__ unsigned scnt[3][kMaxBins];
  __shared__ float slo[3][kMaxBins][3], shi[3][kMaxBins][3];
  const int nb = s.bins;
  const Chunk c = chunks[blockIdx.x];
  const Task &t = tasks[c.task];
  const uint32_t *src = ids_of(s, t.buf);
  for (int i = threadIdx.x; i < 3 * nb; i += blockDim.x) {
    int a = i / nb, b = i % nb;
    scnt[a][b] = 0u;
    for (int k = 0; k < 3; k++) slo[a][b][k] = FLT_MAX, shi[a][b][k] = -FLT_MAX;
  }
  float cmin[3], scale[3];
  for (int a = 0; a < 3; a++) {
    cmin[a] = cb[6 * c.task + a];
    scale[a] = bin_scale(cmin[a], cb[6 * c.task + 3 + a], nb);
  }
  __syncthreads();
  for (uint32_t r0 = c.begin; r0 < c.end; r0 += blockDim.x) { /* whole warps: bin_add votes */
    const uint32_t i = r0 + threadIdx.x;
    const bool valid = i < c.end;
    float4 bl = make_float4(0.f, 0.f, 0.f, 0.f), bh = bl;
    if (valid) {
      const uint32_t id = src[i];
      bl = __ldg(s.lo + id), bh = __ldg(s.hi + id);
    }
    const float3 p = make_float3((bl.x + bh.x) * 0.5f, (bl.y + bh.y) * 0.5f, (bl.z + bh.z) * 0.5f);
    for (int a = 0; a < 3; a++)
      bin_add(scnt[a], slo[a], shi[a], bin_of(comp(p, a), cmin[a], scale[a], nb), valid, bl, bh);
  }
  __syncthreads();
  Bins &g = bins[c.task];
  for (int i = threadIdx.x; i < 3 * nb; i += blockDim.x) {
    int a = i / nb, b = i % nb;
    if (scnt[a][b] == 0u) continue;
    atomicAdd(&g.cnt[a][b], scnt[a][b]);
    for (int k = 0; k < 3; k++) {
      atomic_min_f(&g.lo[a][b][k], slo[a][b][k]);
      atomic_max_f(&g.hi[a][b][k], shi[a][b][k]);
    }
  }
}

/* SAH sweep over bins: best (cost, axis, plane) with a deterministic tie order. */
struct Best {
  float cost;
  int key; /* axis * kMaxBins + plane; planes 1..nb-1 */
};
__device__ __forceinline__ bool better(const Best &a, const Best &b) {
  return a.cost < b.cost || (a.cost == b.cost && a.key < b.key);
}

/* SAH over a node's bins staged in shared memory (cnt, lo, hi): warp a of the block scans axis a, lane b
 * holding bin b, from both ends; a plane's two sides are then lane plane - 1's prefix and lane plane's
 * suffix.  Every thread gets the best plane, and cl..dh the boxes of its sides.  The costs are those of a
 * serial sweep (minima, maxima and counts are exact).  The block has at least three warps; sh: 3 Best.
 * A serial sweep per candidate took k_split 10 to 12 us a level. */
__device__ Best scan_bins(int nb, float area, float cost_trav, const unsigned (*cnt)[kMaxBins],
                          const float (*blo)[kMaxBins][3], const float (*bhi)[kMaxBins][3], bool try_split, Best *sh,
                          float (*side)[6], unsigned *left) {
  const int lane = threadIdx.x & 31, a = threadIdx.x >> 5;
  float pl[3], ph[3], sl[3], shi[3];
  unsigned np = 0, ns = 0;
  Best best{FLT_MAX, 0x7fffffff};
  if (a < 3) {
    const bool in = lane < nb;
    np = ns = in ? cnt[a][lane] : 0u;
    for (int k = 0; k < 3; k++) {
      pl[k] = sl[k] = in ? blo[a][lane][k] : FLT_MAX;
      ph[k] = shi[k] = in ? bhi[a][lane][k] : -FLT_MAX;
    }
    for (int o = 1; o < nb; o <<= 1) {
      const unsigned up = __shfl_up_sync(0xffffffffu, np, o), dn = __shfl_down_sync(0xffffffffu, ns, o);
      const bool u = lane >= o, d = lane + o < 32;
      if (u) np += up;
      if (d) ns += dn;
      for (int k = 0; k < 3; k++) {
        const float x = __shfl_up_sync(0xffffffffu, pl[k], o), y = __shfl_up_sync(0xffffffffu, ph[k], o);
        const float z = __shfl_down_sync(0xffffffffu, sl[k], o), w = __shfl_down_sync(0xffffffffu, shi[k], o);
        if (u) pl[k] = fminf(pl[k], x), ph[k] = fmaxf(ph[k], y);
        if (d) sl[k] = fminf(sl[k], z), shi[k] = fmaxf(shi[k], w);
      }
    }
    /* plane p lies between bins p - 1 and p: lane p - 1 evaluates it */
    float rl[3], rh[3];
    const unsigned nr = __shfl_down_sync(0xffffffffu, ns, 1);
    for (int k = 0; k < 3; k++)
      rl[k] = __shfl_down_sync(0xffffffffu, sl[k], 1), rh[k] = __shfl_down_sync(0xffffffffu, shi[k], 1);
    if (try_split && lane + 1 < nb && np != 0 && nr != 0)
      best = Best{cost_trav + (half_area(pl, ph) * (float)np + half_area(rl, rh) * (float)nr) / area,
                  a * kMaxBins + lane + 1};
    for (int o = 16; o > 0; o >>= 1) {
      Best q{__shfl_xor_sync(0xffffffffu, best.cost, o), __shfl_xor_sync(0xffffffffu, best.key, o)};
      if (better(q, best)) best = q;
    }
    if (lane == 0) sh[a] = best;
  }
  __syncthreads();
  best = sh[0];
  if (better(sh[1], best)) best = sh[1];
  if (better(sh[2], best)) best = sh[2];
  if (best.key != 0x7fffffff && a == best.key / kMaxBins) {
    const int plane = best.key % kMaxBins;
    if (lane == plane - 1) {
      *left = np;
      for (int k = 0; k < 3; k++) side[0][k] = pl[k], side[0][3 + k] = ph[k];
    }
    if (lane == plane)
      for (int k = 0; k < 3; k++) side[1][k] = sl[k], side[1][3 + k] = shi[k];
  }
  __syncthreads();
  return best;
}

__global__ void __launch_bounds__(kBlock) k_split(Shared s, int level) {
  chain();
  __shared__ Best sh[3];
  __shared__ unsigned cnt[3][kMaxBins];
  __shared__ float blo[3][kMaxBins][3], bhi[3][kMaxBins][3];
  __shared__ float side[2][6];
  __shared__ unsigned left;
  __shared__ int child[2];
  const unsigned n_tasks = s.n->level[level].tasks;
  if (blockIdx.x >= n_tasks) return;
  {
    const Task t = s.large[level & 1][blockIdx.x];
    const Bins &B = s.tbins[level & 1][blockIdx.x];
    const float *cb = s.cb[level & 1];
    const int nb = s.bins;
    for (int i = threadIdx.x; i < 3 * nb; i += blockDim.x) {
      const int a = i / nb, b = i % nb;
      cnt[a][b] = B.cnt[a][b];
      for (int k = 0; k < 3; k++) blo[a][b][k] = B.lo[a][b][k], bhi[a][b][k] = B.hi[a][b][k];
    }
    __syncthreads();
    const float area = half_area(t.lo, t.hi);
    const Best best = scan_bins(nb, area, s.cost_trav, cnt, blo, bhi, area > 0.f && t.depth < kMedianDepth, sh, side,
                                &left);
    if (threadIdx.x == 0) {
      SplitInfo sp;
      for (int a = 0; a < 3; a++) {
        sp.cmin[a] = cb[6 * blockIdx.x + a];
        sp.scale[a] = bin_scale(sp.cmin[a], cb[6 * blockIdx.x + 3 + a], nb);
      }
      float llo[3], lhi[3], rlo[3], rhi[3];
      if (best.key != 0x7fffffff) {
        sp.median = 0;
        sp.axis = best.key / kMaxBins;
        sp.bin = best.key % kMaxBins - 1; /* left side: bins <= sp.bin */
        sp.mid = t.begin + left;
        for (int k = 0; k < 3; k++)
          llo[k] = side[0][k], lhi[k] = side[0][3 + k], rlo[k] = side[1][k], rhi[k] = side[1][3 + k];
      } else {
        sp.median = 1;
        sp.axis = 0;
        sp.bin = 0;
        sp.mid = t.begin + (t.end - t.begin) / 2;
        for (int k = 0; k < 3; k++) llo[k] = rlo[k] = t.lo[k], lhi[k] = rhi[k] = t.hi[k];
      }
      sp.left_ptr = t.begin;
      sp.right_ptr = sp.mid;
      const int node = new_node(s, t, sp.mid);
      if (t.parent >= 0) write_ref(s.nodes, t.parent, t.slot, node);
      write_child(s.nodes, node, 0, llo, lhi);
      write_child(s.nodes, node, 1, rlo, rhi);
      const Task L{t.begin, sp.mid, node, 0, t.depth + 1, 1 - t.buf, {llo[0], llo[1], llo[2]}, {lhi[0], lhi[1], lhi[2]}};
      const Task R{sp.mid, t.end, node, 1, t.depth + 1, 1 - t.buf, {rlo[0], rlo[1], rlo[2]}, {rhi[0], rhi[1], rhi[2]}};
      sp.child[0] = child[0] = push_task(s, L, level + 1);
      sp.child[1] = child[1] = push_task(s, R, level + 1);
      s.splits[blockIdx.x] = sp;
    }
    __syncthreads();
    for (int k = 0; k < 2; k++)
      if (child[k] >= 0) init_task(s, (level + 1) & 1, child[k]);
  }
  if (last_block(&s.n->level[level].done, n_tasks)) make_chunks(s, level + 1);
}

__global__ void __launch_bounds__(kBlock) k_partition(Shared s, int level) {
  chain();
  __shared__ unsigned warp_l[kBlock / 32], warp_r[kBlock / 32];
  __shared__ unsigned base_l, base_r;
  __shared__ float red[6 * 32];
  if (blockIdx.x >= s.n->level[level].chunks) return;
  const Chunk c = s.chunks[level & 1][blockIdx.x];
  const Task &t = s.large[level & 1][c.task];
  SplitInfo &sp = s.splits[c.task];
  const int child_l = sp.child[0], child_r = sp.child[1];
  float ll[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, lh[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
  float rl[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, rh[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
  const uint32_t *src = ids_of(s, t.buf);
  uint32_t *dst = ids_of(s, 1 - t.buf);
  const int nb = s.bins;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (uint32_t r0 = c.begin; r0 < c.end; r0 += blockDim.x) {
    const uint32_t i = r0 + threadIdx.x;
    const bool valid = i < c.end;
    uint32_t id = 0;
    bool left = false;
    if (valid) {
      id = src[i];
      const float3 p = centroid(s, id);
      if (sp.median)
        left = i < sp.mid;
      else
        left = bin_of(comp(p, sp.axis), sp.cmin[sp.axis], sp.scale[sp.axis], nb) <= sp.bin;
      for (int k = 0; k < 3; k++) {
        const float v = comp(p, k);
        if (left)
          ll[k] = fminf(ll[k], v), lh[k] = fmaxf(lh[k], v);
        else
          rl[k] = fminf(rl[k], v), rh[k] = fmaxf(rh[k], v);
      }
    }
    const unsigned ml = __ballot_sync(0xffffffffu, valid && left), mr = __ballot_sync(0xffffffffu, valid && !left);
    if (lane == 0) warp_l[w] = __popc(ml), warp_r[w] = __popc(mr);
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned tl = 0, tr = 0;
      for (int j = 0; j < (int)(blockDim.x >> 5); j++) {
        unsigned a = warp_l[j], b = warp_r[j];
        warp_l[j] = tl, warp_r[j] = tr;
        tl += a, tr += b;
      }
      base_l = atomicAdd(&sp.left_ptr, tl);
      base_r = atomicAdd(&sp.right_ptr, tr);
    }
    __syncthreads();
    const unsigned below = (1u << lane) - 1u;
    if (valid) {
      /* positions stay inside [begin, mid) / [mid, end) because partition and binning share
       * bin_of(); the guard keeps a bookkeeping error from ever writing outside the node */
      const unsigned pos = left ? base_l + warp_l[w] + __popc(ml & below) : base_r + warp_r[w] + __popc(mr & below);
      if (left ? (pos < sp.mid) : (pos < t.end))
        dst[pos] = id;
      else
        atomicAdd(&s.n->errors, 1u);
    }
    __syncthreads();
  }
  /* the children's centroid bounds, for the next level */
  float *cb = s.cb[(level + 1) & 1];
  if (child_l >= 0) {
    block_minmax3(ll, lh, red);
    if (threadIdx.x < 3) {
      atomic_min_f(cb + 6 * child_l + threadIdx.x, ll[threadIdx.x]);
      atomic_max_f(cb + 6 * child_l + 3 + threadIdx.x, lh[threadIdx.x]);
    }
  }
  if (child_r >= 0) {
    block_minmax3(rl, rh, red);
    if (threadIdx.x < 3) {
      atomic_min_f(cb + 6 * child_r + threadIdx.x, rl[threadIdx.x]);
      atomic_max_f(cb + 6 * child_r + 3 + threadIdx.x, rh[threadIdx.x]);
    }
  }
}

/* ------------------------------------------------------------------ small nodes */

/* ------------------------------------------------------------------ warp subtrees (<= 32 primitives)
 *
 * A subtree of at most 32 primitives is built by one warp without block barriers.  Its primitives' ids
 * and boxes go to shared memory once, and once per axis they are sorted by centroid (bitonic, ties by
 * primitive id); a node then holds its primitives in each axis's order, scans the sorted boxes from
 * both ends and evaluates the SAH of every split position (an exact sweep, where the larger nodes use
 * bins); the best (cost, axis, position) wins.  A split keeps each axis's order within each side (a
 * stable partition by the set of left primitives), so the children need no sort.  Leaf rules, cost model
 * and the median split below kMedianDepth are those of the CTA path.
 *
 * The work runs on lane segments: a segment of W lanes (W = 32 is the whole warp) builds a node of
 * at most W primitives.  When both children of a split fit in W / 2 lanes the segment forks: its
 * lower half builds the left subtree while its upper half builds the right one, each as a segment of
 * W / 2 lanes, down to single lanes (one-primitive leaves); otherwise the left child continues on
 * the segment and the right one waits on the segment's stack.  A half whose subtree is done waits
 * for its sibling, and the two continue as their parent segment.  The splits do not depend on which
 * lanes compute them or in which order, so the tree is the one a single warp building node after
 * node produces.
 *
 * Bound by chains of dependent shuffles and shared-memory loads at 23 warps per SM (58 % of the issue slots, 64 M
 * warp instructions).  163 k triangles: sorting every node and loading its boxes from memory again took 195 us,
 * this 133. */
/* Right siblings a W-lane segment keeps: it pushes only at nodes of >= W / 2 + 2 primitives (smaller
 * ones fork), nested with strictly decreasing sizes <= W, so at most W / 2 - 1 at once (none for
 * W <= 2).  Per warp: one segment of 32 lanes (15 entries), 2 of 16 (7 each), 4 of 8 (3 each) and 8
 * of 4 (1 each). */
constexpr int kWarpStack = 15 + 2 * 7 + 4 * 3 + 8 * 1;

/* One warp's subtree in shared memory; primitives are named by their lane at the root. */
struct WarpTree {
  Task stack[kWarpStack];
  float box[6][32];          /* lo.xyz, hi.xyz */
  uint32_t id[32];
  uint8_t order[3][32];      /* per axis, the primitives of each node's range in sorted order */
};

__device__ __forceinline__ unsigned seg_mask(int W) {
  return W == 32 ? 0xffffffffu : ((1u << W) - 1u) << ((threadIdx.x & 31) & ~(W - 1));
}

/* The stack of the calling lane's W-lane segment, at level log2(32 / W) (W >= 4). */
__device__ __forceinline__ Task *seg_stack(Task *stacks, int level, int W) {
  const int base = level == 0 ? 0 : (level == 1 ? 15 : (level == 2 ? 29 : 41));
  return stacks + base + ((threadIdx.x & 31) / W) * (W / 2 - 1);
}

/* Sorts the warp's (key, tie) pairs ascending over its first `span` lanes (a power of two, 2..32) and
 * returns, for this lane's rank, the lane that held it.  tie must be unique per lane (the primitive id,
 * so equal centroids sort the same way whatever order the ids arrive in; empty lanes, which come last,
 * use 0xffffffff - lane). */
__device__ __forceinline__ int warp_sort_idx(float key, uint32_t tie, int span) {
  const int lane = threadIdx.x & 31;
  int idx = lane;
  for (int k = 2; k <= span; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      const float ok = __shfl_xor_sync(0xffffffffu, key, j);
      const uint32_t ot = __shfl_xor_sync(0xffffffffu, tie, j);
      const int oi = __shfl_xor_sync(0xffffffffu, idx, j);
      const bool other_less = ok < key || (ok == key && ot < tie);
      const bool keep_min = ((lane & j) == 0) == ((lane & k) == 0);
      if (keep_min ? other_less : !other_less) key = ok, tie = ot, idx = oi;
    }
  return idx;
}

/* Inclusive prefix (from segment lane 0) and suffix (towards the segment's last lane) bounds of the
 * boxes held by the segment's lanes.  Each lane's scan reaches `span` lanes (a power of two): with
 * the node's boxes in lanes 0..n-1, n <= span, and empty boxes above, the prefix of lane i < n and
 * the suffix of lane i (over i..n-1) are exact, the same values as a scan over the whole segment
 * (min and max are exact). */
__device__ __forceinline__ void seg_scan_boxes(const float lo[3], const float hi[3], float pl[3], float ph[3],
                                               float sl[3], float sh[3], int span, int W, unsigned mask) {
  const int lane = threadIdx.x & (W - 1);
  for (int k = 0; k < 3; k++) pl[k] = sl[k] = lo[k], ph[k] = sh[k] = hi[k];
  for (int o = 1; o < span; o <<= 1)
    for (int k = 0; k < 3; k++) {
      const float a = __shfl_up_sync(mask, pl[k], o, W), b = __shfl_up_sync(mask, ph[k], o, W);
      const float c = __shfl_down_sync(mask, sl[k], o, W), d = __shfl_down_sync(mask, sh[k], o, W);
      if (lane >= o) pl[k] = fminf(pl[k], a), ph[k] = fmaxf(ph[k], b);
      if (lane + o < W) sl[k] = fminf(sl[k], c), sh[k] = fmaxf(sh[k], d);
    }
}

__device__ __forceinline__ Best seg_best(Best b, int W, unsigned mask) {
  for (int o = W / 2; o > 0; o >>= 1) {
    Best q{__shfl_xor_sync(mask, b.cost, o, W), __shfl_xor_sync(mask, b.key, o, W)};
    if (better(q, b)) b = q;
  }
  return b;
}

/* Builds the subtree of `root` (<= 32 primitives) with the calling warp; all 32 lanes call it. */
__device__ void warp_build(const Shared &s, Task root, WarpTree &tree) {
  {
    const int lane = threadIdx.x & 31;
    const uint32_t n = root.end - root.begin;
    const bool act = (uint32_t)lane < n;
    float c[3] = {FLT_MAX, FLT_MAX, FLT_MAX};
    uint32_t tie = 0xffffffffu - (uint32_t)lane;
    if (act) {
      const uint32_t id = ids_of(s, root.buf)[root.begin + lane];
      const float4 a = __ldg(s.lo + id), b = __ldg(s.hi + id);
      tree.box[0][lane] = a.x, tree.box[1][lane] = a.y, tree.box[2][lane] = a.z;
      tree.box[3][lane] = b.x, tree.box[4][lane] = b.y, tree.box[5][lane] = b.z;
      tree.id[lane] = tie = id;
      c[0] = (a.x + b.x) * 0.5f, c[1] = (a.y + b.y) * 0.5f, c[2] = (a.z + b.z) * 0.5f;
    }
    /* the sort reaches the smallest power of two >= n lanes */
    const int span = n <= 2u ? 2 : 1 << (32 - __clz((int)n - 1));
    for (int a = 0; a < 3; a++) tree.order[a][lane] = (uint8_t)(n > 1 ? warp_sort_idx(c[a], tie, span) : lane);
    __syncwarp();
  }
  int W = 32, level = 0; /* this lane's segment: width and log2(32 / W) */
  uint32_t depth_sp = 0; /* per level (4 bits each, levels 0..3), the segment's stack depth */
  bool failed = false;
  Task t = root;
  for (int iter = 0;; iter++) {
    const int lane = threadIdx.x & (W - 1);
    unsigned mask = seg_mask(W);
    const uint32_t n = t.end - t.begin, at = t.begin - root.begin;
    const bool act = (uint32_t)lane < n;
    int ord[3];
    for (int a = 0; a < 3; a++) ord[a] = act ? tree.order[a][at + lane] : 0;
    /* a lane processes distinct nodes of a <= 32-primitive subtree, at most 63: past 2 * 63
     * iterations something is broken, and every further node becomes a leaf, so the segments still
     * drain their stacks and meet their siblings (no lane leaves while another waits for it).  The
     * vote keeps the decision uniform over the segment (lanes of a joined segment count differently) */
    if (__any_sync(mask, iter >= 2 * (2 * kWarpPrims - 1)) && !failed) {
      failed = true;
      if (lane == 0) atomicAdd(&s.n->errors, 1u); /* reported as a build failure */
    }
    bool make_leaf = n <= 1 || failed;
    const float area = half_area(t.lo, t.hi);
    Best best{FLT_MAX, 0x7fffffff};
    float cl[3], ch[3], dl[3], dh[3]; /* the best axis's boxes left and right of the split after this lane */
    for (int k = 0; k < 3; k++) cl[k] = dl[k] = FLT_MAX, ch[k] = dh[k] = -FLT_MAX;
    if (!make_leaf && area > 0.f && t.depth < kMedianDepth) {
      /* scans reach the smallest power of two >= n lanes (uniform over the segment) */
      const int span = n <= 2u ? 2 : 1 << (32 - __clz((int)n - 1));
#pragma unroll
      for (int a = 0; a < 3; a++) {
        float bl[3], bh[3], pl[3], ph[3], sl[3], sh[3];
        for (int k = 0; k < 3; k++) {
          bl[k] = act ? tree.box[k][ord[a]] : FLT_MAX;
          bh[k] = act ? tree.box[3 + k][ord[a]] : -FLT_MAX;
        }
        seg_scan_boxes(bl, bh, pl, ph, sl, sh, span, W, mask);
        float rl[3], rh[3];
        for (int k = 0; k < 3; k++)
          rl[k] = __shfl_down_sync(mask, sl[k], 1, W), rh[k] = __shfl_down_sync(mask, sh[k], 1, W);
        Best mine{FLT_MAX, 0x7fffffff};
        if ((uint32_t)lane + 1 < n) { /* split after sorted position lane: left = lane + 1 primitives */
          const float cost =
              s.cost_trav + (half_area(pl, ph) * (float)(lane + 1) + half_area(rl, rh) * (float)(n - 1 - lane)) / area;
          mine = Best{cost, a * 64 + lane};
        }
        mine = seg_best(mine, W, mask);
        if (better(mine, best)) {
          best = mine;
          for (int k = 0; k < 3; k++) cl[k] = pl[k], ch[k] = ph[k], dl[k] = rl[k], dh[k] = rh[k];
        }
      }
    }
    const bool has_split = best.key != 0x7fffffff;
    if (!make_leaf) {
      if ((int)n <= s.max_leaf && (!has_split || (float)n <= best.cost)) make_leaf = true;
      if ((int)n <= s.hard_leaf && !has_split) make_leaf = true;
    }
    if (!make_leaf) {
      /* the split: best SAH position, or the median along the widest centroid extent */
      int axis, left_n;
      if (has_split) {
        axis = best.key / 64;
        left_n = best.key % 64 + 1;
      } else {
        float ext[3];
        for (int k = 0; k < 3; k++) { /* sorted: the last primitive's centroid less the first's */
          const float c = act ? (tree.box[k][ord[k]] + tree.box[3 + k][ord[k]]) * 0.5f : 0.f;
          ext[k] = __shfl_sync(mask, c, (int)n - 1, W) - __shfl_sync(mask, c, 0, W);
        }
        axis = ext[1] > ext[0] ? (ext[2] > ext[1] ? 2 : 1) : (ext[2] > ext[0] ? 2 : 0);
        left_n = (int)n / 2;
      }
      const int mine = axis == 0 ? ord[0] : axis == 1 ? ord[1] : ord[2];
      const unsigned left_set = __reduce_or_sync(mask, act && lane < left_n ? 1u << mine : 0u);
      if (!has_split) { /* boxes of the halves */
        for (int k = 0; k < 3; k++) {
          float a0 = FLT_MAX, a1 = -FLT_MAX, b0 = FLT_MAX, b1 = -FLT_MAX;
          if (act) {
            const float x = tree.box[k][mine], y = tree.box[3 + k][mine];
            if (lane < left_n)
              a0 = x, a1 = y;
            else
              b0 = x, b1 = y;
          }
          for (int o = W / 2; o > 0; o >>= 1) {
            a0 = fminf(a0, __shfl_xor_sync(mask, a0, o, W)), a1 = fmaxf(a1, __shfl_xor_sync(mask, a1, o, W));
            b0 = fminf(b0, __shfl_xor_sync(mask, b0, o, W)), b1 = fmaxf(b1, __shfl_xor_sync(mask, b1, o, W));
          }
          cl[k] = a0, ch[k] = a1, dl[k] = b0, dh[k] = b1;
        }
      } else {
        for (int k = 0; k < 3; k++) {
          cl[k] = __shfl_sync(mask, cl[k], left_n - 1, W), ch[k] = __shfl_sync(mask, ch[k], left_n - 1, W);
          dl[k] = __shfl_sync(mask, dl[k], left_n - 1, W), dh[k] = __shfl_sync(mask, dh[k], left_n - 1, W);
        }
      }
      /* each axis's order within each side: left primitives to the front of the node's range */
      const unsigned below = ((1u << (threadIdx.x & 31)) - 1u) & mask;
      for (int a = 0; a < 3; a++) {
        const bool left = act && ((left_set >> ord[a]) & 1u);
        const unsigned ml = __ballot_sync(mask, left), mr = __ballot_sync(mask, act && !left);
        if (act) tree.order[a][at + (left ? __popc(ml & below) : left_n + __popc(mr & below))] = (uint8_t)ord[a];
      }
      const uint32_t mid = t.begin + (uint32_t)left_n;
      const int node = (int)mid;
      if (lane == 0) {
        new_node(s, t, mid);
        if (t.parent >= 0) write_ref(s.nodes, t.parent, t.slot, node);
        write_child(s.nodes, node, 0, cl, ch);
        write_child(s.nodes, node, 1, dl, dh);
      }
      __syncwarp(mask); /* the children read orders written by other lanes */
      const Task L{t.begin, mid, node, 0, t.depth + 1, t.buf, {cl[0], cl[1], cl[2]}, {ch[0], ch[1], ch[2]}};
      const Task R{mid, t.end, node, 1, t.depth + 1, t.buf, {dl[0], dl[1], dl[2]}, {dh[0], dh[1], dh[2]}};
      if ((uint32_t)left_n <= (uint32_t)(W / 2) && n - (uint32_t)left_n <= (uint32_t)(W / 2)) {
        /* fork: the lower half builds the left subtree, the upper half the right one */
        t = lane < W / 2 ? L : R;
        W >>= 1;
        level++;
        if (level < 4) depth_sp &= ~(15u << (4 * level));
        continue;
      }
      const int sp = (int)((depth_sp >> (4 * level)) & 15u);
      if (sp < W / 2 - 1) {
        if (lane == 0) seg_stack(tree.stack, level, W)[sp] = R;
        depth_sp += 1u << (4 * level);
      } else if (lane == 0) {
        atomicAdd(&s.n->errors, 1u); /* cannot happen (see kWarpStack): reported as a build failure */
      }
      __syncwarp(mask);
      t = L;
      continue;
    }
    if (act) s.order[t.begin + lane] = tree.id[ord[0]];
    if (lane == 0) finish_leaf(s, t);
    /* next: the segment's pending sibling; a segment with none waits for its sibling half and the
     * two continue as their parent */
    for (;;) {
      const int sp = level < 4 ? (int)((depth_sp >> (4 * level)) & 15u) : 0;
      if (sp > 0) {
        __syncwarp(mask);
        t = seg_stack(tree.stack, level, W)[sp - 1];
        depth_sp -= 1u << (4 * level);
        __syncwarp(mask);
        break;
      }
      if (level == 0) return;
      W <<= 1;
      level--;
      mask = seg_mask(W);
      __syncwarp(mask);
    }
  }
}

/* Subtrees of 33 to kCtaPrims primitives, one CTA each (CTAs take them from a counter): one primitive per
 * thread, held in registers through a node's bounds, binning and partition; nodes of at most 32 go to
 * the warps of k_build_warps.  Bound by its barriers (half of the stall cycles; 27 warps per SM).  163 k
 * triangles: with each pass of a node reading its boxes again, and the CTA's own warps building its
 * small subtrees, 345 us; this 80 us and k_build_warps 133. */
__global__ void __launch_bounds__(kCtaPrims) k_build_small(Shared s) {
  chain();
  __shared__ Task stack[kSmallStack];
  __shared__ int sp;
  __shared__ unsigned item;
  __shared__ unsigned scnt[3][kMaxBins];
  __shared__ float slo[3][kMaxBins][3], shi[3][kMaxBins][3];
  __shared__ float red[6 * 32], side[2][6];
  __shared__ unsigned wl[kCtaPrims / 32], wr[kCtaPrims / 32], left_total;
  __shared__ Best best_sh[3];
  const int nb = s.bins, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned n_tasks = s.n->small;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) {
      item = atomicAdd(&s.n->small_next, 1u);
      if (item < n_tasks) stack[0] = s.tasks[item];
      sp = 1;
    }
    __syncthreads();
    if (item >= n_tasks) return;
    while (sp > 0) { /* uniform: read between barriers */
      const Task t = stack[sp - 1];
      const uint32_t n = t.end - t.begin;
      const uint32_t *src = ids_of(s, t.buf);
      uint32_t *dst = ids_of(s, 1 - t.buf);
      const bool act = threadIdx.x < n;
      const uint32_t id = act ? src[t.begin + threadIdx.x] : 0u;
      float4 bl = make_float4(0.f, 0.f, 0.f, 0.f), bh = bl;
      if (act) bl = __ldg(s.lo + id), bh = __ldg(s.hi + id);
      const float3 p = make_float3((bl.x + bh.x) * 0.5f, (bl.y + bh.y) * 0.5f, (bl.z + bh.z) * 0.5f);
      /* centroid bounds; the bins are cleared between its barriers */
      for (int i = threadIdx.x; i < 3 * nb; i += blockDim.x) {
        const int a = i / nb, b = i % nb;
        scnt[a][b] = 0u;
        for (int k = 0; k < 3; k++) slo[a][b][k] = FLT_MAX, shi[a][b][k] = -FLT_MAX;
      }
      float l[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, h[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
      if (act)
        for (int k = 0; k < 3; k++) l[k] = h[k] = comp(p, k);
      block_minmax3(l, h, red);
      int bin[3];
      if (32u * w < n) /* whole warps: bin_add votes */
        for (int a = 0; a < 3; a++) {
          bin[a] = bin_of(comp(p, a), l[a], bin_scale(l[a], h[a], nb), nb);
          bin_add(scnt[a], slo[a], shi[a], bin[a], act, bl, bh);
        }
      __syncthreads();
      const float area = half_area(t.lo, t.hi);
      const Best best = scan_bins(nb, area, s.cost_trav, scnt, slo, shi, area > 0.f && t.depth < kMedianDepth, best_sh,
                                  side, &left_total);
      const bool has_split = best.key != 0x7fffffff;
      const int axis = has_split ? best.key / kMaxBins : 0;
      const uint32_t mid = t.begin + (has_split ? left_total : n / 2);
      const bool left = act && (has_split ? (axis == 0 ? bin[0] : axis == 1 ? bin[1] : bin[2]) < best.key % kMaxBins
                                          : threadIdx.x < n / 2);
      const unsigned ml = __ballot_sync(0xffffffffu, left), mr = __ballot_sync(0xffffffffu, act && !left);
      if (lane == 0) wl[w] = __popc(ml), wr[w] = __popc(mr);
      if (!has_split) { /* the halves' boxes (two more reductions, for the rare median split) */
        float al[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, ah[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        float cl[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, ch[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        if (act) {
          float *ol = left ? al : cl, *oh = left ? ah : ch;
          ol[0] = bl.x, ol[1] = bl.y, ol[2] = bl.z, oh[0] = bh.x, oh[1] = bh.y, oh[2] = bh.z;
        }
        block_minmax3(al, ah, red);
        block_minmax3(cl, ch, red);
        if (threadIdx.x == 0)
          for (int k = 0; k < 3; k++)
            side[0][k] = al[k], side[0][3 + k] = ah[k], side[1][k] = cl[k], side[1][3 + k] = ch[k];
      }
      __syncthreads();
      if (act) {
        unsigned before = 0;
        for (int j = 0; j < w; j++) before += left ? wl[j] : wr[j];
        const uint32_t pos = (left ? t.begin : mid) + before + __popc((left ? ml : mr) & ((1u << lane) - 1u));
        if (left ? (pos < mid) : (pos < t.end))
          dst[pos] = id;
        else
          atomicAdd(&s.n->errors, 1u);
      }
      if (threadIdx.x == 0) {
        const int node = new_node(s, t, mid);
        if (t.parent >= 0) write_ref(s.nodes, t.parent, t.slot, node);
        write_child(s.nodes, node, 0, side[0], side[0] + 3);
        write_child(s.nodes, node, 1, side[1], side[1] + 3);
        int top = sp - 1;
        for (int k = 1; k >= 0; k--) {
          const Task c{k ? mid : t.begin, k ? t.end : mid, node, k, t.depth + 1, 1 - t.buf,
                       {side[k][0], side[k][1], side[k][2]}, {side[k][3], side[k][4], side[k][5]}};
          if (c.end - c.begin <= (uint32_t)kWarpPrims)
            push_task(s, c, 0);
          else if (top < kSmallStack) /* depth-first: at most one pending sibling per level */
            stack[top++] = c;
          else
            atomicAdd(&s.n->errors, 1u); /* a lost subtree: reported as a build failure */
        }
        sp = top;
      }
      __syncthreads();
    }
  }
}

/* Subtrees of at most 32 primitives, one warp each; the warps take them from a counter, so none waits for
 * the other subtrees of its CTA. */
constexpr int kWarpBlock = 128;
__global__ void __launch_bounds__(kWarpBlock, 8) k_build_warps(Shared s) {
  chain();
  __shared__ WarpTree trees[kWarpBlock / 32];
  const unsigned n = s.n->warps;
  for (;;) {
    unsigned item = 0;
    if ((threadIdx.x & 31) == 0) item = atomicAdd(&s.n->warp_next, 1u);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= n) return;
    warp_build(s, s.tasks[s.max_tasks - 1u - item], trees[threadIdx.x >> 5]);
    __syncwarp();
  }
}

/* ------------------------------------------------------------------ depth-first node order
 *
 * Nodes are numbered as they are created, so a subtree's nodes end up interleaved with other
 * subtrees'.  The last passes renumber them in depth-first preorder (left child first), so a node's
 * descendants follow it in memory.  A node is preceded by the nodes that begin at an earlier
 * primitive (its ancestors and what hangs left of its path) and by its ancestors that begin at the
 * same one: its number is the count of nodes over the earlier positions plus its depth below the first
 * node of its own position.  (Subtree sizes passed up the tree, one atomic arrival after the other, and
 * then down each node's path, with a leaf sort and a copy back: 84 us for 93 k nodes; these four passes
 * 23.) */

/* Leaves' primitives in ascending order; nodes counted and their least depth taken per position; the
 * tree's node and leaf counts and depth. */
__global__ void __launch_bounds__(256) k_node_hist(Shared s, uint32_t n, uint32_t *count, uint32_t *least) {
  chain();
  __shared__ uint32_t total[3];
  if (threadIdx.x < 3) total[threadIdx.x] = 0;
  __syncthreads();
  uint32_t nodes = 0, leaves = 0, depth = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint2 at = s.node_at[i], L = s.leaf_at[i];
    if (at.x != 0xffffffffu) {
      atomicAdd(count + at.x, 1u);
      atomicMin(least + at.x, at.y);
      nodes++;
    }
    if (L.x == 0) continue;
    leaves++;
    depth = max(depth, L.y);
    uint32_t *o = s.order + i;
    for (uint32_t a = 1; a < L.x; a++) {
      uint32_t v = o[a];
      int b = (int)a - 1;
      while (b >= 0 && o[b] > v) {
        o[b + 1] = o[b];
        b--;
      }
      o[b + 1] = v;
    }
  }
  nodes = __reduce_add_sync(0xffffffffu, nodes);
  leaves = __reduce_add_sync(0xffffffffu, leaves);
  depth = __reduce_max_sync(0xffffffffu, depth);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&total[0], nodes);
    atomicAdd(&total[1], leaves);
    atomicMax(&total[2], depth);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicAdd(&s.n->nodes, total[0]);
    atomicAdd(&s.n->leaves, total[1]);
    atomicMax(&s.n->max_depth, (int)total[2]);
  }
}

constexpr uint32_t kScanThreads = 256, kScanPer = 4, kScanItems = kScanThreads * kScanPer;

__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t *sh /* kScanThreads / 32 */) {
  v = __reduce_add_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  uint32_t t = 0;
  for (uint32_t j = 0; j < kScanThreads / 32; j++) t += sh[j];
  __syncthreads();
  return t;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_sums(const uint32_t *count, uint32_t n, uint32_t *sums) {
  chain();
  __shared__ uint32_t sh[kScanThreads / 32];
  const uint32_t base = blockIdx.x * kScanItems;
  uint32_t c = 0;
  for (uint32_t k = 0; k < kScanPer; k++) {
    const uint32_t i = base + k * kScanThreads + threadIdx.x;
    if (i < n) c += count[i];
  }
  const uint32_t t = block_sum(c, sh);
  if (threadIdx.x == 0) sums[blockIdx.x] = t;
}

/* count[i] becomes the number of nodes at positions before i. */
__global__ void __launch_bounds__(kScanThreads) k_scan_apply(uint32_t *count, uint32_t n, const uint32_t *sums) {
  chain();
  __shared__ uint32_t sh[kScanThreads / 32];
  uint32_t b = 0;
  for (uint32_t j = threadIdx.x; j < blockIdx.x; j += kScanThreads) b += sums[j];
  uint32_t run = block_sum(b, sh);
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (uint32_t k = 0; k < kScanPer; k++) {
    const uint32_t i = blockIdx.x * kScanItems + k * kScanThreads + threadIdx.x;
    const uint32_t c = i < n ? count[i] : 0u;
    uint32_t x = c;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if ((int)lane >= o) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    uint32_t before = 0, tile = 0;
    for (uint32_t j = 0; j < kScanThreads / 32; j++) {
      if (j < w) before += sh[j];
      tile += sh[j];
    }
    if (i < n) count[i] = run + before + x - c;
    run += tile;
    __syncthreads();
  }
}

__global__ void k_permute(Shared s, uint32_t n, const uint32_t *before, const uint32_t *least, float4 *out) {
  chain();
  const uint32_t n_nodes = s.n->nodes;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (s.node_at[i].x == 0xffffffffu) continue;
    auto number = [&](uint32_t v) {
      const uint2 at = s.node_at[v];
      return at.x < n ? before[at.x] + at.y - least[at.x] : 0u;
    };
    const uint32_t j = number(i);
    float4 n3 = s.nodes[4 * (size_t)i + 3];
    const int32_t r0 = __float_as_int(n3.x), r1 = __float_as_int(n3.y);
    if (r0 >= 0) n3.x = __int_as_float((uint32_t)r0 < n ? (int32_t)number((uint32_t)r0) : 0);
    if (r1 >= 0) n3.y = __int_as_float((uint32_t)r1 < n ? (int32_t)number((uint32_t)r1) : 0);
    if (j >= n_nodes) continue; /* a broken tree: the validation reports it */
    float4 *o = out + 4 * (size_t)j;
    o[0] = s.nodes[4 * (size_t)i + 0];
    o[1] = s.nodes[4 * (size_t)i + 1];
    o[2] = s.nodes[4 * (size_t)i + 2];
    o[3] = n3;
  }
}

}  // namespace

namespace {

/* A launch that may start while its predecessor in the stream still runs (see chain()). */
template <class... P, class... A>
void launch(void (*k)(P...), unsigned grid, unsigned block, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.stream = stream;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k, static_cast<P>(args)...);
}

}  // namespace

cudaError_t build_bvh(const float4 *lo, const float4 *hi, uint32_t n, const BvhBuildParams &p, float4 *nodes,
                      uint32_t *order, cudaStream_t stream, BvhBuildResult *res) {
  auto t0 = std::chrono::steady_clock::now();
  if (n == 0) return cudaErrorInvalidValue;
  Shared s{};
  s.lo = lo;
  s.hi = hi;
  s.order = order;
  s.bins = std::max(4, std::min(kMaxBins, p.bins > 0 ? p.bins : 16));
  s.hard_leaf = std::max(1, std::min(kHardLeaf, p.hard_leaf > 0 ? p.hard_leaf : kHardLeaf));
  s.max_leaf = std::max(1, std::min(s.hard_leaf, p.max_leaf > 0 ? p.max_leaf : 8));
  s.cost_trav = p.cost_trav > 0.f ? p.cost_trav : 1.0f;
  s.small_task = p.small_task >= 64 ? std::min<uint32_t>(p.small_task, kCtaPrims) : kSmallTaskDefault;
  s.chunk = kMaxChunk;
  while (s.chunk > kMinChunk && n / s.chunk < 4u * 148u) s.chunk /= 2;
  const uint32_t max_large = n / s.small_task + 2;
  s.max_tasks = n + n / (kWarpPrims + 1) + 2;
  s.max_chunks = n / s.chunk + max_large + 2;
  const uint32_t scan_blocks = (n + kScanItems - 1) / kScanItems;
  /* all scratch in one pool allocation */
  size_t bytes = 0;
  auto take = [&](size_t b) {
    const size_t off = bytes;
    bytes += (b + 255) & ~(size_t)255;
    return off;
  };
  const size_t o_n = take(sizeof(Counters)), o_scene = take(12 * sizeof(float));
  const size_t o_ids0 = take(4ull * n), o_ids1 = take(4ull * n), o_count = take(4ull * n), o_least = take(4ull * n);
  const size_t o_nodes = take(64ull * n);
  const size_t o_at = take(8ull * n), o_leaves = take(8ull * n), o_tasks = take(sizeof(Task) * (size_t)s.max_tasks);
  const size_t o_splits = take(sizeof(SplitInfo) * (size_t)max_large), o_sums = take(4ull * scan_blocks);
  size_t o_large[2], o_bins[2], o_cb[2], o_chunks[2];
  for (int k = 0; k < 2; k++) {
    o_large[k] = take(sizeof(Task) * (size_t)max_large);
    o_bins[k] = take(sizeof(Bins) * (size_t)max_large);
    o_cb[k] = take(6 * sizeof(float) * (size_t)max_large);
    o_chunks[k] = take(sizeof(Chunk) * (size_t)s.max_chunks);
  }
  char *m = nullptr;
  cudaError_t err = cudaMallocAsync(&m, bytes, stream);
  if (err != cudaSuccess) return err;
  s.n = reinterpret_cast<Counters *>(m + o_n);
  s.scene = reinterpret_cast<float *>(m + o_scene);
  s.ids0 = reinterpret_cast<uint32_t *>(m + o_ids0);
  s.ids1 = reinterpret_cast<uint32_t *>(m + o_ids1);
  s.nodes = reinterpret_cast<float4 *>(m + o_nodes);
  s.node_at = reinterpret_cast<uint2 *>(m + o_at);
  s.leaf_at = reinterpret_cast<uint2 *>(m + o_leaves);
  s.tasks = reinterpret_cast<Task *>(m + o_tasks);
  s.splits = reinterpret_cast<SplitInfo *>(m + o_splits);
  uint32_t *sums = reinterpret_cast<uint32_t *>(m + o_sums);
  uint32_t *count = reinterpret_cast<uint32_t *>(m + o_count), *least = reinterpret_cast<uint32_t *>(m + o_least);
  for (int k = 0; k < 2; k++) {
    s.large[k] = reinterpret_cast<Task *>(m + o_large[k]);
    s.tbins[k] = reinterpret_cast<Bins *>(m + o_bins[k]);
    s.cb[k] = reinterpret_cast<float *>(m + o_cb[k]);
    s.chunks[k] = reinterpret_cast<Chunk *>(m + o_chunks[k]);
  }
  Counters hc{};
  const auto run = [&]() -> cudaError_t {
    cudaMemsetAsync(s.node_at, 0xff, 8ull * n, stream);
    cudaMemsetAsync(s.leaf_at, 0, 8ull * n, stream);
    k_init<<<1, 256, 0, stream>>>(s);
    const uint32_t begin_blocks = std::min<uint32_t>(std::max<uint32_t>(148, std::min<uint32_t>(4 * 148, n / 4096)),
                                                     (n + kBlock - 1) / kBlock);
    launch(k_begin, begin_blocks, kBlock, stream, s, n);
    /* levels of a balanced tree and six more: a level past the last large node leaves its three kernels
     * nothing to do (7 us), and one too few costs another round of everything below (170 us) */
    int level = 0, want = 0;
    if (n > s.small_task)
      for (want = 6; n >> (want - 6) > s.small_task;) want++;
    for (;;) {
      for (; level < want; level++) {
        if (level + 1 >= kMaxLevels) return cudaErrorUnknown; /* the median splits end every tree before */
        const uint32_t tasks = (uint32_t)std::min<uint64_t>(max_large - 1, 1ull << std::min(level, 31));
        const uint32_t chunks = std::min(s.max_chunks, n / s.chunk + tasks);
        launch(k_bin, chunks, kBlock, stream, s, level);
        launch(k_split, tasks, kBlock, stream, s, level);
        launch(k_partition, chunks, kBlock, stream, s, level);
      }
      if (n > (uint32_t)kWarpPrims)
        launch(k_build_small, std::min<uint32_t>(148 * 4, n / (kWarpPrims + 1) + 1), kCtaPrims, stream, s);
      launch(k_build_warps, std::min<uint32_t>(148 * 8, (n + 3) / 4), kWarpBlock, stream, s);
      cudaMemsetAsync(count, 0, 4ull * n, stream);
      cudaMemsetAsync(least, 0xff, 4ull * n, stream);
      const unsigned grid = std::min<uint32_t>(148 * 8, (n + 255) / 256);
      launch(k_node_hist, grid, 256, stream, s, n, count, least);
      launch(k_scan_sums, scan_blocks, kScanThreads, stream, count, n, sums);
      launch(k_scan_apply, scan_blocks, kScanThreads, stream, count, n, sums);
      launch(k_permute, grid, 256, stream, s, n, count, least, nodes);
      cudaError_t e = cudaGetLastError();
      if (e == cudaSuccess) e = cudaMemcpyAsync(&hc, s.n, sizeof(Counters), cudaMemcpyDeviceToHost, stream);
      if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
      if (e != cudaSuccess || hc.errors != 0 || n <= s.small_task || hc.level[level].tasks == 0) return e;
      /* large nodes are left: more levels, then the subtrees they add (the counters the CTAs and warps took
       * theirs from have run past the end) and the order again */
      want = level + 4;
      hc.small_next = hc.small;
      hc.warp_next = hc.warps;
      hc.nodes = hc.leaves = 0;
      e = cudaMemcpyAsync(s.n, &hc, sizeof(Counters), cudaMemcpyHostToDevice, stream);
      if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
      if (e != cudaSuccess) return e;
    }
  };
  err = run();
  cudaFreeAsync(m, stream);
  if (err == cudaSuccess && hc.errors != 0) err = cudaErrorUnknown; /* never expected: reported as a build failure */
  if (err == cudaSuccess && res) {
    res->n_nodes = hc.nodes;
    res->n_leaves = hc.leaves;
    res->max_depth = hc.max_depth;
  }
  if (res) res->ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  return err;
}

}  // namespace nb
