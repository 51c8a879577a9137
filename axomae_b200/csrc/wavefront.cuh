/* What the wavefront's translation units share: its tables and counters, the device code of one path's steps, and
 * the kernels that more than one of them instantiates.
 *
 *   integrator.cu     renders: the wave loop, camera rays, shading, films; the intersector's own calls
 *   wave_adjoint.cu   the replay's waves
 *   wave_modes.cu     trace modes 1 to 3: ray hand-out, counted walks, the persistent wavefront
 *
 * Each is a module of its own on the device, loaded by the first call that launches from it.  Loading takes
 * 0.4 ms a megabyte: in one module of 11 MB a process's first trace() took 5.4 ms, now 2.7, and its first
 * small frame 6.3 ms, now 2.9.
 * integrator.cu describes the whole.
 */
#pragma once

#include <algorithm>

#include "context.cuh"
#include "shading.cuh"
#include "traverse.cuh"

namespace nb {
namespace wave {

struct RenderParams {
  int32_t W, H;
  uint32_t NP;    /* pixels */
  uint32_t count; /* samples traced for this job in the current chunk */
  uint32_t begin; /* first of those samples */
  uint32_t spp_total;
  int32_t max_depth;
  uint32_t seed;
  int32_t rr_start;
  float inv_P[16], inv_V[16];
  uint32_t tile_w, tile_h; /* consecutive paths walk tile_w x tile_h pixel tiles (0: image rows) */
  int32_t vinv;            /* film rows stored top-down (vertical_invert) */
};

struct Job {
  DevScene sc;
  RenderParams rp;
  uint32_t path_begin; /* first path id of this job in the chunk (radiance slot of its first path) */
  uint32_t n_paths;
};

/* One wave's counters.  Wave k uses ring entry k & 3: its kernels read entry k, append survivors to
 * entry k + 1 and clear entry k + 2, so no kernel between waves has to advance them. */
struct WaveState {
  uint32_t n_active; /* rays waiting in the wave's input queue */
  uint32_t next;     /* next path id to start */
  uint32_t hit_count;
  uint32_t hit_back;   /* hits of transmissive materials, from the end of the hit list */
  uint32_t trace_next; /* next queued ray handed out by the persistent trace kernel */
  uint32_t shade_next; /* next hit handed out in the persistent wavefront */
};
constexpr uint32_t kWaveRing = 4;

struct WaveCounters {
  WaveState w[kWaveRing];
  uint32_t total; /* paths in the chunk */
  uint32_t cap;   /* queue capacity */
  uint32_t waves; /* waves that did work */
  uint32_t finish_waves; /* most segments a path took in k_finish: the waves it stands for */
  uint32_t done;         /* persistent wavefront: every path has ended */
  /* device status of the whole loop (never reset between waves): path radiance values that were not
   * finite and were written as 0 (the reference's DENAN, Integrator.cpp:92), and hits whose
   * primitive, instance or material id is out of range (the path ends black, the render fails) */
  uint32_t nonfinite, bad_index;
  unsigned long long traced;
  unsigned long long node_visits, tri_tests; /* trace_mode 2 only: the traversal's own work */
};

/* The chunk's job table as a kernel parameter. */
struct OneJob {
  Job j;
  __device__ __forceinline__ const Job &at(uint32_t) const { return j; }
  __device__ __forceinline__ uint32_t find(uint32_t) const { return 0u; }
};

constexpr uint32_t kParamJobs = 104;

struct ManyJobs {
  uint32_t n;
  Job j[kParamJobs];
  __device__ __forceinline__ const Job &at(uint32_t k) const { return j[k]; }
  /* the last job whose first path id is <= g */
  __device__ __forceinline__ uint32_t find(uint32_t g) const {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (j[mid].path_begin <= g)
        lo = mid;
      else
        hi = mid;
    }
    return lo;
  }
};
static_assert(sizeof(ManyJobs) + 256 <= 32764, "a batch job table must fit the 32 KB kernel parameter space");

struct Queue {
  float4 *o, *d, *beta;
};

struct AdjQueue {
  float4 *rem, *dl;
};

/* Launch shape of one render: rays per wave and the trace / shade block sizes. */
struct LaunchShape {
  uint32_t cap;
  uint32_t trace_block, shade_block;
  uint32_t trace_mode; /* 0: one ray per thread, 1: persistent warps with ray hand-out (binary BVH),
                         2: one ray per thread, counting node visits and triangle tests,
                         3: the persistent wavefront (one cooperative launch per chunk) */
  uint32_t wait_limit_us; /* trace_mode 3: longest grid-barrier wait before the render fails */
  uint32_t finish_rays;   /* rays left at which k_finish takes over (trace modes 1 and 2 stay with their kernel) */
};

/* Replay-loop arguments: the adjoint queues (A, B), the image adjoint and the gradients. */
struct AdjArgs {
  AdjQueue qa, qb;
  const float4 *d_image;
  float *g_alb, *g_rough;
};

/* One wave to enqueue: its number, the most rays and new paths it can hold (its kernels read the exact
 * counts on the device) and whether k_finish takes it over. */
struct WavePlan {
  uint32_t wave, rays, fresh, total, cap;
  bool finish;
};

/* Counters of wave loops. */
struct LoopStats {
  float t_trace = 0.f, t_shade = 0.f;
  uint64_t kernels = 0, traced = 0;
  uint64_t nonfinite = 0, bad_index = 0, node_visits = 0, tri_tests = 0;
  uint32_t waves = 0;
  void add_to(nova_b200_render_stats &s) const {
    s.node_visits += node_visits;
    s.tri_tests += tri_tests;
    s.nonfinite += nonfinite;
    s.bad_index += bad_index;
    s.traced += traced;
    s.segments += traced;
    s.waves += waves;
    s.kernels += kernels;
    s.trace_ms += t_trace;
    s.shade_ms += t_shade;
  }
};

/* wave_adjoint.cu: enqueues one wave of the replay, as integrator.cu's enqueue_wave does one of a render. */
cudaError_t enqueue_adjoint_wave(nova_b200_ctx *c, const OneJob &js, const LaunchShape &ls, int width,
                                 const WavePlan &p, uint64_t &kernels, const AdjArgs &adj);

/* wave_modes.cu: launches the trace pass of trace modes 1 (binary BVH) and 2 on the wave's input queue, and runs a
 * whole chunk in mode 3. */
void launch_mode_trace(nova_b200_ctx *c, const OneJob &js, const LaunchShape &ls, int width, const WavePlan &p);
void launch_mode_trace(nova_b200_ctx *c, const ManyJobs &js, const LaunchShape &ls, int width, const WavePlan &p);
nova_b200_status run_persistent(nova_b200_ctx *x, const OneJob &js, const LaunchShape &ls, int width, uint32_t total,
                                uint32_t cap, LoopStats &st);
nova_b200_status run_persistent(nova_b200_ctx *x, const ManyJobs &js, const LaunchShape &ls, int width, uint32_t total,
                                uint32_t cap, LoopStats &st);

}  // namespace wave
}  // namespace nb

namespace {

using namespace nb;
using namespace nb::wave;

constexpr unsigned kRRDimBase = 200; /* Russian roulette decisions use Sobol dimension 200 + bounce */
constexpr int kMaxDepth = 48;        /* 2 + 4 (depth + 1) Sobol dimensions must stay below 200 */

struct WaveBuffers {
  Queue qa, qb;
  float4 *hits;
  uint2 *hit_slot; /* per hit: its ray's queue slot and the hit triangle's instance */
  WaveCounters *wc;
};

inline WaveBuffers wave_buffers(nova_b200_ctx *c) {
  const uint32_t cap = c->queue_cap;
  float4 *base = static_cast<float4 *>(c->d_queue);
  WaveBuffers b;
  b.qa = Queue{base, base + cap, base + 2 * (size_t)cap};
  b.qb = Queue{base + 3 * (size_t)cap, base + 4 * (size_t)cap, base + 5 * (size_t)cap};
  b.hits = base + 6 * (size_t)cap;
  b.hit_slot = reinterpret_cast<uint2 *>(base + 7 * (size_t)cap);
  b.wc = static_cast<WaveCounters *>(c->d_wave);
  return b;
}

/* The wave's input and output queue: A -> B -> A ... */
inline const Queue &input_queue(const WaveBuffers &b, uint32_t wave) { return wave & 1u ? b.qb : b.qa; }
inline const Queue &output_queue(const WaveBuffers &b, uint32_t wave) { return wave & 1u ? b.qa : b.qb; }

/* Blocks of `block` threads for n items, at least one. */
inline unsigned blocks_for(uint32_t n, uint32_t block) { return std::max(1u, (n + block - 1) / block); }

/* Paths per warp of k_finish: the fewest, down to 2, that make at most 2,048 warps of paths already on
 * their way, or 4,096 of camera rays, half of which end at once (2,960 warps are resident).  A warp takes
 * as long as the union of its lanes' walks, so few paths are spread thin: 16,384 camera paths of depth 4
 * take 146 us with 8 a warp and 185 with 32, 1,024 take 84 with 2 and 157 with 32; 65,536 take 173 with
 * 16, 191 with 32 and 200 with 8, but the late waves of a 1283 x 721 frame lose 50 us with 16. */
inline uint32_t finish_lanes(uint32_t rays, uint32_t wave) {
  const uint32_t warps = wave == 0 ? 4096 : 2048;
  uint32_t lanes = 32;
  while (lanes > 2 && rays / (lanes / 2) <= warps) lanes /= 2;
  return lanes;
}

/* New paths that start in the wave of entry `ws`, and the wave's rays. */
__device__ __forceinline__ uint32_t wave_new(const WaveCounters &wc, const WaveState &ws) {
  return min(wc.cap - ws.n_active, wc.total - ws.next);
}
__device__ __forceinline__ uint32_t wave_rays(const WaveCounters &wc, const WaveState &ws) {
  return ws.n_active + wave_new(wc, ws);
}
__device__ __forceinline__ WaveState &wave_at(WaveCounters *wc, uint32_t k) { return wc->w[k & (kWaveRing - 1u)]; }

/* The next wave's first path and the wave statistics, by one thread of wave k's trace pass. */
__device__ __forceinline__ void advance_wave(WaveCounters *wc, uint32_t k) {
  const WaveState &ws = wave_at(wc, k);
  const uint32_t n_new = wave_new(*wc, ws), n = ws.n_active + n_new;
  wave_at(wc, k + 1).next = ws.next + n_new;
  wc->traced += n;
  if (n) wc->waves++;
}

/* Entry k + 2 cleared for its wave, by one thread of wave k's shading pass. */
__device__ __forceinline__ void clear_wave(WaveCounters *wc, uint32_t k) {
  WaveState &ws = wave_at(wc, k + 2);
  ws.n_active = ws.hit_count = ws.hit_back = ws.trace_next = ws.shade_next = 0;
}

/* The q-th pixel a frame's paths visit: row-major, or tile_w x tile_h tiles in row-major tile
 * order (partial tiles at the right and bottom edges), so a warp's primary rays cover a compact
 * patch of the image. */
__device__ __forceinline__ void tile_pixel(const RenderParams &rp, uint32_t q, uint32_t &x, uint32_t &y) {
  const uint32_t W = (uint32_t)rp.W, H = (uint32_t)rp.H;
  if (rp.tile_w == 0) {
    y = q / W;
    x = q - y * W;
    return;
  }
  const uint32_t tw = rp.tile_w, th = rp.tile_h;
  const uint32_t ty = q / (W * th), r = q - ty * W * th;
  const uint32_t h_r = min(th, H - ty * th);
  const uint32_t tx = r / (tw * h_r), r2 = r - tx * tw * h_r;
  const uint32_t w_c = min(tw, W - tx * tw);
  const uint32_t ly = r2 / w_c;
  x = tx * tw + (r2 - ly * w_c);
  y = ty * th + ly;
}

/* The camera ray of path g of the chunk: pixel (x, y), radiance slot and Sobol index. */
struct CameraPath {
  uint32_t job, x, y, rslot, index;
  V4 o, d;
};

template <class JS>
__device__ __forceinline__ CameraPath camera_path(const JS &js, uint32_t g) {
  CameraPath c;
  c.job = js.find(g);
  const Job &J = js.at(c.job);
  const RenderParams &rp = J.rp;
  const uint32_t p = g - J.path_begin;
  const uint32_t s_local = p / rp.NP, q_pix = p - s_local * rp.NP;
  uint32_t x, y;
  tile_pixel(rp, q_pix, x, y);
  c.x = x;
  c.y = y;
  /* the radiance slot stays keyed by the row-major pixel, whatever order paths start in */
  c.rslot = J.path_begin + s_local * rp.NP + y * (uint32_t)rp.W + x;
  const uint32_t index = ((uint32_t)x * (uint32_t)rp.H + (uint32_t)y) * rp.spp_total + (rp.begin + s_local);
  c.index = index;
  const float r0 = sobol_sample(J.sc.sobol_dv, index, 0, rp.seed);
  const float r1 = sobol_sample(J.sc.sobol_dv, index, 1, rp.seed);
  const float dx = r0 * 0.0005f, dy = r1 * 0.0005f; /* RAND_DX / RAND_DY, Integrator.h:54-55 */
  const int ys = rp.H - (int)y;                     /* screen row, Integrator.h:84 */
  const float ndc_x = (float)(2 * (int)x - rp.W) / (float)rp.W;
  const float ndc_y = (float)(rp.H - 2 * ys) / (float)rp.H;
  const float nx = ndc_x + dx, ny = ndc_y + dy;
  const M4 iP = m4_load(rp.inv_P), iV = m4_load(rp.inv_V);
  V4 o = mul(iP, V4{nx, ny, -1.f, 1.f});
  o = o / o.w;
  o = mul(iV, V4{o.x, o.y, o.z, 1.f});
  V4 d = mul(iP, V4{nx, ny, -1.f, 0.f});
  d = normalize(mul(iV, V4{d.x, d.y, -1.f, 0.f}));
  c.o = o;
  c.d = d;
  return c;
}

/* Camera ray of new path `next + i` into queue slot `n_active + i`; o4, d4: its queue entries. */
template <class JS>
__device__ __forceinline__ void refill_one(const Queue &q, uint32_t next, uint32_t n_active, float4 *L, const JS &js,
                                           uint32_t i, float4 &o4, float4 &d4) {
  const CameraPath c = camera_path(js, next + i);
  const uint32_t slot = n_active + i;
  q.o[slot] = o4 = make_float4(c.o.x, c.o.y, c.o.z, __uint_as_float(c.rslot));
  q.d[slot] = d4 = make_float4(c.d.x, c.d.y, c.d.z, __uint_as_float(c.job << 8));
  q.beta[slot] = make_float4(1.f, 1.f, 1.f, __uint_as_float(c.index));
  if (js.at(c.job).sc.has_emissive) L[c.rslot] = make_float4(0.f, 0.f, 0.f, 0.f);
}

/* The wave's counters; wave 0's refill starts them (no copy from the host before it), so its blocks take
 * them as zero. */
__device__ __forceinline__ WaveState first_state(WaveCounters *wcp, uint32_t wave, uint32_t total, uint32_t cap) {
  if (wave != 0) return wave_at(wcp, wave);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    WaveCounters wc{};
    wc.total = total;
    wc.cap = cap;
    *wcp = wc;
  }
  return WaveState{};
}

/* Non-finite radiance becomes 0 (DENAN), counted in *nonfinite (rare: a plain atomic). */
__device__ __forceinline__ float4 finite_or_zero(V3 L, float alpha, unsigned *nonfinite) {
  if (!finite3(L)) {
    atomicAdd(nonfinite, 1u);
    return make_float4(0.f, 0.f, 0.f, 0.f);
  }
  return make_float4(L.x, L.y, L.z, alpha);
}

/* Loads of data written earlier in the same launch by other blocks: through L2 (ld.global.cg) when P,
 * the persistent wavefront; plain loads otherwise (a kernel boundary orders them). */
template <bool P, class T>
__device__ __forceinline__ T ldq(const T *p) {
  if constexpr (P)
    return __ldcg(p);
  else
    return *p;
}

/* Writes a finished path's radiance (adds the emission gathered so far when the scene has any). */
template <bool P = false>
__device__ __forceinline__ void finish_path(const DevScene &sc, float4 *L, uint32_t g, float4 result,
                                            unsigned *nonfinite) {
  if (sc.has_emissive) {
    const float4 acc = ldq<P>(&L[g]);
    float4 r = make_float4(acc.x + result.x, acc.y + result.y, acc.z + result.z, result.w);
    if (!isfinite(r.x) || !isfinite(r.y) || !isfinite(r.z)) {
      atomicAdd(nonfinite, 1u);
      r = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    L[g] = r;
  } else {
    L[g] = result;
  }
}

/* The hit's primitive, its instance (from the hit list) and the instance's material all index their
 * tables, and the primitive is one of the instance's triangles. */
__device__ __forceinline__ bool hit_ids_valid(const DevScene &sc, int prim, uint32_t inst) {
  if (prim < 0 || (uint32_t)prim >= sc.n_prims || inst >= sc.n_instances) return false;
  const DevInstance &I = sc.instances[inst];
  return (uint32_t)prim - I.prim_offset < I.n_tris && I.material < sc.n_materials;
}

/* Warp-aggregated append: returns the slot of every lane with `flag` set. */
__device__ __forceinline__ unsigned warp_append(bool flag, unsigned *counter) {
  const unsigned lane = threadIdx.x & 31u;
  const unsigned m = __ballot_sync(0xffffffffu, flag);
  unsigned base = 0;
  if (m) {
    if (lane == (unsigned)(__ffs(m) - 1)) base = atomicAdd(counter, (unsigned)__popc(m));
    base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
  }
  return base + __popc(m & ((1u << lane) - 1u));
}

/* Closest hit of every queued ray.  A miss finishes its path here (environment lookup,
 * Integrator.cpp:94-98); hits are appended to a compact hit list so the shading kernel only runs
 * on rays that hit.  At least 10 resident blocks of 128 (48 registers): the walk is latency-bound,
 * and 40 warps per SM beat 32 (-4% on the batched scenes); 12 blocks spill the walk state. */
/* Resident blocks of 128 threads per SM that k_trace is compiled for (the register bound is
 * 65536 / (128 * blocks)).  Binary: 10 blocks (48 registers, next to no spills), 21.6 ms of traversal
 * on an 8-frame batch against 22.3 at 9 and 23.4 at 8.  Two-level: the walk also holds the world ray
 * and the instance, so 10 blocks spill: 3.84 ms on 1000 instances at 720p, 9 blocks (56 registers) 3.64,
 * 8 blocks 3.61. */
template <int WIDTH>
constexpr int kTraceBlocks = WIDTH == 1 ? 9 : 10;

/* The hit list holds non-transmissive hits from its front and transmissive ones from its back (k_shade
 * reads both ranges), so shading warps mostly run one lobe family: the dielectric lobe's refraction
 * code or the reflective lobes'.  The class is the instance's (its material's eta and k,
 * NovaMaterials.h:118-121).  On 32 frames k_shade went from 107.3 to 80.9 ms (films bit-identical);
 * only the order in which hits are shaded changes.  A third list for fully metal materials measured
 * equal (shading -0.6 %, the third append +0.4 % in k_trace). */

/* The closest-hit pass for one warp's lanes (ray i of n queued; the warp's lanes call together: the
 * hit append is a warp ballot).
 *
 * FRESH, for a wave that starts paths: the lanes past the waiting rays make their camera rays themselves, and
 * the queue entries they write are for k_shade.  A k_refill before the pass wrote the same entries for it
 * to read again: 33 M paths at 1920 x 1080 take 8.01 ms so against 8.14, 90 M paths of 8 frames 35.2 against
 * 35.4.  Camera rays made a second time in k_shade instead of kept in the queue: 8.17 and 35.9. */
template <int WIDTH, class JS, bool ADJ, bool COUNT, bool P, bool FRESH = false>
__device__ __forceinline__ void trace_warp(const Queue &q, WaveCounters *wcp, WaveState &ws, float4 *hits,
                                           uint2 *hit_slot, float4 *L, const JS &js, uint32_t i, uint32_t n) {
  {
    bool is_hit = false, back = false;
    TraceResult r{-1, 0.f, 0.f, 0.f, 0u};
    uint64_t nv = 0, tt = 0;
    if (i < n) {
      float4 o, d;
      if (FRESH && i >= ws.n_active)
        refill_one(q, ws.next, ws.n_active, L, js, i - ws.n_active, o, d);
      else
        o = ldq<P>(&q.o[i]), d = ldq<P>(&q.d[i]);
      const DevScene &sc = js.at(__float_as_uint(d.w) >> 8).sc;
      if constexpr (P)
        r = walk<WIDTH>(sc, V3{o.x, o.y, o.z}, V3{d.x, d.y, d.z});
      else
        r = trace_closest_w<WIDTH>(sc, V3{o.x, o.y, o.z}, V3{d.x, d.y, d.z}, COUNT ? &nv : nullptr,
                                   COUNT ? &tt : nullptr);
      if (r.prim >= 0) {
        is_hit = true;
        if constexpr (!COUNT && !P) back = sc.instances[r.inst].lobe_class != 0u;
      } else if (!ADJ) { /* a replayed path's radiance is already known */
        const float4 b4 = ldq<P>(&q.beta[i]);
        const V4 e = env_sample(sc, V3{d.x, d.y, d.z});
        finish_path<P>(sc, L, __float_as_uint(o.w),
                    finite_or_zero(V3{b4.x, b4.y, b4.z} * V3{e.x, e.y, e.z},
                                   (float)(__float_as_uint(d.w) & 0xffu) + e.w, &wcp->nonfinite),
                    &wcp->nonfinite);
      }
    }
    if constexpr (COUNT) { /* one atomic per warp for each counter */
      for (int off = 16; off > 0; off >>= 1) {
        nv += __shfl_down_sync(0xffffffffu, nv, off);
        tt += __shfl_down_sync(0xffffffffu, tt, off);
      }
      if ((threadIdx.x & 31u) == 0) {
        atomicAdd(&wcp->node_visits, (unsigned long long)nv);
        atomicAdd(&wcp->tri_tests, (unsigned long long)tt);
      }
    }
    uint32_t slot;
    if constexpr (!COUNT && !P) {
      /* transmissive hits go to the end of the list, the others to the front, so the shading warps
       * mostly take one lobe family (BSDF.h:69-79) */
      const unsigned f = warp_append(is_hit && !back, &ws.hit_count);
      const unsigned b = warp_append(back, &ws.hit_back);
      slot = back ? wcp->cap - 1u - b : f;
    } else {
      slot = warp_append(is_hit, &ws.hit_count);
    }
    if (is_hit) {
      hits[slot] = make_float4(r.t, r.u, r.v, __int_as_float(r.prim));
      hit_slot[slot] = make_uint2(i, r.inst);
    }
  }
}

template <int WIDTH, class JS, bool ADJ = false, bool COUNT = false, bool FRESH = false>
__global__ void __launch_bounds__(128, kTraceBlocks<WIDTH>)
    k_trace(Queue q, WaveCounters *wcp, uint32_t wave, float4 *hits, uint2 *hit_slot, float4 *L,
            const __grid_constant__ JS js) {
  WaveState &ws = wave_at(wcp, wave);
  const uint32_t n = wave_rays(*wcp, ws);
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) advance_wave(wcp, wave);
  if ((i & ~31u) >= n) return; /* whole warps leave together (the append is a warp ballot) */
  trace_warp<WIDTH, JS, ADJ, COUNT, false, FRESH>(q, wcp, ws, hits, hit_slot, L, js, i, n);
}

/* Shades one path at its hit (t, u, v, prim) on instance `inst`: true when it goes on, with the spawned
 * ray in o4, d4, b4; else its radiance has been written. */
template <class JS, bool P>
__device__ __forceinline__ bool shade_path(float4 &o4, float4 &d4, float4 &b4, const float4 &h, uint32_t inst,
                                           WaveCounters *wcp, float4 *L, const JS &js) {
  const uint32_t g = __float_as_uint(o4.w);
  const uint32_t tag = __float_as_uint(d4.w);
  const int bounce = (int)(tag & 0xffu);
  const Job &J = js.at(tag >> 8);
  const DevScene &sc = J.sc;
  const RenderParams &rp = J.rp;
  const uint32_t index = __float_as_uint(b4.w); /* the path's Sobol index, set by k_refill */
  const V3 ro{o4.x, o4.y, o4.z}, rd{d4.x, d4.y, d4.z};
  V3 beta{b4.x, b4.y, b4.z};
  const int prim = __float_as_int(h.w);
  if (!hit_ids_valid(sc, prim, inst)) {
    atomicAdd(&wcp->bad_index, 1u);
    L[g] = make_float4(0.f, 0.f, 0.f, 0.f);
    return false;
  }
  const DevInstance &I = sc.instances[inst];
  const HitRecord hr = make_record(sc, ro, rd, I, (uint32_t)prim - I.prim_offset, h.x, h.y, h.z);
  const ScatterResult sr = scatter(sc, rd, hr, sc.materials[I.material], index, 2u + 4u * (unsigned)bounce, rp.seed,
                                   (uint32_t)prim, I.material);
  /* a failed scatter returns black, emission included (Integrator.cpp:73-79) */
  if (sr.valid && sc.has_emissive && any_nonzero(sr.emissive)) {
    const V3 em = beta * sr.emissive;
    const float4 acc = ldq<P>(&L[g]);
    L[g] = make_float4(acc.x + em.x, acc.y + em.y, acc.z + em.z, acc.w);
  }
  float4 result = make_float4(0.f, 0.f, 0.f, (float)bounce);
  if (sr.valid) {
    V3 c = sr.weight;
    bool alive = true;
    if (rp.rr_start >= 0 && bounce >= rp.rr_start) {
      const V3 nbt = beta * c;
      const float q = fmin_std(1.f, fmax_std(0.05f, fmax_std(nbt.x, fmax_std(nbt.y, nbt.z))));
      const float urr = sobol_sample(sc.sobol_dv, index, kRRDimBase + (unsigned)bounce, rp.seed);
      if (!(urr < q)) {
        alive = false;
        result = make_float4(0.f, 0.f, 0.f, (float)bounce + 1.f);
      } else {
        c = c / q;
      }
    }
    if (alive) {
      beta = beta * c;
      const float eps = 1e-3f; /* Ray::spawn, ray/Ray.h:22-27 */
      const V3 nd3 = normalize(sr.wi);
      const V3 no3 = hr.position + hr.ng * (eps + eps * fsign(dot(hr.ng, sr.wi)));
      if (bounce + 1 > rp.max_depth) {
        const V4 e = env_sample(sc, nd3);
        result = finite_or_zero(beta * V3{e.x, e.y, e.z}, (float)bounce + 1.f + e.w, &wcp->nonfinite);
      } else {
        o4 = make_float4(no3.x, no3.y, no3.z, o4.w);
        d4 = make_float4(nd3.x, nd3.y, nd3.z, __uint_as_float(tag + 1u));
        b4 = make_float4(beta.x, beta.y, beta.z, b4.w);
        return true;
      }
    }
  }
  finish_path<P>(sc, L, g, result, &wcp->nonfinite);
  return false;
}

/* The shading pass for one warp's lanes (hit i, when the lane has one; the warp's lanes call together:
 * the continuation append is a warp ballot). */
template <class JS, bool P>
__device__ __forceinline__ void shade_warp(const Queue &in, const Queue &out, WaveCounters *wcp, unsigned *out_count,
                                           const float4 *hits, const uint2 *hit_slot, float4 *L, const JS &js,
                                           uint32_t i, bool valid) {
  bool enq = false;
  float4 o4{}, d4{}, b4{};
  if (valid) {
    const uint2 hs = ldq<P>(&hit_slot[i]);
    o4 = ldq<P>(&in.o[hs.x]), d4 = ldq<P>(&in.d[hs.x]), b4 = ldq<P>(&in.beta[hs.x]);
    enq = shade_path<JS, P>(o4, d4, b4, ldq<P>(&hits[i]), hs.y, wcp, L, js);
  }
  const unsigned slot = warp_append(enq, out_count);
  if (enq) {
    out.o[slot] = o4;
    out.d[slot] = d4;
    out.beta[slot] = b4;
  }
}

/* Hit t of a wave: of the front range, or of the back range counted from the end of the list. */
__device__ __forceinline__ uint32_t hit_index(uint32_t t, uint32_t front, uint32_t cap) {
  return t < front ? t : cap - 1u - (t - front);
}

/* ---------------------------------------------------------------- replay adjoint
 *
 * Path-replay backpropagation (detached sampling).  A path's estimate is
 *   I = sum_k beta_k e_k + beta_K env,  beta_k = w_0 ... w_{k-1},  w_k = f_k |cos| / pdf_k.
 * With the sampling densities held fixed, d w_k / d theta = w_k d ln f_k / d theta, and theta_k
 * (the albedo of the triangle hit at vertex k, the roughness of its material) scales everything
 * the path gathers after vertex k's own emission: R_k = I - sum_{m <= k} beta_m e_m.  So
 *   dLoss/dtheta_k += sum_c dLoss/dI_c R_k,c d ln f_k,c / d theta_k.
 * The replay starts with R = I (the path's radiance from the primal pass, read from the radiance
 * buffer) and subtracts emission as it walks the path again from the same Sobol index; vertices
 * add their terms to the gradients with atomics.  Extra path state: R and dLoss/dI (2 x 16 B). */

/* Adds v[0..N) to base[key * N + 0..N) for every active lane.  Lanes of the warp with the same key
 * are summed first (pointer jumping along the lanes that share the key: after five rounds the
 * first lane of each key holds its sum), so a key costs one atomic per value per warp.  Camera
 * paths of neighbouring pixels share triangles and materials, and a large triangle can be hit by a
 * sizeable part of the image: without the warp sum, its atomics serialise.  All 32 lanes must call
 * this together. */
template <int N>
__device__ __forceinline__ void warp_add_by_key(bool active, uint32_t key, const float (&v)[N], float *base) {
  const unsigned full = 0xffffffffu;
  const unsigned lane = threadIdx.x & 31u;
  const unsigned peers = __match_any_sync(full, active ? key : 0xffffffffu);
  const unsigned above = lane == 31u ? 0u : (peers & (0xffffffffu << (lane + 1u)));
  int nxt = above ? __ffs(above) - 1 : 32;
  float sum[N];
#pragma unroll
  for (int k = 0; k < N; k++) sum[k] = active ? v[k] : 0.f;
#pragma unroll
  for (int it = 0; it < 5; it++) {
    const int src = nxt < 32 ? nxt : (int)lane;
    float t[N];
#pragma unroll
    for (int k = 0; k < N; k++) t[k] = __shfl_sync(full, sum[k], src);
    const int nn = __shfl_sync(full, nxt, src);
    if (nxt < 32) {
#pragma unroll
      for (int k = 0; k < N; k++) sum[k] += t[k];
      nxt = nn;
    }
  }
  if (active && lane == (unsigned)(__ffs(peers) - 1)) {
#pragma unroll
    for (int k = 0; k < N; k++)
      if (sum[k] != 0.f) atomicAdd(base + (size_t)key * N + k, sum[k]);
  }
}

/* One vertex's terms of the gradients. */
struct AdjTerms {
  bool active;
  uint32_t prim, mat;
  float albedo[3], rough[1];
};

/* Replays one path's vertex at its hit: its gradient terms, and true when the path goes on, with the
 * spawned ray in o4, d4, b4 and what it still gathers in rem. */
template <class JS>
__device__ __forceinline__ bool shade_adj_path(float4 &o4, float4 &d4, float4 &b4, float4 &rem4, const float4 &l4,
                                               const float4 &h, uint32_t inst, WaveCounters *wcp, const JS &js,
                                               AdjTerms &g) {
  const uint32_t tag = __float_as_uint(d4.w);
  const int bounce = (int)(tag & 0xffu);
  const Job &J = js.at(tag >> 8);
  const DevScene &sc = J.sc;
  const RenderParams &rp = J.rp;
  const uint32_t index = __float_as_uint(b4.w);
  const V3 ro{o4.x, o4.y, o4.z}, rd{d4.x, d4.y, d4.z};
  V3 beta{b4.x, b4.y, b4.z};
  V3 rem{rem4.x, rem4.y, rem4.z};
  const V3 dl{l4.x, l4.y, l4.z};
  const int prim = __float_as_int(h.w);
  if (!hit_ids_valid(sc, prim, inst)) {
    atomicAdd(&wcp->bad_index, 1u);
    return false;
  }
  const DevInstance &I = sc.instances[inst];
  const HitRecord hr = make_record(sc, ro, rd, I, (uint32_t)prim - I.prim_offset, h.x, h.y, h.z);
  Scores scs;
  const ScatterResult sr = scatter(sc, rd, hr, sc.materials[I.material], index, 2u + 4u * (unsigned)bounce, rp.seed,
                                   (uint32_t)prim, I.material, &scs);
  if (!sr.valid) return false;
  if (sc.has_emissive) rem = rem - beta * sr.emissive;
  const V3 cw = dl * rem;
  g.active = true;
  g.prim = (uint32_t)prim;
  g.mat = I.material;
  g.albedo[0] = cw.x * scs.albedo.x;
  g.albedo[1] = cw.y * scs.albedo.y;
  g.albedo[2] = cw.z * scs.albedo.z;
  const float gr = ((cw.x + cw.y) + cw.z) * scs.roughness;
  g.rough[0] = isfinite(gr) ? gr : 0.f;
  V3 c = sr.weight;
  if (rp.rr_start >= 0 && bounce >= rp.rr_start) {
    const V3 nbt = beta * c;
    const float q = fmin_std(1.f, fmax_std(0.05f, fmax_std(nbt.x, fmax_std(nbt.y, nbt.z))));
    const float urr = sobol_sample(sc.sobol_dv, index, kRRDimBase + (unsigned)bounce, rp.seed);
    if (!(urr < q)) return false;
    c = c / q;
  }
  if (bounce + 1 > rp.max_depth) return false;
  beta = beta * c;
  const float eps = 1e-3f;
  const V3 nd3 = normalize(sr.wi);
  const V3 no3 = hr.position + hr.ng * (eps + eps * fsign(dot(hr.ng, sr.wi)));
  o4 = make_float4(no3.x, no3.y, no3.z, o4.w);
  d4 = make_float4(nd3.x, nd3.y, nd3.z, __uint_as_float(tag + 1u));
  b4 = make_float4(beta.x, beta.y, beta.z, b4.w);
  rem4 = make_float4(rem.x, rem.y, rem.z, 0.f);
  return true;
}

/* Adds the warp's terms to the gradients asked for (all 32 lanes call it). */
__device__ __forceinline__ void add_terms(const AdjTerms &g, float *g_alb, float *g_rough) {
  if (g_alb) warp_add_by_key<3>(g.active, g.prim, g.albedo, g_alb);
  if (g_rough) warp_add_by_key<1>(g.active, g.mat, g.rough, g_rough);
}

/* ---------------------------------------------------------------- finishing a draining wavefront
 *
 * Once every path has started and few are left, a wave costs the latency of its longest walk (70 us,
 * 187 rays or 65,536 alike) whatever it holds, and each later bounce pays it again.  k_finish takes the
 * queue instead and runs each path to its end in one thread: a warp waits for its own longest walk of
 * each bounce, not the wave's, and the bounces need no launches.  The device functions are the waves'
 * (same arithmetic per path, so the same films bit for bit).  A 256 x 256 frame of 65 k triangles, one
 * sample, depth 4: five waves 440 us on the device, k_finish alone 235 (216 at 24 % of the issue slots, 6 of 32
 * lanes and 7 warps an SM: a chain of dependent loads); 1283 x 721: 1.04 -> 0.87 ms. */
constexpr int kFinishBlocks = 5; /* 96 registers; 4, 6 and 8 blocks per SM measured within 2 % */

template <int WIDTH, class JS, bool ADJ>
__global__ void __launch_bounds__(128, kFinishBlocks)
    k_finish(Queue q, AdjQueue a, WaveCounters *wcp, uint32_t wave, uint32_t lanes, float4 *L, float *g_alb,
             float *g_rough, const __grid_constant__ JS js) {
  const unsigned full = 0xffffffffu;
  const uint32_t n = wave_rays(*wcp, wave_at(wcp, wave));
  unsigned most = 0, sum = 0;
  const uint32_t lane = threadIdx.x & 31u, first = (blockIdx.x * blockDim.x + threadIdx.x) / 32u * lanes;
  if (first >= n) return;
  {
    const uint32_t i = first + lane;
    bool alive = lane < lanes && i < n;
    float4 o4{}, d4{}, b4{}, rem4{}, l4{};
    if (alive) {
      o4 = q.o[i], d4 = q.d[i], b4 = q.beta[i];
      if constexpr (ADJ) rem4 = a.rem[i], l4 = a.dl[i];
    }
    for (unsigned seg = 1; __any_sync(full, alive); seg++) {
      float4 h{};
      uint32_t inst = 0;
      AdjTerms g{};
      if (alive) {
        const DevScene &sc = js.at(__float_as_uint(d4.w) >> 8).sc;
        const TraceResult r = walk<WIDTH>(sc, V3{o4.x, o4.y, o4.z}, V3{d4.x, d4.y, d4.z});
        h = make_float4(r.t, r.u, r.v, __int_as_float(r.prim));
        inst = r.inst;
        most = max(most, seg);
        sum++;
      }
      __syncwarp();
      if (alive) {
        const DevScene &sc = js.at(__float_as_uint(d4.w) >> 8).sc;
        if (__float_as_int(h.w) < 0) {
          alive = false;
          if constexpr (!ADJ) {
            const V4 e = env_sample(sc, V3{d4.x, d4.y, d4.z});
            finish_path(sc, L, __float_as_uint(o4.w),
                        finite_or_zero(V3{b4.x, b4.y, b4.z} * V3{e.x, e.y, e.z},
                                       (float)(__float_as_uint(d4.w) & 0xffu) + e.w, &wcp->nonfinite),
                        &wcp->nonfinite);
          }
        } else if constexpr (ADJ) {
          alive = shade_adj_path(o4, d4, b4, rem4, l4, h, inst, wcp, js, g);
        } else {
          alive = shade_path<JS, false>(o4, d4, b4, h, inst, wcp, L, js);
        }
      }
      if constexpr (ADJ) {
        __syncwarp();
        add_terms(g, g_alb, g_rough);
      }
    }
  }
  for (int off = 16; off > 0; off >>= 1) {
    sum += __shfl_xor_sync(full, sum, off);
    most = max(most, __shfl_xor_sync(full, most, off));
  }
  if ((threadIdx.x & 31u) == 0 && sum) {
    atomicAdd(&wcp->traced, (unsigned long long)sum);
    atomicMax(&wcp->finish_waves, most);
  }
}

}  // namespace
