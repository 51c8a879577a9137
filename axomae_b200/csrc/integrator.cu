/* Wavefront path tracer: the reference's PathIntegrator::Li (integrator/Integrator.cpp:60-99) as
 * sm_100a kernels over a path queue in HBM, for one frame or a batch of frames of different scenes.
 *
 *   k_refill   (first waves of frames that start small; others make their camera rays in k_trace) fills
 *              free queue slots with camera rays of new paths (Integrator.h:66-85 with the
 *              OptiX raygen's sample index (x * H + y) * spp + s, integrator_optix.cu:43; Sobol
 *              dimensions 0 and 1 jitter NDC)
 *   k_trace    closest hit per queued ray (traverse.cuh); a miss finishes its path with the
 *              environment lookup, hits go to a compact hit list
 *   k_shade    per hit: principled scatter (Sobol dimensions 2 + 4b .. 5 + 4b at bounce b),
 *              throughput update, spawned ray appended to the next queue with warp-aggregated
 *              atomics; after the last allowed scatter the spawned direction looks up the
 *              environment directly (the reference traces that ray but discards the hit,
 *              Integrator.cpp:94-98)
 *   k_finish   once every path has started and few are left: the rest of each path in one thread
 *   k_resolve  per pixel, adds the per-path radiance of the call's samples to the running sum in
 *              sample order and writes sum / samples (writeFramebuffer, api/engine.cpp:351-363)
 *
 * The steps of a path are in wavefront.cuh; the adjoint's waves (wave_adjoint.cu) and trace modes 1 to 3
 * (wave_modes.cu) are modules of their own.
 *
 * Jobs: every path carries its job index (a frame of one context: scene, BVH, camera, sample
 * range) and every kernel reads the chunk's job table, so a batch of frames of different scenes
 * runs as one wavefront.  A single render is a batch of one.  The table travels in the kernel
 * parameter space (__grid_constant__, read through the constant cache): one Job for a single
 * frame, up to kParamJobs for a batch chunk.  The per-path arithmetic does not depend on the batch,
 * and each pixel's samples are added in sample order, so a frame rendered in a batch equals the
 * same frame rendered alone, bit for bit.
 *
 * Wave loop: the counters (waiting rays, next path, hits) live on the device in a ring of wave entries
 * and the kernels read their counts there, so a wave is enqueued while the one before it runs: the host
 * reads a finished wave's counters (pinned memory, event-synchronised), which bound the rays of the
 * waves after it, and sizes the next launches by them.  The job table is a kernel parameter, so a chunk
 * needs no set-up: 32 KB of it cost a launch less than a graph of four waves per chunk did to capture.
 *
 * The recursive estimator e_0 + c_0 (e_1 + c_1 (... env)) is evaluated forward as
 * sum_k beta_k e_k + beta_K env with beta_k = c_0 ... c_{k-1}; a path whose result is not finite
 * contributes 0 (DENAN, Integrator.cpp:92).  Path state: origin + radiance slot, direction + bounce +
 * job, throughput + Sobol sample index (3 x 16 B); hits 16 B + 4 B slot; per-path radiance 16 B,
 * written once.
 */
#include <algorithm>
#include <cfloat>
#include <condition_variable>
#include <cstring>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>
#include "caller_memory.cuh"
#include "context.cuh"
#include "wavefront.cuh"

namespace {

constexpr uint32_t kQueueCapDefault = 1u << 23; /* rays per wave unless tuned */
/* Radiance buffer: up to kRadianceCapBytes of a call's paths; a call with more goes in chunks.  A batch's chunks
 * are as long as the buffer: each drains by itself (32 frames, 485 M paths: 245 ms a step in chunks of 4 GiB,
 * 251 in 544 MiB).  A single frame's are kFrameChunkBytes, which costs it 7 % (2^31 paths: 286 ms in 4 GiB, 300 in
 * 768 MiB, 305 in 576 MiB, 309 in 512), and for one reason only: test_cancel_stops_a_long_render cancels a frame of
 * 2^31 paths 0.3 s after its start and needs it to be still running.  306 ms is what such a frame took before the
 * waves were made shorter. */
constexpr size_t kRadianceCapBytes = 4ull << 30, kFrameChunkBytes = 576ull << 20;

constexpr uint32_t kTileW = 8, kTileH = 4; /* default pixel tile: one warp of camera rays per tile */

/* Tiles of a tuning: 0 x 0 = the default tile, 1 x 1 = image rows (tile_w = 0 below). */
void set_tiles(RenderParams &rp, const nova_b200_tuning &tu) {
  if (tu.tile_w == 0) {
    rp.tile_w = kTileW;
    rp.tile_h = kTileH;
  } else if (tu.tile_w == 1 && tu.tile_h == 1) {
    rp.tile_w = rp.tile_h = 0u;
  } else {
    rp.tile_w = tu.tile_w;
    rp.tile_h = tu.tile_h;
  }
}

template <class JS>
__global__ void __launch_bounds__(256) k_refill(Queue q, WaveCounters *wcp, uint32_t wave, uint32_t total,
                                                uint32_t cap, float4 *L, const __grid_constant__ JS js) {
  const WaveState ws = first_state(wcp, wave, total, cap);
  const uint32_t n_new = min(cap - ws.n_active, total - ws.next);
  float4 o, d;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_new; i += gridDim.x * blockDim.x)
    refill_one(q, ws.next, ws.n_active, L, js, i, o, d);
}

/* What k_refill does to the counters before a first wave that starts its own paths. */
__global__ void k_start(WaveCounters *wcp, uint32_t total, uint32_t cap) { first_state(wcp, 0, total, cap); }

/* Resident blocks of 128 per SM that k_shade is compiled for.  With hits of one lobe family per
 * warp, 8 blocks (64 registers) are best on 32 frames: 79.5 ms per step, against 79.9 at 9, 80.7 at 10
 * (48 registers, more spills) and 81.4 at 12; 8 also suits the heightfield (11.7 against 12.1). */
#ifndef NB_SHADE_MIN_BLOCKS
#define NB_SHADE_MIN_BLOCKS 8
#endif

template <class JS>
__global__ void __launch_bounds__(128, NB_SHADE_MIN_BLOCKS)
    k_shade(Queue in, Queue out, WaveCounters *wcp, uint32_t wave, const float4 *hits, const uint2 *hit_slot, float4 *L,
            const __grid_constant__ JS js) {
  const WaveState &ws = wave_at(wcp, wave);
  const uint32_t nf = ws.hit_count, n = nf + ws.hit_back, cap = wcp->cap;
  unsigned *out_count = &wave_at(wcp, wave + 1).n_active;
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t == 0) clear_wave(wcp, wave);
  if ((t & ~31u) >= n) return;
  shade_warp<JS, false>(in, out, wcp, out_count, hits, hit_slot, L, js, hit_index(t, nf, cap), t < n);
}

/* Adds the chunk's samples of each pixel to its running sum (from zero when `clear`) and writes the mean;
 * nothing once the device status word holds a bad index (the call fails). */
__global__ void k_resolve(const float4 *L, uint32_t NP, uint32_t count, float4 *acc, bool clear, float denom, float *out,
                          int W, int H, int vinv, const WaveCounters *wcp, WaveCounters *back) {
  const uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix == 0 && back) *back = *wcp; /* pinned host memory: read after the stream has been waited for */
  if (pix >= NP || wcp->bad_index) return;
  float4 a = clear ? make_float4(0.f, 0.f, 0.f, 0.f) : acc[pix];
  for (uint32_t s = 0; s < count; s++) {
    const float4 l = L[(size_t)s * NP + pix];
    a.x += l.x, a.y += l.y, a.z += l.z, a.w += l.w;
  }
  acc[pix] = a;
  const uint32_t y = pix / (uint32_t)W, x = pix - y * (uint32_t)W;
  const uint32_t row = vinv ? (uint32_t)H - 1u - y : y;
  reinterpret_cast<float4 *>(out)[(size_t)row * W + x] = make_float4(a.x / denom, a.y / denom, a.z / denom, a.w / denom);
}

/* Resident blocks of 128 threads per SM of the intersector by itself: as in a wave, but for the 8-wide walk,
 * whose spills at 10 blocks cost more here (1 M incoherent rays on 65 k triangles: 297 us at 10, 294 at 9,
 * 265 at 8, 268 at 7; 274 with the three walks in one kernel). */
template <int WIDTH>
constexpr int kTraceApiBlocks = WIDTH == 8 ? 8 : kTraceBlocks<WIDTH>;

/* One kernel per BVH width: with the three walks in one kernel the registers were the largest walk's. */
template <int WIDTH>
__global__ void __launch_bounds__(128, kTraceApiBlocks<WIDTH>)
    k_trace_api(DevScene sc, uint64_t n, const float *o, const float *d, int32_t *prim, float *t, float *u, float *v) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const TraceResult r =
      trace_closest_w<WIDTH>(sc, V3{o[3 * i], o[3 * i + 1], o[3 * i + 2]}, V3{d[3 * i], d[3 * i + 1], d[3 * i + 2]});
  prim[i] = r.prim;
  t[i] = r.t;
  u[i] = r.u;
  v[i] = r.v;
}

/* One shading event per given hit: the hit record, the principled scatter with Sobol dimensions
 * 2 + 4 * bounce .. 5 + 4 * bounce, and the spawned ray (the body of k_shade for one path). */
__global__ void k_scatter_api(DevScene sc, uint64_t n, const float *o, const float *d, const int32_t *prim,
                              const float *t, const float *u, const float *v, const uint32_t *index,
                              const int32_t *bounce, uint32_t seed, float *out_o, float *out_d, float *weight,
                              float *emissive, int32_t *valid) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t p = prim[i];
  if (p < 0 || (uint64_t)p >= sc.n_prims || bounce[i] < 0 || bounce[i] > kMaxDepth) {
    valid[i] = -1;
    return;
  }
  const V3 ro{o[3 * i], o[3 * i + 1], o[3 * i + 2]}, rd{d[3 * i], d[3 * i + 1], d[3 * i + 2]};
  const DevInstance &I = sc.instances[__ldg(sc.prim_inst + p)];
  const HitRecord hr = make_record(sc, ro, rd, I, (uint32_t)p - I.prim_offset, t[i], u[i], v[i]);
  const ScatterResult sr =
      scatter(sc, rd, hr, sc.materials[I.material], index[i], 2u + 4u * (unsigned)bounce[i], seed, (uint32_t)p,
              I.material);
  const float eps = 1e-3f;
  const V3 nd3 = normalize(sr.wi);
  const V3 no3 = hr.position + hr.ng * (eps + eps * fsign(dot(hr.ng, sr.wi)));
  for (int k = 0; k < 3; k++) {
    out_o[3 * i + k] = k == 0 ? no3.x : k == 1 ? no3.y : no3.z;
    out_d[3 * i + k] = k == 0 ? nd3.x : k == 1 ? nd3.y : nd3.z;
    weight[3 * i + k] = k == 0 ? sr.weight.x : k == 1 ? sr.weight.y : sr.weight.z;
    emissive[3 * i + k] = k == 0 ? sr.emissive.x : k == 1 ? sr.emissive.y : sr.emissive.z;
  }
  valid[i] = sr.valid ? 1 : 0;
}

__global__ void k_sobol_api(const uint32_t *dv, uint64_t n, const uint32_t *idx, const uint32_t *dim, uint32_t seed,
                            float *out) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t dm = dim[i];
  out[i] = dm < (uint32_t)kSobolDims ? sobol_sample(dv, idx[i], dm, seed) : __int_as_float(0x7fc00000);
}

/* ------------------------------------------------------------------ host side */

nova_b200_status ensure_film(nova_b200_ctx *c, int W, int H) {
  const size_t npx = (size_t)W * H;
  if (c->film_w != W || c->film_h != H || !c->d_film_acc) {
    cudaFree(c->d_film_acc);
    c->d_film_acc = nullptr;
    NB_CUDA(c, cudaMalloc(&c->d_film_acc, npx * sizeof(float4)), "cudaMalloc(film)");
    c->film_clear = true;
    c->film_w = W;
    c->film_h = H;
    c->film_samples = 0;
  }
  if (c->film_out_cap < npx * 4) {
    cudaFree(c->d_film_out);
    c->d_film_out = nullptr;
    NB_CUDA(c, cudaMalloc(&c->d_film_out, npx * 4 * sizeof(float)), "cudaMalloc(film out)");
    c->film_out_cap = npx * 4;
  }
  return NOVA_B200_SUCCESS;
}

nova_b200_status ensure_wave_buffers(nova_b200_ctx *c, uint32_t cap, size_t radiance) {
  if (c->queue_cap < cap) {
    cudaFree(c->d_queue);
    c->d_queue = nullptr;
    c->queue_cap = 0;
    c->queue_bytes = 0;
    const size_t bytes = (size_t)cap * (16 * 7 + 8);
    NB_CUDA(c, cudaMalloc(&c->d_queue, bytes), "cudaMalloc(queue)");
    c->queue_cap = cap;
    c->queue_bytes = bytes;
  }
  if (c->radiance_cap < radiance) {
    cudaFree(c->d_radiance);
    c->d_radiance = nullptr;
    c->radiance_cap = 0;
    NB_CUDA(c, cudaMalloc(&c->d_radiance, radiance * sizeof(float4)), "cudaMalloc(radiance)");
    c->radiance_cap = radiance;
  }
  if (!c->d_wave) {
    NB_CUDA(c, cudaMalloc(&c->d_wave, sizeof(WaveCounters)), "cudaMalloc(wave counters)");
    NB_CUDA(c, cudaMallocHost(&c->h_wave, 3 * sizeof(WaveCounters)), "cudaMallocHost(wave counters)");
    for (cudaEvent_t &e : c->ev_wave) NB_CUDA(c, cudaEventCreate(&e), "cudaEventCreate");
    for (cudaEvent_t &e : c->ev_done)
      NB_CUDA(c, cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "cudaEventCreate");
  }
  return NOVA_B200_SUCCESS;
}

/* Rays up to which a wavefront with no path left to start goes to k_finish: about two rays for each of
 * its 95,000 resident threads, above which a wave is bound by its rays and no longer by its longest walk.
 * Fewer leave waves to their latency (75,000: a 256 x 256 x 16 adjoint step 1.53 ms against 1.44), more
 * give up the waves' full warps (600,000: 1000 instances at 720p 5.6 ms against 4.5; 300,000: 4.7). */
constexpr uint32_t kFinishRays = 150000;

/* Enqueues one wave for pipeline slot wave & 1 (queues alternating A -> B -> A ...): an event record
 * around the trace and the shading kernel (k_finish counts as the trace), the read-back of the counters
 * into the slot's pinned copy and the slot's completion event. */
template <class JS, int WIDTH>
cudaError_t enqueue_wave(nova_b200_ctx *c, const JS &js, const LaunchShape &ls, const WavePlan &p, uint64_t &kernels) {
  const WaveBuffers b = wave_buffers(c);
  const int slot = (int)(p.wave & 1u);
  const Queue &in = input_queue(b, p.wave), &out = output_queue(b, p.wave);
  cudaEvent_t *ev = c->ev_wave + 3 * slot;
  const bool fused = p.fresh && !p.finish && ls.trace_mode == 0;
  if (fused) {
    if (p.wave == 0) { /* the trace pass makes the camera rays; something has to start its counters */
      k_start<<<1, 1, 0, c->stream>>>(b.wc, p.total, p.cap);
      kernels++;
    }
  } else if (p.fresh) {
    k_refill<JS>
        <<<blocks_for(p.fresh, 256), 256, 0, c->stream>>>(in, b.wc, p.wave, p.total, p.cap, c->d_radiance, js);
    kernels++;
  }
  cudaEventRecord(ev[0], c->stream);
  if (p.finish) {
    const uint32_t lanes = finish_lanes(p.rays, p.wave);
    k_finish<WIDTH, JS, false><<<blocks_for(p.rays, 4u * lanes), 128, 0, c->stream>>>(
        in, AdjQueue{}, b.wc, p.wave, lanes, c->d_radiance, nullptr, nullptr, js);
    kernels++;
    cudaEventRecord(ev[1], c->stream);
    return cudaGetLastError(); /* what follows the last wave brings the counters back */
  }
  const unsigned g_trace = blocks_for(p.rays, ls.trace_block);
  const unsigned g_shade = blocks_for(p.rays, ls.shade_block);
  if (ls.trace_mode == 2 || (ls.trace_mode == 1 && WIDTH == 2))
    launch_mode_trace(c, js, ls, WIDTH, p);
  else if (fused)
    k_trace<WIDTH, JS, false, false, true>
        <<<g_trace, ls.trace_block, 0, c->stream>>>(in, b.wc, p.wave, b.hits, b.hit_slot, c->d_radiance, js);
  else
    k_trace<WIDTH, JS>
        <<<g_trace, ls.trace_block, 0, c->stream>>>(in, b.wc, p.wave, b.hits, b.hit_slot, c->d_radiance, js);
  cudaEventRecord(ev[1], c->stream);
  k_shade<JS><<<g_shade, ls.shade_block, 0, c->stream>>>(in, out, b.wc, p.wave, b.hits, b.hit_slot, c->d_radiance, js);
  kernels += 2;
  cudaEventRecord(ev[2], c->stream);
  cudaMemcpyAsync(static_cast<WaveCounters *>(c->h_wave) + slot, b.wc, sizeof(WaveCounters), cudaMemcpyDeviceToHost,
                  c->stream);
  cudaEventRecord(c->ev_done[slot], c->stream);
  return cudaGetLastError();
}

/* The wave launcher of a job table: run_waves' `launch`. */
template <class JS>
auto wave_launcher(nova_b200_ctx *c, const JS &js, const LaunchShape &ls, int width) {
  return [=, &js, &ls](const WavePlan &p, uint64_t &kernels) {
    if (width == 8) return enqueue_wave<JS, 8>(c, js, ls, p, kernels);
    if (width == 1) return enqueue_wave<JS, 1>(c, js, ls, p, kernels);
    return enqueue_wave<JS, 2>(c, js, ls, p, kernels);
  };
}

/* Runs the device-driven wave loop over `total` paths: uploads the counters, keeps two waves in flight
 * (launch(plan, kernels) enqueues one), reads each finished wave's counters and event times, and stops
 * once every path has ended.  A wave is enqueued while the one before it runs, so its plan holds upper
 * bounds: the rays of that wave and the paths not yet started.  Once no path is left to start and at
 * most `finish_rays` rays are, the plan is k_finish's and the last.  after_last() enqueues what follows the
 * last wave, and behind k_finish copies the counters to the slot it is given, so that one wait of the host
 * covers both. */
template <class Launch, class Last>
nova_b200_status run_waves(nova_b200_ctx *x, uint32_t total, uint32_t cap, uint32_t finish_rays, Launch &&launch,
                           Last &&after_last, LoopStats &ls) {
  WaveCounters *hw = static_cast<WaveCounters *>(x->h_wave); /* pinned read-back slots */
  /* bounds on the next wave to enqueue: its waiting rays, and the paths started before it (exact) */
  uint32_t waiting = 0, started = 0, enqueued = 0, finished = 0;
  bool finish = false;
  for (;;) {
    while (!finish && enqueued < finished + 2) {
      WavePlan p{enqueued, 0, 0, total, cap, false};
      p.rays = (uint32_t)std::min<uint64_t>(cap, (uint64_t)waiting + (total - started));
      if (p.rays == 0) break;
      p.fresh = std::min(cap, total - started);
      p.finish = finish = p.rays <= finish_rays && total - started <= cap - waiting;
      NB_CUDA(x, launch(p, ls.kernels), "wave");
      enqueued++;
      if (finish) after_last(hw + (p.wave & 1u));
      /* at least cap - waiting of them start in this wave; how many exactly is read back */
      started += std::min(cap - waiting, total - started);
      waiting = p.rays;
    }
    const int slot = (int)(finished & 1u);
    const bool last = finish && finished + 1 == enqueued; /* k_finish: with all that is enqueued behind it */
    NB_CUDA(x, last ? cudaStreamSynchronize(x->stream) : cudaEventSynchronize(x->ev_done[slot]), "waves");
    const cudaEvent_t *ev = x->ev_wave + 3 * slot;
    float a = 0.f, b = 0.f;
    cudaEventElapsedTime(&a, ev[0], ev[1]);
    if (!last) cudaEventElapsedTime(&b, ev[1], ev[2]);
    ls.t_trace += a;
    ls.t_shade += b;
    const WaveCounters r = hw[slot];
    finished++;
    auto drain = [&] { /* the wave still in flight; its counters */
      if (enqueued == finished) return cudaSuccess;
      return finish ? cudaStreamSynchronize(x->stream) : cudaEventSynchronize(x->ev_done[finished & 1u]);
    };
    if (r.bad_index) { /* the device status word: stop after this wave, as the reference aborts a tile
                        * once its exception manager holds an error (integrator/Integrator.h:74-78) */
      NB_CUDA(x, drain(), "waves");
      const WaveCounters last = enqueued == finished ? r : hw[slot ^ 1];
      ls.bad_index += std::max(r.bad_index, last.bad_index);
      ls.nonfinite += std::max(r.nonfinite, last.nonfinite);
      char msg[160];
      std::snprintf(msg, sizeof(msg), "device status: %u hits with an out-of-range primitive, instance or material id",
                    (unsigned)std::max(r.bad_index, last.bad_index));
      return nbctx::fail(x, NOVA_B200_RENDERER_EXCEPTION, "%s", msg);
    }
    const WaveState &next = r.w[finished % kWaveRing];
    const bool done = finish ? finished == enqueued : next.n_active == 0 && next.next == total;
    if (done) {
      ls.waves += r.waves + r.finish_waves;
      ls.traced += r.traced;
      ls.nonfinite += r.nonfinite;
      ls.node_visits += r.node_visits;
      ls.tri_tests += r.tri_tests;
      if (!finish) after_last(nullptr);
      return NOVA_B200_SUCCESS;
    }
    if (!finish && x->cancel.load()) { /* nova_b200_cancel: let the wave in flight finish, enqueue nothing
                                        * more (a render whose last wave is enqueued completes) */
      NB_CUDA(x, drain(), "waves");
      return nbctx::fail(x, NOVA_B200_RENDERER_EXCEPTION, "render cancelled%s");
    }
    /* the counts before wave `finished` are known now; a wave already enqueued after it starts what its
     * queue has room for and leaves at most its rays */
    waiting = next.n_active;
    started = next.next;
    for (uint32_t w = finished; w < enqueued; w++) {
      const uint32_t fresh = std::min(cap - waiting, total - started);
      started += fresh;
      waiting += fresh;
    }
  }
}

struct Piece {
  nova_b200_ctx *ctx; /* the job's context: scene, BVH, film */
  const nova_b200_frame *f;
  uint32_t begin, count;
};

/* The frame's own fields (the scene and BVH are checked by validate_frame). */
nova_b200_status validate_frame_fields(nova_b200_ctx *c, const nova_b200_frame *f) {
  using namespace nbctx;
  if (!f) return fail(c, NOVA_B200_INVALID_ARGUMENT, "frame is null%s");
  if (f->width <= 0 || f->height <= 0 || f->spp_total <= 0 || f->sample_begin < 0 || f->sample_count <= 0 ||
      f->sample_begin + f->sample_count > f->spp_total)
    return fail(c, NOVA_B200_INVALID_ARGUMENT, "invalid frame size or sample range%s");
  if (f->max_depth < 0 || f->max_depth > kMaxDepth)
    return fail(c, NOVA_B200_INVALID_ARGUMENT, "max_depth must be in 0..48 (Sobol dimensions)%s");
  if ((uint64_t)f->width * f->height * (uint64_t)f->spp_total >= (1ull << 32))
    return fail(c, NOVA_B200_INVALID_ARGUMENT, "width * height * spp must stay below 2^32 (Sobol index)%s");
  return NOVA_B200_SUCCESS;
}

nova_b200_status validate_frame(nova_b200_ctx *c, const nova_b200_frame *f) {
  using namespace nbctx;
  if (f && !c->bvh_ready) return fail(c, NOVA_B200_SCENE_NOT_PROCESSED, "build the acceleration structure first%s");
  return validate_frame_fields(c, f);
}

/* Pipelined batches: called before a chunk uses job j's scene; blocks until that context's upload
 * and build are done and returns their status. */
using WaitReady = std::function<nova_b200_status(size_t)>;

/* Renders frames (one per job) as one wavefront on the executing context `x`.  Jobs are cut into
 * chunks whose per-path radiance fits the radiance buffer; a job's samples stay in order. */
/* The order frames go into chunks: largest film first.  The films of the last chunk are copied
 * out after its waves end (those of earlier chunks while later ones render), so it holds the
 * smallest; a frame's film does not depend on the chunk it lands in. */
std::vector<uint32_t> chunk_order(const std::vector<const nova_b200_frame *> &frames) {
  std::vector<uint32_t> ord(frames.size());
  for (uint32_t j = 0; j < (uint32_t)ord.size(); j++) ord[j] = j;
  std::stable_sort(ord.begin(), ord.end(), [&](uint32_t a, uint32_t b) {
    return (uint64_t)frames[a]->width * frames[a]->height > (uint64_t)frames[b]->width * frames[b]->height;
  });
  return ord;
}

nova_b200_status render_jobs(nova_b200_ctx *x, const std::vector<nova_b200_ctx *> &ctxs,
                             const std::vector<const nova_b200_frame *> &frames, float *const *films_host,
                             float *const *films_device, nova_b200_render_stats *stats,
                             const WaitReady *wait_ready = nullptr, int pipelined_width = 0,
                             uint32_t first_chunk_jobs = kParamJobs) {
  using namespace nbctx;
  x->cancel.store(false); /* a cancel applies to the call in progress */
  if (x->h_cancel_map) *x->h_cancel_map = 0;
  const size_t nj = ctxs.size();
  const int width = wait_ready ? pipelined_width : ctxs[0]->bvh_width;
  uint64_t max_np = 0, total = 0;
  for (size_t j = 0; j < nj; j++) {
    if (ctxs[j]->device != x->device)
      return fail(x, NOVA_B200_INVALID_ARGUMENT, "all contexts of a batch must use the same device%s");
    if (!wait_ready && ctxs[j]->bvh_width != width)
      return fail(x, NOVA_B200_INVALID_ARGUMENT, "all scenes of a batch must use the same BVH width%s");
    const uint64_t np = (uint64_t)frames[j]->width * frames[j]->height;
    max_np = std::max(max_np, np);
    total += np * (uint64_t)frames[j]->sample_count;
  }
  const uint64_t most = (nj == 1 && total > kRadianceCapBytes / sizeof(float4) ? kFrameChunkBytes : kRadianceCapBytes) /
                        sizeof(float4);
  const uint64_t radiance = std::max<uint64_t>(max_np, std::min(total, most));
  const nova_b200_tuning &tu = x->tuning;
  const uint32_t qc = tu.queue_capacity ? tu.queue_capacity : kQueueCapDefault;
  const uint32_t cap = (uint32_t)std::min<uint64_t>(qc, std::max<uint64_t>(radiance, 1024));
  const LaunchShape ls{cap, tu.trace_block ? tu.trace_block : 128u, tu.shade_block ? tu.shade_block : 128u,
                       tu.trace_mode, tu.wait_limit_us ? tu.wait_limit_us : 1000000u, tu.trace_mode ? 0u : kFinishRays};
  nova_b200_status st = ensure_wave_buffers(x, cap, radiance);
  if (st != NOVA_B200_SUCCESS) return st;
  x->primal_valid = false; /* this render overwrites the radiance buffer */
  for (size_t j = 0; j < nj; j++) {
    nova_b200_ctx *c = ctxs[j];
    if ((st = ensure_film(c, frames[j]->width, frames[j]->height)) != NOVA_B200_SUCCESS) return st;
    if (frames[j]->reset) {
      c->film_clear = true; /* the next resolve starts from zero */
      c->film_samples = 0;
    }
  }
  /* scene uploads and film clears of other contexts ran on their own streams (pipelined: each
   * context's upload and build end with a synchronisation of its stream, and the chunk loop waits
   * for them) */
  if (!wait_ready)
    for (size_t j = 0; j < nj; j++)
      if (ctxs[j] != x) NB_CUDA(x, cudaStreamSynchronize(ctxs[j]->stream), "sync batch context");
  /* cut the work into chunks of at most `radiance` paths and kParamJobs frame pieces */
  std::vector<std::vector<Piece>> chunks(1);
  uint64_t in_chunk = 0;
  const std::vector<uint32_t> ord = chunk_order(frames);
  for (size_t q = 0; q < nj; q++) {
    const size_t j = ord[q];
    const nova_b200_frame *f = frames[j];
    const uint64_t np = (uint64_t)f->width * f->height;
    uint32_t s = 0;
    while (s < (uint32_t)f->sample_count) {
      uint64_t room = (radiance - in_chunk) / np;
      if (room == 0 || chunks.back().size() == (chunks.size() == 1 ? first_chunk_jobs : kParamJobs)) {
        chunks.emplace_back();
        in_chunk = 0;
        room = radiance / np;
      }
      const uint32_t take = (uint32_t)std::min<uint64_t>(room, (uint64_t)f->sample_count - s);
      chunks.back().push_back(Piece{ctxs[j], f, (uint32_t)f->sample_begin + s, take});
      in_chunk += np * take;
      s += take;
    }
  }
  /* A frame's film is final after its last chunk: with several chunks, device films and pinned host
   * films of finished frames are copied out on a second stream while later chunks render. */
  const size_t nc = chunks.size();
  std::vector<size_t> last_chunk(nj, 0);
  std::vector<char> early(nj, 0);
  for (size_t ci = 0; ci < nc; ci++)
    for (const Piece &P : chunks[ci])
      for (size_t j = 0; j < nj; j++)
        if (ctxs[j] == P.ctx) last_chunk[j] = ci;
  if (nc > 1) {
    for (size_t j = 0; j < nj; j++) {
      bool pinned = false;
      if (films_host && films_host[j]) {
        cudaPointerAttributes pa{};
        if (cudaPointerGetAttributes(&pa, films_host[j]) == cudaSuccess)
          pinned = pa.type == cudaMemoryTypeHost;
        else
          cudaGetLastError(); /* not a pointer the runtime knows: treated as pageable */
      }
      const bool host_ok = !(films_host && films_host[j]) || pinned;
      early[j] = host_ok && last_chunk[j] + 1 < nc ? 1 : 0;
    }
    if (!x->copy_stream) {
      NB_CUDA(x, cudaStreamCreateWithFlags(&x->copy_stream, cudaStreamNonBlocking), "film copy stream");
      NB_CUDA(x, cudaEventCreateWithFlags(&x->ev_copy, cudaEventDisableTiming), "film copy event");
    }
  }
  struct CopiesDone { /* every return waits for the film copies already issued */
    cudaStream_t s;
    ~CopiesDone() {
      if (s) cudaStreamSynchronize(s);
    }
  } copies_done{nc > 1 ? x->copy_stream : nullptr};
  /* where a frame's last resolve writes its film: the caller's device film itself where it may, which
   * saves a copy of it; earlier chunks of the frame write the context's, so that a render that fails
   * leaves the caller's alone */
  std::vector<Span> spans(nj, Span{0, 0, false});
  for (size_t j = 0; films_device && j < nj; j++) {
    cudaPointerAttributes at{};
    if (films_device[j] && cudaPointerGetAttributes(&at, films_device[j]) != cudaSuccess) cudaGetLastError();
    spans[j] = Span{reinterpret_cast<uintptr_t>(films_device[j]),
                    (size_t)frames[j]->width * frames[j]->height * 4 * sizeof(float), on_device(at, x->device)};
  }
  const std::vector<char> direct = direct_films(spans);
  auto film_target = [&](size_t j) { return direct[j] ? films_device[j] : ctxs[j]->d_film_out; };
  auto copy_film = [&](size_t j, cudaStream_t stream) -> nova_b200_status {
    const size_t bytes = (size_t)frames[j]->width * frames[j]->height * 4 * sizeof(float);
    const float *film = film_target(j);
    if (films_device && films_device[j] && films_device[j] != film)
      NB_CUDA(x, cudaMemcpyAsync(films_device[j], film, bytes, cudaMemcpyDeviceToDevice, stream), "copy film");
    if (films_host && films_host[j])
      NB_CUDA(x, cudaMemcpyAsync(films_host[j], film, bytes, cudaMemcpyDeviceToHost, stream), "copy film");
    return NOVA_B200_SUCCESS;
  };
  nova_b200_render_stats sum{};
  LoopStats loop;
  NB_CUDA(x, cudaEventRecord(x->ev_begin, x->stream), "event");
  std::vector<Job> hj(kParamJobs);
  ManyJobs many{};
  for (size_t ci = 0; ci < nc; ci++) {
    const auto &chunk = chunks[ci];
    if (x->cancel.load()) return fail(x, NOVA_B200_RENDERER_EXCEPTION, "render cancelled%s");
    if (chunk.empty()) continue;
    if (wait_ready)
      for (const Piece &P : chunk)
        for (size_t j = 0; j < nj; j++)
          if (ctxs[j] == P.ctx && (st = (*wait_ready)(j)) != NOVA_B200_SUCCESS) return st;
    uint32_t pb = 0;
    for (size_t k = 0; k < chunk.size(); k++) {
      const Piece &P = chunk[k];
      Job &J = hj[k];
      J = Job{};
      J.sc = P.ctx->scene;
      RenderParams &rp = J.rp;
      rp.W = P.f->width, rp.H = P.f->height, rp.NP = (uint32_t)((uint64_t)P.f->width * P.f->height);
      rp.count = P.count;
      rp.begin = P.begin;
      rp.spp_total = (uint32_t)P.f->spp_total;
      rp.max_depth = P.f->max_depth;
      rp.seed = P.f->seed;
      rp.rr_start = P.f->rr_start;
      std::copy(P.f->inv_P, P.f->inv_P + 16, rp.inv_P);
      std::copy(P.f->inv_V, P.f->inv_V + 16, rp.inv_V);
      rp.vinv = P.f->vertical_invert;
      set_tiles(rp, tu);
      J.path_begin = pb;
      J.n_paths = rp.NP * P.count;
      pb += J.n_paths;
    }
    const bool single = chunk.size() == 1;
    OneJob one{};
    if (single) {
      one.j = hj[0];
    } else {
      many = ManyJobs{};
      many.n = (uint32_t)chunk.size();
      std::copy(hj.begin(), hj.begin() + chunk.size(), many.j);
    }
    /* the chunk's samples into its films, enqueued behind its last wave */
    auto resolve = [&](WaveCounters *back) {
      for (size_t k = 0; k < chunk.size(); k++) {
        const Piece &P = chunk[k];
        nova_b200_ctx *c = P.ctx;
        const size_t j = (size_t)(std::find(ctxs.begin(), ctxs.end(), c) - ctxs.begin());
        c->film_samples += P.count;
        const uint32_t NP = hj[k].rp.NP;
        k_resolve<<<(NP + 255) / 256, 256, 0, x->stream>>>(
            x->d_radiance + hj[k].path_begin, NP, P.count, c->d_film_acc, c->film_clear, (float)c->film_samples,
            last_chunk[j] == ci ? film_target(j) : c->d_film_out, P.f->width, P.f->height, P.f->vertical_invert,
            static_cast<const WaveCounters *>(x->d_wave), k == 0 ? back : nullptr);
        c->film_clear = false;
        sum.kernels++;
      }
      if (ci + 1 == nc) cudaEventRecord(x->ev_end, x->stream);
    };
    if (ls.trace_mode == 3) { /* the persistent wavefront: one launch runs every wave of the chunk */
      st = single ? run_persistent(x, one, ls, width, pb, cap, loop) : run_persistent(x, many, ls, width, pb, cap, loop);
      if (st == NOVA_B200_SUCCESS) resolve(nullptr);
    } else {
      std::vector<std::pair<uint64_t, bool>> film_state; /* for a failure found after the resolves are enqueued */
      for (const Piece &P : chunk) film_state.emplace_back(P.ctx->film_samples, P.ctx->film_clear);
      st = single ? run_waves(x, pb, cap, ls.finish_rays, wave_launcher(x, one, ls, width), resolve, loop)
                  : run_waves(x, pb, cap, ls.finish_rays, wave_launcher(x, many, ls, width), resolve, loop);
      if (st != NOVA_B200_SUCCESS)
        for (size_t k = 0; k < chunk.size(); k++)
          chunk[k].ctx->film_samples = film_state[k].first, chunk[k].ctx->film_clear = film_state[k].second;
    }
    if (st != NOVA_B200_SUCCESS) return st;
    sum.paths += pb;
    bool any = false;
    for (size_t j = 0; j < nj; j++) any = any || (early[j] && last_chunk[j] == ci);
    if (any) {
      NB_CUDA(x, cudaEventRecord(x->ev_copy, x->stream), "event");
      NB_CUDA(x, cudaStreamWaitEvent(x->copy_stream, x->ev_copy, 0), "event");
      for (size_t j = 0; j < nj; j++)
        if (early[j] && last_chunk[j] == ci && (st = copy_film(j, x->copy_stream)) != NOVA_B200_SUCCESS) return st;
    }
  }
  NB_CUDA(x, cudaGetLastError(), "render kernels");
  for (size_t j = 0; j < nj; j++)
    if (!early[j] && (st = copy_film(j, x->stream)) != NOVA_B200_SUCCESS) return st;
  NB_CUDA(x, cudaStreamSynchronize(x->stream), "render");
  if (x->copy_stream) NB_CUDA(x, cudaStreamSynchronize(x->copy_stream), "film copies");
  if (nj == 1 && chunks.size() == 1 && chunks[0].size() == 1) {
    x->primal_valid = true;
    x->primal_frame = *frames[0];
    x->primal_albedo = x->scene.diff_albedo;
    x->primal_rough = x->scene.diff_rough;
  }
  float total_ms = 0.f;
  cudaEventElapsedTime(&total_ms, x->ev_begin, x->ev_end);
  loop.add_to(sum);
  sum.device_ms = total_ms;
  if (stats) *stats = sum;
  return NOVA_B200_SUCCESS;
}

}  // namespace

nova_b200_status nb_render(nova_b200_ctx *c, const nova_b200_frame *f, float *film_host, float *film_device,
                           nova_b200_render_stats *stats) {
  nova_b200_status st = validate_frame(c, f);
  if (st != NOVA_B200_SUCCESS) return st;
  cudaSetDevice(c->device);
  return render_jobs(c, {c}, {f}, &film_host, &film_device, stats);
}

/* Upload, build and render a batch in one pipelined call: up to 16 host threads upload and build
 * the contexts in batch order (each on its own stream), and the calling thread renders on ctxs[0],
 * starting each chunk as soon as the contexts of its frames are built, so the later scenes' copies
 * and builds overlap the first chunks' waves.  Same result as the three calls one after another. */
nova_b200_status nb_upload_build_render_batch(nova_b200_ctx *const *ctxs, const nova_b200_scene_desc *descs,
                                              const nova_b200_frame *frames, uint32_t n,
                                              const nova_b200_bvh_options *opts, float *const *films_host,
                                              float *const *films_device, nova_b200_render_stats *stats) {
  using namespace nbctx;
  if (!ctxs || !ctxs[0]) return NOVA_B200_INVALID_ARGUMENT;
  nova_b200_ctx *x = ctxs[0];
  if (!descs || !frames || n == 0) return fail(x, NOVA_B200_INVALID_ARGUMENT, "empty batch%s");
  const int width = opts && opts->width ? opts->width : 2;
  std::vector<nova_b200_ctx *> cs(n);
  std::vector<const nova_b200_frame *> fs(n);
  for (uint32_t j = 0; j < n; j++) {
    if (!ctxs[j]) return fail(x, NOVA_B200_INVALID_ARGUMENT, "null context in batch%s");
    if (ctxs[j]->device != x->device)
      return fail(x, NOVA_B200_INVALID_ARGUMENT, "all contexts of a batch must use the same device%s");
    nova_b200_status st = validate_frame_fields(ctxs[j], &frames[j]);
    if (st != NOVA_B200_SUCCESS) {
      x->error = ctxs[j]->error;
      return st;
    }
    for (uint32_t k = 0; k < j; k++)
      if (ctxs[k] == ctxs[j]) return fail(x, NOVA_B200_INVALID_ARGUMENT, "a context appears twice in a batch%s");
    cs[j] = ctxs[j];
    fs[j] = &frames[j];
  }
  constexpr int kPending = -1;
  std::mutex mu;
  std::condition_variable cv;
  std::vector<int> done(n, kPending);
  std::atomic<uint32_t> next{0};
  std::atomic<bool> stop{false};
  /* scenes are built in the order chunks render them, the executing context's own first (its stream
   * carries the render) */
  std::vector<uint32_t> ord = chunk_order(fs);
  std::rotate(ord.begin(), std::find(ord.begin(), ord.end(), 0u), std::find(ord.begin(), ord.end(), 0u) + 1);
  auto work = [&] {
    for (uint32_t q; (q = next.fetch_add(1)) < n;) {
      const uint32_t k = ord[q];
      nova_b200_status st = stop.load() ? NOVA_B200_RENDERER_EXCEPTION : nova_b200_upload_scene(cs[k], &descs[k]);
      if (st == NOVA_B200_SUCCESS) st = nova_b200_build_bvh(cs[k], opts);
      {
        std::lock_guard<std::mutex> lock(mu);
        done[k] = (int)st;
      }
      cv.notify_all();
    }
  };
  const unsigned nt = std::max(1u, std::min(std::min(n, 16u), std::max(1u, std::thread::hardware_concurrency())));
  std::vector<std::thread> pool;
  for (unsigned t = 0; t < nt; t++) pool.emplace_back(work);
  const WaitReady wait_ready = [&](size_t j) -> nova_b200_status {
    nova_b200_status st;
    {
      std::unique_lock<std::mutex> lock(mu);
      cv.wait(lock, [&] { return done[j] != kPending; });
      st = (nova_b200_status)done[j];
    }
    if (st != NOVA_B200_SUCCESS) {
      if (cs[j] != x) x->error = cs[j]->error;
      return st;
    }
    if (cs[j]->bvh_width != width)
      return fail(x, NOVA_B200_INVALID_ARGUMENT, "all scenes of a batch must use the same BVH width%s");
    return NOVA_B200_SUCCESS;
  };
  /* the executing context's own scene must be in place before its stream renders */
  nova_b200_status st = wait_ready(0);
  if (st == NOVA_B200_SUCCESS) {
    cudaSetDevice(x->device);
    /* the first chunk holds only the frames whose scenes the first round of threads builds, so its
     * waves start while the rest build */
    st = render_jobs(x, cs, fs, films_host, films_device, stats, &wait_ready, width, std::min<uint32_t>(nt, kParamJobs));
  }
  stop.store(st != NOVA_B200_SUCCESS); /* a failed render skips the uploads not started yet */
  for (auto &t : pool) t.join();
  if (st == NOVA_B200_SUCCESS)
    for (uint32_t k = 0; k < n; k++)
      if (done[k] != (int)NOVA_B200_SUCCESS) {
        if (k != 0) x->error = cs[k]->error;
        return (nova_b200_status)done[k];
      }
  return st;
}

nova_b200_status nb_render_batch(nova_b200_ctx *const *ctxs, const nova_b200_frame *frames, uint32_t n,
                                 float *const *films_host, float *const *films_device, nova_b200_render_stats *stats) {
  using namespace nbctx;
  if (!ctxs || !ctxs[0]) return NOVA_B200_INVALID_ARGUMENT;
  nova_b200_ctx *x = ctxs[0];
  if (!frames || n == 0) return fail(x, NOVA_B200_INVALID_ARGUMENT, "empty batch%s");
  std::vector<nova_b200_ctx *> cs(n);
  std::vector<const nova_b200_frame *> fs(n);
  for (uint32_t j = 0; j < n; j++) {
    if (!ctxs[j]) return fail(x, NOVA_B200_INVALID_ARGUMENT, "null context in batch%s");
    nova_b200_status st = validate_frame(ctxs[j], &frames[j]);
    if (st != NOVA_B200_SUCCESS) {
      x->error = ctxs[j]->error;
      return st;
    }
    for (uint32_t k = 0; k < j; k++)
      if (ctxs[k] == ctxs[j]) return fail(x, NOVA_B200_INVALID_ARGUMENT, "a context appears twice in a batch%s");
    cs[j] = ctxs[j];
    fs[j] = &frames[j];
  }
  cudaSetDevice(x->device);
  return render_jobs(x, cs, fs, films_host, films_device, stats);
}

/* The frame fields that decide every path of a render (reset and vertical_invert do not). */
bool same_paths(const nova_b200_frame &a, const nova_b200_frame &b) {
  return a.width == b.width && a.height == b.height && a.spp_total == b.spp_total &&
         a.sample_begin == b.sample_begin && a.sample_count == b.sample_count && a.max_depth == b.max_depth &&
         a.seed == b.seed && a.rr_start == b.rr_start && std::memcmp(a.inv_P, b.inv_P, sizeof(a.inv_P)) == 0 &&
         std::memcmp(a.inv_V, b.inv_V, sizeof(a.inv_V)) == 0;
}

nova_b200_status nb_backward(nova_b200_ctx *c, const nova_b200_frame *f, const float *d_image, float *grad_albedo,
                             float *grad_roughness, uint32_t flags, nova_b200_render_stats *stats) {
  using namespace nbctx;
  nova_b200_status st = validate_frame(c, f);
  if (st != NOVA_B200_SUCCESS) return st;
  if (!d_image) return fail(c, NOVA_B200_INVALID_ARGUMENT, "d_image is null%s");
  cudaSetDevice(c->device);
  const uint32_t NP = (uint32_t)((uint64_t)f->width * f->height);
  const uint64_t total = (uint64_t)NP * (uint64_t)f->sample_count;
  const uint64_t radiance = std::max<uint64_t>(NP, std::min<uint64_t>(total, kRadianceCapBytes / sizeof(float4)));
  const nova_b200_tuning &tu = c->tuning;
  const uint32_t qc = tu.queue_capacity ? tu.queue_capacity : kQueueCapDefault;
  const uint32_t cap = (uint32_t)std::min<uint64_t>(qc, std::max<uint64_t>(radiance, 1024));
  const LaunchShape ls{cap, tu.trace_block ? tu.trace_block : 128u, tu.shade_block ? tu.shade_block : 128u,
                       tu.trace_mode == 3 ? 0u : tu.trace_mode, 0u, /* the replay keeps the per-wave kernels */
                       tu.trace_mode == 1 || tu.trace_mode == 2 ? 0u : kFinishRays};
  if ((st = ensure_wave_buffers(c, cap, radiance)) != NOVA_B200_SUCCESS) return st;
  if (c->adj_cap < c->queue_cap) {
    cudaFree(c->d_adj);
    c->d_adj = nullptr;
    c->adj_cap = 0;
    NB_CUDA(c, cudaMalloc(&c->d_adj, sizeof(float4) * 4 * (size_t)c->queue_cap), "cudaMalloc(adjoint queues)");
    c->adj_cap = c->queue_cap;
  }
  AdjArgs adj;
  const size_t qcap = c->adj_cap;
  adj.qa = AdjQueue{c->d_adj, c->d_adj + qcap};
  adj.qb = AdjQueue{c->d_adj + 2 * qcap, c->d_adj + 3 * qcap};
  adj.d_image = reinterpret_cast<const float4 *>(d_image);
  adj.g_alb = grad_albedo;
  adj.g_rough = grad_roughness;
  const int width = c->bvh_width;
  nova_b200_render_stats sum{};
  LoopStats primal, replay;
  NB_CUDA(c, cudaEventRecord(c->ev_begin, c->stream), "event");
  const uint32_t per_chunk = (uint32_t)std::max<uint64_t>(1, radiance / NP);
  const bool reuse = (flags & NOVA_B200_BACKWARD_REUSE_PRIMAL) && c->primal_valid &&
                     per_chunk >= (uint32_t)f->sample_count && same_paths(c->primal_frame, *f) &&
                     c->primal_albedo == c->scene.diff_albedo && c->primal_rough == c->scene.diff_rough;
  if (!reuse) c->primal_valid = false; /* the radiance pass below overwrites the buffer (and may stop midway) */
  c->cancel.store(false);              /* a cancel applies to the call in progress */
  for (uint32_t s0 = 0; s0 < (uint32_t)f->sample_count; s0 += per_chunk) {
    const uint32_t take = std::min<uint32_t>(per_chunk, (uint32_t)f->sample_count - s0);
    OneJob one{};
    Job &J = one.j;
    J.sc = c->scene;
    RenderParams &rp = J.rp;
    rp.W = f->width, rp.H = f->height, rp.NP = NP;
    rp.count = (uint32_t)f->sample_count; /* the image averages all of the frame's samples */
    rp.begin = (uint32_t)f->sample_begin + s0;
    rp.spp_total = (uint32_t)f->spp_total;
    rp.max_depth = f->max_depth;
    rp.seed = f->seed;
    rp.rr_start = f->rr_start;
    std::copy(f->inv_P, f->inv_P + 16, rp.inv_P);
    std::copy(f->inv_V, f->inv_V + 16, rp.inv_V);
    rp.vinv = f->vertical_invert;
    set_tiles(rp, tu);
    J.path_begin = 0;
    J.n_paths = NP * take;
    /* primal: each path's radiance into the radiance buffer */
    auto read_back = [&](WaveCounters *back) {
      if (back) cudaMemcpyAsync(back, c->d_wave, sizeof(WaveCounters), cudaMemcpyDeviceToHost, c->stream);
    };
    if (!reuse &&
        (st = run_waves(c, J.n_paths, cap, ls.finish_rays, wave_launcher(c, one, ls, width), read_back, primal)) != NOVA_B200_SUCCESS)
      return st;
    /* replay with the adjoint */
    const auto replay_wave = [&](const WavePlan &p, uint64_t &kernels) {
      return enqueue_adjoint_wave(c, one, ls, width, p, kernels, adj);
    };
    if ((st = run_waves(c, J.n_paths, cap, ls.finish_rays, replay_wave, read_back, replay)) != NOVA_B200_SUCCESS)
      return st;
    sum.paths += J.n_paths;
  }
  NB_CUDA(c, cudaEventRecord(c->ev_end, c->stream), "event");
  NB_CUDA(c, cudaStreamSynchronize(c->stream), "backward");
  float total_ms = 0.f;
  cudaEventElapsedTime(&total_ms, c->ev_begin, c->ev_end);
  primal.add_to(sum);
  replay.add_to(sum);
  sum.device_ms = total_ms;
  if (stats) *stats = sum;
  /* a one-pass backward leaves this frame's radiance in the buffer */
  c->primal_valid = per_chunk >= (uint32_t)f->sample_count;
  c->primal_frame = *f;
  c->primal_albedo = c->scene.diff_albedo;
  c->primal_rough = c->scene.diff_rough;
  return NOVA_B200_SUCCESS;
}

nova_b200_status nb_trace(nova_b200_ctx *c, uint64_t n, const float *o, const float *d, int32_t *prim, float *t,
                          float *u, float *v) {
  using namespace nbctx;
  if (!c->bvh_ready) return fail(c, NOVA_B200_SCENE_NOT_PROCESSED, "build the acceleration structure first%s");
  if (n == 0) return NOVA_B200_SUCCESS;
  if (!o || !d || !prim || !t || !u || !v) return fail(c, NOVA_B200_INVALID_ARGUMENT, "null buffer%s");
  cudaSetDevice(c->device);
  const unsigned grid = (unsigned)((n + 127) / 128);
  if (c->scene.width == 8)
    k_trace_api<8><<<grid, 128, 0, c->stream>>>(c->scene, n, o, d, prim, t, u, v);
  else if (c->scene.width == 1)
    k_trace_api<1><<<grid, 128, 0, c->stream>>>(c->scene, n, o, d, prim, t, u, v);
  else
    k_trace_api<2><<<grid, 128, 0, c->stream>>>(c->scene, n, o, d, prim, t, u, v);
  NB_CUDA(c, cudaGetLastError(), "k_trace_api");
  NB_CUDA(c, cudaStreamSynchronize(c->stream), "trace");
  return NOVA_B200_SUCCESS;
}

nova_b200_status nb_scatter(nova_b200_ctx *c, uint64_t n, const float *o, const float *d, const int32_t *prim,
                            const float *t, const float *u, const float *v, const uint32_t *index,
                            const int32_t *bounce, uint32_t seed, float *out_o, float *out_d, float *weight,
                            float *emissive, int32_t *valid) {
  using namespace nbctx;
  if (!c->bvh_ready) return fail(c, NOVA_B200_SCENE_NOT_PROCESSED, "build the acceleration structure first%s");
  if (n == 0) return NOVA_B200_SUCCESS;
  if (!o || !d || !prim || !t || !u || !v || !index || !bounce || !out_o || !out_d || !weight || !emissive || !valid)
    return fail(c, NOVA_B200_INVALID_ARGUMENT, "null buffer%s");
  cudaSetDevice(c->device);
  k_scatter_api<<<(unsigned)((n + 127) / 128), 128, 0, c->stream>>>(c->scene, n, o, d, prim, t, u, v, index, bounce,
                                                                     seed, out_o, out_d, weight, emissive, valid);
  NB_CUDA(c, cudaGetLastError(), "k_scatter_api");
  NB_CUDA(c, cudaStreamSynchronize(c->stream), "scatter");
  return NOVA_B200_SUCCESS;
}

nova_b200_status nb_sobol(nova_b200_ctx *c, uint64_t n, const uint32_t *idx, const uint32_t *dim, uint32_t seed,
                          float *out) {
  using namespace nbctx;
  if (n == 0) return NOVA_B200_SUCCESS;
  if (!idx || !dim || !out) return fail(c, NOVA_B200_INVALID_ARGUMENT, "null buffer%s");
  cudaSetDevice(c->device);
  k_sobol_api<<<(unsigned)((n + 255) / 256), 256, 0, c->stream>>>(c->d_sobol, n, idx, dim, seed, out);
  NB_CUDA(c, cudaGetLastError(), "k_sobol_api");
  NB_CUDA(c, cudaStreamSynchronize(c->stream), "sobol");
  return NOVA_B200_SUCCESS;
}
