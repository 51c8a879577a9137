/* Trace modes 1 to 3 of the tuning: persistent warps that hand rays out, walks that count their work, and the
 * persistent wavefront, one cooperative launch for all waves of a chunk.
 */
#include "wavefront.cuh"

namespace {

/* Persistent variant of k_trace (binary BVH): a fixed grid of warps hands out the queued rays with
 * a warp-wide counter, and lanes whose walk has ended take new rays while the warp's other lanes
 * keep walking, so lanes do not idle behind the warp's longest walk.  Work goes in rounds: every lane
 * advances its walk by up to kDynSteps iterations of trace_closest2's loop (an inner node, or a leaf
 * and the pop after it), leaving the round early once kRefillLanes lanes are done; then finished
 * walks report (miss: environment, hit: the compact hit list, one warp append per round) and idle
 * lanes take new rays.  The walk's arithmetic and order are trace_closest2's, so the hits are the
 * same.  A lane keeps its ray's scene tables in registers (WalkScene), so a batch's job table is
 * read once per ray. */
/* Measured on the 32-job batch (trace time per step): 8 blocks per SM and 32 steps 221 ms, 16 steps
 * 222 ms, 8 steps 282 ms; 10 blocks per SM (spills) and 16 steps 245 ms; the per-ray kernel 195 ms.
 * The hits also reach the shading pass in finishing order instead of queue order, which costs
 * k_shade 11 % (121 vs 109 ms). */
#ifndef NB_DYN_STEPS
#define NB_DYN_STEPS 32
#endif
#ifndef NB_DYN_MIN_BLOCKS
#define NB_DYN_MIN_BLOCKS 8
#endif
constexpr int kDynSteps = NB_DYN_STEPS;
constexpr int kRefillLanes = 8;

template <class JS>
__global__ void __launch_bounds__(128, NB_DYN_MIN_BLOCKS) k_trace_dyn(Queue q, WaveCounters *wcp, uint32_t wave,
                                                                      float4 *hits, uint2 *hit_slot, float4 *L,
                                                                      const __grid_constant__ JS js) {
  WaveState &ws_ = wave_at(wcp, wave);
  const uint32_t n = wave_rays(*wcp, ws_);
  if (blockIdx.x == 0 && threadIdx.x == 0) advance_wave(wcp, wave);
  const unsigned full = 0xffffffffu, lane = threadIdx.x & 31u;
  Walk2 w;
  WalkScene ws{nullptr, nullptr, nullptr};
  int32_t stack[kTraversalStack];
  int32_t ray = -1;
  bool exhausted = false;
  /* every round hands out rays or advances a walk; the bound only guards against a bug */
  for (uint32_t round = 0; round < (1u << 30); round++) {
    const bool idle = ray < 0 && !exhausted;
    const unsigned need = __ballot_sync(full, idle);
    if (need) {
      const int leader = __ffs(need) - 1;
      uint32_t base = 0;
      if ((int)lane == leader) base = atomicAdd(&ws_.trace_next, (unsigned)__popc(need));
      base = __shfl_sync(full, base, leader);
      if (idle) {
        const uint32_t i = base + (uint32_t)__popc(need & ((1u << lane) - 1u));
        if (i < n) {
          const float4 o = q.o[i], d = q.d[i];
          const DevScene &sc = js.at(__float_as_uint(d.w) >> 8).sc;
          ws = WalkScene{sc.nodes, sc.tris, sc.instances};
          ray = (int32_t)i;
          w.init(V3{o.x, o.y, o.z}, V3{d.x, d.y, d.z});
        } else {
          exhausted = true;
        }
      }
    }
    if (__ballot_sync(full, ray >= 0) == 0) break; /* every lane idle after a refill: all rays handed out */
    bool fin = false;
    for (int k = 0; k < kDynSteps; k++) {
      if (ray >= 0 && !fin) fin = !w.step(ws, stack);
      if (__popc(__ballot_sync(full, ray < 0 || fin)) >= kRefillLanes) break;
    }
    const bool is_hit = fin && w.r.prim >= 0;
    if (fin && !is_hit) {
      const float4 o = q.o[ray], b4 = q.beta[ray], d = q.d[ray];
      const DevScene &sc = js.at(__float_as_uint(d.w) >> 8).sc;
      const V4 e = env_sample(sc, V3{d.x, d.y, d.z});
      finish_path(sc, L, __float_as_uint(o.w),
                  finite_or_zero(V3{b4.x, b4.y, b4.z} * V3{e.x, e.y, e.z}, (float)(__float_as_uint(d.w) & 0xffu) + e.w,
                                 &wcp->nonfinite),
                  &wcp->nonfinite);
    }
    if (__ballot_sync(full, fin)) {
      const unsigned slot = warp_append(is_hit, &ws_.hit_count);
      if (is_hit) {
        hits[slot] = make_float4(w.r.t, w.r.u, w.r.v, __int_as_float(w.r.prim));
        hit_slot[slot] = make_uint2((uint32_t)ray, w.r.inst);
      }
    }
    if (fin) ray = -1;
  }
}

/* ---------------------------------------------------------------- persistent wavefront (trace_mode 3)
 *
 * One cooperative launch runs every wave of a chunk: refill -> trace -> shade -> wave end, the same
 * device functions as the per-wave kernels, separated by a grid barrier.  Warps take 32 rays (hits)
 * at a time from a counter, so the block scheduler's balancing of the per-wave kernels is kept.
 * Data one phase writes and a later phase reads on another SM is loaded through L2 (ldq<true>).
 *
 * The barrier is this file's own and its wait is bounded: block leaders arrive on a counter and
 * spin on a generation word with a time limit (globaltimer); a leader that waits past the limit sets
 * the status word to 1 and every block leaves at its next barrier, so the kernel always ends and the
 * host reports RENDERER_EXCEPTION.  A cancel (the context's mapped flag) sets status 2 the same way. */
struct PersistSync {
  unsigned arrive, gen, status, pad;
  unsigned long long trace_ns, shade_ns; /* phase times seen by block 0 */
};

__device__ __forceinline__ unsigned ld_volatile(const unsigned *p) { return *(const volatile unsigned *)p; }

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

/* false once any block gave up waiting (or the render was cancelled): the caller returns.  The leader's
 * reading of the status word is shared through shared memory, so a block leaves as a whole. */
__device__ bool grid_barrier(PersistSync *s, unsigned long long limit_ns) {
  __shared__ unsigned s_status;
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned gen = ld_volatile(&s->gen);
    __threadfence();
    if (atomicAdd(&s->arrive, 1u) == gridDim.x - 1u) {
      atomicExch(&s->arrive, 0u);
      __threadfence();
      atomicAdd(&s->gen, 1u);
    } else {
      const unsigned long long t0 = global_ns();
      while (ld_volatile(&s->gen) == gen) {
        if (ld_volatile(&s->status) != 0u) break;
        if (global_ns() - t0 > limit_ns) {
          atomicCAS(&s->status, 0u, 1u);
          break;
        }
        __nanosleep(64);
      }
    }
    __threadfence();
    s_status = ld_volatile(&s->status);
  }
  __syncthreads();
  return s_status == 0u;
}

/* A warp's next 32 items from a counter (lane 0 takes them, the warp shares the base). */
__device__ __forceinline__ uint32_t warp_take(unsigned *counter) {
  uint32_t base = 0;
  if ((threadIdx.x & 31u) == 0) base = atomicAdd(counter, 32u);
  return __shfl_sync(0xffffffffu, base, 0);
}

/* Resident blocks of 128 per SM that k_persist is compiled for.  It holds both the walk and the
 * shading state, so its register budget is the larger of the two phases': on the 32-job batch, 6
 * blocks (80 registers) took 379 ms per step, 5 (96) 408 ms and 4 (128, no spills) 465 ms, against
 * 316 ms for the per-wave kernels (40 resident warps for k_trace, 32 for k_shade when measured). */
#ifndef NB_PERSIST_MIN_BLOCKS
#define NB_PERSIST_MIN_BLOCKS 6
#endif

template <int WIDTH, class JS>
__global__ void __launch_bounds__(128, NB_PERSIST_MIN_BLOCKS) k_persist(Queue qa, Queue qb, WaveCounters *wcp, float4 *hits,
                                                 uint2 *hit_slot, float4 *L, PersistSync *sync,
                                                 const volatile int *cancel, unsigned long long limit_ns,
                                                 const __grid_constant__ JS js) {
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
  const uint32_t lane = threadIdx.x & 31u;
  const bool leader = tid == 0;
  for (uint32_t w = 0;; w++) {
    const Queue &in = (w & 1u) ? qb : qa;
    const Queue &out = (w & 1u) ? qa : qb;
    WaveState &ws = wave_at(wcp, w);
    const uint32_t n_active = __ldcg(&ws.n_active), next = __ldcg(&ws.next);
    const uint32_t total = __ldcg(&wcp->total), cap = __ldcg(&wcp->cap);
    if (__ldcg(&wcp->done)) return;
    const uint32_t n_new = min(cap - n_active, total - next), n = n_active + n_new;
    float4 o, d;
    for (uint32_t i = tid; i < n_new; i += nthreads) refill_one(in, next, n_active, L, js, i, o, d);
    if (!grid_barrier(sync, limit_ns)) return;
    const unsigned long long t0 = leader ? global_ns() : 0ull;
    for (;;) {
      const uint32_t base = warp_take(&ws.trace_next);
      if (base >= n) break;
      trace_warp<WIDTH, JS, false, false, true>(in, wcp, ws, hits, hit_slot, L, js, base + lane, n);
    }
    if (!grid_barrier(sync, limit_ns)) return;
    const unsigned long long t1 = leader ? global_ns() : 0ull;
    const uint32_t nh = __ldcg(&ws.hit_count);
    unsigned *out_count = &wave_at(wcp, w + 1).n_active;
    for (;;) {
      const uint32_t base = warp_take(&ws.shade_next);
      if (base >= nh) break;
      shade_warp<JS, true>(in, out, wcp, out_count, hits, hit_slot, L, js, base + lane, base + lane < nh);
    }
    if (!grid_barrier(sync, limit_ns)) return;
    if (leader) { /* the next entry's first path, the one after it cleared */
      sync->trace_ns += t1 - t0;
      sync->shade_ns += global_ns() - t1;
      if (n) {
        wcp->waves++;
        wcp->traced += n;
      }
      wave_at(wcp, w + 1).next = next + n_new;
      clear_wave(wcp, w);
      wcp->done = (__ldcg(out_count) == 0 && next + n_new == total) ? 1u : 0u;
      if (*cancel) atomicCAS(&sync->status, 0u, 2u);
      __threadfence();
    }
    if (!grid_barrier(sync, limit_ns)) return;
  }
}

/* The persistent wavefront over `total` paths: counters and barrier reset, one cooperative launch of
 * k_persist with every block resident (the occupancy calculator's count per SM), then the counters'
 * read-back.  Status 1 (a barrier wait ran out) and 2 (cancelled) fail the call; the context stays
 * usable either way (the kernel has returned). */
template <int WIDTH, class JS>
nova_b200_status persistent(nova_b200_ctx *x, const JS &js, const LaunchShape &ls, uint32_t total, uint32_t cap,
                                LoopStats &st) {
  using namespace nbctx;
  WaveCounters *hw = static_cast<WaveCounters *>(x->h_wave);
  if (!x->d_persist) {
    NB_CUDA(x, cudaMalloc(&x->d_persist, sizeof(PersistSync)), "cudaMalloc(persistent barrier)");
    void *flag = nullptr;
    NB_CUDA(x, cudaHostAlloc(&flag, sizeof(int), cudaHostAllocMapped), "cudaHostAlloc(cancel flag)");
    x->h_cancel_map = static_cast<volatile int *>(flag);
    *x->h_cancel_map = x->cancel.load() ? 1 : 0;
  }
  void *d_cancel_v = nullptr;
  NB_CUDA(x, cudaHostGetDevicePointer(&d_cancel_v, const_cast<int *>(x->h_cancel_map), 0), "cancel flag");
  int *d_cancel = static_cast<int *>(d_cancel_v);
  hw[2] = WaveCounters{};
  hw[2].total = total;
  hw[2].cap = cap;
  NB_CUDA(x, cudaMemcpyAsync(x->d_wave, hw + 2, sizeof(WaveCounters), cudaMemcpyHostToDevice, x->stream),
          "upload(wave counters)");
  NB_CUDA(x, cudaMemsetAsync(x->d_persist, 0, sizeof(PersistSync), x->stream), "reset(barrier)");
  int sms = 148, occ = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, x->device);
  NB_CUDA(x, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_persist<WIDTH, JS>, 128, 0), "occupancy");
  if (occ < 1) return fail(x, NOVA_B200_RENDERER_EXCEPTION, "persistent wavefront: no resident block fits%s");
  const WaveBuffers b = wave_buffers(x);
  PersistSync *sync = static_cast<PersistSync *>(x->d_persist);
  float4 *L = x->d_radiance;
  const volatile int *cancel = d_cancel;
  const unsigned long long limit_ns = 1000ull * ls.wait_limit_us;
  void *args[] = {const_cast<Queue *>(&b.qa), const_cast<Queue *>(&b.qb), const_cast<WaveCounters **>(&b.wc),
                  const_cast<float4 **>(&b.hits), const_cast<uint2 **>(&b.hit_slot), &L, &sync,
                  const_cast<const volatile int **>(&cancel), const_cast<unsigned long long *>(&limit_ns),
                  const_cast<JS *>(&js)};
  NB_CUDA(x, cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(k_persist<WIDTH, JS>), dim3(sms * occ),
                                         dim3(128), args, 0, x->stream),
          "persistent wavefront launch");
  PersistSync hs{};
  NB_CUDA(x, cudaMemcpyAsync(hw, x->d_wave, sizeof(WaveCounters), cudaMemcpyDeviceToHost, x->stream), "readback");
  NB_CUDA(x, cudaMemcpyAsync(&hs, x->d_persist, sizeof(PersistSync), cudaMemcpyDeviceToHost, x->stream), "readback");
  NB_CUDA(x, cudaStreamSynchronize(x->stream), "persistent wavefront");
  const WaveCounters r = hw[0];
  st.kernels += 1;
  st.t_trace += (float)(hs.trace_ns * 1e-6);
  st.t_shade += (float)(hs.shade_ns * 1e-6);
  st.waves += r.waves;
  st.traced += r.traced;
  st.nonfinite += r.nonfinite;
  st.bad_index += r.bad_index;
  if (hs.status == 2u) return fail(x, NOVA_B200_RENDERER_EXCEPTION, "render cancelled%s");
  if (hs.status != 0u) {
    char msg[160];
    std::snprintf(msg, sizeof(msg), "persistent wavefront: a grid barrier waited longer than %u us", ls.wait_limit_us);
    return fail(x, NOVA_B200_RENDERER_EXCEPTION, "%s", msg);
  }
  if (r.bad_index) {
    char msg[160];
    std::snprintf(msg, sizeof(msg), "device status: %u hits with an out-of-range primitive, instance or material id",
                  (unsigned)r.bad_index);
    return fail(x, NOVA_B200_RENDERER_EXCEPTION, "%s", msg);
  }
  if (!r.done) return fail(x, NOVA_B200_RENDERER_EXCEPTION, "persistent wavefront ended before its paths%s");
  return NOVA_B200_SUCCESS;
}

template <class JS>
nova_b200_status persistent_w(nova_b200_ctx *x, const JS &js, const LaunchShape &ls, int width, uint32_t total,
                              uint32_t cap, LoopStats &st) {
  if (width == 8) return persistent<8>(x, js, ls, total, cap, st);
  if (width == 1) return persistent<1>(x, js, ls, total, cap, st);
  return persistent<2>(x, js, ls, total, cap, st);
}

template <int WIDTH, class JS>
void counted(nova_b200_ctx *c, const JS &js, const LaunchShape &ls, const WavePlan &p) {
  const WaveBuffers b = wave_buffers(c);
  k_trace<WIDTH, JS, false, true><<<blocks_for(p.rays, ls.trace_block), ls.trace_block, 0, c->stream>>>(
      input_queue(b, p.wave), b.wc, p.wave, b.hits, b.hit_slot, c->d_radiance, js);
}

template <class JS>
void mode_trace(nova_b200_ctx *c, const JS &js, const LaunchShape &ls, int width, const WavePlan &p) {
  if (ls.trace_mode == 1) {
    const WaveBuffers b = wave_buffers(c);
    int sms = 148, occ = 1;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_trace_dyn<JS>, 128, 0);
    k_trace_dyn<JS><<<std::min(blocks_for(p.rays, 128), (unsigned)(sms * std::max(1, occ))), 128, 0, c->stream>>>(
        input_queue(b, p.wave), b.wc, p.wave, b.hits, b.hit_slot, c->d_radiance, js);
  } else if (width == 8) {
    counted<8>(c, js, ls, p);
  } else if (width == 1) {
    counted<1>(c, js, ls, p);
  } else {
    counted<2>(c, js, ls, p);
  }
}

}  // namespace

void nb::wave::launch_mode_trace(nova_b200_ctx *c, const OneJob &js, const LaunchShape &ls, int width,
                                 const WavePlan &p) {
  mode_trace(c, js, ls, width, p);
}
void nb::wave::launch_mode_trace(nova_b200_ctx *c, const ManyJobs &js, const LaunchShape &ls, int width,
                                 const WavePlan &p) {
  mode_trace(c, js, ls, width, p);
}
nova_b200_status nb::wave::run_persistent(nova_b200_ctx *x, const OneJob &js, const LaunchShape &ls, int width,
                                          uint32_t total, uint32_t cap, LoopStats &st) {
  return persistent_w(x, js, ls, width, total, cap, st);
}
nova_b200_status nb::wave::run_persistent(nova_b200_ctx *x, const ManyJobs &js, const LaunchShape &ls, int width,
                                          uint32_t total, uint32_t cap, LoopStats &st) {
  return persistent_w(x, js, ls, width, total, cap, st);
}
