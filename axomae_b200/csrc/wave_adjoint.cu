/* The replay adjoint's waves (nova_b200_backward): camera rays with what each path still gathers, the vertices'
 * gradient terms, and the last paths.  The method is described at shade_adj_path's section of wavefront.cuh.
 */
#include "wavefront.cuh"

namespace {

template <class JS>
__global__ void __launch_bounds__(256) k_refill_adj(Queue q, AdjQueue a, WaveCounters *wcp, uint32_t wave,
                                                    uint32_t total, uint32_t cap, const float4 *L,
                                                    const float4 *d_image, const __grid_constant__ JS js) {
  const WaveState ws = first_state(wcp, wave, total, cap);
  const uint32_t n_new = min(cap - ws.n_active, total - ws.next);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_new; i += gridDim.x * blockDim.x) {
    const CameraPath c = camera_path(js, ws.next + i);
    const RenderParams &rp = js.at(c.job).rp;
    const uint32_t slot = ws.n_active + i;
    q.o[slot] = make_float4(c.o.x, c.o.y, c.o.z, __uint_as_float(c.rslot));
    q.d[slot] = make_float4(c.d.x, c.d.y, c.d.z, __uint_as_float(c.job << 8));
    q.beta[slot] = make_float4(1.f, 1.f, 1.f, __uint_as_float(c.index));
    const float4 I = L[c.rslot];
    a.rem[slot] = make_float4(I.x, I.y, I.z, 0.f);
    /* the film pixel of (x, y): rows flipped when the frame asks for it (k_resolve) */
    const uint32_t row = rp.vinv ? (uint32_t)rp.H - 1u - c.y : c.y;
    const float4 g = d_image[(size_t)row * rp.W + c.x];
    const float inv = 1.f / (float)rp.count; /* the image is the mean of the frame's samples */
    a.dl[slot] = make_float4(g.x * inv, g.y * inv, g.z * inv, 0.f);
  }
}

template <class JS>
__global__ void __launch_bounds__(128, 8)
    k_shade_adj(Queue in, Queue out, AdjQueue ain, AdjQueue aout, WaveCounters *wcp, uint32_t wave, const float4 *hits,
                const uint2 *hit_slot, float *g_alb, float *g_rough, const __grid_constant__ JS js) {
  const WaveState &ws = wave_at(wcp, wave);
  const uint32_t nf = ws.hit_count, n = nf + ws.hit_back, cap = wcp->cap;
  unsigned *out_count = &wave_at(wcp, wave + 1).n_active;
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t == 0) clear_wave(wcp, wave);
  if ((t & ~31u) >= n) return;
  bool enq = false;
  float4 o4{}, d4{}, b4{}, rem4{}, l4{};
  AdjTerms g{};
  if (t < n) {
    const uint32_t i = hit_index(t, nf, cap);
    const uint2 hs = hit_slot[i];
    o4 = in.o[hs.x], d4 = in.d[hs.x], b4 = in.beta[hs.x];
    rem4 = ain.rem[hs.x], l4 = ain.dl[hs.x];
    enq = shade_adj_path(o4, d4, b4, rem4, l4, hits[i], hs.y, wcp, js, g);
  }
  add_terms(g, g_alb, g_rough);
  const unsigned slot = warp_append(enq, out_count);
  if (enq) {
    out.o[slot] = o4;
    out.d[slot] = d4;
    out.beta[slot] = b4;
    aout.rem[slot] = rem4;
    aout.dl[slot] = l4;
  }
}
template <int WIDTH>
cudaError_t enqueue(nova_b200_ctx *c, const OneJob &js, const LaunchShape &ls, const WavePlan &p, uint64_t &kernels,
                    const AdjArgs &adj) {
  const WaveBuffers b = wave_buffers(c);
  const int slot = (int)(p.wave & 1u);
  const Queue &in = input_queue(b, p.wave), &out = output_queue(b, p.wave);
  const AdjQueue &ain = slot ? adj.qb : adj.qa, &aout = slot ? adj.qa : adj.qb;
  cudaEvent_t *ev = c->ev_wave + 3 * slot;
  if (p.fresh) {
    k_refill_adj<OneJob><<<blocks_for(p.fresh, 256), 256, 0, c->stream>>>(in, ain, b.wc, p.wave, p.total, p.cap,
                                                                          c->d_radiance, adj.d_image, js);
    kernels++;
  }
  cudaEventRecord(ev[0], c->stream);
  if (p.finish) {
    const uint32_t lanes = finish_lanes(p.rays, p.wave);
    k_finish<WIDTH, OneJob, true><<<blocks_for(p.rays, 4u * lanes), 128, 0, c->stream>>>(
        in, ain, b.wc, p.wave, lanes, c->d_radiance, adj.g_alb, adj.g_rough, js);
    kernels++;
    cudaEventRecord(ev[1], c->stream);
    return cudaGetLastError(); /* what follows the last wave brings the counters back */
  }
  k_trace<WIDTH, OneJob, true><<<blocks_for(p.rays, ls.trace_block), ls.trace_block, 0, c->stream>>>(
      in, b.wc, p.wave, b.hits, b.hit_slot, nullptr, js);
  cudaEventRecord(ev[1], c->stream);
  k_shade_adj<OneJob><<<blocks_for(p.rays, ls.shade_block), ls.shade_block, 0, c->stream>>>(
      in, out, ain, aout, b.wc, p.wave, b.hits, b.hit_slot, adj.g_alb, adj.g_rough, js);
  kernels += 2;
  cudaEventRecord(ev[2], c->stream);
  cudaMemcpyAsync(static_cast<WaveCounters *>(c->h_wave) + slot, b.wc, sizeof(WaveCounters), cudaMemcpyDeviceToHost,
                  c->stream);
  cudaEventRecord(c->ev_done[slot], c->stream);
  return cudaGetLastError();
}

}  // namespace

cudaError_t nb::wave::enqueue_adjoint_wave(nova_b200_ctx *c, const OneJob &js, const LaunchShape &ls, int width,
                                           const WavePlan &p, uint64_t &kernels, const AdjArgs &adj) {
  if (width == 8) return enqueue<8>(c, js, ls, p, kernels, adj);
  if (width == 1) return enqueue<1>(c, js, ls, p, kernels, adj);
  return enqueue<2>(c, js, ls, p, kernels, adj);
}
