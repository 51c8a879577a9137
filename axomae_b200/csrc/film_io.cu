/* Film outputs and the Radiance .hdr image format: the callers on either side of the render.
 *
 * Device kernels (one thread per pixel or per four floats; each reads its inputs once and writes
 * its outputs once, so they are bound by HBM bandwidth):
 *   k_accumulate     Engine::writeFramebuffer (corelib/nova/api/engine.cpp:351-363): the running
 *                    sum of one-sample frames and its mean, accumulated / (frame_index + 1).
 *   k_display_blend  NovaRenderer::copyBufferToPbo (sources/renderer/nova/NovaRenderer_draw.cpp:35-45):
 *                    the editor's display value old + 0.8 (new - old), old = accumulated / (frame + 1).
 *   k_snapshot       NovaRenderer::getSnapshotFloat (sources/renderer/nova/NovaRenderer.cpp:139-153)
 *                    through TextureOperations::processTexture / uvSample / bilinearInterpolate /
 *                    wrapAroundPixelCoords (sources/processing/TextureProcessing.h:157-250): a resample
 *                    of the film to another size with the reference's float / double conversions.
 *   k_rgbe_encode    float pixel -> shared-exponent RGBE bytes of the Radiance format (G. Ward,
 *   k_rgbe_decode    "Real Pixels", Graphics Gems II, 1991) and back, rounded the way the stb_image
 *                    routines the reference calls do it (stbi_write_hdr in IO::Loader::writeHdr,
 *                    stbi_loadf in IO::Loader::loadRadianceFile, sources/IO/Loader_image.cpp:50-62,
 *                    146-192; stb is an un-vendored submodule of the reference, github.com/nothings/stb).
 *
 *   k_rle_find, k_rle_walk, k_rle_link, k_rle_rows  where the rows of a run-length file start, and their
 *                    packets expanded.
 *
 * Host code: the file's text header, and the packet walk of small or irregular run-length files.
 */
#include <climits>
#include <cstring>
#include <fstream>
#include <memory>
#include <string>
#include <vector>

#include "context.cuh"

namespace {

/* ---- device kernels ---------------------------------------------------------------------- */

__global__ void k_accumulate(const float *partial, float *accum, float *final_buf, uint64_t n, float denom) {
  const uint64_t i4 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i4 + 4 <= n) {
    const float4 p = *reinterpret_cast<const float4 *>(partial + i4);
    float4 a = *reinterpret_cast<const float4 *>(accum + i4);
    a.x += p.x, a.y += p.y, a.z += p.z, a.w += p.w;
    *reinterpret_cast<float4 *>(accum + i4) = a;
    if (final_buf)
      *reinterpret_cast<float4 *>(final_buf + i4) = make_float4(a.x / denom, a.y / denom, a.z / denom, a.w / denom);
  } else {
    for (uint64_t i = i4; i < n; i++) {
      const float a = accum[i] + partial[i];
      accum[i] = a;
      if (final_buf) final_buf[i] = a / denom;
    }
  }
}

__device__ __forceinline__ float blend(float acc, float now, float denom) {
  const float old = acc / denom;
  return old + 0.8f * (now - old);
}

/* From the end of the film: what k_accumulate left of it in the L2 is the end, and the display image goes past
 * it (3840 x 2160: 77 -> 71 us a call; 398 MB). */
__global__ void k_display_blend(const float *partial, const float *accum, float *out, uint64_t n, float denom) {
  const uint64_t i4 = ((uint64_t)(gridDim.x - 1u - blockIdx.x) * blockDim.x + threadIdx.x) * 4;
  if (i4 + 4 <= n) {
    const float4 p = *reinterpret_cast<const float4 *>(partial + i4);
    const float4 a = *reinterpret_cast<const float4 *>(accum + i4);
    __stcs(reinterpret_cast<float4 *>(out + i4), make_float4(blend(a.x, p.x, denom), blend(a.y, p.y, denom),
                                                             blend(a.z, p.z, denom), blend(a.w, p.w, denom)));
  } else {
    for (uint64_t i = i4; i < n; i++) out[i] = blend(accum[i], partial[i], denom);
  }
}

struct Film {
  const float *data;
  int w, h, ch;
  /* TextureOperations::discreteSample with wrapAroundPixelCoords (TextureProcessing.h:174-181, 233-250) */
  __device__ float3 texel(int x, int y) const {
    const int xc = x >= w ? x % w : (x < 0 ? w + (x % w) : x);
    const int yc = y >= h ? y % h : (y < 0 ? h + (y % h) : y);
    const float *p = data + ((size_t)yc * w + xc) * ch;
    return make_float3(p[0], p[1], p[2]);
  }
};

/* uvToPixel (math_texturing.h:19-21): float coordinate times the size, converted to unsigned the
 * way x86-64 code does it (64-bit truncation, low 32 bits). */
__device__ __forceinline__ unsigned uv_to_pixel(float coord, unsigned dim) {
  return (unsigned)(long long)__fmul_rn(coord, (float)dim);
}

__device__ __forceinline__ float wrap_uv(double c) {
  /* wrapAroundTexCoords<double> (TextureProcessing.h:214-230), returned as a float vec2 */
  const double ci = floor(c);
  return (float)((c > 1.0 || c < 0.0) ? c - ci : c);
}

__global__ void k_snapshot(Film src, float *dst, int dw, int dh) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
  if (i >= dw || j >= dh) return;
  /* processTexture: u = i / dest_width, v = j / dest_height in double (math_texturing.h:14-17) */
  const float wu = wrap_uv((double)i / (double)dw), wv = wrap_uv((double)j / (double)dh);
  /* pixel coordinates: unsigned -> double -> float (glm::dvec2 into glm::vec2) */
  const float px = (float)(double)uv_to_pixel(wu, (unsigned)src.w);
  const float py = (float)(double)uv_to_pixel(wv, (unsigned)src.h);
  const float tlx = floorf(px), tly = floorf(py);
  const float trx = __fadd_rn(floorf(px), 1.f), bly = __fadd_rn(floorf(py), 1.f);
  /* bilinearInterpolate (TextureProcessing.h:183-199), literally: the weights come out 0 and 1 for
   * whole-pixel coordinates, and the arithmetic keeps the reference's signed zeros and NaN spread */
  const float u = __fdiv_rn(__fsub_rn(px, tlx), __fsub_rn(trx, tlx));
  const float v = __fdiv_rn(__fsub_rn(py, tly), __fsub_rn(bly, tly));
  const float hd = __fsub_rn(1.f, u);
  const float3 tl = src.texel((int)tlx, (int)tly), tr = src.texel((int)trx, (int)tly);
  const float3 bl = src.texel((int)tlx, (int)bly), br = src.texel((int)trx, (int)bly);
  const float vd = __fsub_rn(1.f, v);
  auto lerp2 = [&](float a, float b, float c, float d) {
    const float top = __fadd_rn(__fmul_rn(hd, a), __fmul_rn(u, b));
    const float bot = __fadd_rn(__fmul_rn(hd, c), __fmul_rn(u, d));
    return __fadd_rn(__fmul_rn(vd, top), __fmul_rn(v, bot));
  };
  /* dest index uses the source's channel stride; channel 3 is never written (:167-171) */
  float *o = dst + ((size_t)j * dw + i) * src.ch;
  o[0] = lerp2(tl.x, tr.x, bl.x, br.x);
  o[1] = lerp2(tl.y, tr.y, bl.y, br.y);
  o[2] = lerp2(tl.z, tr.z, bl.z, br.z);
}

/* Float RGB -> RGBE.  m = max(r, g, b) taken as max(r, max(g, b)) with "a > b ? a : b" (so a NaN
 * operand is passed over unless it is the first); m < 1e-32 -> all zero; else m = f 2^e with f in
 * [0.5, 1), scale = f * 256 / m, byte_c = low byte of the int32 truncation of c * scale, byte_e =
 * low byte of e + 128.  A non-finite m gives RGB 0 and exponent byte 128.  The truncations follow
 * x86-64 conversion (int32 truncation toward zero, NaN -> 0 in the low byte). */
__device__ __forceinline__ uchar4 rgbe_encode(float r, float g, float b) {
  const float gb = g > b ? g : b;
  const float m = r > gb ? r : gb;
  if (m < 1e-32f) return make_uchar4(0, 0, 0, 0);
  if (!isfinite(m)) return make_uchar4(0, 0, 0, 128);
  /* m is a normal float here (>= 1e-32): its exponent field gives e directly */
  const uint32_t bits = __float_as_uint(m);
  const int e = (int)((bits >> 23) & 0xffu) - 126;
  const float f = __uint_as_float((bits & 0x807fffffu) | (126u << 23));
  const float scale = __fdiv_rn(__fmul_rn(f, 256.f), m);
  auto byte = [](float x) -> unsigned char {
    return isnan(x) ? (unsigned char)0 : (unsigned char)((unsigned)(int)x & 0xffu);
  };
  return make_uchar4(byte(__fmul_rn(r, scale)), byte(__fmul_rn(g, scale)), byte(__fmul_rn(b, scale)),
                     (unsigned char)((unsigned)(e + 128) & 0xffu));
}

/* Encodes rows in file order (flip: bottom row first).  planar = 1 writes each row as four planes
 * of width bytes (R, G, B, E: the order of run-length scanlines), 0 as interleaved pixels.  vec4:
 * 4-channel pixels at a 16-byte aligned address, read as one float4. */
__global__ void k_rgbe_encode(const float *src, int w, int h, int ch, int flip, int planar, int vec4,
                              unsigned char *dst) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, row = blockIdx.y;
  if (x >= w || row >= h) return;
  const int srow = flip ? h - 1 - row : row;
  const size_t px = (size_t)srow * w + x;
  float r, g, b;
  if (vec4) {
    const float4 v = __ldg(reinterpret_cast<const float4 *>(src) + px);
    r = v.x, g = v.y, b = v.z;
  } else if (ch >= 3) {
    const float *p = src + px * ch;
    r = p[0], g = p[1], b = p[2];
  } else {
    r = g = b = src[px * ch];
  }
  const uchar4 q = rgbe_encode(r, g, b);
  if (planar) {
    unsigned char *o = dst + (size_t)row * w * 4;
    o[x] = q.x, o[w + x] = q.y, o[2 * w + x] = q.z, o[3 * w + x] = q.w;
  } else {
    reinterpret_cast<uchar4 *>(dst)[(size_t)row * w + x] = q;
  }
}

/* RGBE -> float: exponent byte 0 -> (0, 0, 0); else c = byte 2^(e - 136), exact; alpha 1 (the
 * loader widens 3-channel files to RGBA with alpha 1, Loader_image.cpp:161-170). */
__device__ __forceinline__ float4 rgbe_decode(uint32_t word) {
  const uint32_t e = word >> 24;
  if (e == 0) return make_float4(0.f, 0.f, 0.f, 1.f);
  const double s = __longlong_as_double((long long)((int)e - 136 + 1023) << 52);
  return make_float4((float)((word & 0xffu) * s), (float)(((word >> 8) & 0xffu) * s),
                     (float)(((word >> 16) & 0xffu) * s), 1.f);
}

/* Four pixels per thread: one 16-byte load of RGBE words, four float4 stores (both buffers 16-byte
 * aligned); the last thread takes the ragged end pixel by pixel.  ok: null, or 0 for "nothing to decode". */
__global__ void k_rgbe_decode(const uint32_t *src, uint64_t n, float4 *dst, const uint32_t *ok) {
  if (ok && *ok == 0u) return;
  const uint64_t i4 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i4 + 4 <= n) {
    const uint4 q = __ldg(reinterpret_cast<const uint4 *>(src + i4));
    dst[i4] = rgbe_decode(q.x);
    dst[i4 + 1] = rgbe_decode(q.y);
    dst[i4 + 2] = rgbe_decode(q.z);
    dst[i4 + 3] = rgbe_decode(q.w);
  } else {
    for (uint64_t i = i4; i < n; i++) dst[i] = rgbe_decode(src[i]);
  }
}

/* Run-length packing, one warp per (row, plane) of the planar RGBE rows: runs of 3 or more equal
 * bytes become run packets (count + 128, value; count <= 127), the rest dump packets (count,
 * bytes; count <= 128).  The greedy scan is the serial one (next run start = first position whose
 * byte equals the next two; a run ends at the first different byte), with 32 positions tested per
 * step by a ballot; dump bytes are copied by all lanes.  Each warp writes its packets into its own
 * region of `cap` bytes (cap bounds the packets of any row: width + width / 128 + 2) and their size
 * into sizes; a region that would overflow sets *err and is cut. */
__global__ void k_rle_pack(const unsigned char *planar, int w, int n_planes, int cap, unsigned char *regions,
                           uint32_t *sizes, unsigned *err) {
  const int e = (int)((blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (e >= n_planes) return; /* whole warps leave together */
  const unsigned char *p = planar + (size_t)e * w; /* planes are consecutive: row-major (row, plane) */
  unsigned char *o = regions + (size_t)e * cap;
  int n = 0, x = 0;
  bool over = false;
  while (x < w) {
    int lit = w;
    for (int base = x; base < w; base += 32) {
      const int i = base + lane;
      const bool t = i + 2 < w && p[i] == p[i + 1] && p[i] == p[i + 2];
      const unsigned m = __ballot_sync(0xffffffffu, t);
      if (m) {
        lit = base + __ffs(m) - 1;
        break;
      }
    }
    while (x < lit) {
      const int cnt = min(lit - x, 128);
      if (n + 1 + cnt > cap) {
        over = true;
        break;
      }
      if (lane == 0) o[n] = (unsigned char)cnt;
      for (int k = lane; k < cnt; k += 32) o[n + 1 + k] = p[x + k];
      n += 1 + cnt;
      x += cnt;
    }
    if (over) break;
    if (lit < w) {
      const unsigned char v = p[lit];
      int end = w;
      for (int base = lit; base < w; base += 32) {
        const int i = base + lane;
        const unsigned m = __ballot_sync(0xffffffffu, i >= w || p[i] != v);
        if (m) {
          end = min(base + __ffs(m) - 1, w);
          break;
        }
      }
      while (x < end) {
        const int cnt = min(end - x, 127);
        if (n + 2 > cap) {
          over = true;
          break;
        }
        if (lane == 0) o[n] = (unsigned char)(128 + cnt), o[n + 1] = v;
        n += 2;
        x += cnt;
      }
      if (over) break;
    }
  }
  if (lane == 0) {
    if (over) atomicAdd(err, 1u);
    sizes[e] = (uint32_t)n;
  }
}

/* Exclusive scan of the packed sizes into file offsets, one block of 1024 threads: element
 * (row, plane 0) also carries the row's 4-byte header.  offsets[n] = total bytes. */
__global__ void __launch_bounds__(1024) k_rle_scan(const uint32_t *sizes, int n, uint64_t *offsets) {
  __shared__ uint64_t part[1024];
  const int t = threadIdx.x;
  const int chunk = (n + 1023) / 1024;
  const int b = min(t * chunk, n), e = min(b + chunk, n);
  uint64_t sum = 0;
  for (int i = b; i < e; i++) sum += sizes[i] + ((i & 3) == 0 ? 4u : 0u);
  part[t] = sum;
  __syncthreads();
  for (int d = 1; d < 1024; d <<= 1) { /* inclusive Hillis-Steele scan */
    const uint64_t v = t >= d ? part[t - d] : 0;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  uint64_t run = part[t] - sum;
  for (int i = b; i < e; i++) {
    offsets[i] = run;
    run += sizes[i] + ((i & 3) == 0 ? 4u : 0u);
  }
  if (t == 1023) offsets[n] = part[1023];
}

/* One warp per (row, plane): its packets to their file offset; plane 0 writes the row header
 * (2, 2, width >> 8, width & 255) first. */
__global__ void k_rle_gather(const unsigned char *regions, const uint32_t *sizes, const uint64_t *offsets, int w,
                             int cap, int n_planes, unsigned char *out) {
  const int e = (int)((blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (e >= n_planes) return;
  uint64_t dst = offsets[e];
  if ((e & 3) == 0) {
    if (lane < 4) out[dst + lane] = lane < 2 ? 2 : (lane == 2 ? (unsigned char)(w >> 8) : (unsigned char)(w & 255));
    dst += 4;
  }
  const unsigned char *src = regions + (size_t)e * cap;
  const uint32_t n = sizes[e];
  for (uint32_t j = lane; j < n; j += 32) out[dst + j] = src[j];
}

/* Run-length expansion, one warp per (row, plane): the packets starting at file offset starts[e]
 * (found and checked on the host) into byte `plane` of each RGBE pixel of the row; lane 0 reads
 * each packet's count, all lanes copy or fill.  The body buffer is zero-padded past the file's end,
 * which the loader reads as zeros. */
__global__ void k_rle_unpack(const unsigned char *body, const uint64_t *starts, int w, int n_planes,
                             unsigned char *rgbe) {
  const int e = (int)((blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (e >= n_planes) return;
  const unsigned char *p = body + starts[e];
  unsigned char *o = rgbe + (size_t)(e >> 2) * w * 4 + (e & 3);
  int x = 0;
  while (x < w) {
    int cnt = __shfl_sync(0xffffffffu, lane == 0 ? (int)p[0] : 0, 0);
    if (cnt == 0) break; /* excluded by the host's check; never loops without progress */
    if (cnt > 128) {
      cnt = min(cnt - 128, w - x);
      const unsigned char v = p[1];
      for (int k = lane; k < cnt; k += 32) o[4 * (size_t)(x + k)] = v;
      p += 2;
    } else {
      cnt = min(cnt, w - x);
      for (int k = lane; k < cnt; k += 32) o[4 * (size_t)(x + k)] = p[1 + k];
      p += 1 + cnt;
    }
    x += cnt;
  }
}

/* A run-length file's rows on the device.  Where a row starts is known only when the one before has been
 * walked, so every byte position that holds the row header (2, 2, width >> 8, width & 255) is walked as a
 * row (k_rle_find, k_rle_walk; a few of them are packet data), and k_rle_link follows the ends from the
 * first to the last row.  A chain that does not close (a cut or damaged file, a flat one) clears the status
 * word: the host then reads the file again, as it reads small ones. */

/* Two kernels: WRITE = false counts a block's matches, WRITE = true places the first `most` of them in file
 * order.  `chunk` (bytes per block) is a multiple of a tile, 16 bytes a thread; the body is padded by 256
 * zeros.  Bound by the body's bytes. */
constexpr int kFindThreads = 256, kFindTile = 16 * kFindThreads, kFindBlocks = 2048;

template <bool WRITE>
__global__ void __launch_bounds__(kFindThreads)
    k_rle_find(const unsigned char *body, uint32_t n, uint32_t pattern, uint32_t chunk, uint32_t *counts, uint32_t most,
               uint32_t *starts) {
  __shared__ uint32_t warp_sum[kFindThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  /* exclusive prefix of v over the block and the block's total */
  auto scan = [&](uint32_t v, uint32_t &total) {
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    __syncthreads();
    if (lane == 31) warp_sum[w] = x;
    __syncthreads();
    uint32_t before = 0;
    total = 0;
    for (int k = 0; k < kFindThreads / 32; k++) {
      const uint32_t t = warp_sum[k];
      if (k < w) before += t;
      total += t;
    }
    return before + x - v;
  };
  uint32_t base = 0, found = 0, total;
  if (WRITE) {
    uint32_t mine = 0;
    for (uint32_t b = threadIdx.x; b < blockIdx.x; b += kFindThreads) mine += counts[b];
    scan(mine, base);
    if (base >= most || counts[blockIdx.x] == 0u) return;
  }
  const uint64_t first = (uint64_t)blockIdx.x * chunk, last = min((uint64_t)n, first + chunk);
  for (uint64_t tile = first; tile < last; tile += kFindTile) {
    const uint64_t p = tile + 16u * threadIdx.x;
    uint32_t match = 0;
    if (p < n) {
      const uint4 q = __ldg(reinterpret_cast<const uint4 *>(body + p));
      const uint32_t v[5] = {q.x, q.y, q.z, q.w, __ldg(reinterpret_cast<const uint32_t *>(body + p + 16))};
#pragma unroll
      for (int k = 0; k < 16; k++)
        if (__funnelshift_r(v[k >> 2], v[(k >> 2) + 1], 8 * (k & 3)) == pattern && p + k + 4 <= n) match |= 1u << k;
    }
    if (!WRITE) {
      found += __popc(match);
    } else {
      uint32_t at = base + scan(__popc(match), total);
      for (; match; match &= match - 1u, at++)
        if (at < most) starts[at] = (uint32_t)p + __ffs(match) - 1u;
      base += total;
    }
  }
  if (!WRITE) {
    scan(found, total);
    if (threadIdx.x == 0) counts[blockIdx.x] = total;
  }
}

/* The bytes [start, start + bytes) of the body to shared memory by the whole block, 16 at a time; the first
 * of them lands at start & 15. */
__device__ __forceinline__ void stage_row(const unsigned char *body, uint32_t start, uint32_t bytes, uint4 *staged) {
  const uint4 *src = reinterpret_cast<const uint4 *>(body + (start & ~15u));
  for (uint32_t i = threadIdx.x; 16u * i < (start & 15u) + bytes; i += blockDim.x) staged[i] = __ldg(src + i);
  __syncthreads();
}

/* One block per position placed (0xffffffff: none): its row's bytes (2 per value at most) into shared
 * memory, then one thread walks the packet headers of the four planes, which follow one another: where each
 * plane starts and the row ends, in `walked`; an end of 0 when this is no row. */
struct WalkedRow {
  uint32_t plane[4], end;
};
__global__ void __launch_bounds__(128) k_rle_walk(const unsigned char *body, uint32_t n, const uint32_t *starts, int w,
                                                  uint32_t cap, WalkedRow *walked) {
  extern __shared__ uint4 staged[];
  const uint32_t start = starts[blockIdx.x];
  if (start == 0xffffffffu) return;
  const uint32_t shift = start & 15u, bytes = min(min(n - start, 8u * (uint32_t)w + 4u), cap - shift);
  stage_row(body, start, bytes, staged);
  if (threadIdx.x != 0) return;
  const unsigned char *sm = reinterpret_cast<const unsigned char *>(staged) + shift;
  WalkedRow r;
  uint32_t p = 4u;
  bool fine = true;
  for (int k = 0; k < 4; k++) {
    r.plane[k] = p;
    for (uint32_t left = (uint32_t)w; fine && left > 0u;) {
      const uint32_t head = p < bytes ? sm[p] : 0u, cnt = head > 128u ? head - 128u : head;
      fine = cnt != 0u && cnt <= left;
      p += head > 128u ? 2u : 1u + cnt;
      left -= cnt;
    }
  }
  r.end = fine && p <= bytes ? start + p : 0u;
  walked[blockIdx.x] = r;
}

/* Which of the walked positions are the image's h rows: the first, and each one that starts where the row
 * before ends.  One block; without matches in packet data position j is row j, which all threads check at
 * once, else one warp follows the links, 32 positions in its lanes.  *ok becomes 0 when the rows do not chain. */
__global__ void __launch_bounds__(1024) k_rle_link(const uint32_t *starts, const WalkedRow *walked, uint32_t most,
                                                   uint32_t h, uint32_t *next, uint32_t *rows, uint32_t *ok) {
  constexpr uint32_t kNone = 0xffffffffu;
  bool plain = true;
  for (uint32_t i = threadIdx.x; i < most && starts[i] != kNone; i += blockDim.x) {
    const uint32_t end = walked[i].end;
    uint32_t to = kNone;
    if (end != 0u && i + 1u < most) {
      uint32_t lo = i + 1u, hi = most; /* the first position at or after the end (0xffffffff: past the last) */
      if (starts[lo] < end)
        while (lo < hi) {
          const uint32_t mid = lo + (hi - lo) / 2u;
          if (starts[mid] < end)
            lo = mid + 1u;
          else
            hi = mid;
        }
      if (lo < most && starts[lo] == end) to = lo;
    }
    next[i] = to;
    if (i < h) {
      rows[i] = i;
      plain = plain && (i + 1u < h ? to == i + 1u : end != 0u);
    }
  }
  if (__syncthreads_and(plain && (h <= most && starts[h - 1u] != kNone))) return;
  if (threadIdx.x >= 32u) return;
  uint32_t at = 0, mine = 0, base = kNone;
  for (uint32_t j = 0; j < h; j++) {
    if (base == kNone || at - base >= 32u) {
      base = at;
      mine = at + threadIdx.x < most && starts[at + threadIdx.x] != kNone ? next[at + threadIdx.x] : kNone;
    }
    if (threadIdx.x == 0) rows[j] = at;
    if (j + 1u == h) {
      if (threadIdx.x == 0 && walked[at].end == 0u) *ok = 0u;
      return;
    }
    at = __shfl_sync(0xffffffffu, mine, at - base);
    if (at == kNone) {
      if (threadIdx.x == 0) *ok = 0u;
      return;
    }
  }
}

/* Run-length expansion of the linked rows, one block per row: its bytes into shared memory, then one warp per
 * plane walks 32 packets, one to a lane, and writes their values: packet by packet when they are long, else 32
 * values at a time, each lane finding its packet by bisection over the lanes (exponents come in packets of a
 * few values: packet by packet they took 44 us).  1024 x 512 of random values, 118,000 packets in 2 MB: 21 us (the walk before it 17). */
__global__ void __launch_bounds__(128) k_rle_rows(const unsigned char *body, const uint32_t *starts,
                                                  const WalkedRow *walked, const uint32_t *rows, int w,
                                                  unsigned char *rgbe, const uint32_t *ok) {
  extern __shared__ uint4 staged[];
  if (*ok == 0u) return;
  const uint32_t i = rows[blockIdx.x], start = starts[i];
  const WalkedRow &r = walked[i];
  stage_row(body, start, r.end - start, staged);
  const unsigned char *sm = reinterpret_cast<const unsigned char *>(staged) + (start & 15u);
  const int lane = threadIdx.x & 31, plane = threadIdx.x >> 5;
  unsigned char *o = rgbe + (size_t)blockIdx.x * w * 4 + plane;
  uint32_t p = r.plane[plane];
  for (int x = 0; x < w;) {
    const int x0 = x;
    int first = INT_MAX; /* the lane's packet: its first value, and where its bytes are (a run's: bit 31) */
    uint32_t src = 0;
    int packets = 0;
    for (; packets < 32 && x < w; packets++) {
      const uint32_t head = sm[p];
      const bool run = head > 128u;
      const uint32_t cnt = run ? head - 128u : head;
      if (lane == packets) first = x, src = (p + 1u) | (run ? 0x80000000u : 0u);
      p += run ? 2u : 1u + cnt;
      x += (int)cnt;
    }
    if (x - x0 >= 32 * packets) { /* long packets: one after the other */
      for (int k = 0; k < packets; k++) {
        const uint32_t from = __shfl_sync(0xffffffffu, src, k);
        const int at = __shfl_sync(0xffffffffu, first, k);
        const int end = k + 1 < packets ? __shfl_sync(0xffffffffu, first, k + 1) : x;
        for (int t = at + lane; t < end; t += 32)
          o[4 * (size_t)t] = sm[(from & 0x7fffffffu) + (from >> 31 ? 0u : (uint32_t)(t - at))];
      }
      continue;
    }
    for (int b = x0; b < x; b += 32) {
      const int t = b + lane;
      int l = 0; /* the last packet that starts at or before t */
      for (int step = 16; step > 0; step >>= 1)
        if (__shfl_sync(0xffffffffu, first, l + step) <= t) l += step;
      const uint32_t from = __shfl_sync(0xffffffffu, src, l);
      const int at = __shfl_sync(0xffffffffu, first, l);
      if (t < x) o[4 * (size_t)t] = sm[(from & 0x7fffffffu) + (from >> 31 ? 0u : (uint32_t)(t - at))];
    }
  }
}

/* ---- host: the file format ----------------------------------------------------------------- */

constexpr int kMaxDim = 1 << 24; /* the largest width / height the loader accepts */

bool rle_width(int w) { return w >= 8 && w < 32768; }

struct Reader {
  const std::vector<unsigned char> &b;
  size_t pos = 0;
  /* reading past the end yields zeros, as the reference's loader does */
  unsigned char get() { return pos < b.size() ? b[pos++] : (unsigned char)0; }
  std::string line() {
    std::string s;
    while (pos < b.size() && b[pos] != '\n' && s.size() < 1023) s.push_back((char)b[pos++]);
    while (pos < b.size() && b[pos] != '\n') pos++; /* an over-long line is cut, the rest skipped */
    if (pos < b.size()) pos++;
    return s;
  }
};

struct Header {
  int w = 0, h = 0;
  size_t data = 0; /* offset of the first scanline byte */
};

/* IO::Loader::loadHdrEnvmap's magic check (Loader_image.cpp:64-90) then the Radiance header as the
 * stb loader parses it: first line "#?RADIANCE" or "#?RGBE", lines up to an empty one with
 * "FORMAT=32-bit_rle_rgbe" among them, then "-Y <height> +X <width>". */
nova_b200_status parse_header(nova_b200_ctx *c, const std::vector<unsigned char> &bytes, Header &hd) {
  using namespace nbctx;
  char magic[32] = {0};
  std::memcpy(magic, bytes.data(), std::min<size_t>(31, bytes.size()));
  if (bytes.size() >= 4 && (unsigned char)magic[0] == 0x76 && (unsigned char)magic[1] == 0x2f &&
      (unsigned char)magic[2] == 0x31 && (unsigned char)magic[3] == 0x01)
    return fail(c, NOVA_B200_INVALID_ARGUMENT, "OpenEXR files are not supported by this library%s");
  if (!std::strstr(magic, "#?RADIANCE"))
    return fail(c, NOVA_B200_INVALID_ARGUMENT, "Must be an HDR/EXR format .%s");
  Reader r{bytes};
  const std::string first = r.line();
  if (first != "#?RADIANCE" && first != "#?RGBE") return fail(c, NOVA_B200_INVALID_ARGUMENT, "not an HDR file%s");
  bool format = false;
  for (;;) {
    if (r.pos >= bytes.size()) return fail(c, NOVA_B200_INVALID_ARGUMENT, "HDR header has no end%s");
    const std::string t = r.line();
    if (t.empty()) break;
    if (t == "FORMAT=32-bit_rle_rgbe") format = true;
  }
  if (!format) return fail(c, NOVA_B200_INVALID_ARGUMENT, "unsupported HDR format (not 32-bit_rle_rgbe)%s");
  const std::string res = r.line();
  const char *p = res.c_str();
  if (std::strncmp(p, "-Y ", 3)) return fail(c, NOVA_B200_INVALID_ARGUMENT, "unsupported HDR data layout%s");
  char *end = nullptr;
  const long h = std::strtol(p + 3, &end, 10);
  p = end;
  while (*p == ' ') p++;
  if (std::strncmp(p, "+X ", 3)) return fail(c, NOVA_B200_INVALID_ARGUMENT, "unsupported HDR data layout%s");
  const long w = std::strtol(p + 3, nullptr, 10);
  if (w <= 0 || h <= 0 || w > kMaxDim || h > kMaxDim)
    return fail(c, NOVA_B200_INVALID_ARGUMENT, "HDR image size out of range%s");
  hd.w = (int)w, hd.h = (int)h, hd.data = r.pos;
  return NOVA_B200_SUCCESS;
}

/* Where the scanlines are.  Rows of a width in [8, 32768) are run-length packets: a row header
 * (2, 2, width >> 8, width & 255), then for each of R, G, B, E packets that are either a run
 * (count + 128, value) or a dump (count, count bytes), count in 1..remaining.  The host walks the
 * packet headers only (one byte per packet; dump data is skipped) to check them and to find where
 * each (row, plane) starts; the device expands them.  A row whose first bytes are not a run-length
 * header means the file is flat from there: those 4 bytes are pixel 0 of row 0 and the rest follow
 * in order (the stb loader's rule, kept as is).  Reading past the end yields zeros. */
struct Layout {
  bool flat = false;
  std::vector<unsigned char> flat_rgbe; /* flat files: the interleaved RGBE pixels */
  std::vector<uint64_t> starts;         /* run-length files: file offset of each (row, plane) */
};

nova_b200_status scan_rows(nova_b200_ctx *c, const std::vector<unsigned char> &bytes, const Header &hd,
                           Layout &L) {
  using namespace nbctx;
  const size_t w = (size_t)hd.w, h = (size_t)hd.h;
  Reader r{bytes, hd.data};
  auto flat_from = [&](size_t first_byte) {
    L.flat = true;
    L.flat_rgbe.assign(w * h * 4, 0);
    const size_t avail = r.pos < bytes.size() ? bytes.size() - r.pos : 0;
    const size_t n = std::min(avail, w * h * 4 - first_byte);
    if (n) std::memcpy(&L.flat_rgbe[first_byte], &bytes[r.pos], n);
  };
  if (!rle_width(hd.w)) {
    flat_from(0);
    return NOVA_B200_SUCCESS;
  }
  L.starts.resize(4 * h);
  for (size_t j = 0; j < h; j++) {
    const unsigned char c1 = r.get(), c2 = r.get(), c3 = r.get();
    if (c1 != 2 || c2 != 2 || (c3 & 0x80)) {
      const unsigned char c4 = r.get();
      flat_from(4);
      L.flat_rgbe[0] = c1, L.flat_rgbe[1] = c2, L.flat_rgbe[2] = c3, L.flat_rgbe[3] = c4;
      return NOVA_B200_SUCCESS;
    }
    const size_t len = ((size_t)c3 << 8) | r.get();
    if (len != w) return fail(c, NOVA_B200_INVALID_ARGUMENT, "invalid decoded scanline length%s");
    for (int k = 0; k < 4; k++) {
      L.starts[4 * j + k] = r.pos;
      size_t i = 0;
      while (i < w) {
        unsigned count = r.get();
        const size_t left = w - i;
        const bool run = count > 128;
        if (run) count -= 128;
        if (count == 0 || count > left) return fail(c, NOVA_B200_INVALID_ARGUMENT, "bad RLE data in HDR%s");
        if (run)
          r.get();
        else
          r.pos = std::min(r.pos + count, bytes.size() + 256); /* dump data: skipped, zeros past the end */
        i += count;
      }
    }
  }
  return NOVA_B200_SUCCESS;
}

/* Opens a file, unbuffered (it is read in large pieces), and reads all of its `size` bytes up to `whole`, else the
 * first kHeadBytes. */
constexpr size_t kHeadBytes = 1 << 16;

nova_b200_status read_head(nova_b200_ctx *c, const char *path, std::ifstream &f, size_t whole,
                           std::vector<unsigned char> &bytes, size_t &size) {
  using namespace nbctx;
  if (!path) return fail(c, NOVA_B200_INVALID_ARGUMENT, "path is null%s");
  f.rdbuf()->pubsetbuf(nullptr, 0);
  f.open(path, std::ios::binary | std::ios::ate);
  if (!f) return fail(c, NOVA_B200_INVALID_ARGUMENT, "cannot open %s", path);
  const std::streamoff end = f.tellg();
  if (end < 0) return fail(c, NOVA_B200_INVALID_ARGUMENT, "cannot read %s", path);
  size = (size_t)end;
  bytes.resize(size <= whole ? size : std::min(size, kHeadBytes));
  f.seekg(0);
  if (!bytes.empty() && !f.read(reinterpret_cast<char *>(bytes.data()), (std::streamsize)bytes.size()))
    return fail(c, NOVA_B200_INVALID_ARGUMENT, "cannot read %s", path);
  return NOVA_B200_SUCCESS;
}

/* The rest of a file whose head is in `bytes`. */
nova_b200_status read_rest(nova_b200_ctx *c, const char *path, std::ifstream &f, std::vector<unsigned char> &bytes,
                           size_t size) {
  const size_t have = bytes.size();
  if (size <= have) return NOVA_B200_SUCCESS;
  bytes.resize(size);
  f.clear();
  f.seekg((std::streamoff)have);
  if (!f.read(reinterpret_cast<char *>(bytes.data() + have), (std::streamsize)(size - have)))
    return nbctx::fail(c, NOVA_B200_INVALID_ARGUMENT, "cannot read %s", path);
  return NOVA_B200_SUCCESS;
}

nova_b200_status check_read(nova_b200_ctx *c, const Header &hd, const float *rgba_device, uint64_t capacity) {
  using namespace nbctx;
  const uint64_t npx = (uint64_t)hd.w * hd.h;
  if (npx > (1ull << 31)) return fail(c, NOVA_B200_INVALID_ARGUMENT, "HDR image larger than 2^31 pixels%s");
  if (capacity < npx * 4) return fail(c, NOVA_B200_INVALID_ARGUMENT, "output holds fewer than width * height * 4 floats%s");
  if (rgba_device && (reinterpret_cast<uintptr_t>(rgba_device) & 15))
    return fail(c, NOVA_B200_INVALID_ARGUMENT, "rgba_device must be 16-byte aligned%s");
  return NOVA_B200_SUCCESS;
}

/* hdr_read of a run-length file of more than kDeviceBytes or kDevicePixels: the bytes go to the device in pieces
 * as they are read, and the device finds, checks and expands the rows.  *done stays false when this is no
 * such file, or one whose rows it could not chain: nothing has been written then, and the caller reads
 * the file the other way, which also says what is wrong with it.
 *
 * The other way's walk of the packets on the host costs 2.5 ns a packet, this one five short kernels and their
 * gaps.  Random values (few packets a byte): 128 KB 83 us the other way and 101 this way, 320 KB 121 and 120,
 * 513 KB 155 and 136, 2 MB 555 and 317, 32 MB 8.4 and 3.1 ms; one colour (66 values a byte, so the pixels
 * tell): 0.5 Mpixel 81 and 92, 2 Mpixel 160 and 120, 8 Mpixel 450 and 241.  Pieces of 64 to 256 KB are
 * slower and uneven (2 MB: 330 to 370 us), pinned ones 290, but pinning 1 MB costs a new context 1.3 ms. */
constexpr size_t kFilePiece = 1 << 20, kRowSmem = 200 << 10;
constexpr size_t kDeviceBytes = 5 << 16, kDevicePixels = 1 << 20;

nova_b200_status read_rows_on_device(nova_b200_ctx *c, std::ifstream &f, const std::vector<unsigned char> &head,
                                     const Header &hd, size_t size, float *rgba_host, float *rgba_device,
                                     uint64_t capacity, bool *done) {
  using namespace nbctx;
  *done = false;
  if (size <= kHeadBytes || hd.data + 4 > head.size() || !rle_width(hd.w)) return NOVA_B200_SUCCESS;
  const uint32_t pattern = 2u | 2u << 8 | (uint32_t)(hd.w >> 8) << 16 | (uint32_t)(hd.w & 255) << 24;
  uint32_t word;
  std::memcpy(&word, &head[hd.data], 4);
  const uint64_t n = size - hd.data;
  if (n <= kDeviceBytes && (uint64_t)hd.w * hd.h < kDevicePixels) return NOVA_B200_SUCCESS;
  if (word != pattern || n >= 0xffffffffull || n < 4ull * (uint64_t)hd.h) return NOVA_B200_SUCCESS;
  nova_b200_status st = check_read(c, hd, rgba_device, capacity);
  if (st) return st;
  cudaSetDevice(c->device);
  const uint64_t npx = (uint64_t)hd.w * hd.h;
  const uint32_t h = (uint32_t)hd.h;
  const uint64_t tiles = (n + kFindTile - 1) / kFindTile, per = (tiles + kFindBlocks - 1) / kFindBlocks;
  const uint32_t chunk = (uint32_t)(per * kFindTile), blocks = (uint32_t)((tiles + per - 1) / per);
  const uint32_t cap = (uint32_t)std::min<size_t>((8 * (size_t)hd.w + 4 + 15 + 15) & ~(size_t)15, kRowSmem);
  unsigned char *d_body = nullptr, *d_rgbe = nullptr;
  /* positions taken for rows; packet data that looks like one is rare, and the rest is left to the host */
  const uint32_t most = (uint32_t)std::min<uint64_t>((uint64_t)h + h / 2 + 1024, n / 4);
  WalkedRow *d_walked = nullptr;
  uint32_t *d_ok = nullptr;
  float4 *d_out = reinterpret_cast<float4 *>(rgba_device), *tmp = nullptr;
  cudaError_t e = cudaMallocAsync(&d_body, n + 256, c->stream);
  if (e == cudaSuccess) e = cudaMallocAsync(&d_rgbe, npx * 4, c->stream);
  if (e == cudaSuccess) e = cudaMallocAsync(&d_walked, sizeof(WalkedRow) * most, c->stream);
  if (e == cudaSuccess) e = cudaMallocAsync(&d_ok, sizeof(uint32_t) * (1 + 2 * (size_t)most + h + blocks), c->stream);
  uint32_t *d_starts = d_ok + 1, *d_next = d_starts + most, *d_rows = d_next + most, *d_counts = d_rows + h;
  if (e == cudaSuccess && !d_out) {
    e = cudaMallocAsync(&tmp, npx * sizeof(float4), c->stream);
    d_out = tmp;
  }
  if (e == cudaSuccess) e = cudaMemsetAsync(d_body + n, 0, 256, c->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(d_ok, 0xff, sizeof(uint32_t) * (1 + (size_t)most), c->stream);
  bool read = true;
  const uint64_t held = head.size() - hd.data; /* bytes of the body that have been read */
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_body, &head[hd.data], held, cudaMemcpyHostToDevice, c->stream);
  const std::unique_ptr<char[]> piece(new char[(size_t)std::min<uint64_t>(n - held, kFilePiece)]);
  for (uint64_t off = held; e == cudaSuccess && read && off < n; off += kFilePiece) {
    const size_t bytes = (size_t)std::min<uint64_t>(kFilePiece, n - off);
    read = (bool)f.read(piece.get(), (std::streamsize)bytes);
    if (read) e = cudaMemcpyAsync(d_body + off, piece.get(), bytes, cudaMemcpyHostToDevice, c->stream);
  }
  uint32_t ok = 0;
  if (e == cudaSuccess && read) {
    cudaEventRecord(c->ev_begin, c->stream);
    const unsigned char *body = d_body;
    k_rle_find<false><<<blocks, kFindThreads, 0, c->stream>>>(body, (uint32_t)n, pattern, chunk, d_counts, most, d_starts);
    k_rle_find<true><<<blocks, kFindThreads, 0, c->stream>>>(body, (uint32_t)n, pattern, chunk, d_counts, most, d_starts);
    for (const void *kernel : {(const void *)k_rle_walk, (const void *)k_rle_rows})
      if (cap > 48 << 10 && e == cudaSuccess)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowSmem);
    if (e == cudaSuccess) {
      k_rle_walk<<<most, 128, cap, c->stream>>>(body, (uint32_t)n, d_starts, hd.w, cap, d_walked);
      k_rle_link<<<1, 1024, 0, c->stream>>>(d_starts, d_walked, most, h, d_next, d_rows, d_ok);
      k_rle_rows<<<h, 128, cap, c->stream>>>(body, d_starts, d_walked, d_rows, hd.w, d_rgbe, d_ok);
      k_rgbe_decode<<<(unsigned)((npx + 1023) / 1024), 256, 0, c->stream>>>(
          reinterpret_cast<const uint32_t *>(d_rgbe), npx, d_out, d_ok);
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    cudaEventRecord(c->ev_end, c->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(c->h_counters, d_ok, sizeof(uint32_t), cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e == cudaSuccess) ok = c->h_counters[0];
    if (ok && rgba_host)
      e = cudaMemcpyAsync(rgba_host, d_out, npx * sizeof(float4), cudaMemcpyDeviceToHost, c->stream);
  }
  for (void *ptr : {(void *)d_body, (void *)d_rgbe, (void *)d_walked, (void *)d_ok, (void *)tmp})
    if (ptr) cudaFreeAsync(ptr, c->stream);
  const cudaError_t synced = cudaStreamSynchronize(c->stream);
  if (e == cudaSuccess) e = synced;
  if (e != cudaSuccess) return cuda_fail(c, e, "hdr_read");
  *done = ok != 0;
  return NOVA_B200_SUCCESS;
}

nova_b200_status check_ctx(nova_b200_ctx *c) { return c ? NOVA_B200_SUCCESS : NOVA_B200_INVALID_ARGUMENT; }

}  // namespace

extern "C" nova_b200_status nova_b200_film_accumulate(nova_b200_ctx *c, const float *partial, float *accum,
                                                      float *final_buf, uint64_t n, uint32_t frame_index) {
  using namespace nbctx;
  if (check_ctx(c)) return NOVA_B200_INVALID_ARGUMENT;
  if (!partial || !accum) return fail(c, NOVA_B200_INVALID_ARGUMENT, "null buffer%s");
  if ((reinterpret_cast<uintptr_t>(partial) | reinterpret_cast<uintptr_t>(accum) |
       reinterpret_cast<uintptr_t>(final_buf)) & 15)
    return fail(c, NOVA_B200_INVALID_ARGUMENT, "film buffers must be 16-byte aligned%s");
  if (n == 0) return NOVA_B200_SUCCESS;
  cudaSetDevice(c->device);
  const uint64_t threads = (n + 3) / 4;
  cudaEventRecord(c->ev_begin, c->stream);
  k_accumulate<<<(unsigned)((threads + 255) / 256), 256, 0, c->stream>>>(partial, accum, final_buf, n,
                                                                          (float)(frame_index + 1));
  NB_CUDA(c, cudaGetLastError(), "k_accumulate");
  cudaEventRecord(c->ev_end, c->stream);
  NB_CUDA(c, cudaStreamSynchronize(c->stream), "film_accumulate");
  return NOVA_B200_SUCCESS;
}

extern "C" nova_b200_status nova_b200_display_blend(nova_b200_ctx *c, const float *partial, const float *accum,
                                                    float *out, uint64_t n, uint32_t current_frame) {
  using namespace nbctx;
  if (check_ctx(c)) return NOVA_B200_INVALID_ARGUMENT;
  if (!partial || !accum || !out) return fail(c, NOVA_B200_INVALID_ARGUMENT, "null buffer%s");
  if ((reinterpret_cast<uintptr_t>(partial) | reinterpret_cast<uintptr_t>(accum) | reinterpret_cast<uintptr_t>(out)) &
      15)
    return fail(c, NOVA_B200_INVALID_ARGUMENT, "film buffers must be 16-byte aligned%s");
  if (n == 0) return NOVA_B200_SUCCESS;
  cudaSetDevice(c->device);
  const uint64_t threads = (n + 3) / 4;
  cudaEventRecord(c->ev_begin, c->stream);
  k_display_blend<<<(unsigned)((threads + 255) / 256), 256, 0, c->stream>>>(partial, accum, out, n,
                                                                             (float)(current_frame + 1));
  NB_CUDA(c, cudaGetLastError(), "k_display_blend");
  cudaEventRecord(c->ev_end, c->stream);
  NB_CUDA(c, cudaStreamSynchronize(c->stream), "display_blend");
  return NOVA_B200_SUCCESS;
}

extern "C" nova_b200_status nova_b200_snapshot(nova_b200_ctx *c, const float *film, int32_t w, int32_t h,
                                               int32_t channels, float *dst, int32_t dw, int32_t dh) {
  using namespace nbctx;
  if (check_ctx(c)) return NOVA_B200_INVALID_ARGUMENT;
  if (!film || !dst) return fail(c, NOVA_B200_INVALID_ARGUMENT, "null buffer%s");
  if (w <= 0 || h <= 0 || dw <= 0 || dh <= 0 || w > kMaxDim || h > kMaxDim || dw > kMaxDim || dh > 65535)
    return fail(c, NOVA_B200_INVALID_ARGUMENT, "invalid snapshot size%s");
  if (channels < 3 || channels > 4) return fail(c, NOVA_B200_INVALID_ARGUMENT, "channels must be 3 or 4%s");
  cudaSetDevice(c->device);
  cudaEventRecord(c->ev_begin, c->stream);
  k_snapshot<<<dim3((unsigned)((dw + 127) / 128), (unsigned)dh), 128, 0, c->stream>>>(Film{film, w, h, channels}, dst,
                                                                                    dw, dh);
  NB_CUDA(c, cudaGetLastError(), "k_snapshot");
  cudaEventRecord(c->ev_end, c->stream);
  NB_CUDA(c, cudaStreamSynchronize(c->stream), "snapshot");
  return NOVA_B200_SUCCESS;
}

extern "C" nova_b200_status nova_b200_hdr_info(nova_b200_ctx *c, const char *path, int32_t *width, int32_t *height) {
  /* the header from the first 64 KB; the whole file only when the header runs past them */
  std::vector<unsigned char> bytes;
  std::ifstream f;
  size_t size = 0;
  nova_b200_status st = read_head(c, path, f, 0, bytes, size);
  if (st) return st;
  Header hd;
  st = parse_header(c, bytes, hd);
  if (bytes.size() < size && (st || hd.data >= bytes.size())) {
    if ((st = read_rest(c, path, f, bytes, size))) return st;
    st = parse_header(c, bytes, hd);
  }
  if (st) return st;
  if (width) *width = hd.w;
  if (height) *height = hd.h;
  return NOVA_B200_SUCCESS;
}

extern "C" nova_b200_status nova_b200_hdr_read(nova_b200_ctx *c, const char *path, float *rgba_host,
                                               float *rgba_device, uint64_t capacity) {
  using namespace nbctx;
  if (check_ctx(c)) return NOVA_B200_INVALID_ARGUMENT;
  std::ifstream f;
  std::vector<unsigned char> bytes;
  size_t size = 0;
  /* a file that the host's walk takes unless it has many pixels is read at once: in two pieces, with the header
   * parsed for each, 320 x 240 took 3 us more of 138 */
  nova_b200_status st = read_head(c, path, f, kDeviceBytes, bytes, size);
  if (st) return st;
  Header hd;
  st = parse_header(c, bytes, hd);
  if (!st) {
    bool done = false;
    st = read_rows_on_device(c, f, bytes, hd, size, rgba_host, rgba_device, capacity, &done);
    if (st || done) return st;
  }
  if (bytes.size() < size) {
    if ((st = read_rest(c, path, f, bytes, size))) return st;
    st = parse_header(c, bytes, hd);
  }
  if (st) return st;
  if ((st = check_read(c, hd, rgba_device, capacity))) return st;
  const uint64_t npx = (uint64_t)hd.w * hd.h;
  Layout L;
  if ((st = scan_rows(c, bytes, hd, L))) return st;
  cudaSetDevice(c->device);
  const int n_planes = 4 * hd.h;
  /* run-length files: the body (padded with zeros) and the plane offsets go to the device */
  const size_t body_n = L.flat ? 0 : bytes.size() - hd.data + 256;
  unsigned char *d_rgbe = nullptr, *d_body = nullptr;
  uint64_t *d_starts = nullptr;
  float4 *d_out = reinterpret_cast<float4 *>(rgba_device), *tmp = nullptr;
  NB_CUDA(c, cudaMallocAsync(&d_rgbe, npx * 4, c->stream), "cudaMalloc(hdr bytes)");
  cudaError_t e = cudaSuccess;
  if (L.flat) {
    e = cudaMemcpyAsync(d_rgbe, L.flat_rgbe.data(), npx * 4, cudaMemcpyHostToDevice, c->stream);
  } else {
    const size_t file_n = bytes.size() - hd.data;
    for (auto &o : L.starts) o -= hd.data;
    e = cudaMallocAsync(&d_body, body_n, c->stream);
    if (e == cudaSuccess) e = cudaMallocAsync(&d_starts, n_planes * sizeof(uint64_t), c->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(d_body + file_n, 0, body_n - file_n, c->stream);
    if (e == cudaSuccess && file_n)
      e = cudaMemcpyAsync(d_body, bytes.data() + hd.data, file_n, cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(d_starts, L.starts.data(), n_planes * sizeof(uint64_t), cudaMemcpyHostToDevice, c->stream);
  }
  if (e == cudaSuccess && !d_out) {
    e = cudaMallocAsync(&tmp, npx * sizeof(float4), c->stream);
    d_out = tmp;
  }
  if (e == cudaSuccess) {
    cudaEventRecord(c->ev_begin, c->stream);
    if (!L.flat)
      k_rle_unpack<<<(unsigned)(((uint64_t)n_planes * 32 + 127) / 128), 128, 0, c->stream>>>(d_body, d_starts, hd.w,
                                                                                               n_planes, d_rgbe);
    const uint64_t threads = (npx + 3) / 4;
    k_rgbe_decode<<<(unsigned)((threads + 255) / 256), 256, 0, c->stream>>>(reinterpret_cast<const uint32_t *>(d_rgbe),
                                                                              npx, d_out, nullptr);
    e = cudaGetLastError();
    cudaEventRecord(c->ev_end, c->stream);
  }
  if (e == cudaSuccess && rgba_host)
    e = cudaMemcpyAsync(rgba_host, d_out, npx * sizeof(float4), cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  cudaFreeAsync(d_rgbe, c->stream);
  if (d_body) cudaFreeAsync(d_body, c->stream);
  if (d_starts) cudaFreeAsync(d_starts, c->stream);
  if (tmp) cudaFreeAsync(tmp, c->stream);
  if (e != cudaSuccess) return cuda_fail(c, e, "hdr_read");
  NB_CUDA(c, cudaStreamSynchronize(c->stream), "hdr_read");
  return NOVA_B200_SUCCESS;
}

extern "C" nova_b200_status nova_b200_hdr_write(nova_b200_ctx *c, const char *path, const float *pixels_host,
                                                const float *pixels_device, int32_t w, int32_t h, int32_t channels,
                                                int32_t flip) {
  using namespace nbctx;
  if (check_ctx(c)) return NOVA_B200_INVALID_ARGUMENT;
  if (!path) return fail(c, NOVA_B200_INVALID_ARGUMENT, "path is null%s");
  if (!pixels_host && !pixels_device) return fail(c, NOVA_B200_INVALID_ARGUMENT, "no pixels%s");
  if (w <= 0 || h <= 0 || w > kMaxDim || h > 65535) return fail(c, NOVA_B200_INVALID_ARGUMENT, "invalid image size%s");
  if (channels < 1 || channels > 4) return fail(c, NOVA_B200_INVALID_ARGUMENT, "channels must be 1 to 4%s");
  const uint64_t npx = (uint64_t)w * h;
  const bool rle = rle_width(w);
  const bool vec4 = channels == 4 && !(reinterpret_cast<uintptr_t>(pixels_device) & 15);
  cudaSetDevice(c->device);
  const int n_planes = 4 * h;
  const int cap = w + w / 64 + 8; /* > width + width / 128 + 2, the most packets a row plane takes */
  const size_t regions_n = rle ? (size_t)n_planes * cap : 0, out_cap = rle ? regions_n + 4 * (size_t)h : npx * 4;
  unsigned char *d_rgbe = nullptr, *d_regions = nullptr, *d_out = nullptr;
  uint32_t *d_sizes = nullptr;
  uint64_t *d_offsets = nullptr;
  unsigned *d_err = nullptr;
  float *d_src = const_cast<float *>(pixels_device), *tmp = nullptr;
  NB_CUDA(c, cudaMallocAsync(&d_rgbe, npx * 4, c->stream), "cudaMalloc(hdr bytes)");
  cudaError_t e = cudaSuccess;
  if (!d_src) {
    e = cudaMallocAsync(&tmp, npx * channels * sizeof(float), c->stream);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(tmp, pixels_host, npx * channels * sizeof(float), cudaMemcpyHostToDevice, c->stream);
    d_src = tmp;
  }
  if (rle) {
    if (e == cudaSuccess) e = cudaMallocAsync(&d_regions, regions_n, c->stream);
    if (e == cudaSuccess) e = cudaMallocAsync(&d_out, out_cap, c->stream);
    if (e == cudaSuccess) e = cudaMallocAsync(&d_sizes, n_planes * sizeof(uint32_t), c->stream);
    if (e == cudaSuccess) e = cudaMallocAsync(&d_offsets, (n_planes + 1) * sizeof(uint64_t) + 16, c->stream);
    if (e == cudaSuccess) {
      d_err = reinterpret_cast<unsigned *>(d_offsets + n_planes + 1);
      e = cudaMemsetAsync(d_err, 0, sizeof(unsigned), c->stream);
    }
  }
  if (e == cudaSuccess) {
    cudaEventRecord(c->ev_begin, c->stream);
    k_rgbe_encode<<<dim3((unsigned)((w + 127) / 128), (unsigned)h), 128, 0, c->stream>>>(
        d_src, w, h, channels, flip, rle ? 1 : 0, (vec4 || (tmp && channels == 4)) ? 1 : 0, d_rgbe);
    if (rle) {
      k_rle_pack<<<(unsigned)(((uint64_t)n_planes * 32 + 127) / 128), 128, 0, c->stream>>>(d_rgbe, w, n_planes, cap,
                                                                                             d_regions, d_sizes, d_err);
      k_rle_scan<<<1, 1024, 0, c->stream>>>(d_sizes, n_planes, d_offsets);
      k_rle_gather<<<(unsigned)(((uint64_t)n_planes * 32 + 255) / 256), 256, 0, c->stream>>>(
          d_regions, d_sizes, d_offsets, w, cap, n_planes, d_out);
    }
    e = cudaGetLastError();
    cudaEventRecord(c->ev_end, c->stream);
  }
  /* the packed size and the overflow flag, then exactly the packed bytes */
  uint64_t tail[2] = {npx * 4, 0};
  if (e == cudaSuccess && rle)
    e = cudaMemcpyAsync(tail, d_offsets + n_planes, sizeof(uint64_t) + sizeof(unsigned), cudaMemcpyDeviceToHost,
                        c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  std::string out = "#?RADIANCE\n# nova_b200\nFORMAT=32-bit_rle_rgbe\n\n-Y " + std::to_string(h) + " +X " +
                    std::to_string(w) + "\n";
  const size_t head_n = out.size(), body_n = (size_t)tail[0];
  const bool overflow = rle && (uint32_t)tail[1] != 0;
  if (e == cudaSuccess && !overflow && body_n <= out_cap) {
    out.resize(head_n + body_n);
    e = cudaMemcpyAsync(&out[head_n], rle ? d_out : d_rgbe, body_n, cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  }
  for (void *ptr : {(void *)d_rgbe, (void *)d_regions, (void *)d_out, (void *)d_sizes, (void *)d_offsets, (void *)tmp})
    if (ptr) cudaFreeAsync(ptr, c->stream);
  if (e != cudaSuccess) return cuda_fail(c, e, "hdr_write");
  if (overflow || body_n > out_cap) return fail(c, NOVA_B200_RENDERER_EXCEPTION, "run-length packing overflow%s");
  /* IO::Loader::writeHdr appends the extension (Loader_image.cpp:51-52) */
  const std::string file = std::string(path) + ".hdr";
  std::ofstream f(file, std::ios::binary);
  if (!f) return fail(c, NOVA_B200_INVALID_ARGUMENT, "cannot write %s", file.c_str());
  f.write(out.data(), (std::streamsize)out.size());
  if (!f) return fail(c, NOVA_B200_RENDERER_EXCEPTION, "write failed: %s", file.c_str());
  return NOVA_B200_SUCCESS;
}

extern "C" nova_b200_status nova_b200_bake_texture(nova_b200_ctx *c, const char *type, int32_t out_w, int32_t out_h,
                                                   int32_t samples, const char *path_in, const char *path_out) {
  return nova_b200_bake_texture_flags(c, type, out_w, out_h, samples, path_in, path_out, 0u);
}

extern "C" nova_b200_status nova_b200_bake_texture_flags(nova_b200_ctx *c, const char *type, int32_t out_w,
                                                         int32_t out_h, int32_t samples, const char *path_in,
                                                         const char *path_out, uint32_t flags) {
  using namespace nbctx;
  if (check_ctx(c)) return NOVA_B200_INVALID_ARGUMENT;
  if (!type || std::strcmp(type, "irradiance") != 0)
    return fail(c, NOVA_B200_INVALID_ARGUMENT, "bake type must be \"irradiance\"%s");
  auto pow2 = [](int32_t v) { return v > 0 && (v & (v - 1)) == 0; };
  if (!pow2(out_w) || !pow2(out_h))
    return fail(c, NOVA_B200_INVALID_ARGUMENT, "irradiance size must be a power of two (TextureProcessing.cpp:11)%s");
  if (samples <= 0) return fail(c, NOVA_B200_INVALID_ARGUMENT, "samples must be positive%s");
  if (!path_out) return fail(c, NOVA_B200_INVALID_ARGUMENT, "path_out is null%s");
  int32_t w = 0, h = 0;
  nova_b200_status st = nova_b200_hdr_info(c, path_in, &w, &h);
  if (st) return st;
  cudaSetDevice(c->device);
  const size_t src_n = (size_t)w * h * 4, out_n = (size_t)out_w * out_h * 4;
  float *src = nullptr, *out = nullptr;
  NB_CUDA(c, cudaMallocAsync(&src, src_n * sizeof(float), c->stream), "cudaMalloc(environment map)");
  cudaError_t e = cudaMallocAsync(&out, out_n * sizeof(float), c->stream);
  /* the reference's output starts as zeros and its alpha channel is never written */
  if (e == cudaSuccess) e = cudaMemsetAsync(out, 0, out_n * sizeof(float), c->stream);
  if (e != cudaSuccess) {
    cudaFreeAsync(src, c->stream);
    return cuda_fail(c, e, "cudaMalloc(irradiance map)");
  }
  st = nova_b200_hdr_read(c, path_in, nullptr, src, src_n);
  if (!st)
    st = (flags & NOVA_B200_BAKE_GPU_KERNEL) ? nb_bake_texunit(c, src, w, h, 4, out_w, out_h, samples, out)
                                             : nb_bake(c, src, w, h, 4, out_w, out_h, samples, out);
  if (!st) st = nova_b200_hdr_write(c, path_out, nullptr, out, out_w, out_h, 4, 0);
  cudaFreeAsync(src, c->stream);
  cudaFreeAsync(out, c->stream);
  cudaStreamSynchronize(c->stream);
  return st;
}

extern "C" nova_b200_status nova_b200_last_call_ms(nova_b200_ctx *c, float *device_ms) {
  using namespace nbctx;
  if (check_ctx(c) || !device_ms) return NOVA_B200_INVALID_ARGUMENT;
  cudaSetDevice(c->device);
  NB_CUDA(c, cudaEventElapsedTime(device_ms, c->ev_begin, c->ev_end), "last_call_ms");
  return NOVA_B200_SUCCESS;
}
