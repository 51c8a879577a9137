/* Diffuse irradiance bake of an equirectangular float environment map on the device.
 *
 * Follows the reference's CPU path (sources/processing/TextureProcessing.cpp:10-64,
 * TextureProcessing.h:174-303) so results match it texel for texel: one thread per output texel
 * (x, y) -> direction from (x / W, y / H) -> tangent frame with right = (1, 0, 0) -> `samples`
 * cosine-weighted directions from the pgc3d hash (math_importance_sampling.h:7-22) seeded with the
 * texel's own approximate spherical pixel -> approximate spherical uv (atan2 polynomial, acos
 * table) -> bilinear source lookup with wrap-around -> mean.  The output keeps the source's
 * channel stride; channel 3 is left untouched (the reference never writes it).
 *
 * The reference's CUDA kernel (sources/processing/cuda/CubemapProcessing.cu:129-175) differs from
 * its CPU path (hash seeded with the output texel, exact acos/atan2, hardware filtering); this
 * kernel reproduces the CPU path, which is the one the oracle restates.
 */
#include <algorithm>

#include "context.cuh"
#include "shading.cuh"

namespace {

using namespace nb;

/* float -> unsigned as compiled x86-64 code does it (64-bit truncation, low 32 bits kept), so
 * negative coordinates seed the hash the same way. */
__device__ __forceinline__ unsigned to_pixel(float coord, unsigned dim) {
  return (unsigned)(long long)(coord * (float)dim);
}

__device__ __forceinline__ void pgc3d(unsigned x, unsigned y, unsigned z, float out[3]) {
  x = x * 1664525u + 1013904223u;
  y = y * 1664525u + 1013904223u;
  z = z * 1664525u + 1013904223u;
  x += y * z;
  y += z * x;
  z += x * y;
  x ^= x >> 16u;
  y ^= y >> 16u;
  z ^= z >> 16u;
  x += y * z;
  y += z * x;
  z += x * y;
  out[0] = __uint2float_rn(x) * kOneOverUintMax;
  out[1] = __uint2float_rn(y) * kOneOverUintMax;
  out[2] = __uint2float_rn(z) * kOneOverUintMax;
}

struct Src {
  const float *data;
  int w, h, ch;
  bool vec4; /* 4 channels on a 16-byte aligned base: one 16-byte load per texel instead of three */
  __device__ V3 texel(int x, int y) const {
    int xc = x >= w ? x % w : (x < 0 ? w + (x % w) : x);
    int yc = y >= h ? y % h : (y < 0 ? h + (y % h) : y);
    const size_t i = (size_t)yc * w + xc;
    if (vec4) { /* the lookups scatter (each texel hashes its own directions): fewer L1 wavefronts */
      const float4 q = __ldg(reinterpret_cast<const float4 *>(data) + i);
      return {q.x, q.y, q.z};
    }
    const float *p = data + i * ch;
    return {__ldg(p), __ldg(p + 1), __ldg(p + 2)};
  }
  /* FINITE: no texel of the map is infinite or NaN, and both sizes are below 2^23.  The filter's
   * coordinates are whole pixels, so its weights are 1, 0, 0, 0; with finite neighbours the three
   * products with 0 add a zero, and the value is the first texel's. */
  template <bool FINITE>
  __device__ V3 uv_sample(float u, float v) const {
    float ui = floorf(u), vi = floorf(v);
    float uw = (u > 1.f || u < 0.f) ? u - ui : u;
    float vw = (v > 1.f || v < 0.f) ? v - vi : v;
    if constexpr (FINITE) return texel((int)to_pixel(uw, (unsigned)w), (int)to_pixel(vw, (unsigned)h));
    float px = (float)(double)to_pixel(uw, (unsigned)w);
    float py = (float)(double)to_pixel(vw, (unsigned)h);
    float tlx = floorf(px), tly = floorf(py), trx = floorf(px) + 1, bly = floorf(py) + 1;
    const float fu = (px - tlx) / (trx - tlx);
    const float fv = (py - tly) / (bly - tly);
    const float hd = 1 - fu;
    V3 tl = texel((int)tlx, (int)tly), tr = texel((int)trx, (int)tly);
    V3 bl = texel((int)tlx, (int)bly), br = texel((int)trx, (int)bly);
    V3 top = hd * tl + fu * tr;
    V3 bot = hd * bl + fu * br;
    return (1 - fv) * top + fv * bot;
  }
};

__device__ __forceinline__ void to_uv(const float *lut, float x, float y, float z, float &u, float &v) {
  float phi = atan2_approx(y, x);
  float theta = acos_lt(lut, z);
  u = (float)((double)phi * kInv2PiD);
  v = (float)((double)theta * kInvPiD);
}

/* *flag = 1 when a component of the map (n floats, n4 of them as float4) is infinite or NaN. */
__global__ void k_any_nonfinite(const float *data, size_t n, size_t n4, unsigned *flag) {
  bool bad = false;
  const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x, step = gridDim.x * (size_t)blockDim.x;
  for (size_t i = t; i < n4; i += step) {
    const float4 q = __ldg(reinterpret_cast<const float4 *>(data) + i);
    bad |= !(isfinite(q.x) && isfinite(q.y) && isfinite(q.z) && isfinite(q.w));
  }
  for (size_t i = 4 * n4 + t; i < n; i += step) bad |= !isfinite(__ldg(data + i));
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) *flag = 1u;
}

/* The frame of an output texel and the hash seed of its directions. */
struct TexelFrame {
  V3 tangent, bitangent, normal;
  unsigned px, py;
};

/* sin and cos, each rounded once, of theta = asin(x) rounded to float, x in [0, 1].  Instead of two
 * evaluations at theta: x and sqrt(1 - x^2) are the sine and cosine of asin(x), and the rounding moved
 * the angle by d < 2^-24, whose third-order terms lie far below double precision. */
__device__ __forceinline__ void sincos_of_asin(float x, float &s, float &c) {
  const double X = (double)x, a = asin(X);
  const float theta = (float)a;
  if (x >= 1.f) { /* the cosine is the rounding's alone */
    s = sin_rn(theta);
    c = cos_rn(theta);
    return;
  }
  const double d = (double)theta - a, C = sqrt((1.0 - X) * (1.0 + X)), h = 0.5 * d * d;
  s = (float)(X + (C * d - X * h));
  c = (float)(C - (X * d + C * h));
}

template <bool FINITE>
__device__ __forceinline__ V3 bake_sample(const Src &src, const float *lut, const TexelFrame &f, unsigned s) {
  float r[3];
  pgc3d(f.px, f.py, s, r);
  const float phi = (float)(2.0 * kPiD * (double)r[0]);
  float sth, cth, sph, cph;
  sincos_of_asin(sqrtf(r[1]), sth, cth);
  sincos_rn(phi, sph, cph);
  V3 cdir{sth * cph, sth * sph, cth};
  cdir = cdir.x * f.tangent + cdir.y * f.bitangent + cdir.z * f.normal;
  float su, sv;
  to_uv(lut, cdir.x, cdir.y, cdir.z, su, sv);
  return src.uv_sample<FINITE>(su, sv);
}

/* The mean of a texel's samples: the G lanes of its group take every G-th sample and add the group's
 * values in sample order (each lane all of them), so the sum is the serial one. */
template <bool FINITE, int G>
__device__ __forceinline__ V3 bake_sum(const Src &src, const float *lut, const TexelFrame &f, unsigned samples) {
  const unsigned lane = threadIdx.x & (G - 1);
  V3 irr{0.f, 0.f, 0.f};
  unsigned s = 0;
  for (; s + G <= samples; s += G) {
    const V3 v = bake_sample<FINITE>(src, lut, f, s + lane);
#pragma unroll
    for (int k = 0; k < G; k++)
      irr = irr + V3{__shfl_sync(0xffffffffu, v.x, k, G), __shfl_sync(0xffffffffu, v.y, k, G),
                     __shfl_sync(0xffffffffu, v.z, k, G)};
  }
  if (s < samples) { /* the last group's lanes past the end add nothing */
    const V3 v = bake_sample<FINITE>(src, lut, f, s + lane);
    for (unsigned k = 0; s + k < samples; k++)
      irr = irr + V3{__shfl_sync(0xffffffffu, v.x, k, G), __shfl_sync(0xffffffffu, v.y, k, G),
                     __shfl_sync(0xffffffffu, v.z, k, G)};
  }
  return irr;
}

/* G lanes per output texel.  Bound by instruction issue (81 % of the slots, 28 of 32 lanes): about 380 a
 * sample.  512 x 256 texels x 128 samples of a 2048 x 1024 map, one call:
 * 507 us with four texel loads and five double-precision functions a sample, 264 us with one load and
 * three (the source read for non-finite texels included).  256 x 128 texels, where one thread per texel
 * fills a tenth of the GPU: 347 us with one lane, 99 with eight. */
template <int G>
__global__ void __launch_bounds__(128) k_bake(Src src, const float *lut, const unsigned *nonfinite, int log_w, int H,
                                              unsigned samples, float *out) {
  const size_t texels = (size_t)H << log_w;
  const size_t t = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) / G;
  const size_t id = min(t, texels - 1); /* lanes past the end keep the warp whole */
  const int W = 1 << log_w, y = (int)(id >> log_w), x = (int)(id & (size_t)(W - 1));
  const float u0 = (float)((double)x / (double)W), v0 = (float)((double)y / (double)H);
  const float phi0 = (float)(2.0 * kPiD * (double)u0), theta0 = (float)(kPiD * (double)v0);
  const float st = sin_rn(theta0);
  TexelFrame f;
  f.normal = V3{st * cos_rn(phi0), st * sin_rn(phi0), cos_rn(theta0)};
  float tu, tv;
  to_uv(lut, f.normal.x, f.normal.y, f.normal.z, tu, tv);
  f.px = to_pixel(tu, (unsigned)W), f.py = to_pixel(tv, (unsigned)H);
  const V3 right{1.f, 0.f, 0.f};
  const float dd = dot(right, f.normal);
  f.tangent = V3{0.f, 1.f, 0.f};
  if (1.0 - (double)fabsf(dd) > 1e-6) f.tangent = normalize(cross(right, f.normal));
  f.bitangent = cross(f.normal, f.tangent);
  V3 irr = *nonfinite ? bake_sum<false, G>(src, lut, f, samples) : bake_sum<true, G>(src, lut, f, samples);
  irr = irr / (float)samples;
  if (t >= texels || (threadIdx.x & (G - 1)) != 0) return;
  float *o = out + id * src.ch;
  o[0] = irr.x;
  o[1] = irr.y;
  o[2] = irr.z;
}

/* Lanes per texel: the fewest of 1, 2, 4, 8 that give every thread the GPU holds a lane.  Each lane adds all of
 * its group's samples (6 instructions a sample and lane) and makes the texel's frame, so more lanes than that
 * cost.  128 samples of a 2048 x 1024 map with 1, 2, 4 and 8 lanes: 32,768 texels 176, 109, 93 and 92 us, 65,536
 * 195, 157, 151 and 155, 131,072 284, 266, 266 and 278 (33 samples 91, 90, 97 and 113), 262,144 499, 482, 492 and
 * 522, 524,288 927, 915, 943 and 1017.  Where the loads miss the L2 more lanes hide more of them: 131,072 texels of
 * an 8192 x 4096 map 715 us with 4, 683 with 8. */
int bake_lanes(uint64_t texels) {
  int g = 1;
  while (g < 8 && texels * g < 148ull * 2048) g *= 2;
  return g;
}

}  // namespace

nova_b200_status nb_bake(nova_b200_ctx *c, const float *src, int32_t sw, int32_t sh, int32_t ch, int32_t ow,
                         int32_t oh, int32_t samples, float *out) {
  using namespace nbctx;
  auto pow2 = [](int32_t v) { return v > 0 && (v & (v - 1)) == 0; };
  if (!src || !out) return fail(c, NOVA_B200_INVALID_ARGUMENT, "null buffer%s");
  if (!pow2(ow) || !pow2(oh))
    return fail(c, NOVA_B200_INVALID_ARGUMENT, "irradiance size must be a power of two (TextureProcessing.cpp:11)%s");
  if (sw < 1 || sh < 1 || ch < 3 || ch > 4 || samples <= 0)
    return fail(c, NOVA_B200_INVALID_ARGUMENT, "invalid source map or sample count%s");
  cudaSetDevice(c->device);
  const bool vec4 = ch == 4 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0;
  const Src map{src, sw, sh, ch, vec4};
  const uint64_t texels = (uint64_t)ow * (uint64_t)oh;
  const int log_w = __builtin_ctz((unsigned)ow);
  /* reading the map once to learn that it is finite pays when at least as many samples are taken from it */
  const bool scan = texels * (uint64_t)samples >= (uint64_t)sw * (uint64_t)sh && sw < (1 << 23) && sh < (1 << 23);
  unsigned *flag = c->d_counters;
  NB_CUDA(c, cudaMemsetAsync(flag, scan ? 0 : 1, sizeof(unsigned), c->stream), "memset(bake flag)");
  if (scan) {
    const size_t n = (size_t)sw * sh * ch, n4 = (reinterpret_cast<uintptr_t>(src) & 15u) == 0 ? n / 4 : 0;
    const size_t items = n4 ? n4 : n;
    k_any_nonfinite<<<(unsigned)std::min<size_t>(148 * 8, (items + 255) / 256), 256, 0, c->stream>>>(src, n, n4, flag);
  }
  const int g = bake_lanes(texels);
  const unsigned grid = (unsigned)((texels * g + 127) / 128);
  if (g == 1)
    k_bake<1><<<grid, 128, 0, c->stream>>>(map, c->d_acos, flag, log_w, oh, (unsigned)samples, out);
  else if (g == 2)
    k_bake<2><<<grid, 128, 0, c->stream>>>(map, c->d_acos, flag, log_w, oh, (unsigned)samples, out);
  else if (g == 4)
    k_bake<4><<<grid, 128, 0, c->stream>>>(map, c->d_acos, flag, log_w, oh, (unsigned)samples, out);
  else
    k_bake<8><<<grid, 128, 0, c->stream>>>(map, c->d_acos, flag, log_w, oh, (unsigned)samples, out);
  NB_CUDA(c, cudaGetLastError(), "k_bake");
  NB_CUDA(c, cudaStreamSynchronize(c->stream), "bake");
  return NOVA_B200_SUCCESS;
}
