/* Diffuse irradiance bake with the semantics of the reference's CUDA kernel: the path its command line
 * takes with --gpu (sources/controller/cmd/API.cpp:29,52 -> TextureProcessing.cpp:19-45 ->
 * GPU_compute_irradiance, sources/processing/cuda/CubemapProcessing.cu:244-284, kernel :129-175).
 *
 * It differs from the CPU path (bake.cu) in three ways, all kept here:
 *   - the pgc3d hash is seeded with the output texel's own indices (i, j), not with the pixel of its
 *     approximate spherical coordinates;
 *   - directions map to uv with the exact acos / atan2f (the device's own functions), not the fast
 *     polynomial and the acos table;
 *   - the source is read through a float4 texture object with hardware bilinear filtering, wrap
 *     addressing and normalised coordinates (CubemapProcessing.cu:216-230), so the filter weights
 *     are the texture unit's 8-bit-fraction fixed point ones.
 * The output is RGBA with alpha 1 (gpgpu_device_write_buffer, :121-127).  Angles are evaluated as
 * the reference's expressions are written: products with PI (a double constant) in double, the
 * trigonometry in float.  This file is compiled with the default multiply-add contraction, like the
 * reference's CUDA sources (its CMake flags only add --expt-relaxed-constexpr -std=c++17).
 */
#include "caller_memory.cuh"
#include "context.cuh"

namespace {

constexpr double kPi = 3.14159265358979323846; /* PI, internal/common/math/math_spherical.h:8 (double) */

struct F3 {
  float x, y, z;
};

__device__ __forceinline__ F3 sph_to_cart(float phi, float theta) {
  return F3{sinf(theta) * cosf(phi), sinf(theta) * sinf(phi), cosf(theta)};
}

__device__ __forceinline__ float dot3(F3 a, F3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

__device__ __forceinline__ F3 cross3(F3 a, F3 b) {
  return F3{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}

__device__ __forceinline__ F3 normalize3(F3 a) {
  const float d = sqrtf(a.x * a.x + a.y * a.y + a.z * a.z);
  return F3{a.x / d, a.y / d, a.z / d};
}

__device__ __forceinline__ F3 scale(float k, F3 v) { return F3{v.x * k, v.y * k, v.z * k}; }
__device__ __forceinline__ F3 add(F3 a, F3 b) { return F3{a.x + b.x, a.y + b.y, a.z + b.z}; }

/* The 3D hash of the kernel (integer arithmetic, then unsigned -> float times 1 / float(2^32 - 1)). */
__device__ __forceinline__ F3 pgc3d(unsigned x, unsigned y, unsigned z) {
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
  const float cste = 1.f / float(0xFFFFFFFFu);
  return F3{(float)x * cste, (float)y * cste, (float)z * cste};
}

/* G lanes per output texel take every G-th sample; the group's values are added in sample order by every
 * lane, so the sum is the serial one.  One thread per texel in the reference's 32 x 32 blocks put a
 * 256 x 128 map on 45 of 148 SMs (205 us for 128 samples; the whole call takes 90 us now). */
template <int G>
__global__ void __launch_bounds__(128) k_bake_texunit(float *out, cudaTextureObject_t tex, int log_w, unsigned H,
                                                      unsigned samples) {
  const unsigned W = 1u << log_w, lane = threadIdx.x & (G - 1);
  const size_t t = (blockDim.x * (size_t)blockIdx.x + threadIdx.x) / G, texels = (size_t)H << log_w;
  const size_t id = min(t, texels - 1); /* lanes past the end keep the warp whole */
  const int j = (int)(id >> log_w), i = (int)(id & (size_t)(W - 1u));
  const float u = (float)i / (float)W;
  const float v = (float)j / (float)H;
  const float phi0 = (float)(2 * kPi * u), theta0 = (float)(kPi * v); /* uvToSpherical */
  const F3 normal = sph_to_cart(phi0, theta0);
  const F3 some{1.f, 0.f, 0.f};
  const float dd = dot3(some, normal);
  F3 tangent{0.f, 1.f, 0.f};
  if (1.0 - fabsf(dd) > 1e-6) tangent = normalize3(cross3(some, normal));
  const F3 bitangent = cross3(normal, tangent);
  F3 irr{0.f, 0.f, 0.f};
  for (unsigned s0 = 0; s0 < samples; s0 += G) {
    const F3 r = pgc3d((unsigned)i, (unsigned)j, s0 + lane);
    const float phi = (float)(2 * kPi * r.x);
    const float theta = asinf(sqrtf(r.y));
    F3 c = sph_to_cart(phi, theta);
    c = add(add(scale(c.x, tangent), scale(c.y, bitangent)), scale(c.z, normal));
    const float th = acosf(c.z), ph = atan2f(c.y, c.x); /* cartesianToSpherical */
    const float tu = (float)(ph / (2 * kPi)), tv = (float)(th / kPi); /* sphericalToUv */
    const float4 q = tex2D<float4>(tex, tu, tv);
#pragma unroll
    for (int k = 0; k < G; k++) {
      const F3 x{__shfl_sync(0xffffffffu, q.x, k, G), __shfl_sync(0xffffffffu, q.y, k, G),
                 __shfl_sync(0xffffffffu, q.z, k, G)};
      if (s0 + k < samples) irr = add(irr, x);
    }
  }
  irr.x /= samples;
  irr.y /= samples;
  irr.z /= samples;
  if (t >= texels || lane != 0) return;
  float *o = out + id * 4;
  o[0] = irr.x;
  o[1] = irr.y;
  o[2] = irr.z;
  o[3] = 1.f;
}

/* RGB source -> RGBA rows of `pitch` bytes with alpha 1, as TextureProcessing.cpp:24-32 prepares it. */
__global__ void k_to_rgba(const float *src, int w, size_t n, char *dst, size_t pitch) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
    const size_t y = k / (size_t)w, x = k - y * (size_t)w;
    reinterpret_cast<float4 *>(dst + y * pitch)[x] = make_float4(src[3 * k], src[3 * k + 1], src[3 * k + 2], 1.f);
  }
}

/* The fewest of 1, 2, 4, 8 lanes per texel that fill the GPU's threads twice over. */
void launch_bake(nova_b200_ctx *c, float *out, cudaTextureObject_t tex, unsigned W, unsigned H, unsigned samples) {
  const uint64_t texels = (uint64_t)W * H, fill = 2ull * 148 * 2048;
  const int log_w = __builtin_ctz(W);
  auto grid = [&](unsigned g) { return (unsigned)((texels * g + 127) / 128); };
  if (texels >= fill)
    k_bake_texunit<1><<<grid(1), 128, 0, c->stream>>>(out, tex, log_w, H, samples);
  else if (texels * 2 >= fill)
    k_bake_texunit<2><<<grid(2), 128, 0, c->stream>>>(out, tex, log_w, H, samples);
  else if (texels * 4 >= fill)
    k_bake_texunit<4><<<grid(4), 128, 0, c->stream>>>(out, tex, log_w, H, samples);
  else
    k_bake_texunit<8><<<grid(8), 128, 0, c->stream>>>(out, tex, log_w, H, samples);
}

}  // namespace

nova_b200_status nb_bake_texunit(nova_b200_ctx *c, const float *src, int32_t sw, int32_t sh, int32_t ch, int32_t ow,
                                 int32_t oh, int32_t samples, float *out) {
  using namespace nbctx;
  auto pow2 = [](int32_t v) { return v > 0 && (v & (v - 1)) == 0; };
  if (!src || !out) return fail(c, NOVA_B200_INVALID_ARGUMENT, "null buffer%s");
  if (!pow2(ow) || !pow2(oh))
    return fail(c, NOVA_B200_INVALID_ARGUMENT, "irradiance size must be a power of two (TextureProcessing.cpp:11)%s");
  if (sw < 1 || sh < 1 || ch < 3 || ch > 4 || samples <= 0)
    return fail(c, NOVA_B200_INVALID_ARGUMENT, "invalid source map or sample count%s");
  int max_w = 0, max_h = 0;
  cudaDeviceGetAttribute(&max_w, cudaDevAttrMaxTexture2DWidth, c->device);
  cudaDeviceGetAttribute(&max_h, cudaDevAttrMaxTexture2DHeight, c->device);
  if (sw > max_w || sh > max_h) return fail(c, NOVA_B200_INVALID_ARGUMENT, "source map larger than a 2D texture%s");
  cudaSetDevice(c->device);
  /* The texture reads linear memory where its limits allow: the caller's own map when it lies on this GPU,
   * its base and rows are aligned and the bake does not write over it, else an aligned copy from the pool.
   * RGBA maps are copied by the copy engine's rules, which take another GPU's memory too.  An array of its
   * own per call took cudaMallocArray and cudaFreeArray, 0.4 of the call's 0.55 ms at 1024 x 512 (and now
   * and then tens of ms); the texture unit filters both alike.  Larger maps still get the array. */
  const size_t texels = (size_t)sw * sh;
  int lin_w = 0, lin_h = 0, lin_pitch = 0, tex_align = 512, pitch_align = 32;
  cudaDeviceGetAttribute(&lin_w, cudaDevAttrMaxTexture2DLinearWidth, c->device);
  cudaDeviceGetAttribute(&lin_h, cudaDevAttrMaxTexture2DLinearHeight, c->device);
  cudaDeviceGetAttribute(&lin_pitch, cudaDevAttrMaxTexture2DLinearPitch, c->device);
  cudaDeviceGetAttribute(&tex_align, cudaDevAttrTextureAlignment, c->device);
  cudaDeviceGetAttribute(&pitch_align, cudaDevAttrTexturePitchAlignment, c->device);
  auto aligned = [](size_t v, int a) { return v % (size_t)a == 0; };
  const size_t row = (size_t)sw * sizeof(float4);
  cudaPointerAttributes at{};
  if (cudaPointerGetAttributes(&at, src) != cudaSuccess) cudaGetLastError();
  const nb::Span map{reinterpret_cast<uintptr_t>(src), row * sh, nb::on_device(at, c->device)};
  const nb::Span target{reinterpret_cast<uintptr_t>(out), sizeof(float4) * (size_t)ow * oh, true};
  const bool direct = ch == 4 && map.here && !nb::overlap(map, target) && aligned(map.begin, tex_align) &&
                      aligned(row, pitch_align);
  const size_t pitch = direct ? row : (row + tex_align - 1) / tex_align * tex_align;
  const bool linear = sw <= lin_w && sh <= lin_h && pitch <= (size_t)lin_pitch;
  const cudaChannelFormatDesc fmt = cudaCreateChannelDesc(32, 32, 32, 32, cudaChannelFormatKindFloat);
  char *rgba = nullptr;
  cudaArray_t array = nullptr;
  cudaTextureObject_t tex = 0;
  cudaResourceDesc res{};
  cudaError_t e = cudaSuccess;
  if (!(linear ? direct : ch == 4)) {
    char *base = nullptr;
    e = cudaMallocAsync(&base, (linear ? pitch : row) * sh + tex_align, c->stream);
    rgba = base;
    if (e == cudaSuccess) {
      base += (tex_align - reinterpret_cast<uintptr_t>(base) % tex_align) % tex_align;
      if (ch == 4)
        e = cudaMemcpy2DAsync(base, pitch, src, row, row, (size_t)sh, cudaMemcpyDeviceToDevice, c->stream);
      else
        k_to_rgba<<<592, 256, 0, c->stream>>>(src, sw, texels, base, linear ? pitch : row);
      src = reinterpret_cast<const float *>(base);
    }
  }
  if (linear) {
    res.resType = cudaResourceTypePitch2D;
    res.res.pitch2D.devPtr = const_cast<float *>(src);
    res.res.pitch2D.desc = fmt;
    res.res.pitch2D.width = (size_t)sw;
    res.res.pitch2D.height = (size_t)sh;
    res.res.pitch2D.pitchInBytes = pitch;
  } else {
    if (e == cudaSuccess) e = cudaMallocArray(&array, &fmt, (size_t)sw, (size_t)sh);
    if (e == cudaSuccess)
      e = cudaMemcpy2DToArrayAsync(array, 0, 0, src, row, row, (size_t)sh, cudaMemcpyDeviceToDevice, c->stream);
    res.resType = cudaResourceTypeArray;
    res.res.array.array = array;
  }
  if (e == cudaSuccess) {
    cudaTextureDesc td{}; /* CubemapProcessing.cu:223-229 */
    td.addressMode[0] = cudaAddressModeWrap;
    td.addressMode[1] = cudaAddressModeWrap;
    td.filterMode = cudaFilterModeLinear;
    td.readMode = cudaReadModeElementType;
    td.normalizedCoords = 1;
    e = cudaCreateTextureObject(&tex, &res, &td, nullptr);
  }
  if (e == cudaSuccess) {
    cudaEventRecord(c->ev_begin, c->stream);
    launch_bake(c, out, tex, (unsigned)ow, (unsigned)oh, (unsigned)samples);
    cudaEventRecord(c->ev_end, c->stream);
    e = cudaGetLastError();
  }
  const cudaError_t es = cudaStreamSynchronize(c->stream);
  if (tex) cudaDestroyTextureObject(tex);
  if (array) cudaFreeArray(array);
  if (rgba) cudaFreeAsync(rgba, c->stream);
  if (e != cudaSuccess) return cuda_fail(c, e, "bake (texture unit)");
  if (es != cudaSuccess) return cuda_fail(c, es, "bake (texture unit)");
  return NOVA_B200_SUCCESS;
}
