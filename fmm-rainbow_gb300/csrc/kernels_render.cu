// Headless point-splat renderer: the reference's display passes restated as
// CUDA kernels writing an RGBA8 image into device memory (no window, no
// swapchain, no graphics API).
//
// Reference (iskamag/fmm-rainbow):
//   render_vertex / render_fragment   src/rainbow_fmm.wgsl:780-900
//   reconstruct_field + blur passes   src/rainbow_fmm.wgsl:914-970
//   resolve_fragment                  src/rainbow_fmm.wgsl:972-1009
//   pass sequence, texture sizes      app.js:650-710, 216-251 (accumulation at
//                                     half the canvas size, linear clamp sampler)
//
// Differences by design: the additive rgba16float blend becomes a per-pixel
// fixed-point sum (64-bit integer atomics at 2^24 per unit), which is exact
// and independent of the order points arrive in; the blur and resolve
// intermediates are binary32 instead of binary16; bilinear taps use the exact
// fractional position.
#include <cuda_runtime.h>

#include "rfmm_device.cuh"
#include "rfmm_kernels.h"
#include "rfmm_math.h"

namespace rfmm {

namespace {

constexpr float kTau = 6.28318530718f;
constexpr float kFix = 16777216.0f;        // 2^24 fixed-point units per 1.0
constexpr float kFixInv = 1.0f / 16777216.0f;

__device__ __forceinline__ float mixf(float a, float b, float t) { return a * (1.0f - t) + b * t; }

__device__ __forceinline__ float smoothstepf_d(float lo, float hi, float x) {
  const float t = clampf_d((x - lo) / (hi - lo), 0.0f, 1.0f);
  return t * t * (3.0f - 2.0f * t);
}

__device__ __forceinline__ float len3(float x, float y, float z) { return sqrtf((x * x + y * y) + z * z); }

// Fixed-point accumulation texture -> float4 (r, g, b, a).
__device__ __forceinline__ float4 fetch_accum(const unsigned long long *acc, uint32_t w, uint32_t h,
                                              int x, int y) {
  x = min(max(x, 0), (int)w - 1);
  y = min(max(y, 0), (int)h - 1);
  const ulonglong2 *p = reinterpret_cast<const ulonglong2 *>(acc + 4ull * ((size_t)y * w + (size_t)x));
  const ulonglong2 rg = p[0], ba = p[1];
  return make_float4((float)rg.x * kFixInv, (float)rg.y * kFixInv, (float)ba.x * kFixInv,
                     (float)ba.y * kFixInv);
}

__device__ __forceinline__ float4 fetch_tex(const float4 *tex, uint32_t w, uint32_t h, int x, int y) {
  x = min(max(x, 0), (int)w - 1);
  y = min(max(y, 0), (int)h - 1);
  return tex[(size_t)y * w + (size_t)x];
}

__device__ __forceinline__ float4 lerp4(float4 a, float4 b, float f) {
  return make_float4(a.x * (1.0f - f) + b.x * f, a.y * (1.0f - f) + b.y * f,
                     a.z * (1.0f - f) + b.z * f, a.w * (1.0f - f) + b.w * f);
}

__device__ __forceinline__ float4 add4(float4 a, float4 b) {
  return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

__device__ __forceinline__ float4 scale4(float4 a, float s) {
  return make_float4(a.x * s, a.y * s, a.z * s, a.w * s);
}

}  // namespace

// The body an instance draws (wgsl:806-808).
__device__ __forceinline__ uint32_t instance_body(uint32_t i, uint32_t n) {
  return (i * 747796405u + 2891336453u) % n;
}

// Draws of every body: counts[body] instances map to it.
__global__ void __launch_bounds__(256) k_draw_counts(uint32_t instances, uint32_t n, uint32_t *__restrict__ counts) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < instances) atomicAdd(&counts[instance_body(i, n)], 1u);
}

// render_vertex + render_fragment: every drawn body's camera-space position
// and colour, and its additive splat into the pixel its point covers.  All
// instances of a body add the same fixed-point values, so bodies are drawn
// once in resident order, times their number of draws (`counts`, by caller id;
// null: `draws` for every body): whole-sector body reads and neighbouring
// pixels, where drawing by instance reads 32 random bytes per point.  The four
// sums of a pixel are one 32-byte sector, so the lanes of a quad exchange
// their points' components and add all four of one point per instruction
// (a quarter of the sector updates).  1,048,576 points on 1920 x 1080: 54 us
// and 10 for the id -> slot map before, 23.6 now; what is left is about half
// the colour arithmetic (400 instructions a point), half the updates.  Body
// counts that do not divide 2^32 pay for a fill, the counting pass and a
// scattered read per body: whole frames of 1,048,576 points 145 -> 63 us, of
// 1,000,003 144 -> 74.
__global__ void __launch_bounds__(256) k_splat(const SceneDesc *__restrict__ scenes, uint32_t scene,
                                               const float4 *__restrict__ part,
                                               const uint32_t *__restrict__ ids,
                                               const uint32_t *__restrict__ counts, uint32_t draws,
                                               RenderCamera cam, unsigned long long *__restrict__ acc) {
  const SceneDesc &S = scenes[scene];
  grid_dependency_wait();
  const uint32_t local = blockIdx.x * blockDim.x + threadIdx.x, slot = S.body_off + local;
  uint32_t times = 0u;
  if (local < S.n) {
    times = draws;
    if (counts != nullptr) {
      const uint32_t id = ids[slot];
      times = id < S.n ? counts[id] : 0u;
    }
  }
  float4 pl = make_float4(0.0f, 0.0f, 0.0f, 0.0f), vh = pl;
  if (times != 0u) load_body(part, slot, pl, vh);
  constexpr uint32_t kNoPixel = 0xFFFFFFFFu;
  uint32_t pixel = kNoPixel;
  unsigned long long sum[4] = {0ull, 0ull, 0ull, 0ull};
  if (times != 0u) {

  // rotate_camera (wgsl:785-798); the four trigonometric values come in.
  const float yx = cam.cos_yaw * pl.x + cam.sin_yaw * pl.z;
  const float yy = pl.y;
  const float yz = -cam.sin_yaw * pl.x + cam.cos_yaw * pl.z;
  const float rx = yx, ry = cam.cos_pitch * yy - cam.sin_pitch * yz,
              rz = cam.sin_pitch * yy + cam.cos_pitch * yz;
  const float view_z = cam.zoom * kHalf - rz;
  const float perspective = (1.92f * kHalf) / view_z;
  const float cx = rx * perspective / cam.aspect, cy = ry * perspective;
  const float depth = 0.46f + rz * 0.08f;

  const float velocity = len3(vh.x, vh.y, vh.z);
  const float speed = fmaxf(velocity, 0.0001f);
  const float excitation = clampf_d(vh.w, 0.0f, 1.0f);
  const float signed_radial =
      clampf_d(((pl.x * vh.x + pl.y * vh.y) + pl.z * vh.z) / (fmaxf(len3(pl.x, pl.y, pl.z), 0.0001f) * speed),
               -1.0f, 1.0f);
  const float infall = clampf_d(-signed_radial, 0.0f, 1.0f);
  const float outflow = clampf_d(signed_radial, 0.0f, 1.0f);
  float sp[3] = {mixf(0.50f, 0.24f, infall), mixf(0.42f, 0.56f, infall), mixf(0.58f, 1.00f, infall)};
  sp[0] = mixf(sp[0], 1.00f, outflow);
  sp[1] = mixf(sp[1], 0.50f, outflow);
  sp[2] = mixf(sp[2], 0.20f, outflow);
  const float heat = smoothstepf_d(0.18f, 0.85f, excitation);
  const float phase[3] = {0.00f, 0.67f, 0.33f};
  float col[3];
  const float luminosity = 0.30f + excitation * 0.90f;
  const float speed_gain = 0.62f + fminf(velocity * 1.4f, 1.0f) * 0.30f;
  for (int k = 0; k < 3; k++) {
    const float rainbow = 0.5f + 0.5f * rf_cosf(kTau * (pl.w + phase[k]));
    const float tint = rf_powf(rainbow, 0.85f);
    const float s = mixf(sp[k] * tint, sp[k], heat);
    col[k] = s * (speed_gain + excitation * 0.90f) + heat * heat * 0.55f;
  }
  float influence = 0.0f;
  float cc[3] = {0.82f, 1.0f, 0.28f};
  if (S.control_point[3] > 0.5f) {
    const float dx = S.control_point[0] - pl.x, dy = S.control_point[1] - pl.y,
                dz = S.control_point[2] - pl.z;
    const float radius = fmaxf(S.control_radius, 0.02f);
    influence = rf_expf(-2.0f * ((dx * dx + dy * dy) + dz * dz) / (radius * radius));
    const float mode = S.control_axis_mode[3];
    if (mode > 1.5f && mode < 2.5f) {
      cc[0] = 1.0f; cc[1] = 0.38f; cc[2] = 0.18f;
    } else if (mode >= 2.5f) {
      cc[0] = 0.82f; cc[1] = 0.34f; cc[2] = 1.0f;
    }
  }
  for (int k = 0; k < 3; k++) col[k] = mixf(col[k], cc[k], influence * 0.68f);
  const float depth_fade = clampf_d(0.62f + rz * 0.25f, 0.28f, 1.0f) * (0.76f + excitation * 0.48f) *
                           luminosity * (1.0f + influence * 0.72f);

  // Clip volume (x, y in [-1, 1], z in [0, 1]) and the 1-pixel point's pixel.
  if (cx >= -1.0f && cx <= 1.0f && cy >= -1.0f && cy <= 1.0f && depth >= 0.0f && depth <= 1.0f) {
    const float fx = (cx + 1.0f) * 0.5f * (float)cam.acc_w;
    const float fy = (1.0f - cy) * 0.5f * (float)cam.acc_h;
    const int px = min((int)floorf(fx), (int)cam.acc_w - 1), py = min((int)floorf(fy), (int)cam.acc_h - 1);
    const float weight = cam.exposure * depth_fade * cam.population_scale;
    pixel = (uint32_t)py * cam.acc_w + (uint32_t)px;
#pragma unroll
    for (int k = 0; k < 3; k++) sum[k] = times * __float2ull_rn(col[k] * weight * kFix);
    sum[3] = times * __float2ull_rn(weight * kFix);
  }
  }
  // 4 x 4 exchange inside each quad: afterwards lane c of the quad holds
  // component c of the quad's points 0..3.
  constexpr uint32_t kAll = 0xFFFFFFFFu;
  const bool odd = threadIdx.x & 1u, high = threadIdx.x & 2u;
#pragma unroll
  for (int k = 0; k < 4; k += 2) {
    const unsigned long long got = __shfl_xor_sync(kAll, odd ? sum[k] : sum[k + 1], 1);
    if (odd) sum[k] = got; else sum[k + 1] = got;
  }
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const unsigned long long got = __shfl_xor_sync(kAll, high ? sum[k] : sum[k + 2], 2);
    if (high) sum[k] = got; else sum[k + 2] = got;
  }
#pragma unroll
  for (uint32_t k = 0; k < 4u; k++) {
    const uint32_t to = __shfl_sync(kAll, pixel, (threadIdx.x & 28u) | k);
    if (to != kNoPixel) atomicAdd(acc + 4ull * to + (threadIdx.x & 3u), sum[k]);
  }
}

// One separable pass of reconstruct_field (wgsl:914-945): five bilinear taps
// along `axis` at +-1.384615 and +-3.230769 steps, step = point_size /
// (canvas size * 3.230769) in texture coordinates.  The first pass reads the
// fixed-point accumulation, the second the first pass's output.
// With kFromAccum the row is converted to binary32 once, in shared memory:
// `halo` texels to either side of the CTA's 256 hold every tap (0: a radius
// beyond kMaxHalo, taps convert what they read).  Ten strided reads and 40
// 64-bit conversions per texel made it 38 us at 960 x 540; 10.6 now.
constexpr uint32_t kMaxHalo = 128u;
template <bool kFromAccum>
__global__ void __launch_bounds__(256) k_blur(const unsigned long long *__restrict__ acc,
                                              const float4 *__restrict__ src, RenderCamera cam,
                                              int axis, uint32_t halo, float4 *__restrict__ dst) {
  __shared__ float4 s_row[kFromAccum ? 256u + 2u * kMaxHalo : 1u];
  const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  const uint32_t w = cam.acc_w, h = cam.acc_h;
  const int row0 = (int)(blockIdx.x * blockDim.x) - (int)halo;
  grid_dependency_wait();
  if (kFromAccum && halo != 0u) {
    for (uint32_t i = threadIdx.x; i < 256u + 2u * halo; i += 256u) s_row[i] = fetch_accum(acc, w, h, row0 + (int)i, (int)y);
    __syncthreads();
  }
  if (x >= w || y >= h) return;
  const float dim = axis == 0 ? (float)w : (float)h;
  const float out_dim = axis == 0 ? cam.canvas_w : cam.canvas_h;
  const float step = fmaxf(cam.point_size, 1.0f) / (out_dim * 3.230769f);
  const float uv = ((axis == 0 ? (float)x : (float)y) + 0.5f) / dim;
  auto tap = [&](float u) -> float4 {
    const float t = u * dim - 0.5f;
    const float f0 = floorf(t);
    const float f = t - f0;
    const int i0 = (int)f0;
    float4 a, b;
    if (kFromAccum && halo != 0u) {
      a = s_row[i0 - row0];
      b = s_row[i0 + 1 - row0];
    } else if (axis == 0) {
      a = kFromAccum ? fetch_accum(acc, w, h, i0, (int)y) : fetch_tex(src, w, h, i0, (int)y);
      b = kFromAccum ? fetch_accum(acc, w, h, i0 + 1, (int)y) : fetch_tex(src, w, h, i0 + 1, (int)y);
    } else {
      a = kFromAccum ? fetch_accum(acc, w, h, (int)x, i0) : fetch_tex(src, w, h, (int)x, i0);
      b = kFromAccum ? fetch_accum(acc, w, h, (int)x, i0 + 1) : fetch_tex(src, w, h, (int)x, i0 + 1);
    }
    return lerp4(a, b, f);
  };
  float4 field = scale4(tap(uv), 0.227027f);
  field = add4(field, scale4(tap(uv + step * 1.384615f), 0.316216f));
  field = add4(field, scale4(tap(uv - step * 1.384615f), 0.316216f));
  field = add4(field, scale4(tap(uv + step * 3.230769f), 0.070270f));
  field = add4(field, scale4(tap(uv - step * 3.230769f), 0.070270f));
  dst[(size_t)y * w + x] = field;
}

// resolve_fragment (wgsl:972-1009) for every canvas pixel: bilinear sample of
// the blurred field, density-normalised colour, filmic curve, gamma 0.82,
// written as RGBA8 (row 0 = top of the canvas).
// The pass also clears the accumulation for the next frame (its readers are
// complete), under the arithmetic that bounds it.
__global__ void __launch_bounds__(256) k_resolve(const float4 *__restrict__ tex, RenderCamera cam,
                                                 unsigned long long *__restrict__ acc, uchar4 *__restrict__ out,
                                                 const Counters *__restrict__ ctr, volatile uint32_t *error_out) {
  const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  grid_dependency_wait();
  report_error(ctr, error_out);
  {
    const uint32_t sums = 4u * cam.acc_w * cam.acc_h, row = gridDim.x * blockDim.x;
    for (uint32_t i = y * row + x; i < sums; i += gridDim.y * row) acc[i] = 0ull;
  }
  const uint32_t W = (uint32_t)cam.canvas_w, H = (uint32_t)cam.canvas_h;
  if (x >= W || y >= H) return;
  const uint32_t w = cam.acc_w, h = cam.acc_h;
  const float u = ((float)x + 0.5f) / cam.canvas_w, v = ((float)y + 0.5f) / cam.canvas_h;
  const float tx = u * (float)w - 0.5f, ty = v * (float)h - 0.5f;
  const float fx0 = floorf(tx), fy0 = floorf(ty);
  const float fx = tx - fx0, fy = ty - fy0;
  const int ix = (int)fx0, iy = (int)fy0;
  const float4 top = lerp4(fetch_tex(tex, w, h, ix, iy), fetch_tex(tex, w, h, ix + 1, iy), fx);
  const float4 bot = lerp4(fetch_tex(tex, w, h, ix, iy + 1), fetch_tex(tex, w, h, ix + 1, iy + 1), fx);
  const float4 a = lerp4(top, bot, fy);
  const float bg[3] = {0.006f, 0.008f, 0.015f};
  float rgb[3] = {bg[0], bg[1], bg[2]};
  if (!(a.w < 0.00001f)) {
    const float avg[3] = {a.x / a.w, a.y / a.w, a.z / a.w};
    const float luma = (avg[0] * 0.2126f + avg[1] * 0.7152f) + avg[2] * 0.0722f;
    const float density = sqrtf(a.w / (a.w + 1.0f));
    for (int k = 0; k < 3; k++) {
      const float vivid = fmaxf(0.0f, mixf(luma, avg[k], 1.16f));
      const float mapped = 1.0f - rf_expf(-vivid * density * 1.58f);
      rgb[k] = rf_powf(clampf_d(mapped + bg[k], 0.0f, 1.0f), 0.82f);
    }
  }
  out[(size_t)y * W + x] = make_uchar4((unsigned char)__float2int_rn(rgb[0] * 255.0f),
                                       (unsigned char)__float2int_rn(rgb[1] * 255.0f),
                                       (unsigned char)__float2int_rn(rgb[2] * 255.0f), 255);
}

void launch_render(const LaunchCtx &L, uint32_t scene, uint32_t n, const uint32_t *ids, uint32_t *counts,
                   const RenderCamera &cam, unsigned long long *acc, float4 *tex_a, float4 *tex_b, uchar4 *out,
                   uint32_t *error_out) {
  // i -> (a i + c) mod 2^32 mod n with odd a permutes 0..n-1 when n divides
  // 2^32: every body is drawn instances / n times.
  const bool even = (n & (n - 1u)) == 0u && cam.instances % n == 0u;
  if (!even) {
    cudaMemsetAsync(counts, 0, 4ull * n, L.stream);
    k_draw_counts<<<(cam.instances + 255u) / 256u, 256, 0, L.stream>>>(cam.instances, n, counts);
  }
  launch_step_kernel(L, k_splat, dim3((n + 255u) / 256u), dim3(256), 0, L.scenes, scene, (const float4 *)L.part, ids,
                     (const uint32_t *)(even ? nullptr : counts), even ? cam.instances / n : 0u, cam, acc);
  // Farthest tap of the horizontal pass, in texels.
  const float reach = (cam.point_size > 1.0f ? cam.point_size : 1.0f) * (float)cam.acc_w / cam.canvas_w;
  const uint32_t halo = reach < (float)kMaxHalo - 4.0f ? (uint32_t)reach + 3u : 0u;
  const dim3 grid_a((cam.acc_w + 255u) / 256u, cam.acc_h);
  launch_step_kernel(L, k_blur<true>, grid_a, dim3(256), 0, (const unsigned long long *)acc, (const float4 *)nullptr, cam,
                     0, halo, tex_a);
  launch_step_kernel(L, k_blur<false>, grid_a, dim3(256), 0, (const unsigned long long *)nullptr, (const float4 *)tex_a, cam,
                     1, 0u, tex_b);
  const dim3 grid_c(((uint32_t)cam.canvas_w + 255u) / 256u, (uint32_t)cam.canvas_h);
  launch_step_kernel(L, k_resolve, grid_c, dim3(256), 0, (const float4 *)tex_b, cam, acc, out, (const Counters *)L.ctr,
                     (volatile uint32_t *)error_out);
}

}  // namespace rfmm
