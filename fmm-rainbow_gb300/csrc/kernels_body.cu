// Body passes: integrate (L2P + self leaf + kick/drift) fused with the next
// step's deposit, the sort-key and gather passes that keep bodies resident in
// leaf (Morton) order, the standalone deposit, and the galaxy seed.
//
// Reference passes (iskamag/fmm-rainbow src/rainbow_fmm.wgsl):
//   deposit     408-422   leaf cell + i32(round(pos * scale)) atomics
//   integrate   613-771   adaptive descent, local expansion, self leaf,
//                         control field, symplectic Euler, soft wall, hue
//   initialize  232-374   seeded galaxy
//
// Bodies live in HBM in leaf-key order (a permutation of the caller's order,
// undone on download).  Every result is independent of that order: each
// body's update reads only its own state and the tree, and the moment sums
// are exact integers.  Sorted order makes a warp's bodies share leaves, so
// the tree gathers broadcast and the deposit is one reduction per run.
#include <cuda_runtime.h>

#include <type_traits>

#include "rfmm_device.cuh"
#include "rfmm_kernels.h"
#include "rfmm_math.h"

RFMM_KERNEL_NS_BEGIN

// Leaf (level `depth`) cell of a position, local to the scene's tree.
__device__ __forceinline__ uint32_t leaf_cell(float x, float y, float z, uint32_t depth) {
  uint32_t cx, cy, cz;
  cells_of_position(x, y, z, depth, cx, cy, cz);
  return level_offset_d(depth) + lin3_lv(cx, cy, cz, depth);
}

// 3-D Morton interleave of leaf coordinates (x in bit 0).
__device__ __forceinline__ uint32_t spread3(uint32_t v) {
  v &= 0x3FFu;
  v = (v | (v << 16)) & 0x030000FFu;
  v = (v | (v << 8)) & 0x0300F00Fu;
  v = (v | (v << 4)) & 0x030C30C3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}

__device__ __forceinline__ uint32_t morton3(uint32_t x, uint32_t y, uint32_t z) {
  return spread3(x) | (spread3(y) << 1) | (spread3(z) << 2);
}

__device__ __forceinline__ float length3(float x, float y, float z) {
  return sqrt_sum((x * x + y * y) + z * z);
}

// Soft absorbing band and last-resort clamp for one axis (wgsl:740-751).
__device__ __forceinline__ void soft_wall(float &p, float &v, float world_edge, float edge_band) {
  const float over = fabsf(p) - (world_edge - edge_band);
  if (over > 0.0f) {
    const float absorb = clampf_d(over / edge_band, 0.0f, 1.0f);
    v = v * (1.0f - absorb * 0.16f);
  }
  if (fabsf(p) > world_edge) {
    p = clampf_d(p, -world_edge, world_edge);
    v = v * -0.55f;
  }
}

// Near-field P2P inputs: the leaf-sorted position snapshot, the per-leaf
// start table (Morton order, absolute slots, 8^depth + 1 entries per scene at
// the scene's cell offset) and the body's own slot.
struct P2PView {
  const float4 *pos;
  const uint32_t *starts;
  uint32_t self;
};

// The cell a body samples its field from (wgsl:625-639): the first level
// whose cell holds at most 16 bodies, else the leaf level.  Resolved once per
// leaf by the upward pass; bodies of unresolved leaves (sparse subtrees)
// descend here.  Returns the global cell index; `level` and the leaf
// coordinates (lx, ly, lz) describe it (coordinates at the level are the
// leaf coordinates shifted right by depth - level).
__device__ __forceinline__ uint32_t sample_cell(const SceneDesc &S, float px, float py, float pz,
                                                const uint4 *__restrict__ mom,
                                                const uint32_t *__restrict__ choice,
                                                uint32_t &level, uint32_t &lx, uint32_t &ly,
                                                uint32_t &lz) {
  const uint32_t D = S.depth;
  // Leaf coordinates; floor(u * 2^l) == floor(u * 2^D) >> (D - l).
  cells_of_position(px, py, pz, D, lx, ly, lz);
  uint32_t chosen = D, cell_index = 0u;
  const uint32_t pick = __ldg(&choice[S.cell_off + level_offset_d(D) + lin3_lv(lx, ly, lz, D)]);
  if (pick != kChoiceUnresolved) {
    chosen = pick >> 28;
    cell_index = S.cell_off + (pick & 0x0FFFFFFFu);
  } else {
#pragma unroll
    for (uint32_t l = 6u; l >= 1u; l--) {
      if (l <= D) {
        const uint32_t sh = D - l;
        const uint32_t idx = S.cell_off + level_offset_d(l) + lin3_lv(lx >> sh, ly >> sh, lz >> sh, l);
        const uint32_t c = __ldg(&mom[idx].x);
        if ((int32_t)c <= (int32_t)kAdaptive || l == D) {
          chosen = l;
          cell_index = idx;
        }
      }
    }
  }
  level = chosen;
  return cell_index;
}

// Softened pair sums over the bodies of the 3x3x3 cells (level `l`) around
// cell (cx, cy, cz): cells z-, y-, x-major from -1 to +1, bodies of a cell in
// (leaf Morton code, caller id) order, the body itself skipped.
template <bool kPhi>
__device__ __forceinline__ void p2p_sums(const SceneDesc &S, const P2PView &V, uint32_t l,
                                         uint32_t cx, uint32_t cy, uint32_t cz, float px, float py,
                                         float pz, float &sx, float &sy, float &sz, float &sp) {
  const int dim = 1 << l;
  const uint32_t sh3 = 3u * (S.depth - l);
  const float eps2 = S.softening * S.softening;
  sx = 0.0f;
  sy = 0.0f;
  sz = 0.0f;
  sp = 0.0f;
  for (int oz = -1; oz <= 1; oz++) {
    const int nz = (int)cz + oz;
    if (nz < 0 || nz >= dim) continue;
    for (int oy = -1; oy <= 1; oy++) {
      const int ny = (int)cy + oy;
      if (ny < 0 || ny >= dim) continue;
      for (int ox = -1; ox <= 1; ox++) {
        const int nx = (int)cx + ox;
        if (nx < 0 || nx >= dim) continue;
        const uint32_t m = morton3((uint32_t)nx, (uint32_t)ny, (uint32_t)nz);
        const uint32_t lo = __ldg(&V.starts[S.cell_off + (m << sh3)]);
        const uint32_t hi = __ldg(&V.starts[S.cell_off + ((m + 1u) << sh3)]);
        for (uint32_t j = lo; j < hi; j++) {
          if (j == V.self) continue;
          const float4 q = __ldg(&V.pos[j]);
          const float dx = q.x - px, dy = q.y - py, dz = q.z - pz;
          const float r2 = ((dx * dx + dy * dy) + dz * dz) + eps2;
          const float inv = inv_sqrt(r2);
          const float w = (inv * inv) * inv;
          sx = sx + dx * w;
          sy = sy + dy * w;
          sz = sz + dz * w;
          if (kPhi) sp = sp + inv;
        }
      }
    }
  }
}

// FMM acceleration at a body (wgsl:619-657): adaptive descent to the sample
// cell, local expansion about its centre, softened self-leaf monopole (or,
// with kP2P, the exact near-field pair sums instead).  With `phi`, also the
// potential of the same expansion (diagnostics only; integrate never
// evaluates it).  Returns the sample cell's count.
template <bool kPhi, bool kP2P = false>
__device__ __forceinline__ uint32_t body_acceleration(const SceneDesc &S, float px, float py, float pz,
                                                      const uint4 *__restrict__ mom,
                                                      const float4 *__restrict__ src,
                                                      const float4 *__restrict__ aux,
                                                      const uint32_t *__restrict__ choice,
                                                      const float *__restrict__ fields, float &ax,
                                                      float &ay, float &az, float &pulse,
                                                      float *phi, const P2PView *V = nullptr) {
    const uint32_t D = S.depth;
    uint32_t chosen, lx, ly, lz;
    const uint32_t cell_index = sample_cell(S, px, py, pz, mom, choice, chosen, lx, ly, lz);
    const float4 ax4 = __ldg(&aux[cell_index]);
    const uint32_t count = __float_as_uint(ax4.z);
    const uint32_t csh = D - chosen;
    const float cx = cell_center_lv(lx >> csh, chosen);
    const float cy = cell_center_lv(ly >> csh, chosen);
    const float cz = cell_center_lv(lz >> csh, chosen);

    const float4 *fp = reinterpret_cast<const float4 *>(fields + (size_t)cell_index * 12u);
    const float4 fa = __ldg(fp), fj0 = __ldg(fp + 1), fj1 = __ldg(fp + 2);
    const float rx = px - cx, ry = py - cy, rz = pz - cz;
    ax = fa.x + (fj0.x * rx + fj0.y * ry + fj0.z * rz);
    ay = fa.y + (fj0.y * rx + fj0.w * ry + fj1.x * rz);
    az = fa.z + (fj0.z * rx + fj1.x * ry + fj1.y * rz);

    if (kP2P) {
      float sx, sy, sz, sp = 0.0f;
      p2p_sums<kPhi>(S, *V, chosen, lx >> csh, ly >> csh, lz >> csh, px, py, pz, sx, sy, sz, sp);
      const float gm = S.gravity / S.n_f;
      ax = ax + gm * sx;
      ay = ay + gm * sy;
      az = az + gm * sz;
      if (kPhi) *phi = (fa.w - ((fa.x * rx + fa.y * ry) + fa.z * rz)) - gm * sp;
      pulse = ax4.y;
      return count;
    }

    // Self leaf: softened monopole of the other count-1 bodies (wgsl:646-657).
    // x / 2^l == x * 2^-l exactly, so the eps division is a scaling.
    if (count > 1u) {
      const float4 s = __ldg(&src[cell_index]);
      const float dx = s.x - px, dy = s.y - py, dz = s.z - pz;
      const float eps = fmaxf(S.softening, (0.62f * kHalf) * pow2_neg(chosen));
      const float inv_r = inv_sqrt((dx * dx + dy * dy) + dz * dz + eps * eps);
      const float gsm = ax4.x;  // G * f32(count - 1) / f32(N)
#ifdef RFMM_FAST_FLOAT
      // One weight for the three components (reassociated: fast variant only).
      const float w = gsm * ((inv_r * inv_r) * inv_r);
      ax = ax + dx * w;
      ay = ay + dy * w;
      az = az + dz * w;
#else
      ax = ax + gsm * dx * inv_r * inv_r * inv_r;
      ay = ay + gsm * dy * inv_r * inv_r * inv_r;
      az = az + gsm * dz * inv_r * inv_r * inv_r;
#endif
    }

    if (kPhi) {
      float p = fa.w - ((fa.x * rx + fa.y * ry) + fa.z * rz);
      if (count > 1u) {
        const float4 s = __ldg(&src[cell_index]);
        const float dx = s.x - px, dy = s.y - py, dz = s.z - pz;
        const float eps = fmaxf(S.softening, (0.62f * kHalf) * pow2_neg(chosen));
        p = p - ax4.x / sqrtf((dx * dx + dy * dy) + dz * dz + eps * eps);
      }
      *phi = p;
    }
    pulse = ax4.y;  // clamp((f32(count) - 16) / 72, 0, 1)
    return count;
}

// What integrate needs of a scene's descriptor and level constants, worked out
// once per scene change instead of once per body.
struct alignas(16) StepScene {
  float cell_scale;     // 2^(D - 1) / 1.6: leaf cells per unit length
  float cell_half;      // 2^(D - 1) - 0.5
  float cell_margin;    // 0.5 - 2^(D - 22)
  float inner;          // |coordinate| up to which the short deposit path runs
  uint32_t cell_base;   // index of the scene's leaf (0, 0, 0), less the biased coordinates' bits
  uint32_t dim, dim2;   // 2^D and 2^(2D)
  uint32_t cell_off;
  uint32_t n, body_off;
  uint32_t level_exp;   // (127 - D) << 23
  float softening;
  float dt, gain_up, gain_down;  // dt_eff; clamp(dt * 10, 0, 1) and clamp(dt * 1.05, 0, 1)
  float scale;          // fixed-point deposit scale
};
constexpr float kBias = 0x1.8p23f;  // v + kBias rounds v to an integer, in the sum's low bits
constexpr uint32_t kBiasBits = 0x4B400000u;

__device__ __forceinline__ StepScene step_scene(const SceneDesc &S) {
  const float world_edge = kHalf * 0.985f, edge_band = 0.12f * kHalf;
  const uint32_t D = S.depth;
  StepScene C;
  C.cell_scale = __int_as_float(__float_as_int(0.3125f) + (int)(D << 23));  // RN(1 / 3.2) 2^D
  C.cell_half = __int_as_float((int)(126u + D) << 23) - 0.5f;
  C.cell_margin = 0.5f - __int_as_float((int)(105u + D) << 23);
  // Inside the soft wall's band; none with a scale whose fixed-point
  // coordinates could pass 2^22.
  C.inner = fabsf(S.scale) <= 0x1p21f ? world_edge - edge_band : -1.0f;
  C.dim = 1u << D;
  C.dim2 = 1u << (2u * D);
  C.cell_base = S.cell_off + level_offset_d(D) - kBiasBits * (1u + C.dim + C.dim2);
  C.cell_off = S.cell_off;
  C.n = S.n;
  C.body_off = S.body_off;
  C.level_exp = (127u - D) << 23;
  C.softening = S.softening;
  C.dt = S.dt_eff;
  C.gain_up = clampf_d(S.dt_eff * 10.0f, 0.0f, 1.0f);
  C.gain_down = clampf_d(S.dt_eff * 1.05f, 0.0f, 1.0f);
  C.scale = S.scale;
  return C;
}

// max(|x|, |y|, |z|), NaN if one of them is.
__device__ __forceinline__ float max_abs3(float x, float y, float z) {
  float m;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(fabsf(x)), "f"(fabsf(y)), "f"(fabsf(z)));
  return m;
}

// The leaves positions lie in, as biased coordinates (t - kBias is the cell
// per axis).  w = p 2^D / 3.2 + 2^(D - 1) - 0.5 by one multiply-add differs
// from u 2^D - 0.5 (u: unit_coord) by at most 2^(D - 23), as in
// cells_of_position, so where its distance d from the nearest integer stays
// below 0.5 - 2^(D - 22) that integer is floor(u 2^D).  ok: whether it does on
// every axis.
template <class V, int kN>
__device__ __forceinline__ void biased_cells(const StepScene &C, const V (&p)[3], V (&t)[3], bool (&ok)[kN]) {
  V scale, half, bias, unbias;
  splat(scale, C.cell_scale);
  splat(half, C.cell_half);
  splat(bias, kBias);
  splat(unbias, -kBias);
  float d[3][kN];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const V w = fma2(p[c], scale, half);
    t[c] = add2(w, bias);
    halves(sub2(w, add2(t[c], unbias)), d[c]);
  }
#pragma unroll
  for (int h = 0; h < kN; h++) ok[h] = max_abs3(d[0][h], d[1][h], d[2][h]) <= C.cell_margin;
}
// RN(RN(p scale) + kBias): the fixed-point coordinate in the sum's low bits.
// Two roundings in every variant, as the deposit of an upload makes them.
__device__ __forceinline__ float biased_fixed(float p, float scale, float) {
  return __fadd_rn(__fmul_rn(p, scale), kBias);
}
__device__ __forceinline__ f32x2 biased_fixed(f32x2 p, float scale, f32x2 mz) {
  return add2(mul2(p, pack2(scale, scale), mz), pack2(kBias, kBias));
}
__device__ __forceinline__ float biased_cell_slow(const StepScene &C, float p) {
  return (float)cell_of_unit(unit_coord(p), C.dim) + kBias;
}
__device__ __forceinline__ uint32_t leaf_index(const StepScene &C, float tx, float ty, float tz) {
  return __float_as_uint(tz) * C.dim2 + (__float_as_uint(ty) * C.dim + (__float_as_uint(tx) + C.cell_base));
}

// Interactive control field (wgsl:659-689): its influence at a position, and
// its acceleration added to a.
__device__ __forceinline__ float control_force(const SceneDesc &S, float px, float py, float pz, float &ax, float &ay,
                                               float &az) {
  const float cdx = S.control_point[0] - px, cdy = S.control_point[1] - py,
              cdz = S.control_point[2] - pz;
  const float d2 = (cdx * cdx + cdy * cdy) + cdz * cdz;
  const float cr = fmaxf(S.control_radius, 0.02f);
  const float control_influence = rf_expf(-2.0f * d2 / (cr * cr));
  const float strength = S.control_strength;
  const float inv = inv_sqrt(d2 + cr * cr * 0.018f);
  const float dirx = cdx * inv, diry = cdy * inv, dirz = cdz * inv;
  const float mode = S.control_axis_mode[3];
  if (mode < 1.5f) {
    ax = ax + dirx * strength * control_influence;
    ay = ay + diry * strength * control_influence;
    az = az + dirz * strength * control_influence;
  } else if (mode < 2.5f) {
    ax = ax - dirx * strength * control_influence;
    ay = ay - diry * strength * control_influence;
    az = az - dirz * strength * control_influence;
  } else {
    const float al = length3(S.control_axis_mode[0], S.control_axis_mode[1], S.control_axis_mode[2]);
    const float nx = S.control_axis_mode[0] / al, ny = S.control_axis_mode[1] / al,
                nz = S.control_axis_mode[2] / al;
    const float tx = ny * cdz - nz * cdy, ty = nz * cdx - nx * cdz, tz = nx * cdy - ny * cdx;
    const float tl = length3(tx, ty, tz);
    if (tl > 0.00001f) {
      ax = ax + tx / tl * strength * control_influence;
      ay = ay + ty / tl * strength * control_influence;
      az = az + tz / tl * strength * control_influence;
    }
  }
  return control_influence;
}

// Walls, biased cells and fixed-point coordinates of a body for which the
// short path does not hold.
__device__ __forceinline__ void outer_deposit(const StepScene &C, float4 &p0, float4 &p1, float &tx, float &ty,
                                              float &tz, uint32_t (&q)[3]) {
  const float world_edge = kHalf * 0.985f, edge_band = 0.12f * kHalf;
  soft_wall(p0.x, p1.x, world_edge, edge_band);
  soft_wall(p0.y, p1.y, world_edge, edge_band);
  soft_wall(p0.z, p1.z, world_edge, edge_band);
  q[0] = (uint32_t)f2i_rn_sat(p0.x * C.scale) + kBiasBits;
  q[1] = (uint32_t)f2i_rn_sat(p0.y * C.scale) + kBiasBits;
  q[2] = (uint32_t)f2i_rn_sat(p0.z * C.scale) + kBiasBits;
  tx = biased_cell_slow(C, p0.x);
  ty = biased_cell_slow(C, p0.y);
  tz = biased_cell_slow(C, p0.z);
}

// The integrate (wgsl:613-771) of a lane's kN bodies, V holding one value of
// each: adaptive sample cells, local expansions about their centres, softened
// self-leaf monopoles (kP2P: the pair sums `near` instead), control field,
// symplectic Euler.  Writes the new states into lo, hi and the new positions'
// leaf cells and fixed-point coordinates plus kBiasBits (the next deposit).
template <bool kP2P, class V, int kN>
__device__ __forceinline__ void integrate_bodies(const SceneDesc &S, const StepScene &C, V mz, float4 (&lo)[kN],
                                                 float4 (&hi)[kN], const uint4 *__restrict__ mom,
                                                 const float4 *__restrict__ src, const float4 *__restrict__ aux,
                                                 const uint32_t *__restrict__ choice,
                                                 const float *__restrict__ fields, const float4 *near,
                                                 uint32_t (&key)[kN], uint32_t (&q)[kN][3]) {
  auto mul = [&](V x, V y) { return mul2(x, y, mz); };
  auto all = [](float c) {
    V v;
    splat(v, c);
    return v;
  };
  auto per = [](auto &&f) {  // f(h) of every body h
    float v[kN];
#pragma unroll
    for (int h = 0; h < kN; h++) v[h] = f(h);
    return joined(v);
  };
  auto sum_sq = [&](const V (&x)[3]) { return add2(add2(mul(x[0], x[0]), mul(x[1], x[1])), mul(x[2], x[2])); };

  V p[3] = {per([&](int h) { return lo[h].x; }), per([&](int h) { return lo[h].y; }),
            per([&](int h) { return lo[h].z; })};
  V t[3];
  bool ok[kN], every = true;
  biased_cells(C, p, t, ok);
#pragma unroll
  for (int h = 0; h < kN; h++)  // (unit_coord clamps above 1.59)
    every = every && ok[h] && max_abs3(lo[h].x, lo[h].y, lo[h].z) <= 1.59f;
  if (!every) {
    t[0] = per([&](int h) { return biased_cell_slow(C, lo[h].x); });
    t[1] = per([&](int h) { return biased_cell_slow(C, lo[h].y); });
    t[2] = per([&](int h) { return biased_cell_slow(C, lo[h].z); });
  }
  float u[3][kN];
#pragma unroll
  for (int c = 0; c < 3; c++) halves(t[c], u[c]);

  // The cells the fields are sampled from (wgsl:625-639), see sample_cell;
  // e: their levels, in a float's exponent field.
  uint32_t pick[kN], e[kN], cell[kN];
  bool resolved = true;
#pragma unroll
  for (int h = 0; h < kN; h++) pick[h] = __ldg(&choice[leaf_index(C, u[0][h], u[1][h], u[2][h])]);
#pragma unroll
  for (int h = 0; h < kN; h++) {
    e[h] = (pick[h] >> 5) & 0x07800000u;
    cell[h] = C.cell_off + (pick[h] & 0x0FFFFFFFu);
    resolved = resolved && pick[h] != kChoiceUnresolved;
  }
  if (!resolved) {
#pragma unroll
    for (int h = 0; h < kN; h++) {
      uint32_t level, lx, ly, lz;
      cell[h] = sample_cell(S, lo[h].x, lo[h].y, lo[h].z, mom, choice, level, lx, ly, lz);
      e[h] = level << 23;
    }
  }
  float4 x[kN], f[kN], j[kN], k[kN];
#pragma unroll
  for (int h = 0; h < kN; h++) {
    x[h] = __ldg(&aux[cell[h]]);
    const float4 *fp = reinterpret_cast<const float4 *>(fields + (size_t)cell[h] * 12u);
    f[h] = __ldg(fp);
    j[h] = __ldg(fp + 1);
    k[h] = __ldg(fp + 2);
  }
  // Their centres, negated: the leaf coordinate scaled down and rounded down
  // is the cell's, ((c + 0.5) 2^(1 - l) - 1) kHalf its centre.  The two
  // products with powers of two are exact, so one rounding each serves.
  V r[3];
  {
    const V down = per([&](int h) { return __uint_as_float(C.level_exp + e[h]); });
    const V width = per([&](int h) { return __uint_as_float(0x40000000u - e[h]); });
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const V at = add2(fma2_down(add2(t[c], all(-kBias)), down, all(kBias)), all(-kBias));
      r[c] = add2(p[c], mul(fma2(add2(at, all(0.5f)), width, all(-1.0f)), all(-kHalf)));
    }
  }
  V a[3];
  {
    const V xx = per([&](int h) { return j[h].x; }), xy = per([&](int h) { return j[h].y; }),
            xz = per([&](int h) { return j[h].z; }), yy = per([&](int h) { return j[h].w; }),
            yz = per([&](int h) { return k[h].x; }), zz = per([&](int h) { return k[h].y; });
    auto dot = [&](V g, V tx, V ty, V tz) { return add2(g, add2(add2(mul(tx, r[0]), mul(ty, r[1])), mul(tz, r[2]))); };
    a[0] = dot(per([&](int h) { return f[h].x; }), xx, xy, xz);
    a[1] = dot(per([&](int h) { return f[h].y; }), xy, yy, yz);
    a[2] = dot(per([&](int h) { return f[h].z; }), xz, yz, zz);
  }

  if (kP2P) {
    const V gm = all(S.gravity / S.n_f);
    a[0] = add2(a[0], mul(gm, per([&](int h) { return near[h].x; })));
    a[1] = add2(a[1], mul(gm, per([&](int h) { return near[h].y; })));
    a[2] = add2(a[2], mul(gm, per([&](int h) { return near[h].z; })));
  } else {
    // Self leaf: softened monopole of the other count-1 bodies (wgsl:646-657).
    bool any = false, others[kN];
#pragma unroll
    for (int h = 0; h < kN; h++) {
      others[h] = __float_as_uint(x[h].z) > 1u;
      any = any || others[h];
    }
    if (any) {
      float4 s[kN];
#pragma unroll
      for (int h = 0; h < kN; h++) s[h] = __ldg(&src[cell[h]]);
      const V d[3] = {sub2(per([&](int h) { return s[h].x; }), p[0]), sub2(per([&](int h) { return s[h].y; }), p[1]),
                      sub2(per([&](int h) { return s[h].z; }), p[2])};
      const V eps = per([&](int h) { return fmaxf(C.softening, __uint_as_float(__float_as_uint(0.62f * kHalf) - e[h])); });
      const V inv = inv_sqrt2(add2(sum_sq(d), mul(eps, eps)), mz);
      const V gsm = per([&](int h) { return x[h].x; });  // G * f32(count - 1) / f32(N)
#ifdef RFMM_FAST_FLOAT
      const V w = mul(gsm, mul(mul(inv, inv), inv));  // one weight (reassociated: fast variant only)
#endif
#pragma unroll
      for (int c = 0; c < 3; c++) {
#ifdef RFMM_FAST_FLOAT
        const V with = add2(a[c], mul(d[c], w));
#else
        const V with = add2(a[c], mul(mul(mul(mul(gsm, d[c]), inv), inv), inv));
#endif
        float without[kN], sum[kN];
        halves(a[c], without);
        halves(with, sum);
        a[c] = per([&](int h) { return others[h] ? sum[h] : without[h]; });
      }
    }
  }

  V influence = all(0.0f);
  if (S.control_point[3] > 0.5f) {
    float g[3][kN];
#pragma unroll
    for (int c = 0; c < 3; c++) halves(a[c], g[c]);
    influence = per([&](int h) { return control_force(S, lo[h].x, lo[h].y, lo[h].z, g[0][h], g[1][h], g[2][h]); });
#pragma unroll
    for (int c = 0; c < 3; c++) a[c] = joined(g[c]);
  }

  // Symplectic Euler with excitation and hue state (wgsl:691-769).
  auto clamped = [&](V v, float low, float high) {
    float w[kN];
    halves(v, w);
    return per([&](int h) { return clampf_d(w[h], low, high); });
  };
  // max(RN(sqrt(v)), 1e-4) is the root of max(v, RN(1e-4^2)): the root is
  // monotonic and RN(sqrt(RN(1e-4^2))) = 1e-4.
  auto length_floor = [&](V v) {
    float w[kN];
    halves(v, w);
    return sqrt2<true>(per([&](int h) { return fmaxf(w[h], 0.0001f * 0.0001f); }), mz);
  };
  V v[3] = {per([&](int h) { return hi[h].x; }), per([&](int h) { return hi[h].y; }),
            per([&](int h) { return hi[h].z; })};
  const V radius = length_floor(sum_sq(p)), speed = length_floor(sum_sq(v));
  float pv[kN], rv[kN];
  halves(add2(add2(mul(p[0], v[0]), mul(p[1], v[1])), mul(p[2], v[2])), pv);
  halves(mul(radius, speed), rv);
  float sr[kN];
#pragma unroll
  for (int h = 0; h < kN; h++) sr[h] = clampf_d(pv[h] / rv[h], -1.0f, 1.0f);
  const V signed_radial = joined(sr), rf = per([&](int h) { return fabsf(sr[h]); });
  const V strength =
      clamped(mul(mul(sqrt2<false>(sum_sq(a), mz), add2(radius, all(0.12f))), all(0.58f)), 0.0f, 1.0f);
  const V pulse = per([&](int h) { return x[h].y; });  // clamp((f32(count) - 16) / 72, 0, 1)
  const V target = clamped(add2(add2(add2(add2(all(0.025f), mul(mul(mul(rf, rf), rf), all(0.56f))),
                                          mul(pulse, all(0.26f))),
                                     mul(strength, all(0.13f))),
                                mul(influence, all(0.42f))),
                           0.0f, 1.0f);
  float goal[kN];
  halves(target, goal);
  const V gain = per([&](int h) { return goal[h] > hi[h].w ? C.gain_up : C.gain_down; });
  const V exc = add2(mul(per([&](int h) { return hi[h].w; }), sub2(all(1.0f), gain)), mul(target, gain));

  const V dt = all(C.dt);
#pragma unroll
  for (int c = 0; c < 3; c++) {
    v[c] = add2(v[c], mul(a[c], dt));
    p[c] = add2(p[c], mul(v[c], dt));
  }
  // Clamped to [0, kWidth] before the division instead of [0, 1] after it
  // (the quotient is monotonic and kWidth / kWidth = 1), n = 0 or |n| > 2^-27
  // and finite: the corrected estimate is the rounded quotient.
  constexpr float kWidth = 0.70f - 0.30f, kWidthRcp = 0x1.400002p+1f;  // RN(1 / kWidth)
  const V n = clamped(add2(exc, all(-0.30f)), 0.0f, kWidth), quot = mul(n, all(kWidthRcp));
  const V st = fma2(fma2(quot, all(-kWidth), n), all(kWidthRcp), quot);
  const V drift = sub2(all(1.0f), mul(mul(st, st), sub2(all(3.0f), mul(all(2.0f), st))));
  const V hue = add2(per([&](int h) { return lo[h].w; }),
                     mul(mul(dt, drift), add2(add2(add2(all(0.012f), mul(signed_radial, all(0.030f))),
                                                   mul(exc, all(0.036f))),
                                              mul(influence, all(0.080f)))));
  {
    float o[8][kN];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      halves(p[c], o[c]);
      halves(v[c], o[4 + c]);
    }
    halves(hue, o[3]);
    halves(exc, o[7]);
#pragma unroll
    for (int h = 0; h < kN; h++) {
      lo[h] = make_float4(o[0][h], o[1][h], o[2][h], o[3][h] - floorf(o[3][h]));
      hi[h] = make_float4(o[4][h], o[5][h], o[6][h], o[7][h]);
    }
  }

  // The next step's deposit (wgsl:414-421 on the new position).  Inside the
  // soft wall's band on every axis the walls change nothing, and adding
  // kBias rounds the fixed-point coordinates to the nearest even integer.
  biased_cells(C, p, t, ok);
  float b[3][kN];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    halves(t[c], u[c]);
    halves(biased_fixed(p[c], C.scale, mz), b[c]);
  }
#pragma unroll
  for (int h = 0; h < kN; h++) {
#pragma unroll
    for (int c = 0; c < 3; c++) q[h][c] = __float_as_uint(b[c][h]);
    if (!(ok[h] && max_abs3(lo[h].x, lo[h].y, lo[h].z) <= C.inner))
      outer_deposit(C, lo[h], hi[h], u[0][h], u[1][h], u[2][h], q[h]);
    key[h] = leaf_index(C, u[0][h], u[1][h], u[2][h]);
  }
}

// Persistent integrate: CTA c of G walks body tiles c, c + G, c + 2G, ...
// (each tile is 256 leaf-sorted, spatially compact bodies; interleaving the
// tiles spreads dense and sparse regions, whose per-body costs differ, evenly
// over the CTAs), integrates every body and accumulates the next step's
// deposit in a shared-memory table flushed once at the end.
//
// kP2P: near field by exact pair sums over the leaf-sorted position snapshot;
// no deposit (the end-of-step sort deposits the new positions).
// One body per lane, a tile per CTA of 256: with the level constants in
// StepScene, biased cells and rounding by kBias, 510 instead of 585
// instructions per 32 bodies (1,048,576 Plummer bodies 21.1 -> 20.7 us,
// uniform 18.3 -> 16.2, 5,242,880 clustered 90.7 -> 83.5, fast 73.3 -> 70.2,
// 256 scenes 321 -> 295), still bound by instruction issue.  Two packed bodies
// per lane, a tile per CTA of 128: 344 instructions, one run scan for both;
// what bounds it is the latency of six warps per sub-partition (issue active
// 63 %).  One / two, exact: 250,000 Plummer bodies 6.1 / 8.6, 524,288 11.7 /
// 12.2 (uniform 9.45 / 9.15), 700,000 13.4 / 13.4, 1,048,576 20.4 / 18.9
// (uniform 16.2 / 15.4), 5,242,880 clustered 83.3 / 76.6, 256 scenes 295 /
// 279: pairs pay from about 16 tiles per SM.  What counts is the tiles with
// bodies in them: a server's slots are mostly empty (one request of 250,000 bodies
// in slots of 2^20: 5.9 / 7.6 a step).  The fast variant's contracted chains are
// shorter and gain nothing from packing (clustered 71 / 73).
//
// Resident CTAs per SM: five of 256 (6 / 5: clustered 84.3 / 83.5, 256 scenes
// 300 / 295), six of 128 (5 / 6 / 7: Plummer 21.9 / 19.0 / 20.7, clustered 84 /
// 77 / 79, 256 scenes 299 / 279 / 272).  Loading a pair's next tile ahead costs
// the registers of a CTA; an L2 prefetch of it 77 -> 80.
constexpr uint32_t kPairTiles = 16u;  // per SM
template <uint32_t kBodies>
constexpr uint32_t kIntegrateCtas = kBodies == 1u ? 5u : 6u;
template <bool kP2P, uint32_t kBodies>
__global__ void __launch_bounds__(kTile / kBodies, kIntegrateCtas<kBodies>) k_integrate(const SceneDesc *__restrict__ scenes,
                                                   const uint32_t *__restrict__ tile_scene,
                                                   float4 *__restrict__ part,
                                                   const uint4 *__restrict__ mom,
                                                   const float4 *__restrict__ src,
                                                   const float4 *__restrict__ aux,
                                                   const uint32_t *__restrict__ choice,
                                                   const float *__restrict__ fields,
                                                   uint4 *__restrict__ mom_next, uint32_t tiles,
                                                   const uint32_t *__restrict__ tile_list,
                                                   Counters *__restrict__ ctr, int dynamic,
                                                   const float4 *__restrict__ near4, float minus_zero,
                                                   unsigned long long *__restrict__ stamp) {
  __shared__ DepositTable T;
  __shared__ SceneDesc S;
  __shared__ StepScene C;
  auto enter_scene = [&](uint32_t s) {
    __syncthreads();
    if (threadIdx.x < sizeof(SceneDesc) / 4u)
      reinterpret_cast<uint32_t *>(&S)[threadIdx.x] = reinterpret_cast<const uint32_t *>(scenes + s)[threadIdx.x];
    if (threadIdx.x == 32u) C = step_scene(scenes[s]);
    __syncthreads();
  };
  __shared__ uint32_t s_next;
  if (!kP2P) T.clear();
  // Before the wait for this step's fields: the tile lists and scene
  // descriptors change only by host copies, and the bodies were last written
  // by a launch that was complete before the tree passes between began their
  // work (each of them waited for its predecessor), so the first tile's
  // descriptor and bodies are loaded while those passes drain (a step 0.2 to
  // 0.5 us shorter).
  const uint32_t ntiles = tile_list != nullptr ? min(ctr->tiles_active, tiles) : tiles;
  // Static schedule: interleaved tiles.  Dynamic: tiles are taken one at a
  // time from a counter (reset by this step's upward pass).
  auto grab = [&]() -> uint32_t {
    __syncthreads();
    if (threadIdx.x == 0) s_next = atomicAdd(&ctr->tile_cursor, 1u);
    __syncthreads();
    return s_next;
  };
  // Static schedule: runs of `run` consecutive tiles, interleaved over the
  // CTAs (CTA c takes runs c, c + G, ...).  Single tiles balance best; with
  // at least 16 tiles per CTA (many scenes, whose tiles are contiguous) runs
  // of 4 make the tile's scene change, and its descriptor reload, rarer.
  const uint32_t end = ntiles;
  const uint32_t run_log2 = end >= 16u * gridDim.x ? 2u : 0u;
  uint32_t k = 0u;  // this CTA's static tile count so far
  auto static_tile = [&](uint32_t kk) {
    return (((kk >> run_log2) * gridDim.x + blockIdx.x) << run_log2) + (kk & ((1u << run_log2) - 1u));
  };
  if (dynamic) grid_dependency_wait();  // its counter belongs to the tree passes
  uint32_t i = dynamic ? grab() : static_tile(k);
  uint32_t cur = 0xFFFFFFFFu;
  using V = std::conditional_t<kBodies == 1u, float, f32x2>;
  V mz;
  splat(mz, minus_zero);
  float4 next_lo[kBodies], next_hi[kBodies];
  auto load = [&](uint32_t tile) {
#pragma unroll
    for (uint32_t h = 0; h < kBodies; h++)
      load_body(part, tile * kTile + kBodies * threadIdx.x + h, next_lo[h], next_hi[h]);
  };
  uint32_t next_tile = i < end ? (tile_list != nullptr ? tile_list[i] : i) : 0u;
  if (i < end) {
    load(next_tile);
    cur = tile_scene[next_tile];
    enter_scene(cur);
  }
  grid_dependency_wait();  // fields of this step are complete
  stamp_begin(stamp);
  while (i < end) {
    const uint32_t tile = next_tile, slot = tile * kTile + kBodies * threadIdx.x;
    float4 lo[kBodies], hi[kBodies];
#pragma unroll
    for (uint32_t h = 0; h < kBodies; h++) {
      lo[h] = next_lo[h];
      hi[h] = next_hi[h];
    }
    i = dynamic ? grab() : static_tile(++k);
    // One body per lane: the next tile's are loaded meanwhile; two leave no
    // registers for that.
    if (i < end) next_tile = tile_list != nullptr ? tile_list[i] : i;
    if (kBodies == 1u && i < end) load(next_tile);
    // The CTA's last tile: the next step's upward pass may launch now (it
    // waits for this whole grid before reading anything); its CTAs take SM
    // slots as this grid's CTAs leave.
    if (i >= end) grid_dependents_may_launch();
    const uint32_t sc = tile_scene[tile];
    if (sc != cur) {
      enter_scene(sc);
      cur = sc;
    }
    const uint32_t body = slot - C.body_off;
    uint32_t key[kBodies], q[kBodies][3];
#pragma unroll
    for (uint32_t h = 0; h < kBodies; h++) {
      key[h] = DepositTable::kEmpty;
      q[h][0] = q[h][1] = q[h][2] = kBiasBits;
    }
    if (body < C.n) {
      integrate_bodies<kP2P>(S, C, mz, lo, hi, mom, src, aux, choice, fields, kP2P ? near4 + slot : nullptr, key, q);
#pragma unroll
      for (uint32_t h = 0; h < kBodies; h++) {
        if (h == 0u || body + h < C.n)
          store_body(part, slot + h, lo[h], hi[h]);
        else
          key[h] = DepositTable::kEmpty;
      }
    }
    if (kBodies > 1u && i < end) load(next_tile);
    if (!kP2P) {
      if constexpr (kBodies == 1u)
        deposit_body<kBiasBits>(T, key[0], key[0] != DepositTable::kEmpty, q[0][0], q[0][1], q[0][2], mom_next);
      else
        deposit_two<kBiasBits>(T, key[0], key[1], q[0], q[1], mom_next);
    }
  }
  if (!kP2P) {
    __syncthreads();
    T.flush(mom_next);
  }
  stamp_end(stamp);
  grid_dependents_may_launch();
}

// ------------------------------------------------------------ P2P near field
//
// Exact softened pair sums of every body over the bodies of the 3x3x3 cells
// around its sample cell (kNearP2P), written per slot for the integrate that
// follows.  What bounds it is the FP32 pipe: 23 operations per pair in the
// exact contract, 11 in the fast variant, with packed three-operand
// multiply-adds at 3.2 instead of 2 cycles (measured: their register reads)
// about 29 and 13 cycles per warp and source.
//
// Warps work alone: a warp takes kUnit consecutive leaf-sorted slots from a
// counter, so the expensive core regions spread over every SM sub-partition
// (a CTA per 256 slots left most of them idle at 120,001 bodies).  Lanes
// 0..26 look up the 27 neighbour ranges at once; their sources form one
// sequence (cells z-, y-, x-major, bodies in slot order) that the warp stages
// in chunks of kP2PChunk as x, y and z rows in shared memory, two sources to
// a packed operation (the packed forms keep each half's rounding and save
// issue slots).  The next chunk's loads are in flight meanwhile.  A warp
// whose bodies sample several cells does one cell after the other.
//
// The exact variant adds every term in that order, so the sums equal
// p2p_sums bit for bit.  The body itself and the padding of the last chunk
// add +0, which changes no sum (sums start at +0 and never become -0).  The
// inner loop has no range check: it runs when every source of the chunk lies
// within 2^60, every body of the warp within 2^59 and softening^2 between
// 2^-80 and 2^120, so that 2^-80 <= r^2 < 2^127 and a padding term underflows
// to +0; otherwise (non-finite or astronomically distant bodies, no
// softening) p2p_chunk_checked evaluates the plain expressions.
//
// kSplit lanes share a body: each evaluates its share of the sources.  The
// fast variant sums the shares at the end.  In the exact variant the terms
// cross through shared memory and lane c of a body's lanes adds component c
// in order.  A cell holding one of the warp's bodies is summed by all 32
// lanes, one holding up to eight by four lanes each (outlying bodies share a
// warp with few of their cell's but have up to every body of the scene as a
// source: one such warp used to end the launch).
//
// Measured, ms per launch, one CTA per 256 slots with IEEE 1/sqrt before ->
// now: Plummer 1,048,576 exact 167 -> 102, fast 88 -> 55; Plummer 120,001
// exact 50 -> 6.7; clusters 600,007 fast 26 -> 11.7.

constexpr uint32_t kP2PChunk = 128u;       // sources per staged chunk: four per lane
constexpr uint32_t kP2PWarps = 4u;         // warps per CTA (independent)
constexpr float kP2PFar = 0x1p60f;         // padding coordinate: its term underflows to +0
#ifdef RFMM_FAST_FLOAT
constexpr uint32_t kP2PBodies = 2u;        // bodies per lane
#else
constexpr uint32_t kP2PBodies = 1u;
#endif
// Resident CTAs per SM.  Exact, unsplit: with 16 sources in flight three warps
// per sub-partition fill the pipe, and fewer units are half done when the
// last are taken (3 / 4 CTAs with 16 sources, 4 with 8, ms: Plummer 120,001
// 6.7 / 7.1 / 7.5, 1,048,576 102 / 104 / 108, clusters 600,007 21.6 / 21.8 /
// 24.6); the fast variant needs four (3 / 4: Plummer 120,001 3.7 / 3.4).
template <uint32_t kSplit>
constexpr uint32_t kP2PCtas = kSplit == 1u && kP2PBodies == 1u ? 3u : 4u;
template <uint32_t kSplit>
constexpr uint32_t kP2PUnit = 32u / kSplit * kP2PBodies;  // slots per work unit
// One warp's staged sources: x, y and z rows of a chunk, and the neighbour
// ranges as a sequence (first sequence index of each range, and what to add to
// a sequence index to get its slot).
struct alignas(16) P2PStage {
  float x[kP2PChunk], y[kP2PChunk], z[kP2PChunk];
  uint32_t first[28], shift[27];
};
static_assert(sizeof(P2PStage) % 16u == 0u && kP2PChunk % 8u == 0u, "rows are read up to 16 bytes at a time");

// Terms on their way to the adding lanes (exact variant).  kSplit 4: 16
// sources of body b, component c from kP2PTermBody b + kP2PTermComp c on (the
// strides put the 16-byte accesses of eight lanes on distinct banks), two
// buffers in turn; kSplit 32: one row of 128 sources per component.
constexpr uint32_t kP2PTermBody = 80u, kP2PTermComp = 20u;
struct alignas(16) P2PTerms {
  float v[2][8u * kP2PTermBody];
};
static_assert(8u * kP2PTermBody >= 3u * kP2PChunk, "kSplit 32 uses one buffer");

// One source's contribution (the expression p2p_sums evaluates).
__device__ __forceinline__ void p2p_pair(float qx, float qy, float qz, float px, float py, float pz,
                                         float eps2, float &sx, float &sy, float &sz) {
  const float dx = qx - px, dy = qy - py, dz = qz - pz;
  const float r2 = ((dx * dx + dy * dy) + dz * dz) + eps2;
  const float inv = inv_sqrt(r2);
  const float w = (inv * inv) * inv;
  sx = sx + dx * w;
  sy = sy + dy * w;
  sz = sz + dz * w;
}

// Sums of one lane's body over a staged chunk of `m` sources.  `self` is the
// chunk index of the body itself (anything >= m: not in this chunk).
__device__ __noinline__ float3 p2p_chunk_checked(const P2PStage &T, uint32_t m, uint32_t self, float px,
                                                 float py, float pz, float eps2, float3 s) {
  for (uint32_t k = 0; k < m; k++)
    if (k != self) p2p_pair(T.x[k], T.y[k], T.z[k], px, py, pz, eps2, s.x, s.y, s.z);
  return s;
}

// One body's side of the packed loop: minus its position, twice.
struct P2PBody {
  f32x2 nx, ny, nz;
};

#ifdef RFMM_FAST_FLOAT
// Even and odd sources of a chunk in the halves of the partial sums.
__device__ __forceinline__ void p2p_two(f32x2 qx, f32x2 qy, f32x2 qz, const P2PBody &b, f32x2 eps2, f32x2 mz,
                                        f32x2 &sx, f32x2 &sy, f32x2 &sz) {
  const f32x2 dx = add2(qx, b.nx), dy = add2(qy, b.ny), dz = add2(qz, b.nz);
  const f32x2 r2 = fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, eps2)));
  float x0, x1;
  unpack2(r2, x0, x1);
  const f32x2 inv = pack2(rsqrt_estimate(x0), rsqrt_estimate(x1));
  const f32x2 w = mul2(mul2(inv, inv, mz), inv, mz);
  sx = fma2(dx, w, sx);
  sy = fma2(dy, w, sy);
  sz = fma2(dz, w, sz);
}
#else
// The terms of two consecutive sources.
__device__ __forceinline__ void p2p_two(f32x2 qx, f32x2 qy, f32x2 qz, const P2PBody &b, f32x2 eps2, f32x2 mz,
                                        f32x2 &tx, f32x2 &ty, f32x2 &tz) {
  const f32x2 dx = add2(qx, b.nx), dy = add2(qy, b.ny), dz = add2(qz, b.nz);
  const f32x2 r2 = add2(add2(add2(mul2(dx, dx, mz), mul2(dy, dy, mz)), mul2(dz, dz, mz)), eps2);
  float x0, x1;
  unpack2(r2, x0, x1);
  const f32x2 inv = inv_sqrt2_in_range(r2, x0, x1, mz);
  const f32x2 w = mul2(mul2(inv, inv, mz), inv, mz);
  tx = mul2(dx, w, mz);
  ty = mul2(dy, w, mz);
  tz = mul2(dz, w, mz);
}
__device__ __forceinline__ float add_both(float s, f32x2 t) {
  float a, b;
  unpack2(t, a, b);
  return __fadd_rn(__fadd_rn(s, a), b);
}
#endif

// Slot range [lo, hi) of neighbour j (0..26, in the reference's z-, y-,
// x-major order) of cell (cx, cy, cz) at level l; false when j lies outside
// the grid.
__device__ __forceinline__ bool neighbour_range(const SceneDesc &S, const uint32_t *starts,
                                                uint32_t l, uint32_t cx, uint32_t cy, uint32_t cz,
                                                uint32_t j, uint32_t &lo, uint32_t &hi) {
  const int dim = 1 << l;
  const int nx = (int)cx + (int)(j % 3u) - 1, ny = (int)cy + (int)((j / 3u) % 3u) - 1,
            nz = (int)cz + (int)(j / 9u) - 1;
  if (nx < 0 || ny < 0 || nz < 0 || nx >= dim || ny >= dim || nz >= dim) return false;
  const uint32_t sh3 = 3u * (S.depth - l);
  const uint32_t m = morton3((uint32_t)nx, (uint32_t)ny, (uint32_t)nz);
  lo = __ldg(&starts[S.cell_off + (m << sh3)]);
  hi = __ldg(&starts[S.cell_off + ((m + 1u) << sh3)]);
  return true;
}

// One pass of a warp over the `total` sources of a cell's neighbourhood: the
// sums of kB bodies per lane, kSplit lanes to a body (the same values in each
// of them).  `self[b]` is the slot of body b, `slot` arguments index pos4.
template <uint32_t kSplit, uint32_t kB>
__device__ __forceinline__ void p2p_pass(P2PStage &T, P2PTerms &U, const float4 *__restrict__ pos4, uint32_t total,
                                         float eps2, f32x2 mz, bool plain, const float (&px)[kB],
                                         const float (&py)[kB], const float (&pz)[kB], const uint32_t (&self)[kB],
                                         float3 (&out)[kB]) {
  constexpr uint32_t kAll = 0xFFFFFFFFu, kNone = 0xFFFFFFFFu, kPer = kP2PChunk / 32u;
  const uint32_t lane = threadIdx.x & 31u, sub = lane % kSplit;
  P2PBody body[kB];
  float3 acc[kB];
#pragma unroll
  for (uint32_t b = 0; b < kB; b++) {
    body[b] = {pack2(-px[b], -px[b]), pack2(-py[b], -py[b]), pack2(-pz[b], -pz[b])};
    acc[b] = make_float3(0.0f, 0.0f, 0.0f);
  }
  const f32x2 e2 = pack2(eps2, eps2);
  uint32_t range[kPer];
  float4 q[kPer];
#pragma unroll
  for (uint32_t i = 0; i < kPer; i++) range[i] = 0u;
  auto fetch = [&](uint32_t base) {
#pragma unroll
    for (uint32_t i = 0; i < kPer; i++) {
      const uint32_t v = base + 32u * i + lane;
      q[i] = make_float4(kP2PFar, kP2PFar, kP2PFar, 0.0f);
      if (v < total) {
        while (v >= T.first[range[i] + 1u]) range[i]++;
        q[i] = __ldg(&pos4[v + T.shift[range[i]]]);
      }
    }
  };
  fetch(0u);
  for (uint32_t base = 0; base < total; base += kP2PChunk) {
    bool near = plain;
    __syncwarp();  // the previous chunk is consumed
#pragma unroll
    for (uint32_t i = 0; i < kPer; i++) {
      T.x[32u * i + lane] = q[i].x;
      T.y[32u * i + lane] = q[i].y;
      T.z[32u * i + lane] = q[i].z;
      near = near && fabsf(q[i].x) <= kP2PFar && fabsf(q[i].y) <= kP2PFar && fabsf(q[i].z) <= kP2PFar;
    }
    near = __all_sync(kAll, near);
    __syncwarp();
    if (base + kP2PChunk < total) fetch(base + kP2PChunk);
    const uint32_t m = min(kP2PChunk, total - base);
    if (!near) {
      // Plain expressions; the first of a body's lanes sums for all.
#pragma unroll
      for (uint32_t b = 0; b < kB; b++) {
        uint32_t at = kNone;  // the body's sequence index, if its slot is among these sources
        for (uint32_t j = 0; j < 27u; j++) {
          const uint32_t v = self[b] - T.shift[j];
          const uint32_t end = j < 26u ? T.first[j + 1u] : total;
          if (v >= T.first[j] && v < end) at = v;
        }
#ifdef RFMM_FAST_FLOAT
        if (sub == 0u) acc[b] = p2p_chunk_checked(T, m, at - base, px[b], py[b], pz[b], eps2, acc[b]);
#else
        const uint32_t l0 = lane - sub;
        float3 s = acc[b];
        if (kSplit > 1u)
          s = make_float3(__shfl_sync(kAll, acc[b].x, l0), __shfl_sync(kAll, acc[b].x, l0 + 1u),
                          __shfl_sync(kAll, acc[b].x, l0 + 2u));
        s = p2p_chunk_checked(T, m, at - base, px[b], py[b], pz[b], eps2, s);
        if (kSplit > 1u) acc[b].x = sub == 0u ? s.x : (sub == 1u ? s.y : s.z);
        else acc[b] = s;
#endif
      }
      __syncwarp();
      continue;
    }
#ifdef RFMM_FAST_FLOAT
    // Fresh partial sums per chunk (the order of addition is free here).
    f32x2 ax[kB], ay[kB], az[kB];
#pragma unroll
    for (uint32_t b = 0; b < kB; b++) ax[b] = ay[b] = az[b] = 0ull;
#pragma unroll 2
    for (uint32_t k = 0; k < m; k += 2u * kSplit) {
      const f32x2 qx = *reinterpret_cast<const f32x2 *>(&T.x[k + 2u * sub]);
      const f32x2 qy = *reinterpret_cast<const f32x2 *>(&T.y[k + 2u * sub]);
      const f32x2 qz = *reinterpret_cast<const f32x2 *>(&T.z[k + 2u * sub]);
#pragma unroll
      for (uint32_t b = 0; b < kB; b++) p2p_two(qx, qy, qz, body[b], e2, mz, ax[b], ay[b], az[b]);
    }
#pragma unroll
    for (uint32_t b = 0; b < kB; b++) {
      float u, v;
      unpack2(ax[b], u, v);
      acc[b].x = acc[b].x + (u + v);
      unpack2(ay[b], u, v);
      acc[b].y = acc[b].y + (u + v);
      unpack2(az[b], u, v);
      acc[b].z = acc[b].z + (u + v);
    }
#else
    if constexpr (kSplit == 1u) {
#pragma unroll 4
      for (uint32_t k = 0; k < m; k += 4u) {
        const ulonglong2 qx = *reinterpret_cast<const ulonglong2 *>(&T.x[k]);
        const ulonglong2 qy = *reinterpret_cast<const ulonglong2 *>(&T.y[k]);
        const ulonglong2 qz = *reinterpret_cast<const ulonglong2 *>(&T.z[k]);
        f32x2 tx, ty, tz, ux, uy, uz;
        p2p_two(qx.x, qy.x, qz.x, body[0], e2, mz, tx, ty, tz);
        p2p_two(qx.y, qy.y, qz.y, body[0], e2, mz, ux, uy, uz);
        acc[0].x = add_both(add_both(acc[0].x, tx), ux);
        acc[0].y = add_both(add_both(acc[0].y, ty), uy);
        acc[0].z = add_both(add_both(acc[0].z, tz), uz);
      }
    } else {
      // A group of 4 kSplit sources, four to a lane; acc[0].x is the running
      // sum of component `sub` (lanes 3 and up of a body: unused).
      constexpr uint32_t kGroup = 4u * kSplit, kRow = kSplit == 4u ? kP2PTermComp : kGroup;
      const uint32_t row0 = (lane / kSplit) * kP2PTermBody;
      const uint32_t put = row0 + 4u * sub, get = row0 + min(sub, 2u) * kRow;
      auto eval = [&](uint32_t k, ulonglong2 &tx, ulonglong2 &ty, ulonglong2 &tz) {
        const ulonglong2 qx = *reinterpret_cast<const ulonglong2 *>(&T.x[k + 4u * sub]);
        const ulonglong2 qy = *reinterpret_cast<const ulonglong2 *>(&T.y[k + 4u * sub]);
        const ulonglong2 qz = *reinterpret_cast<const ulonglong2 *>(&T.z[k + 4u * sub]);
        p2p_two(qx.x, qy.x, qz.x, body[0], e2, mz, tx.x, ty.x, tz.x);
        p2p_two(qx.y, qy.y, qz.y, body[0], e2, mz, tx.y, ty.y, tz.y);
      };
      auto store = [&](float *buf, ulonglong2 tx, ulonglong2 ty, ulonglong2 tz) {
        *reinterpret_cast<ulonglong2 *>(buf + put) = tx;
        *reinterpret_cast<ulonglong2 *>(buf + put + kRow) = ty;
        *reinterpret_cast<ulonglong2 *>(buf + put + 2u * kRow) = tz;
        __syncwarp();
      };
      auto add4 = [&](const float *at) {
        const float4 t = *reinterpret_cast<const float4 *>(at);
        acc[0].x = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc[0].x, t.x), t.y), t.z), t.w);
      };
      ulonglong2 tx, ty, tz;
      eval(0u, tx, ty, tz);
      store(U.v[0], tx, ty, tz);
      if constexpr (kSplit == 4u) {
        // The next group's terms are evaluated while this one's are added;
        // each buffer is read before the barrier that precedes its next store.
#pragma unroll 2
        for (uint32_t k = 0; k < m; k += kGroup) {
          const float *buf = U.v[(k / kGroup) & 1u] + get;
          const bool more = k + kGroup < m;
          if (more) eval(k + kGroup, tx, ty, tz);
#pragma unroll
          for (uint32_t i = 0; i < kGroup; i += 4u) add4(buf + i);
          if (more) store(U.v[(k / kGroup + 1u) & 1u], tx, ty, tz);
        }
        __syncwarp();
      } else {
#pragma unroll 8
        for (uint32_t i = 0; i < m; i += 4u) add4(U.v[0] + get + i);
        __syncwarp();
      }
    }
#endif
  }
#pragma unroll
  for (uint32_t b = 0; b < kB; b++) {
    if constexpr (kSplit > 1u) {
#ifdef RFMM_FAST_FLOAT
#pragma unroll
      for (uint32_t o = 1u; o < kSplit; o <<= 1) {
        acc[b].x = acc[b].x + __shfl_xor_sync(kAll, acc[b].x, o);
        acc[b].y = acc[b].y + __shfl_xor_sync(kAll, acc[b].y, o);
        acc[b].z = acc[b].z + __shfl_xor_sync(kAll, acc[b].z, o);
      }
#else
      const uint32_t l0 = lane - sub;
      const float c = acc[b].x;
      acc[b] = make_float3(__shfl_sync(kAll, c, l0), __shfl_sync(kAll, c, l0 + 1u), __shfl_sync(kAll, c, l0 + 2u));
#endif
    }
    out[b] = acc[b];
  }
}

template <uint32_t kSplit>
__global__ void __launch_bounds__(32 * kP2PWarps, kP2PCtas<kSplit>) k_near_p2p(const SceneDesc *__restrict__ scenes,
                                                  const uint32_t *__restrict__ tile_scene,
                                                  const float4 *__restrict__ pos4,
                                                  const uint32_t *__restrict__ starts,
                                                  const uint4 *__restrict__ mom,
                                                  const uint32_t *__restrict__ choice,
                                                  uint32_t tiles,
                                                  const uint32_t *__restrict__ tile_list,
                                                  Counters *__restrict__ ctr,
                                                  float4 *__restrict__ near_out, float minus_zero,
                                                  unsigned long long *__restrict__ stamp) {
  constexpr uint32_t kUnit = kP2PUnit<kSplit>, kUnitsPerTile = kTile / kUnit, kBody = 32u / kSplit;
  static_assert(kTile % kUnit == 0u, "a unit never crosses a tile");
  constexpr uint32_t kAll = 0xFFFFFFFFu, kNone = 0xFFFFFFFFu;
  __shared__ P2PStage stage[kP2PWarps];
  __shared__ P2PTerms terms[kP2PBodies == 1u ? kP2PWarps : 1u];  // the fast variant has no use for it
  const uint32_t lane = threadIdx.x & 31u, sub = lane % kSplit;
  P2PStage &T = stage[threadIdx.x >> 5];
  P2PTerms &U = terms[kP2PBodies == 1u ? threadIdx.x >> 5 : 0u];
  const f32x2 mz = pack2(minus_zero, minus_zero);
  grid_dependency_wait();  // the upward pass resolved this step's sample cells
  stamp_begin(stamp);
  const uint32_t ntiles = tile_list != nullptr ? min(ctr->tiles_active, tiles) : tiles;
  const uint32_t nunits = ntiles * kUnitsPerTile;
  for (;;) {
    // A unit's cost is its bodies times the sources around their sample
    // cells, two orders of magnitude apart between sparse and core leaves:
    // units come from a counter (reset by this step's upward pass).
    uint32_t unit = 0u;
    if (lane == 0u) unit = atomicAdd(&ctr->p2p_cursor, 1u);
    unit = __shfl_sync(kAll, unit, 0);
    if (unit >= nunits) break;
    // From both ends of the slots inwards: the ends of the Morton order hold
    // the outlying bodies, whose warps take longest (last, they ended the
    // launch: Plummer 120,001 exact 8.7 -> 7.5 ms, clusters 600,007 31.9 ->
    // 24.6, fast 15.4 -> 11.7).
    unit = (unit & 1u) ? nunits - 1u - (unit >> 1) : unit >> 1;
    const uint32_t entry = unit / kUnitsPerTile;
    const uint32_t tile = tile_list != nullptr ? tile_list[entry] : entry;
    const SceneDesc &S = scenes[tile_scene[tile]];
    const uint32_t slot0 = tile * kTile + (unit % kUnitsPerTile) * kUnit + lane / kSplit;
    const float eps2 = S.softening * S.softening;

    float px[kP2PBodies], py[kP2PBodies], pz[kP2PBodies];
    uint32_t level[kP2PBodies], cx[kP2PBodies], cy[kP2PBodies], cz[kP2PBodies], key[kP2PBodies], self[kP2PBodies];
    float3 sum[kP2PBodies];
    bool plain = eps2 >= 0x1p-80f && eps2 <= 0x1p120f;
#pragma unroll
    for (uint32_t b = 0; b < kP2PBodies; b++) {
      const uint32_t slot = slot0 + kBody * b;
      self[b] = slot;
      px[b] = py[b] = pz[b] = 0.0f;
      level[b] = cx[b] = cy[b] = cz[b] = 0u;
      key[b] = kNone;
      if (slot - S.body_off < S.n) {
        const float4 p = pos4[slot];
        px[b] = p.x;
        py[b] = p.y;
        pz[b] = p.z;
        key[b] = sample_cell(S, p.x, p.y, p.z, mom, choice, level[b], cx[b], cy[b], cz[b]);
        const uint32_t csh = S.depth - level[b];
        cx[b] >>= csh;
        cy[b] >>= csh;
        cz[b] >>= csh;
      }
      plain = plain && fabsf(px[b]) < 0.5f * kP2PFar && fabsf(py[b]) < 0.5f * kP2PFar &&
              fabsf(pz[b]) < 0.5f * kP2PFar;
      sum[b] = make_float3(0.0f, 0.0f, 0.0f);
    }
    plain = __all_sync(kAll, plain);

    // One sample cell after the other.
    bool done[kP2PBodies];
#pragma unroll
    for (uint32_t b = 0; b < kP2PBodies; b++) done[b] = key[b] == kNone;
    for (;;) {
      uint32_t gkey = kNone, gl = 0u, gx = 0u, gy = 0u, gz = 0u;
#pragma unroll
      for (uint32_t b = 0; b < kP2PBodies; b++) {
        const uint32_t open = __ballot_sync(kAll, !done[b]);
        if (gkey == kNone && open != 0u) {
          const uint32_t lead = (uint32_t)__ffs(open) - 1u;
          gkey = __shfl_sync(kAll, key[b], lead);
          gl = __shfl_sync(kAll, level[b], lead);
          gx = __shfl_sync(kAll, cx[b], lead);
          gy = __shfl_sync(kAll, cy[b], lead);
          gz = __shfl_sync(kAll, cz[b], lead);
        }
      }
      if (gkey == kNone) break;
      // The neighbour ranges as one sequence of `total` sources.
      uint32_t lo = 0u, hi = 0u;
      if (lane < 27u && !neighbour_range(S, starts, gl, gx, gy, gz, lane, lo, hi)) lo = hi = 0u;
      uint32_t upto = hi - lo;
#pragma unroll
      for (uint32_t off = 1u; off < 32u; off <<= 1) {
        const uint32_t t = __shfl_up_sync(kAll, upto, off);
        if (lane >= off) upto += t;
      }
      const uint32_t total = __shfl_sync(kAll, upto, 31);
      __syncwarp();  // the previous cell's ranges and chunk are consumed
      if (lane < 27u) {
        T.first[lane] = upto - (hi - lo);
        T.shift[lane] = lo - (upto - (hi - lo));
      }
      if (lane == 27u) T.first[27] = kNone;
      __syncwarp();

      // The unit's bodies in this cell (a body's first lane counts for it).
      uint32_t members[kP2PBodies], count = 0u;
#pragma unroll
      for (uint32_t b = 0; b < kP2PBodies; b++) {
        members[b] = __ballot_sync(kAll, key[b] == gkey && sub == 0u);
        count += __popc(members[b]);
      }
      if (count == 1u) {
#pragma unroll
        for (uint32_t b = 0; b < kP2PBodies; b++) {
          if (members[b] == 0u) continue;
          const uint32_t owner = (uint32_t)__ffs(members[b]) - 1u;
          const float ox[1] = {__shfl_sync(kAll, px[b], owner)}, oy[1] = {__shfl_sync(kAll, py[b], owner)},
                      oz[1] = {__shfl_sync(kAll, pz[b], owner)};
          const uint32_t oself[1] = {__shfl_sync(kAll, self[b], owner)};
          float3 o[1];
          p2p_pass<32u, 1u>(T, U, pos4, total, eps2, mz, plain, ox, oy, oz, oself, o);
          if (lane / kSplit == owner / kSplit) sum[b] = o[0];
        }
      } else if (kSplit == 1u && count <= 8u) {
        // Four lanes to a body: quad j takes the cell's j-th body.
#pragma unroll
        for (uint32_t b = 0; b < kP2PBodies; b++) {
          if (members[b] == 0u) continue;
          const uint32_t rank = __popc(members[b] & ((1u << lane) - 1u));
          const uint32_t owner = __fns(members[b], 0u, (int)min(lane >> 2, (uint32_t)__popc(members[b]) - 1u) + 1);
          const float ox[1] = {__shfl_sync(kAll, px[b], owner)}, oy[1] = {__shfl_sync(kAll, py[b], owner)},
                      oz[1] = {__shfl_sync(kAll, pz[b], owner)};
          const uint32_t oself[1] = {__shfl_sync(kAll, self[b], owner)};
          float3 o[1];
          p2p_pass<4u, 1u>(T, U, pos4, total, eps2, mz, plain, ox, oy, oz, oself, o);
          const float rx = __shfl_sync(kAll, o[0].x, 4u * rank & 31u), ry = __shfl_sync(kAll, o[0].y, 4u * rank & 31u),
                      rz = __shfl_sync(kAll, o[0].z, 4u * rank & 31u);
          if (key[b] == gkey) sum[b] = make_float3(rx, ry, rz);
        }
      } else {
        float3 o[kP2PBodies];
        p2p_pass<kSplit, kP2PBodies>(T, U, pos4, total, eps2, mz, plain, px, py, pz, self, o);
#pragma unroll
        for (uint32_t b = 0; b < kP2PBodies; b++)
          if (key[b] == gkey) sum[b] = o[b];
      }
#pragma unroll
      for (uint32_t b = 0; b < kP2PBodies; b++) done[b] = done[b] || key[b] == gkey;
    }
#pragma unroll
    for (uint32_t b = 0; b < kP2PBodies; b++)
      if (key[b] != kNone && sub == 0u) near_out[slot0 + kBody * b] = make_float4(sum[b].x, sum[b].y, sum[b].z, 0.0f);
  }
  stamp_end(stamp);
  grid_dependents_may_launch();
}

// Standalone P2M: deposit the current positions into `moments` (leaf level
// must be zero).  Persistent like k_integrate.
__global__ void __launch_bounds__(256) k_deposit(const SceneDesc *__restrict__ scenes,
                                                 const uint32_t *__restrict__ tile_scene,
                                                 const float4 *__restrict__ part,
                                                 uint4 *__restrict__ moments, uint32_t tiles,
                                                 const uint32_t *__restrict__ tile_list,
                                                 const Counters *__restrict__ ctr) {
  __shared__ DepositTable T;
  __shared__ SceneDesc S;
  const uint32_t ntiles = tile_list != nullptr ? min(ctr->tiles_active, tiles) : tiles;
  uint32_t t0, t1;
  cta_tile_range(ntiles, t0, t1);
  T.clear();
  uint32_t cur = 0xFFFFFFFFu;
  for (uint32_t i = t0; i < t1; i++) {
    const uint32_t tile = tile_list != nullptr ? tile_list[i] : i;
    const uint32_t slot = tile * kTile + threadIdx.x;
    const float4 p = part[2u * slot];
    const uint32_t sc = tile_scene[tile];
    if (sc != cur) {
      load_scene(S, scenes, sc);
      cur = sc;
    }
    const bool active = slot - S.body_off < S.n;
    uint32_t key = DepositTable::kEmpty;
    uint32_t qx = 0, qy = 0, qz = 0;
    if (active) {
      key = S.cell_off + leaf_cell(p.x, p.y, p.z, S.depth);
      qx = (uint32_t)f2i_rn_sat(p.x * S.scale);
      qy = (uint32_t)f2i_rn_sat(p.y * S.scale);
      qz = (uint32_t)f2i_rn_sat(p.z * S.scale);
    }
    deposit_body(T, key, active, qx, qy, qz, moments);
  }
  __syncthreads();
  T.flush(moments);
}

// FMM acceleration and potential of every body of one scene, written in the
// caller's body order (diagnostics and force-error checks; not on the step).
__global__ void __launch_bounds__(256) k_accel(const SceneDesc *__restrict__ scenes,
                                               const uint32_t *__restrict__ tile_scene,
                                               const float4 *__restrict__ part,
                                               const uint32_t *__restrict__ ids,
                                               const uint4 *__restrict__ mom,
                                               const float4 *__restrict__ src,
                                               const float4 *__restrict__ aux,
                                               const uint32_t *__restrict__ choice,
                                               const float *__restrict__ fields,
                                               float4 *__restrict__ out, uint32_t tile_base,
                                               const float4 *__restrict__ pos4,
                                               const uint32_t *__restrict__ starts) {
  const uint32_t tile = tile_base + blockIdx.x;
  const SceneDesc &S = scenes[tile_scene[tile]];
  const uint32_t slot = tile * kTile + threadIdx.x;
  if (slot - S.body_off >= S.n) return;
  const uint32_t id = ids[slot];
  if (id >= S.n) return;
  const float4 p = part[2u * slot];
  float ax, ay, az, pulse, phi;
  if (S.near_mode == kNearP2P) {
    const P2PView V{pos4, starts, slot};
    body_acceleration<true, true>(S, p.x, p.y, p.z, mom, src, aux, choice, fields, ax, ay, az, pulse,
                                  &phi, &V);
  } else {
    body_acceleration<true>(S, p.x, p.y, p.z, mom, src, aux, choice, fields, ax, ay, az, pulse, &phi);
  }
  out[S.body_off + id] = make_float4(ax, ay, az, phi);
}

// Resident slot of every body of one scene: slot_of[body_off + id] = slot.
__global__ void __launch_bounds__(256) k_slot_of(const SceneDesc *__restrict__ scenes,
                                                 const uint32_t *__restrict__ tile_scene,
                                                 const uint32_t *__restrict__ ids,
                                                 uint32_t *__restrict__ slot_of, uint32_t tile_base) {
  const uint32_t tile = tile_base + blockIdx.x;
  const SceneDesc &S = scenes[tile_scene[tile]];
  const uint32_t slot = tile * kTile + threadIdx.x;
  if (slot - S.body_off >= S.n) return;
  const uint32_t id = ids[slot];
  if (id < S.n) slot_of[S.body_off + id] = slot;
}

// FMM acceleration + potential of selected bodies (caller ids) of one scene.
__global__ void __launch_bounds__(256) k_accel_targets(
    const SceneDesc *__restrict__ scenes, uint32_t scene, const float4 *__restrict__ part,
    const uint32_t *__restrict__ slot_of, const uint32_t *__restrict__ targets, uint32_t nt,
    const uint4 *__restrict__ mom, const float4 *__restrict__ src, const float4 *__restrict__ aux,
    const uint32_t *__restrict__ choice, const float *__restrict__ fields, float4 *__restrict__ out,
    const float4 *__restrict__ pos4, const uint32_t *__restrict__ starts) {
  const SceneDesc &S = scenes[scene];
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt || targets[t] >= S.n) return;
  const uint32_t slot = slot_of[S.body_off + targets[t]];
  const float4 p = part[2u * slot];
  float ax, ay, az, pulse, phi;
  if (S.near_mode == kNearP2P) {
    const P2PView V{pos4, starts, slot};
    body_acceleration<true, true>(S, p.x, p.y, p.z, mom, src, aux, choice, fields, ax, ay, az, pulse,
                                  &phi, &V);
  } else {
    body_acceleration<true>(S, p.x, p.y, p.z, mom, src, aux, choice, fields, ax, ay, az, pulse, &phi);
  }
  out[t] = make_float4(ax, ay, az, phi);
}

void launch_accel_targets(const LaunchCtx &L, uint32_t scene, uint32_t tile_base, uint32_t tiles,
                          const uint32_t *ids, uint32_t *slot_of, const uint32_t *targets,
                          uint32_t nt, float4 *out) {
  k_slot_of<<<tiles, kTile, 0, L.stream>>>(L.scenes, L.tile_scene, ids, slot_of, tile_base);
  k_accel_targets<<<(nt + 255u) / 256u, 256, 0, L.stream>>>(
      L.scenes, scene, L.part, slot_of, targets, nt, L.mom, L.src, L.aux, L.choice, L.fields, out,
      L.pos4, L.starts_out);
}

void launch_accel(const LaunchCtx &L, const uint32_t *ids, float4 *out, uint32_t tile_base,
                  uint32_t tiles) {
  k_accel<<<tiles, kTile, 0, L.stream>>>(L.scenes, L.tile_scene, L.part, ids, L.mom, L.src, L.aux,
                                         L.choice, L.fields, out, tile_base, L.pos4, L.starts_out);
}

// Sort keys of the bodies, a tile at a time, and the totals of the keys'
// 8-bit digits for the sort's passes (counted per CTA in shared memory, one
// global addition per CTA and digit).  The grid also clears the tree buffers
// that the deposit after the sort starts from, so no separate fills run.
__global__ void __launch_bounds__(256) k_keys(const SceneDesc *__restrict__ scenes,
                                              const uint32_t *__restrict__ tile_scene,
                                              const float4 *__restrict__ part,
                                              uint32_t *__restrict__ keys, uint32_t *__restrict__ ids,
                                              int fresh_ids, uint32_t tiles,
                                              const __grid_constant__ SceneMask fresh,
                                              const uint32_t *__restrict__ tile_map, uint32_t digits,
                                              uint32_t *__restrict__ totals, const ClearTree clear) {
  __shared__ uint32_t s_total[4][256];
#pragma unroll
  for (uint32_t d = 0; d < 4u; d++) s_total[d][threadIdx.x] = 0u;
  grid_dependency_wait();
  __syncthreads();
  for (uint32_t i = blockIdx.x; i < tiles; i += gridDim.x) {
    const uint32_t tile = tile_map != nullptr ? tile_map[i] : i;
    const uint32_t sc = tile_scene[tile];
    const SceneDesc &S = scenes[sc];
    const uint32_t slot = tile * kTile + threadIdx.x;
    const uint32_t local = slot - S.body_off;
    const uint32_t F = S.key_level;
    uint32_t key = S.key_base | ((1u << (3u * F)) - 1u);  // padding sorts after its scene's bodies
    if (local < S.n) {
      // The key cell: in kNearP2P the leaf only (bodies of a leaf keep their
      // input, caller, order), else a fine cell; floor(u * 2^F) >> (F - depth)
      // == floor(u * 2^depth), so the fine key refines the leaf key.
      const float4 p = part[2u * slot];
      const uint32_t level = S.near_mode == kNearP2P ? S.depth : F;
      uint32_t cx, cy, cz;
      cells_of_position(p.x, p.y, p.z, level, cx, cy, cz);
      key = S.key_base | (morton3(cx, cy, cz) << (3u * (F - level)));
    }
    keys[i * kTile + threadIdx.x] = key;
    for (uint32_t d = 0; d < digits; d++) atomicAdd(&s_total[d][(key >> (8u * d)) & 255u], 1u);
    if (fresh_ids == 1 || (fresh_ids == 2 && ((fresh.bits[sc >> 5] >> (sc & 31u)) & 1u))) ids[slot] = local;
  }
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < clear.words; i += gridDim.x * blockDim.x) {
#pragma unroll
    for (uint32_t b = 0; b < 4u; b++) clear.buf[b][i] = zero;
  }
  __syncthreads();
  for (uint32_t d = 0; d < digits; d++) {
    const uint32_t c = s_total[d][threadIdx.x];
    if (c != 0u) atomicAdd(&totals[256u * d + threadIdx.x], c);
  }
}

// Apply the sort's permutation to the bodies and deposit them (persistent
// grid, per-CTA deposit table): output tile i is tile i, or tile_map[i] (each
// scene's tiles are permuted among themselves); perm holds slots of part_in.
// With `src`, the one scene's bodies come from the caller's buffer of src_n
// bodies instead (slot = caller index).  Caller ids: ids_in of the source slot,
// or without ids_in the source slot's place in its scene.  What bounds it is
// the chain perm -> 32 random bytes, so the next tile's bodies and the
// permutation after that are requested a tile ahead.  With that, the ids from
// the place and the caller's buffer read in place: upload, sort and deposit
// 18 -> 14 us at 4,096 bodies, 96 -> 78 at 1,048,576, 389 -> 311 at 5,242,880.
__global__ void __launch_bounds__(256) k_gather(const SceneDesc *__restrict__ scenes,
                                                const uint32_t *__restrict__ tile_scene,
                                                const uint32_t *__restrict__ perm,
                                                const float4 *__restrict__ part_in,
                                                const float4 *__restrict__ src, uint32_t src_n,
                                                const uint32_t *__restrict__ ids_in,
                                                float4 *__restrict__ part_out,
                                                uint32_t *__restrict__ ids_out,
                                                uint4 *__restrict__ deposit_into, uint32_t tiles,
                                                uint32_t slots, float4 *__restrict__ pos_out,
                                                const uint32_t *__restrict__ tile_map) {
  __shared__ DepositTable T;
  __shared__ SceneDesc S;
  uint32_t t0, t1;
  cta_tile_range(tiles, t0, t1);
  T.clear();
  grid_dependency_wait();  // the permutation is complete
  auto load = [&](uint32_t from, float4 &a, float4 &b) {
    a = b = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (from < (src != nullptr ? src_n : slots)) load_body(src != nullptr ? src : part_in, from, a, b);
  };
  const uint32_t tid = threadIdx.x;
  uint32_t from = t0 < t1 ? perm[t0 * kTile + tid] : 0u, next = t0 + 1u < t1 ? perm[(t0 + 1u) * kTile + tid] : 0u;
  float4 n0, n1;
  if (t0 < t1) load(from, n0, n1);
  uint32_t cur = 0xFFFFFFFFu;
  for (uint32_t i = t0; i < t1; i++) {
    const uint32_t tile = tile_map != nullptr ? tile_map[i] : i;
    const uint32_t slot = tile * kTile + tid, here = from;
    const float4 p0 = n0, p1 = n1;
    if (i + 1u < t1) {
      from = next;
      load(from, n0, n1);
      if (i + 2u < t1) next = perm[(i + 2u) * kTile + tid];
    }
    const uint32_t sc = tile_scene[tile];
    if (sc != cur) {
      load_scene(S, scenes, sc);
      cur = sc;
    }
    const bool active = slot - S.body_off < S.n;
    uint32_t key = DepositTable::kEmpty;
    uint32_t qx = 0, qy = 0, qz = 0;
    if (active) {
      store_body(part_out, slot, p0, p1);
      ids_out[slot] = ids_in != nullptr && here < slots ? ids_in[here] : here - S.body_off;
      if (pos_out != nullptr) pos_out[slot] = p0;
      key = S.cell_off + leaf_cell(p0.x, p0.y, p0.z, S.depth);
      qx = (uint32_t)f2i_rn_sat(p0.x * S.scale);
      qy = (uint32_t)f2i_rn_sat(p0.y * S.scale);
      qz = (uint32_t)f2i_rn_sat(p0.z * S.scale);
    }
    deposit_body(T, key, active, qx, qy, qz, deposit_into);
  }
  __syncthreads();
  T.flush(deposit_into);
}

// Copy of a result buffer with the error word behind it (k_unpermute's
// error_out): one launch where a copy and a second copy of the word ran.
__global__ void __launch_bounds__(256) k_copy_out(const uint4 *__restrict__ from, uint4 *__restrict__ to, uint32_t words,
                                                  const Counters *__restrict__ ctr, volatile uint32_t *error_out) {
  report_error(ctr, error_out);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < words; i += gridDim.x * blockDim.x) to[i] = from[i];
}

void launch_copy_out(const LaunchCtx &L, const void *from, void *to, size_t bytes, uint32_t *error_out) {
  const uint32_t words = (uint32_t)(bytes / 16u), ctas = (words + 255u) / 256u;
  k_copy_out<<<ctas < 16u * L.sms ? ctas : 16u * L.sms, 256, 0, L.stream>>>(static_cast<const uint4 *>(from),
                                                                          static_cast<uint4 *>(to), words, L.ctr, error_out);
}

// Scatter bodies back to the caller's order: out[body_off + id - out_base] =
// part[slot].  With `error_out` (mapped host memory) the engine's error word
// and its detail go there too, for a caller that waits for this launch.
__global__ void __launch_bounds__(256) k_unpermute(const SceneDesc *__restrict__ scenes,
                                                   const uint32_t *__restrict__ tile_scene,
                                                   const float4 *__restrict__ part,
                                                   const uint32_t *__restrict__ ids,
                                                   float4 *__restrict__ out, uint32_t tile_base,
                                                   const uint32_t *__restrict__ tile_map,
                                                   const uint32_t *__restrict__ tile_count, uint32_t out_base,
                                                   const Counters *__restrict__ ctr,
                                                   volatile uint32_t *error_out) {
  report_error(ctr, error_out);
  const uint32_t tile = tile_map != nullptr ? tile_map[blockIdx.x] : tile_base + blockIdx.x;
  const SceneDesc &S = scenes[tile_scene[tile]];
  // The scene's body count: from the caller when given (a retiring serving
  // slot's descriptor may already read empty), else from the descriptor.
  const uint32_t n = tile_count != nullptr ? tile_count[blockIdx.x] : S.n;
  const uint32_t slot = tile * kTile + threadIdx.x;
  if (slot - S.body_off >= n) return;
  const uint32_t id = ids[slot];
  if (id >= n) return;  // defensive: ids are a permutation of 0..n-1
  float4 a, b;
  load_body(part, slot, a, b);
  store_body(out, S.body_off + id - out_base, a, b);
}

// ------------------------------------------------------ galaxy seeding

__device__ __forceinline__ uint32_t hash32(uint32_t x) {  // wgsl:205-210
  x = ((x >> 16) ^ x) * 0x45d9f3bu;
  x = ((x >> 16) ^ x) * 0x45d9f3bu;
  return (x >> 16) ^ x;
}

__device__ __forceinline__ float random01(uint32_t seed) {
  return (float)hash32(seed) * (1.0f / 4294967296.0f);
}

__device__ float seeded_enclosed_mass(float radius) {  // wgsl:216-230
  const float bulge = 0.05f * rf_powf(clampf_d(radius / 0.11f, 0.0f, 1.0f), 3.0f);
  const float halo = 0.70f * rf_powf(clampf_d(radius / 0.70f, 0.0f, 1.0f), 3.0f);
  const float disc = 0.18f * rf_powf(clampf_d((radius - 0.055f) / 0.60f, 0.0f, 1.0f), 1.0f / 0.72f);
  const float polar = 0.07f * rf_powf(clampf_d((radius - 0.22f) / 0.31f, 0.0f, 1.0f), 1.0f / 0.86f);
  return fmaxf(bulge + halo + disc + polar, 0.0001f);
}

__device__ __forceinline__ void cross3(const float a[3], const float b[3], float o[3]) {
  o[0] = a[1] * b[2] - a[2] * b[1];
  o[1] = a[2] * b[0] - a[0] * b[2];
  o[2] = a[0] * b[1] - a[1] * b[0];
}

__global__ void __launch_bounds__(256) k_initialize(const SceneDesc *__restrict__ scenes,
                                                    const uint32_t *__restrict__ tile_scene,
                                                    float4 *__restrict__ out, uint32_t tile_base) {
  constexpr float kTau = 6.28318530718f;
  const uint32_t tile = tile_base + blockIdx.x;
  const SceneDesc &S = scenes[tile_scene[tile]];
  const uint32_t slot = tile * kTile + threadIdx.x;
  const uint32_t i = slot - S.body_off;
  if (i >= S.n) return;
  const float u0 = random01(i * 11u + 1u), u1 = random01(i * 11u + 2u), u2 = random01(i * 11u + 3u);
  const float u3 = random01(i * 11u + 4u), u4 = random01(i * 11u + 5u), u5 = random01(i * 11u + 6u);
  float pos[3], vel[3], excitation;
  if (u5 < 0.75f) {
    const float z = u0 * 2.0f - 1.0f, phi = kTau * u1;
    const float outer = u5 < 0.05f ? 0.11f : 0.70f;
    const float radius = outer * rf_powf(u2, 0.3333333f);
    const float ring = sqrtf(fmaxf(0.0f, 1.0f - z * z));
    const float rd[3] = {ring * rf_cosf(phi), z, ring * rf_sinf(phi)};
    for (int k = 0; k < 3; k++) pos[k] = radius * rd[k];
    const float tz = u3 * 2.0f - 1.0f, tphi = kTau * u4;
    const float tring = sqrtf(fmaxf(0.0f, 1.0f - tz * tz));
    const float rnd[3] = {tring * rf_cosf(tphi), tz, tring * rf_sinf(tphi)};
    float tangent[3];
    cross3(rd, rnd, tangent);
    if (length3(tangent[0], tangent[1], tangent[2]) < 0.001f) {
      const float up[3] = {0.0f, 1.0f, 0.0f};
      cross3(rd, up, tangent);
    }
    if (length3(tangent[0], tangent[1], tangent[2]) < 0.001f) {
      const float ex[3] = {1.0f, 0.0f, 0.0f};
      cross3(rd, ex, tangent);
    }
    const float orbital = 0.985f * sqrtf(S.gravity * seeded_enclosed_mass(radius) / (radius + 0.018f));
    const float tl = length3(tangent[0], tangent[1], tangent[2]);
    for (int k = 0; k < 3; k++) vel[k] = orbital * (tangent[k] / tl);
    excitation = u5 < 0.05f ? 0.09f : 0.025f + u4 * 0.025f;
  } else if (u5 < 0.93f) {
    const float radius = 0.055f + 0.60f * rf_powf(u0, 0.72f);
    const float arm = (float)(i & 3u) * (kTau / 4.0f);
    const float angle = arm + radius * 7.8f + (u1 - 0.5f) * (0.045f + radius * 0.055f);
    const float thickness = (u2 + u3 + u4 - 1.5f) * (0.0035f + radius * 0.010f);
    const float flat[3] = {radius * rf_cosf(angle), radius * rf_sinf(angle) * 0.72f, thickness};
    const float tilt = 0.20f;
    pos[0] = flat[0];
    pos[1] = flat[1] * rf_cosf(tilt) - flat[2] * rf_sinf(tilt);
    pos[2] = flat[1] * rf_sinf(tilt) + flat[2] * rf_cosf(tilt);
    const float orbital = 0.99f * sqrtf(S.gravity * seeded_enclosed_mass(radius) / (radius + 0.018f));
    const float tangent[3] = {-rf_sinf(angle), rf_cosf(angle) * 0.72f * rf_cosf(tilt),
                              rf_cosf(angle) * 0.72f * rf_sinf(tilt)};
    const float pl = length3(pos[0], pos[1], pos[2]);
    const float tl = length3(tangent[0], tangent[1], tangent[2]);
    const float sw = rf_sinf(angle * 3.0f - radius * 13.0f);
    for (int k = 0; k < 3; k++) vel[k] = orbital * (tangent[k] / tl) + (pos[k] / pl) * orbital * 0.035f * sw;
    excitation = 0.08f + u3 * 0.05f;
  } else {
    const float lineage = (float)(i & 3u);
    const float radius = 0.22f + 0.31f * rf_powf(u0, 0.86f) + (lineage - 1.5f) * 0.007f;
    const float angle = kTau * u1 + radius * 3.5f;
    const float thickness = (u2 + u3 + u4 - 1.5f) * (0.004f + radius * 0.009f);
    const float flat[3] = {radius * rf_cosf(angle), thickness, radius * rf_sinf(angle)};
    const float tilt = -0.54f + lineage * 0.36f;
    pos[0] = flat[0] * rf_cosf(tilt) - flat[1] * rf_sinf(tilt);
    pos[1] = flat[0] * rf_sinf(tilt) + flat[1] * rf_cosf(tilt);
    pos[2] = flat[2];
    const float tangent[3] = {-rf_sinf(angle) * rf_cosf(tilt), -rf_sinf(angle) * rf_sinf(tilt), rf_cosf(angle)};
    const float orbital = 0.99f * sqrtf(S.gravity * seeded_enclosed_mass(radius) / (radius + 0.018f));
    const float tl = length3(tangent[0], tangent[1], tangent[2]);
    for (int k = 0; k < 3; k++) vel[k] = -orbital * (tangent[k] / tl);
    excitation = 0.20f + u4 * 0.08f;
  }
  float hue = 0.0f;
  if (u5 >= 0.75f) {
    const float speed = fmaxf(length3(vel[0], vel[1], vel[2]), 0.0001f);
    const float radius = fmaxf(length3(pos[0], pos[1], pos[2]), 0.0001f);
    const float pv = (pos[0] * vel[0] + pos[1] * vel[1]) + pos[2] * vel[2];
    const float radial_motion = clampf_d(pv / (radius * speed), -1.0f, 1.0f);
    float am[3];
    cross3(pos, vel, am);
    const float spin = am[1] / fmaxf(length3(am[0], am[1], am[2]), 0.0001f);
    const float h = rf_atan2f(vel[1], vel[0]) / kTau + (vel[2] / speed) * 0.14f + spin * 0.075f +
                    radial_motion * 0.065f + excitation * 0.085f + (float)(i & 3u) * 0.018f;
    hue = h - floorf(h);
  }
  out[2u * slot] = make_float4(pos[0], pos[1], pos[2], hue);
  out[2u * slot + 1u] = make_float4(vel[0], vel[1], vel[2], excitation);
}

// --------------------------------------------------------------- launches

template <uint32_t kBodies>
static uint32_t integrate_ctas_per_sm() {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_integrate<false, kBodies>, kTile / kBodies, 0) !=
          cudaSuccess ||
      n < 1)
    n = 1;
  return (uint32_t)n;
}
uint32_t integrate_resident(bool pairs) {
#ifndef RFMM_FAST_FLOAT
  if (pairs) return integrate_ctas_per_sm<2u>();
#endif
  return integrate_ctas_per_sm<1u>();
}

// Persistent body-pass grid: whole waves of resident CTAs, at most one per tile.
static uint32_t body_grid(const LaunchCtx &L, uint32_t tiles) {
  return tiles < L.body_ctas ? tiles : L.body_ctas;
}

template <uint32_t kBodies>
static void launch_integrate_bodies(const LaunchCtx &L, uint32_t tiles) {
  static const uint32_t per_sm = integrate_ctas_per_sm<kBodies>();
  const uint32_t grid = body_grid(L, tiles), wave = L.sms * per_sm;
  launch_step_kernel(L, L.p2p ? k_integrate<true, kBodies> : k_integrate<false, kBodies>,
                     dim3(grid < wave ? grid : wave), dim3(kTile / kBodies), 0, L.scenes, L.tile_scene, L.part,
                     (const uint4 *)L.mom, (const float4 *)L.src, (const float4 *)L.aux, (const uint32_t *)L.choice,
                     (const float *)L.fields, L.mom_next, tiles, L.tile_list, L.ctr, L.integrate_dynamic ? 1 : 0,
                     (const float4 *)L.near4, -0.0f, stamp_rec(L, 3u));
}

bool integrate_pairs(uint32_t tiles, uint32_t sms) {
#ifdef RFMM_FAST_FLOAT
  return false;
#else
  return tiles > kPairTiles * sms;
#endif
}

void launch_integrate(const LaunchCtx &L, uint32_t tiles) {
#ifndef RFMM_FAST_FLOAT
  if (L.integrate_pairs) {
    launch_integrate_bodies<2u>(L, tiles);
    return;
  }
#endif
  launch_integrate_bodies<1u>(L, tiles);
}

// One wave of the pair-sum kernel's resident CTAs, at most one warp per unit.
template <uint32_t kSplit>
static void launch_near_p2p_split(const LaunchCtx &L, uint32_t tiles) {
  static const uint32_t per_sm = [] {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_near_p2p<kSplit>, 32 * kP2PWarps, 0) != cudaSuccess ||
        n < 1)
      n = 1;
    return (uint32_t)n;
  }();
  const uint32_t units = tiles * (kTile / kP2PUnit<kSplit>), wave = (L.sms ? L.sms : 1u) * per_sm;
  const uint32_t ctas = (units + kP2PWarps - 1u) / kP2PWarps;
  launch_step_kernel(L, k_near_p2p<kSplit>, dim3(ctas < wave ? ctas : wave), dim3(32u * kP2PWarps), 0, L.scenes,
                     L.tile_scene, (const float4 *)L.pos4, (const uint32_t *)L.starts_out,
                     (const uint4 *)L.mom, (const uint32_t *)L.choice, tiles, L.tile_list, L.ctr,
                     L.near4, -0.0f, stamp_rec(L, 5u));
}

void launch_near_p2p(const LaunchCtx &L, uint32_t tiles) {
  // Units of 8 bodies while units of 32 would leave warps idle: up to 8 per
  // SM (38,912 slots on 152).  Exact, ms, 8 / 32, in slot order: Plummer
  // 16,384 0.55 / 0.68, 32,768 1.79 / 1.78, 120,001 9.6 / 8.8; uniform 16,384
  // 0.13 / 0.18.  The fast variant's split costs nothing, so it always takes
  // 16 (16 / 64, in slot order: Plummer 16,384 0.33 / 0.76, 1,048,576 59.8 /
  // 54.6, clusters 600,007 15.0 / 24.2).
#ifdef RFMM_FAST_FLOAT
  launch_near_p2p_split<4>(L, tiles);
#else
  if (tiles * (kTile / 32u) <= 8u * L.sms)
    launch_near_p2p_split<4>(L, tiles);
  else
    launch_near_p2p_split<1>(L, tiles);
#endif
}

void launch_deposit(const LaunchCtx &L, uint4 *moments, uint32_t tiles) {
  k_deposit<<<body_grid(L, tiles), kTile, 0, L.stream>>>(L.scenes, L.tile_scene, L.part, moments,
                                                         tiles, L.tile_list, L.ctr);
}

void launch_keys(const LaunchCtx &L, const SortScratch &s, uint32_t bits, uint32_t *ids, int fresh_ids,
                 uint32_t tiles, const SceneMask *fresh, const uint32_t *tile_map, const ClearTree *clear) {
  static const SceneMask kNone{};
  // A CTA per tile, or per 256 words to clear where those are more (255 bodies
  // in a forced depth-6 tree: 309 us per upload with one CTA per tile, 19 now).
  const uint32_t wave = 8u * L.sms, clears = clear != nullptr ? (clear->words + kTile - 1u) / kTile : 0u;
  const uint32_t ctas = tiles > clears ? tiles : clears;
  launch_step_kernel(L, k_keys, dim3(ctas < wave ? ctas : wave), dim3(kTile), 0, L.scenes, L.tile_scene,
                     (const float4 *)L.part, s.keys[0], ids, fresh_ids, tiles, fresh != nullptr ? *fresh : kNone,
                     tile_map, (bits + 7u) / 8u, s.totals, clear != nullptr ? *clear : ClearTree{});
}

void launch_gather(const LaunchCtx &L, const uint32_t *perm, const float4 *part_in, const float4 *src,
                   uint32_t src_n, const uint32_t *ids_in, float4 *part_out, uint32_t *ids_out, uint4 *deposit_into,
                   uint32_t tiles, uint32_t slots, float4 *pos_out, const uint32_t *tile_map) {
  launch_step_kernel(L, k_gather, dim3(body_grid(L, tiles)), dim3(kTile), 0, L.scenes, L.tile_scene, perm, part_in, src,
                     src_n, ids_in, part_out, ids_out, deposit_into, tiles, slots, pos_out, tile_map);
}

// Per-leaf body ranges of the leaf-sorted scenes (kNearP2P): entry m of a
// scene's table (at its cell offset) is the first slot whose leaf Morton code
// is >= m, for m in [0, 8^depth]; found by binary search in the sorted keys.
__global__ void __launch_bounds__(256) k_leaf_starts(const SceneDesc *__restrict__ scenes,
                                                     const uint32_t *__restrict__ keys,
                                                     uint32_t *__restrict__ starts) {
  const SceneDesc &S = scenes[blockIdx.y];
  if (S.n == 0u || S.near_mode != kNearP2P) return;
  const uint32_t leaves = 1u << (3u * S.depth);
  for (uint32_t m = blockIdx.x * blockDim.x + threadIdx.x; m <= leaves; m += gridDim.x * blockDim.x) {
    uint32_t lo = m < leaves ? 0u : S.n, hi = S.n;  // entry 8^depth ends the last leaf
    if (m < leaves) {
      const uint32_t target = S.key_base | (m << (3u * (S.key_level - S.depth)));
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (keys[S.body_off + mid] < target) {
          lo = mid + 1u;
        } else {
          hi = mid;
        }
      }
    }
    starts[S.cell_off + m] = S.body_off + lo;
  }
}

void launch_leaf_starts(const LaunchCtx &L, const uint32_t *sorted_keys, uint32_t scenes) {
  k_leaf_starts<<<dim3(64, scenes), 256, 0, L.stream>>>(L.scenes, sorted_keys, L.starts_out);
}

void launch_unpermute(const LaunchCtx &L, const uint32_t *ids, float4 *out, uint32_t tile_base,
                      uint32_t tiles, const uint32_t *tile_map, const uint32_t *tile_count, uint32_t out_base,
                      uint32_t *error_out) {
  k_unpermute<<<tiles, kTile, 0, L.stream>>>(L.scenes, L.tile_scene, L.part, ids, out, tile_base, tile_map, tile_count,
                                             out_base, L.ctr, error_out);
}

// Scene descriptors written from kernel parameters (a few at a time, on the
// caller's stream, without touching the other entries of the table).
struct SceneWrites {
  static constexpr uint32_t kMax = 16u;
  uint32_t count;
  uint32_t index[kMax];
  SceneDesc desc[kMax];
};

__global__ void __launch_bounds__(32) k_write_scenes(SceneDesc *__restrict__ scenes,
                                                     const __grid_constant__ SceneWrites w) {
  for (uint32_t i = 0; i < w.count; i++) {
    const uint32_t *src = reinterpret_cast<const uint32_t *>(&w.desc[i]);
    uint32_t *dst = reinterpret_cast<uint32_t *>(scenes + w.index[i]);
    for (uint32_t k = threadIdx.x; k < sizeof(SceneDesc) / 4u; k += blockDim.x) dst[k] = src[k];
  }
}

void launch_write_scenes(cudaStream_t stream, SceneDesc *scenes, const uint32_t *index,
                         const SceneDesc *desc, uint32_t count) {
  for (uint32_t at = 0; at < count; at += SceneWrites::kMax) {
    SceneWrites w{};
    w.count = count - at < SceneWrites::kMax ? count - at : SceneWrites::kMax;
    for (uint32_t i = 0; i < w.count; i++) {
      w.index[i] = index[at + i];
      w.desc[i] = desc[at + i];
    }
    k_write_scenes<<<1, 32, 0, stream>>>(scenes, w);
  }
}

// Zero the moments (both buffers), sources and records of every cell of the
// scenes set in `which` (a rebuilt scene starts from cleared trees: the
// upward pass skips subtrees that are empty in both moment buffers).  Every
// CTA takes a share of each scene's cells.
__global__ void __launch_bounds__(256) k_clear_scenes(const SceneDesc *__restrict__ scenes, uint32_t nscenes,
                                                      const __grid_constant__ SceneMask which,
                                                      uint4 *__restrict__ mom0, uint4 *__restrict__ mom1,
                                                      float4 *__restrict__ src, float4 *__restrict__ aux) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t w = 0; w < (nscenes + 31u) / 32u; w++) {
    for (uint32_t bits = which.bits[w]; bits != 0u; bits &= bits - 1u) {
      const SceneDesc &S = scenes[32u * w + (uint32_t)(__ffs(bits) - 1)];
      for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < S.cells; c += stride) {
        const uint32_t i = S.cell_off + c;
        mom0[i] = make_uint4(0u, 0u, 0u, 0u);
        mom1[i] = make_uint4(0u, 0u, 0u, 0u);
        src[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        aux[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
    }
  }
}

void launch_clear_scenes(const LaunchCtx &L, uint32_t nscenes, const SceneMask &which, uint4 *mom0,
                         uint4 *mom1, float4 *src, float4 *aux) {
  k_clear_scenes<<<4u * L.sms, 256, 0, L.stream>>>(L.scenes, nscenes, which, mom0, mom1, src, aux);
}

void launch_initialize(const LaunchCtx &L, float4 *part_out, uint32_t tile_base, uint32_t tiles) {
  k_initialize<<<tiles, kTile, 0, L.stream>>>(L.scenes, L.tile_scene, part_out, tile_base);
}

// Bulk upload, one CTA per 256-slot tile: two 16-byte loads and stores per body.
__global__ void __launch_bounds__(256) k_upload_scenes(const SceneDesc *__restrict__ scenes,
                                                       const uint32_t *__restrict__ tile_scene,
                                                       float4 *__restrict__ part, uint32_t tile_base,
                                                       uint32_t scene_base,
                                                       const __grid_constant__ UploadSources src) {
  const uint32_t tile = tile_base + blockIdx.x;
  const uint32_t sc = tile_scene[tile];
  const float4 *from = src.p[sc - scene_base];
  const SceneDesc &S = scenes[sc];
  const uint32_t slot = tile * kTile + threadIdx.x, local = slot - S.body_off;
  if (from != nullptr && local < S.n) {
    part[2u * slot] = from[2u * local];
    part[2u * slot + 1u] = from[2u * local + 1u];
  }
}

void launch_upload_scenes(const LaunchCtx &L, float4 *part, uint32_t tile_base, uint32_t tiles,
                          uint32_t scene_base, const UploadSources &src) {
  k_upload_scenes<<<tiles, kTile, 0, L.stream>>>(L.scenes, L.tile_scene, part, tile_base, scene_base,
                                                 src);
}

RFMM_KERNEL_NS_END
