// Particle-pair passes over a cell sort of the particles: the solid position regularisation
// (src/three/solid-sampling.js:5-42, regularizeSolids; the reference's GPU twin is
// gpu/solver.py:565-648) and the particle-pair heat exchange with the enthalpy phase change
// (src/thermal.js:35-56, src/three/phase-change.js:12-18; GPU twin gpu/solver.py:775-811).
//
// Regularisation pass:
//   k_reg_count    thread per particle: neighbour cell, target spacing from V J Jp and the scene's
//                  largest, cell population
//   scan           exclusive prefix sum of the populations (k_scan_blocks / k_scan_top / k_scan_add)
//   k_reg_scatter  particle slots grouped by cell, with a packed copy of what the pair test reads
//                  (position, target, inverse mass, index, material) in cell order, so neighbour
//                  candidates are read as contiguous runs
//   k_reg_pairs    thread per particle in cell order: its own shift, gathered over the rows of cells
//                  within half the sum of its own and the scene's largest target (ball_rows). The
//                  reference visits each pair once (i < j) and adds +shift to i and -shift to j; the pair
//                  term is antisymmetric, so gathering every neighbour from each side gives the
//                  same sums without atomics. The largest shift of each scene over its budget.
//   k_reg_apply    x += shift / max(1, largest / budget) for unpinned particles, clamped to the box
// HBM traffic per particle: about 110 B (position, D, V, m, aux, id reads; the cell, target, shift
// and packed scratch) plus the neighbour reads, contiguous runs of the packed copy that L1/L2 serve.
#include "mpm_internal.h"
#include "pairs.h"

namespace mpm {

namespace {

__device__ __forceinline__ void position(const Particles& p, long long h, const SceneDev& sc, float x[3]) {
  // metres from the scene's grid origin (exact integer cell part, FP32 fraction)
  const unsigned q[3] = {p.qx[h], p.qy[h], p.qz[h]};
  for (int a = 0; a < 3; ++a) x[a] = static_cast<float>(q[a]) * kInvFixedOne * sc.H;
}

__device__ __forceinline__ unsigned cell_id(const RegScene& rs, const float x[3], float inv_hc) {
  int cc[3];
  for (int a = 0; a < 3; ++a) cc[a] = min(rs.nc[a] - 1, max(0, static_cast<int>(floorf(x[a] * inv_hc))));
  return static_cast<unsigned>(rs.cell_base + ((long long)cc[2] * rs.nc[1] + cc[1]) * rs.nc[0] + cc[0]);
}

// Visits the cell-ordered particles that may lie within rho of x: fn(first, end) for each row of cells
// (fixed y and z) that the ball reaches, over the row's part along x that it reaches. Cells of one row
// are consecutive, so a row is one contiguous run. The bounds are widened by 1e-3 cells and 1e-6 of the
// grid's extent, above the FP32 rounding of a cell's coordinate, so no pair is missed.
template <typename Fn>
__device__ __forceinline__ void ball_rows(const RegScene& rs, const unsigned* start, const float x[3], float rho,
                                          float hc, float inv_hc, Fn&& fn) {
  const float margin = (1e-3f + 1e-6f * static_cast<float>(max(rs.nc[0], max(rs.nc[1], rs.nc[2])))) * hc;
  const float r = rho + margin;
  const int z0 = max(0, static_cast<int>(floorf((x[2] - r) * inv_hc))), z1 = min(rs.nc[2] - 1, static_cast<int>(floorf((x[2] + r) * inv_hc)));
  const int y0 = max(0, static_cast<int>(floorf((x[1] - r) * inv_hc))), y1 = min(rs.nc[1] - 1, static_cast<int>(floorf((x[1] + r) * inv_hc)));
  for (int z = z0; z <= z1; ++z) {
    const float lz = static_cast<float>(z) * hc;
    const float dz = fmaxf(0.f, fmaxf(lz - x[2], z == rs.nc[2] - 1 ? 0.f : x[2] - lz - hc));
    for (int y = y0; y <= y1; ++y) {
      const float ly = static_cast<float>(y) * hc;
      const float dy = fmaxf(0.f, fmaxf(ly - x[1], y == rs.nc[1] - 1 ? 0.f : x[1] - ly - hc));
      const float left = r * r - dz * dz - dy * dy;
      if (left < 0.f) continue;
      const float w = sqrtf(left) + margin;
      const int x0 = min(rs.nc[0] - 1, max(0, static_cast<int>(floorf((x[0] - w) * inv_hc))));
      const int x1 = min(rs.nc[0] - 1, max(0, static_cast<int>(floorf((x[0] + w) * inv_hc))));
      const long long row = rs.cell_base + ((long long)z * rs.nc[1] + y) * rs.nc[0];
      fn(start[row + x0], start[row + x1 + 1]);
    }
  }
}

__global__ void k_reg_count(Ctx c, RegDev r, unsigned* cell_of, float* target, float* inv_mass, unsigned* count,
                            unsigned* tmax) {
  for (long long h = blockIdx.x * (long long)blockDim.x + threadIdx.x; h < c.n; h += (long long)gridDim.x * blockDim.x) {
    const int s = c.nscenes == 1 ? 0 : find_scene_by_particle(c.scenes, c.nscenes, h);
    const SceneDev& sc = c.scenes[s];
    const RegScene& rs = r.scenes[s];
    float x[3];
    position(c.p, h, sc, x);
    const unsigned cell = cell_id(rs, x, r.inv_hc);
    cell_of[h] = cell;
    atomicAdd(&count[cell], 1u);
    // spacing 2.8 cbrt(clamp(V J Jp, 1/64, 8)) in the reference's units (solid-sampling.js:5-8)
    const int mi = c.single_material ? sc.mat_base : c.p.mat[h];
    const int model = c.mats[mi].model;
    float D[9];
    for (int e = 0; e < 9; ++e) D[e] = c.p.Dc[e][h];
    const float J = 1.f + det_minus_one(D);
    const float jp = (c.has_aux && (model == 2 || model == 8 || model == 9)) ? 1.f + c.p.aux[h] : 1.f;
    const float vol = fminf(8.f, fmaxf(0.015625f, c.p.V[h] * J * jp * r.inv_volume_unit));
    const float t = r.spacing * cbrtf(vol);
    target[h] = t;
    {  // one atomic per scene in the warp
      const unsigned act = __activemask(), peers = __match_any_sync(act, s);
      const unsigned m = __reduce_max_sync(peers, __float_as_uint(t));
      if ((threadIdx.x & 31) == __ffs(peers) - 1) atomicMax(&tmax[s], m);
    }
    inv_mass[h] = (c.has_pinned && c.p.pinned[h]) ? 0.f : 1.f / c.p.m[h];
  }
}

__global__ void k_reg_scatter(Ctx c, const unsigned* cell_of, const unsigned* start, unsigned* count,
                              const float* target, const float* inv_mass, unsigned* sorted, uint4* pos_sorted,
                              uint2* inv_sorted, unsigned short* mat_sorted) {
  for (long long h = blockIdx.x * (long long)blockDim.x + threadIdx.x; h < c.n; h += (long long)gridDim.x * blockDim.x) {
    const unsigned cell = cell_of[h];
    const unsigned k = start[cell] + atomicSub(&count[cell], 1u) - 1u;  // counts end at zero for the next pass
    sorted[k] = static_cast<unsigned>(h);
    pos_sorted[k] = make_uint4(c.p.qx[h], c.p.qy[h], c.p.qz[h], __float_as_uint(target[h]));
    inv_sorted[k] = make_uint2(__float_as_uint(inv_mass[h]), c.p.id[h]);
    if (!c.single_material) mat_sorted[k] = c.p.mat[h];
  }
}

__device__ __forceinline__ float scene_dt(const RegDev& r, int s) { return r.dt_scene ? r.dt_scene[s] : r.dt; }

__global__ void __launch_bounds__(256) k_reg_pairs(Ctx c, RegDev r, const unsigned* start, const unsigned* tmax, const unsigned* sorted, const uint4* pos_sorted, const uint2* inv_sorted,
                            const unsigned short* mat_sorted, float4* shift, unsigned* largest) {
  for (long long ks = blockIdx.x * (long long)blockDim.x + threadIdx.x; ks < c.n; ks += (long long)gridDim.x * blockDim.x) {
    const unsigned i = sorted[ks];  // home slot
    const int s = c.nscenes == 1 ? 0 : find_scene_by_particle(c.scenes, c.nscenes, i);
    const SceneDev& sc = c.scenes[s];
    const RegScene& rs = r.scenes[s];
    const float dt = scene_dt(r, s);
    const float gain = -expm1f(-r.rate * dt);
    const uint4 pi = pos_sorted[ks];
    const uint2 bi = inv_sorted[ks];
    const unsigned qi[3] = {pi.x, pi.y, pi.z};
    const float ti = __uint_as_float(pi.w), inv_i = __uint_as_float(bi.x);
    const unsigned id_i = bi.y;
    const int mat_i = c.single_material ? 0 : mat_sorted[ks];
    const float to_m = sc.H * kInvFixedOne;
    float acc[3] = {0.f, 0.f, 0.f};
    if (inv_i > 0.f) {  // a pinned particle's own shift is never applied
      float xi[3];
      for (int a = 0; a < 3; ++a) xi[a] = static_cast<float>(qi[a]) * kInvFixedOne * sc.H;
      // no partner's target is above the scene's largest
      ball_rows(rs, start, xi, 0.5f * (ti + __uint_as_float(tmax[s])), r.hc, r.inv_hc, [&](unsigned b, unsigned e) {
        for (unsigned k = b; k < e; ++k) {
          const uint4 pj = pos_sorted[k];
          // exact fixed-point differences, then metres
          float d[3] = {static_cast<float>(static_cast<int>(qi[0] - pj.x)) * to_m,
                        static_cast<float>(static_cast<int>(qi[1] - pj.y)) * to_m,
                        static_cast<float>(static_cast<int>(qi[2] - pj.z)) * to_m};
          const float r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
          const float t = 0.5f * (ti + __uint_as_float(pj.w));
          if (r2 > 1.000001f * t * t || k == ks) continue;
          float rr = sqrtf(r2);
          if (!(rr < t)) continue;
          if (!c.single_material && mat_sorted[k] != mat_i) continue;  // one part
          const uint2 bj = inv_sorted[k];
          const float total = inv_i + __uint_as_float(bj.x);
          float q;
          if (rr < r.eps) {
            // the reference's hashed direction of the pair (lower index first), +/- by side
            const unsigned id_j = bj.y;
            const unsigned lo = min(id_i, id_j), hi = max(id_i, id_j);
            const unsigned hsh = (lo + 1u) * 73856093u ^ (hi + 1u) * 19349663u;
            const float sign = id_i < id_j ? 1.f : -1.f;
            d[0] = sign * (static_cast<float>(hsh & 1023u) / 511.5f - 1.f);
            d[1] = sign * (static_cast<float>((hsh >> 10) & 1023u) / 511.5f - 1.f);
            d[2] = sign * (static_cast<float>((hsh >> 20) & 1023u) / 511.5f - 1.f);
            rr = sqrtf(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
            q = t * gain / (rr * total);
          } else {
            q = (t - rr) * gain / (rr * total);
          }
          acc[0] += d[0] * q;
          acc[1] += d[1] * q;
          acc[2] += d[2] * q;
        }
      });
    }
    const float sx = acc[0] * inv_i, sy = acc[1] * inv_i, sz = acc[2] * inv_i;
    shift[i] = make_float4(sx, sy, sz, 0.f);
    // the reference takes the largest shift over every solid, pinned ones included (a pinned
    // particle's is zero here since its inverse mass is zero)
    const float over = sqrtf(sx * sx + sy * sy + sz * sz) / (r.max_speed * dt);
    if (over > 1.f) atomicMax(&largest[s], __float_as_uint(over));
  }
}

__global__ void k_reg_apply(Ctx c, RegDev r, const float4* shift, const unsigned* largest) {
  for (long long h = blockIdx.x * (long long)blockDim.x + threadIdx.x; h < c.n; h += (long long)gridDim.x * blockDim.x) {
    if (c.has_pinned && c.p.pinned[h]) continue;
    const int s = c.nscenes == 1 ? 0 : find_scene_by_particle(c.scenes, c.nscenes, h);
    const SceneDev& sc = c.scenes[s];
    const float scale = fmaxf(1.f, __uint_as_float(largest[s]));
    const float4 d = shift[h];
    const float k = sc.invH * kFixedOne / scale;
    unsigned* qs[3] = {c.p.qx, c.p.qy, c.p.qz};
    const float dd[3] = {d.x, d.y, d.z};
    for (int a = 0; a < 3; ++a) {
      long long q = static_cast<long long>(qs[a][h]) + __float2ll_rn(dd[a] * k);
      const long long lo = sc.clamp ? (long long)sc.qlo[a] : 0;
      const long long hi = sc.clamp ? (long long)sc.qhi[a] : ((long long)sc.dims[a] - 1) << kFracBits;
      qs[a][h] = static_cast<unsigned>(q < lo ? lo : (q > hi ? hi : q));
    }
  }
}

// Exclusive scan of n unsigned counts into out, in three launches (4096 per block).
constexpr int kScanThreads = 1024, kScanItems = 4;
constexpr int kScanSpan = kScanThreads * kScanItems;

__device__ __forceinline__ unsigned block_exclusive_scan(unsigned v, unsigned* warp_sums, unsigned* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[w] = x;
  __syncthreads();
  if (w == 0) {
    unsigned s = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : 0u;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    warp_sums[lane] = s;  // inclusive over warps
  }
  __syncthreads();
  const unsigned before = (w > 0 ? warp_sums[w - 1] : 0u) + x - v;
  if (total) *total = warp_sums[(blockDim.x >> 5) - 1];
  return before;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_blocks(const unsigned* in, long long n, unsigned* out,
                                                             unsigned* block_sums) {
  __shared__ unsigned ws[32];
  __shared__ unsigned tot;
  const long long base = (long long)blockIdx.x * kScanSpan + (long long)threadIdx.x * kScanItems;
  unsigned v[kScanItems], sum = 0;
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = base + k < n ? in[base + k] : 0u;
    sum += v[k];
  }
  unsigned t = 0;
  unsigned run = block_exclusive_scan(sum, ws, threadIdx.x == 0 ? &t : nullptr);
  if (threadIdx.x == 0) tot = t;
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k < n) out[base + k] = run;
    run += v[k];
  }
  __syncthreads();
  if (threadIdx.x == 0) block_sums[blockIdx.x] = tot;
}

// One block scans the block sums in place (up to kScanSpan of them), chunk by chunk.
__global__ void __launch_bounds__(kScanThreads) k_scan_top(unsigned* block_sums, int nb) {
  __shared__ unsigned ws[32];
  unsigned carry = 0;
  for (int base = 0; base < nb; base += kScanSpan) {
    const int b = base + threadIdx.x * kScanItems;
    unsigned v[kScanItems], sum = 0;
    for (int k = 0; k < kScanItems; ++k) {
      v[k] = b + k < nb ? block_sums[b + k] : 0u;
      sum += v[k];
    }
    __shared__ unsigned tot;
    unsigned t = 0;
    unsigned run = carry + block_exclusive_scan(sum, ws, threadIdx.x == 0 ? &t : nullptr);
    if (threadIdx.x == 0) tot = t;
    for (int k = 0; k < kScanItems; ++k) {
      if (b + k < nb) block_sums[b + k] = run;
      run += v[k];
    }
    __syncthreads();
    carry += tot;
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kScanThreads) k_scan_add(unsigned* out, long long n, const unsigned* block_sums) {
  const long long i = (long long)blockIdx.x * kScanSpan;
  const unsigned add = block_sums[blockIdx.x];
  for (int k = threadIdx.x; k < kScanSpan; k += blockDim.x)
    if (i + k < n) out[i + k] += add;
}

// ---- particle-pair heat exchange -------------------------------------------------------------
// k_heat_count / scan / k_heat_scatter: cell sort with a packed copy of position, temperature, conductivity and heat capacity in cell order
// k_heat_budget: per particle the sum of its conductances g over pairs (eps < r < radius), and its
//   budget min(1, 0.45 m cp / (dt sum g)) (1 without contacts)
// k_heat_flow: per particle heat_i = sum_j (T_j - T_i) g dt min(b_i, b_j) — each pair's +Q / -Q
//   gathered from both sides — then the enthalpy update, ambient loss and phase decode of the
//   particle; |Q| summed over pairs (each seen twice: halved) in FP64.

__global__ void k_heat_count(Ctx c, HeatDev hd, unsigned* cell_of, unsigned* count) {
  for (long long h = blockIdx.x * (long long)blockDim.x + threadIdx.x; h < c.n; h += (long long)gridDim.x * blockDim.x) {
    const int s = c.nscenes == 1 ? 0 : find_scene_by_particle(c.scenes, c.nscenes, h);
    const SceneDev& sc = c.scenes[s];
    const RegScene& rs = hd.scenes[s];
    float x[3];
    position(c.p, h, sc, x);
    const unsigned cell = cell_id(rs, x, hd.inv_hc);
    cell_of[h] = cell;
    atomicAdd(&count[cell], 1u);
  }
}

__global__ void k_heat_scatter(Ctx c, const unsigned* cell_of, const unsigned* start, unsigned* count, unsigned* sorted,
                               uint4* pos_sorted, float2* prop_sorted) {
  for (long long h = blockIdx.x * (long long)blockDim.x + threadIdx.x; h < c.n; h += (long long)gridDim.x * blockDim.x) {
    const unsigned cell = cell_of[h];
    const unsigned k = start[cell] + atomicSub(&count[cell], 1u) - 1u;  // counts end at zero for the next pass
    const int s = c.nscenes == 1 ? 0 : find_scene_by_particle(c.scenes, c.nscenes, h);
    const int mi = c.single_material ? c.scenes[s].mat_base : c.p.mat[h];
    sorted[k] = static_cast<unsigned>(h);
    pos_sorted[k] = make_uint4(c.p.qx[h], c.p.qy[h], c.p.qz[h], __float_as_uint(c.p.T[h]));
    prop_sorted[k] = make_float2(c.mats_ext[mi].conductivity, c.p.m[h] * c.mats[mi].cp);
  }
}

// Visits the neighbours j of sorted particle ks within (eps, radius): fn(k, g) with the pair's
// conductance g = (1 - r / radius) geometry heat_rate 2 k_i k_j / (k_i + k_j).
template <typename Fn>
__device__ __forceinline__ void heat_pairs(const Ctx& c, const HeatDev& hd, const unsigned* start, const uint4* pos_sorted,
                                           const float2* prop_sorted, long long ks, unsigned i, Fn&& fn) {
  const int s = c.nscenes == 1 ? 0 : find_scene_by_particle(c.scenes, c.nscenes, i);
  const SceneDev& sc = c.scenes[s];
  const uint4 pi = pos_sorted[ks];
  const float ki = prop_sorted[ks].x;
  const float to_m = sc.H * kInvFixedOne;
  const float r2_max = hd.radius * hd.radius * 1.000001f;
  const float xi[3] = {static_cast<float>(pi.x) * kInvFixedOne * sc.H, static_cast<float>(pi.y) * kInvFixedOne * sc.H,
                       static_cast<float>(pi.z) * kInvFixedOne * sc.H};
  ball_rows(hd.scenes[s], start, xi, hd.radius, hd.hc, hd.inv_hc, [&](unsigned b, unsigned e) {
#pragma unroll 2
    for (unsigned k = b; k < e; ++k) {
      const uint4 pj = pos_sorted[k];
      const float dx = static_cast<float>(static_cast<int>(pi.x - pj.x)) * to_m;
      const float dy = static_cast<float>(static_cast<int>(pi.y - pj.y)) * to_m;
      const float dz = static_cast<float>(static_cast<int>(pi.z - pj.z)) * to_m;
      const float r2 = dx * dx + dy * dy + dz * dz;
      if (r2 > r2_max) continue;
      const float r = sqrtf(r2);
      if (!(r > hd.eps && r < hd.radius) || k == ks) continue;
      const float kj = prop_sorted[k].x;
      // no division inside one material
      const float kh = ki == kj ? ki : ki + kj > 0.f ? 2.f * ki * kj / (ki + kj) : 0.f;
      // 1 - r / radius by the reciprocal's two parts, each product unrounded: the weight keeps its digits
      // where it goes to zero
      const float weight = fmaf(-r, hd.inv_radius_lo, fmaf(-r, hd.inv_radius, 1.f));
      fn(k, weight * hd.geom_rate * kh);
    }
  });
}

// 128-thread CTAs at 48 registers: the search is a chain of cached loads, and 40 resident warps per SM hide
// them better than 36 or 32, though at 48 registers 24 bytes spill. Exchange at 357,120 particles 749 us (780,
// 855), at 195,776 474 (529, 560); where the particles no longer fill those warps it is the spills that show: at
// 131,376 351 (336, 330), at 39,600 303 (290, 289).
constexpr int kHeatThreads = 128;

__global__ void __launch_bounds__(kHeatThreads, 10) k_heat_budget(Ctx c, HeatDev hd, const unsigned* start, const unsigned* sorted, const uint4* pos_sorted, const float2* prop_sorted, float* budget) {
  for (long long ks = blockIdx.x * (long long)blockDim.x + threadIdx.x; ks < c.n; ks += (long long)gridDim.x * blockDim.x) {
    const unsigned i = sorted[ks];
    double gsum = 0.0;
    heat_pairs(c, hd, start, pos_sorted, prop_sorted, ks, i, [&](unsigned, float g) { gsum += g; });
    const double mcp = prop_sorted[ks].y;
    budget[ks] = gsum > 0.0 ? static_cast<float>(fmin(1.0, 0.45 * mcp / (hd.dt * gsum))) : 1.f;
  }
}

__global__ void __launch_bounds__(kHeatThreads, 10) k_heat_flow(Ctx c, HeatDev hd, const unsigned* start, const unsigned* sorted, const uint4* pos_sorted, const float2* prop_sorted,
                            const float* budget, double* exchanged) {
  double absq = 0.0;
  for (long long ks = blockIdx.x * (long long)blockDim.x + threadIdx.x; ks < c.n; ks += (long long)gridDim.x * blockDim.x) {
    const unsigned i = sorted[ks];
    const double Ti = __uint_as_float(pos_sorted[ks].w);
    const float bi = budget[ks];
    double heat = 0.0;
    heat_pairs(c, hd, start, pos_sorted, prop_sorted, ks, i, [&](unsigned k, float g) {
      const double q = ((double)__uint_as_float(pos_sorted[k].w) - Ti) * g * hd.dt * fminf(bi, budget[k]);
      heat += q;
      absq += fabs(q);
    });
    // enthalpy update, ambient loss and the phase decode (src/thermal.js:51-55,
    // src/three/phase-change.js:12-18, src/three/simulation.js:260-270)
    const int s = c.nscenes == 1 ? 0 : find_scene_by_particle(c.scenes, c.nscenes, i);
    const int mi = c.single_material ? c.scenes[s].mat_base : c.p.mat[i];
    const MaterialExt& xt = c.mats_ext[mi];
    const double cp = c.mats[mi].cp, L = xt.latent;
    double hh = cp * Ti + (double)c.p.latent[i] * L + heat / c.p.m[i];
    if (hd.ambient) hh -= (Ti - hd.ambient_T) * cp * hd.dt * hd.ambient_rate;
    const unsigned char was = c.p.melted[i];
    unsigned char liquid = 0;
    double T;
    float f = 0.f;
    if (L > 0.0) {
      const double st = cp * xt.melting_point, en = st + L;
      if (hh <= st) { T = hh / cp; }
      else if (hh >= en) { T = (hh - L) / cp; f = 1.f; liquid = 1; }
      else { T = xt.melting_point; f = static_cast<float>((hh - st) / L); liquid = was; }
    } else {
      T = cp > 0.0 ? hh / cp : Ti;
    }
    c.p.T[i] = static_cast<float>(T);
    c.p.latent[i] = f;
    if (liquid != was) {
      // MPM3.resetParticle on a phase switch; a molten particle is released (Simulation3.pin(i, false))
      c.p.melted[i] = liquid;
      for (int e = 0; e < 9; ++e) {
        c.p.Cc[e][i] = 0.f;
        c.p.Dc[e][i] = 0.f;
      }
      c.p.ep[i] = 0.f;
      c.p.aux[i] = 0.f;
      if (liquid) c.p.pinned[i] = 0;
    }
  }
  // each pair was seen from both sides
  for (int o = 16; o > 0; o >>= 1) absq += __shfl_xor_sync(0xffffffffu, absq, o);
  if ((threadIdx.x & 31) == 0 && absq != 0.0) atomicAdd(exchanged, 0.5 * absq);
}

}  // namespace

// Exclusive prefix sum of the cells' counts into start (cells + 1 entries).
static void scan_cells(const unsigned* count, long long cells, unsigned* start, unsigned* block_sums, cudaStream_t st) {
  const unsigned nb = static_cast<unsigned>(reg_scan_blocks(cells));
  k_scan_blocks<<<nb, kScanThreads, 0, st>>>(count, cells + 1, start, block_sums);
  k_scan_top<<<1, kScanThreads, 0, st>>>(block_sums, static_cast<int>(nb));
  k_scan_add<<<nb, kScanThreads, 0, st>>>(start, cells + 1, block_sums);
}

void launch_exchange_heat(const Ctx& c, const HeatDev& hd, const HeatBufs& b, cudaStream_t st) {
  if (c.n <= 0) return;
  const long long n = c.n;
  const unsigned blocks = static_cast<unsigned>((n + 255) / 256 < 65536 ? (n + 255) / 256 : 65536);
  cudaMemsetAsync(b.exchanged, 0, sizeof(double), st);
  k_heat_count<<<blocks, 256, 0, st>>>(c, hd, b.cell_of, b.count);
  scan_cells(b.count, hd.cells, b.start, b.block_sums, st);
  k_heat_scatter<<<blocks, 256, 0, st>>>(c, b.cell_of, b.start, b.count, b.sorted, b.pos_sorted, b.prop_sorted);
  k_heat_budget<<<2 * blocks, kHeatThreads, 0, st>>>(c, hd, b.start, b.sorted, b.pos_sorted, b.prop_sorted, b.budget);
  k_heat_flow<<<2 * blocks, kHeatThreads, 0, st>>>(c, hd, b.start, b.sorted, b.pos_sorted, b.prop_sorted, b.budget, b.exchanged);
}

// blocks of the scan over cells + 1 counts
size_t reg_scan_blocks(long long cells) { return static_cast<size_t>((cells + 1 + kScanSpan - 1) / kScanSpan); }

void launch_regularize(const Ctx& c, const RegDev& r, const RegBufs& b, cudaStream_t st) {
  if (c.n <= 0) return;
  const long long n = c.n;
  const unsigned blocks = static_cast<unsigned>((n + 255) / 256 < 65536 ? (n + 255) / 256 : 65536);
  cudaMemsetAsync(b.largest, 0, 2 * sizeof(unsigned) * c.nscenes, st);  // and tmax
  k_reg_count<<<blocks, 256, 0, st>>>(c, r, b.cell_of, b.target, b.inv_mass, b.count, b.tmax);
  scan_cells(b.count, r.cells, b.start, b.block_sums, st);
  k_reg_scatter<<<blocks, 256, 0, st>>>(c, b.cell_of, b.start, b.count, b.target, b.inv_mass, b.sorted,
                                        b.pos_sorted, b.inv_sorted, b.mat_sorted);
  k_reg_pairs<<<blocks, 256, 0, st>>>(c, r, b.start, b.tmax, b.sorted, b.pos_sorted, b.inv_sorted, b.mat_sorted, b.shift,
                                      b.largest);
  k_reg_apply<<<blocks, 256, 0, st>>>(c, r, b.shift, b.largest);
}

}  // namespace mpm
