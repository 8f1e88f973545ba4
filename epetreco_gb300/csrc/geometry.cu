// geometry.cu -- per-angle trig table, cuRAND uniforms and world rays.
//
// Rays follow RandRayGen with the per-channel seeding of the workqueue
// kernel: curand_init(seed, channel, 0) and six curand_uniform draws per ray,
// the first three placing the start point in crystal 0 and the last three
// the end point in crystal 1 (getSystemMatrixFromWorkqueue.cu:189-230).
// With EPET_RAYS_REGULAR they follow ReguRayGen (RayGenerators.hpp:46-66):
// the six box coordinates are 0.5, so every ray joins the crystal centres,
// and no generator is seeded.
#include <curand_kernel.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "internal.h"

namespace epet {

__global__ void k_trig(epet_setup s, float* sc) {
  int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a < s.na) angle_sincos(s, a, &sc[2 * a], &sc[2 * a + 1]);
}

// Six box coordinates of one ray: cuRAND uniforms, or 0.5 each for regular rays.
__device__ __forceinline__ void draw6(curandState& st, bool regular, float* u) {
#pragma unroll
  for (int k = 0; k < 6; k++) u[k] = regular ? 0.5f : curand_uniform(&st);
}

// One thread per channel: the cuRAND stream of a channel is sequential, so a
// channel's 6*nrays draws stay on one thread; channels spread over threads.
// The uniforms-only form (a test and debugging interface) seeds every
// channel with curand_init(seed, channel, 0) directly.
__device__ __forceinline__ void emit_rays(const Geo& G, int cnl, curandState st, bool uniforms,
                                          float2* o) {
  const bool regular = G.p.ray_mode == EPET_RAYS_REGULAR;
  int id[5];
  channel_decode(G.p.setup, cnl, id);
  float sn, cs;
  angle_sincos(G.p.setup, id[0], &sn, &cs);
  const CrystalMat m0 = crystal_matrix(G.p.setup, sn, cs, 0, id[1], id[2]);
  const CrystalMat m1 = crystal_matrix(G.p.setup, sn, cs, 1, id[3], id[4]);
  // rays in pairs: 48 bytes as three 16-byte stores when the row's block is
  // 16-byte aligned (half as many scattered stores as 8-byte ones)
  const bool wide = (reinterpret_cast<uintptr_t>(o) & 15) == 0;
  for (int r = 0; r < G.p.nrays; r++) {
    float u[6];
    draw6(st, regular, u);
    float w[6];
    if (uniforms) {
#pragma unroll
      for (int k = 0; k < 6; k++) w[k] = u[k];
    } else {
      crystal_apply(m0, u[0], u[1], u[2], w);
      crystal_apply(m1, u[3], u[4], u[5], w + 3);
    }
    if (wide && r + 1 < G.p.nrays) {
      float u2[6], w2[6];
      draw6(st, regular, u2);
      if (uniforms) {
#pragma unroll
        for (int k = 0; k < 6; k++) w2[k] = u2[k];
      } else {
        crystal_apply(m0, u2[0], u2[1], u2[2], w2);
        crystal_apply(m1, u2[3], u2[4], u2[5], w2 + 3);
      }
      float4* q = reinterpret_cast<float4*>(o + 3 * r);
      q[0] = make_float4(w[0], w[1], w[2], w[3]);
      q[1] = make_float4(w[4], w[5], w2[0], w2[1]);
      q[2] = make_float4(w2[2], w2[3], w2[4], w2[5]);
      r++;
    } else {
      o[3 * r + 0] = make_float2(w[0], w[1]);
      o[3 * r + 1] = make_float2(w[2], w[3]);
      o[3 * r + 2] = make_float2(w[4], w[5]);
    }
  }
}

__global__ void __launch_bounds__(128) k_uniforms(Geo G, const int32_t* __restrict__ rows,
                                                  int64_t m, float* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  curandState st = {};
  if (G.p.ray_mode != EPET_RAYS_REGULAR)
    curand_init(G.p.seed, (unsigned long long)rows[i], 0ull, &st);
  emit_rays(G, rows[i], st, true,
            reinterpret_cast<float2*>(out + i * (int64_t)G.p.nrays * 6));
}

// World rays.  Thread t handles rows t*K .. t*K+K-1 (K = kPer): the first channel's
// generator comes from curand_init, the next ones from the previous
// channel's initial state advanced by the channel difference in
// subsequences (skipahead_sequence): curand_init(seed, c, 0) is the seeded
// state advanced c subsequences, so this yields the same states while a
// typical step (consecutive channel ids) applies one jump matrix instead of
// one per set bit of the channel id.
//
// The lines between the forms (launch_rays) are measured, in us, on random
// rows of 228,488 channels | of 5.1M | on consecutive channels, whose jumps
// cost least:
//  * one row a thread: bound by a thread's own latency, which more rows in
//    series add to (3,000 rows of 20 rays: 149, four rows a thread 248).
//    30,000 rows of 10 rays with 1 / 2 / 4 rows: 151 / 150 / 201 | 186 / 201 /
//    286 | 118 / 112 / 111; of 100: 178 / 185 / 285 | 211 / 237 / 382 | 141 /
//    137 / 170; 50,000 of 10: 162 / 166 / 188 | 201 / 231 / 280 | 152 / 124 /
//    116.  A single row: 121 / 110 / 106, so it takes the next form;
//  * two rows: 70,000 of 10 rays 200 / 170 / 180 | 239 / 231 / 271 | 180 / 135
//    / 120; 120,000 of 100 rays 379 / 331 / 354 | 465 / 441 / 474 | 365 / 278 /
//    262: the more rays, the farther their stores spread;
//  * four rows: beyond.  A thread's own stores are 16 bytes into 32 rows at a
//    time, half a sector each; staged, a warp collects kStageRays rays of its
//    32 rows in shared memory and writes each row's share as one run of whole
//    sectors (rows of an even number of rays on 16-byte boundaries).  Direct /
//    staged, 120,000 rows of 100 rays: 348 / 357 | 471 / 523 | 262 / 253; 200,000
//    of 100: 441 / 386 | 626 / 603 | 373 / 327; 200,000 and 300,000 of 40: - |
//    477 / 507, 588 / 599 | 243 / 243, 314 / 300; 500,000 and a million of 20: - |
//    802 / 827, 1287 / 1278 | 410 / 399, 740 / 674; two million of 10: - | 1888 /
//    2014 | 1117 / 1151.
constexpr int kRaysThreads = 128, kRaysThreadsFew = 64;
constexpr int kRaysOnePerSm = 300;                      // rows an SM up to which a thread has one
constexpr int kRaysTwoPerSm = 330, kRaysTwoPerRay = 5;  // and two: 330 + 5 a ray (at most 100)
// Staged beyond so many rows an SM and from so many rays a row and an SM.
constexpr int kRaysStagedPerSm = 1300, kRaysStagedRays = 20, kRaysStagedSum = 65000;
constexpr int kStageRays = 8, kStageVec = kStageRays * 24 / 16;  // rays and 16-byte pieces a row
template <int kPer, int kT, bool kStaged>
__global__ void __launch_bounds__(kT)
k_rays(Geo G, const int32_t* __restrict__ rows, int64_t m, float* __restrict__ out) {
  // (a row of 13 pieces: the lanes' 16-byte stores fall in distinct banks)
  __shared__ float4 stage[kStaged ? kT / 32 : 1][32][kStageVec + 1];
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t i0 = t * kPer;
  const int64_t i1 = i0 + kPer < m ? i0 + kPer : m;
  const bool regular = G.p.ray_mode == EPET_RAYS_REGULAR;
  const int R = G.p.nrays;
  curandState base = {};
  int prev = 0;
  if (i0 < m) {
    prev = rows[i0];
    if (!regular) curand_init(G.p.seed, (unsigned long long)prev, 0ull, &base);
  }
  const int lane = threadIdx.x & 31;
  float4(*st)[kStageVec + 1] = stage[kStaged ? threadIdx.x >> 5 : 0];
  for (int j = 0; j < kPer; j++) {
    const int64_t i = i0 + j;
    const bool live = i < i1;
    int cnl = 0;
    if (live) {
      cnl = rows[i];
      if (j > 0 && !regular) {
        if (cnl > prev) skipahead_sequence((unsigned long long)(cnl - prev), &base);
        else if (cnl != prev) curand_init(G.p.seed, (unsigned long long)cnl, 0ull, &base);
        prev = cnl;
      }
    }
    if (!kStaged) {
      if (live) emit_rays(G, cnl, base, false, reinterpret_cast<float2*>(out + i * (int64_t)R * 6));
      continue;
    }
    curandState state = base;
    int id[5];
    channel_decode(G.p.setup, cnl, id);
    float sn, cs;
    angle_sincos(G.p.setup, id[0], &sn, &cs);
    const CrystalMat m0 = crystal_matrix(G.p.setup, sn, cs, 0, id[1], id[2]);
    const CrystalMat m1 = crystal_matrix(G.p.setup, sn, cs, 1, id[3], id[4]);
    const int64_t row0 = (t - lane) * kPer + j;  // lane r's row: row0 + r kPer
    for (int r0 = 0; r0 < R; r0 += kStageRays) {
      const int nr = min(kStageRays, R - r0);  // even
#pragma unroll 1
      for (int r = 0; r < nr; r += 2) {
        float u[6], w[12];
#pragma unroll
        for (int k = 0; k < 2; k++) {
          draw6(state, regular, u);
          crystal_apply(m0, u[0], u[1], u[2], w + 6 * k);
          crystal_apply(m1, u[3], u[4], u[5], w + 6 * k + 3);
        }
        float4* q = &st[lane][r * 3 / 2];
        q[0] = make_float4(w[0], w[1], w[2], w[3]);
        q[1] = make_float4(w[4], w[5], w[6], w[7]);
        q[2] = make_float4(w[8], w[9], w[10], w[11]);
      }
      __syncwarp();
      const int nv = nr * 3 / 2;  // pieces of a row
      for (int k = lane; k < 32 * nv; k += 32) {
        const int r = nv == kStageVec ? k / kStageVec : k / nv, c = k - r * nv;
        const int64_t row = row0 + (int64_t)r * kPer;
        if (row < m)
          reinterpret_cast<float4*>(out + (row * R + r0) * 6)[c] = st[r][c];
      }
      __syncwarp();
    }
  }
}

// How far, in voxels, rounding can put a cell that a ray visits outside the
// walk's window of its channel, for a ray that crosses the grid between its
// end points while every line joining the crystals spans the grid (the only
// rays whose cells are not tested; k_walk).  u = 2^-24, first order in u:
//  * a crossing's parameter is RN(RN(P - r0) / RN(r1 - r0)), three roundings,
//    so at any parameter of a cell's interval the line through the ray's float
//    end points lies within 3 u |P - r0| <= 3 u D of the cell along every axis
//    (D: the largest coordinate difference of two points of the heads).  Along
//    the slab axis that is a way off the slab, and the hull's edges move by
//    their slope times it: 3 u kappa D (kappa: of one channel, the longest over
//    the shortest distance along the slab axis between points of its crystals);
//  * the end points and the hull's corners are affine in the box coordinates,
//    each rounded by at most u (R + 2 sqrt2 e) (R: the largest coordinate, e:
//    the largest crystal edge): twice that, and again times the hull's slope S
//    for its part along the slab axis;
//  * a hull edge at a slab plane is ah + t w with t = RN(RN(X - as) RN(1 /
//    RN(ds))): four roundings of t, one of w, one of the product, one of the
//    sum: u (6 D + R).  (Between the planes the edges are straight, and a hull
//    is convex: past a corner an edge's extension bounds it.);
//  * its index, RN(RN(f - o) RN(1 / d)), and the planes RN(o + RN(k d)): u (3 +
//    1) times the grid's extent, and u R.
// 1 % more covers the second order.  Two 13 x 13 heads at 0.25 m (kappa 1.12,
// S 1.12, D 0.52 m): 8.8 m u, so that pitches from 0.53 mm need no test; the
// workloads' 2 mm leave a factor of 3.8.
static double window_error(const epet_problem& p) {
  const epet_setup& s = p.setup;
  const epet_grid& g = p.grid;
  const double e = std::max({(double)s.segx, (double)s.segy, (double)s.segz});
  const double half_z = 0.5 * s.segz * std::max(s.n0z, s.n1z);
  const double half_y = 0.5 * s.segy * std::max(s.n0y, s.n1y);
  const double apart = std::fabs((double)s.pos1x - s.pos0x);
  const double Dy = 0.5 * s.segy * ((double)s.n0y + s.n1y);
  const double D = std::max(std::hypot(apart + s.segx, 0.5 * s.segz * ((double)s.n0z + s.n1z)), Dy);
  double R = std::max(half_y, std::hypot(std::max(std::fabs((double)s.pos0x),
                                                  std::fabs((double)s.pos1x)) + 0.5 * s.segx,
                                         half_z));
  double pitch = g.d[0], extent = 0.0;
  for (int a = 0; a < 3; a++) {
    const double o = g.o[a], n_d = (double)g.n[a] * g.d[a];
    pitch = std::min(pitch, (double)g.d[a]);
    extent = std::max(extent, n_d);
    R = std::max({R, std::fabs(o), std::fabs(o + n_d)});
  }
  // Along the slab axis, the horizontal one that the line follows more closely,
  // the crystals' centres are at least apart / sqrt2 from each other, and
  // points of the crystals at most q nearer or farther.
  const double A = apart * std::sqrt(0.5), q = std::hypot((double)s.segx, (double)s.segz);
  if (!(A > q)) return INFINITY;
  const double kappa = (A + q) / (A - q), S = std::max(kappa, Dy / (A - q));
  const double roundings = (9.0 + 3.0 * kappa) * D +
                           2.0 * (1.0 + S) * (R + 2.0 * std::sqrt(2.0) * e) + 2.0 * R +
                           4.0 * extent;
  return 1.01 * std::ldexp(roundings, -24) / pitch;
}

Geo make_geo(const epet_problem& p) {
  Geo G;
  G.p = p;
  // 0.5*(absolute(vxlEdges)+absolute(pxlEdges)) with absolute = sqrtf of the
  // left-to-right sum of squares (getSystemMatrixDeviceOnly.cu:55-58); this
  // file is compiled with host contraction disabled.
  volatile float a0 = p.grid.d[0] * p.grid.d[0];
  volatile float a1 = p.grid.d[1] * p.grid.d[1];
  volatile float a2 = p.grid.d[2] * p.grid.d[2];
  volatile float av = sqrtf((a0 + a1) + a2);
  volatile float b0 = p.setup.segx * p.setup.segx;
  volatile float b1 = p.setup.segy * p.setup.segy;
  volatile float b2 = p.setup.segz * p.setup.segz;
  volatile float bv = sqrtf((b0 + b1) + b2);
  volatile float sr = av + bv;
  G.sum_radii = 0.5f * sr;
  G.V = p.grid.n[0] * p.grid.n[1] * p.grid.n[2];
  G.nyz = p.grid.n[1] * p.grid.n[2];
  // Fixed-point chord sums: a cell gets at most nrays chords (one per ray),
  // each split as hi * 2^b + lo with lo < 2^b; b and the scale 2^s are chosen
  // so that nrays * 2^b <= 2^32 and nrays * max(hi) < 2^32, i.e. both halves
  // sum in 32 bits without carries, exactly and in any order.  A chord is at
  // most the voxel diagonal (av, +1% for rounding).
  int lg = 0;
  while ((1ll << lg) < (long long)p.nrays + 1) lg++;  // ceil(log2(nrays + 1))
  const int b = 32 - lg;                               // lo bits
  const int units_bits = 64 - 2 * lg;                  // chord units < 2^units_bits
  int s = (int)floor(log2(ldexp(1.0, units_bits) / ((double)av * 1.01 + 1e-30)));
  if (s > 100) s = 100;
  G.fx_scale = ldexpf(1.0f, s);
  G.fx_inv = ldexpf(1.0f, -s);
  G.fx_split = b;
  for (int a = 0; a < 3; a++) G.inv_pitch[a] = 1.f / p.grid.d[a];
  G.check_window = !(window_error(p) < kWinPad);
  return G;
}

template <int kPer, int kT, bool kStaged>
static void launch_rays_as(const Geo& G, const int32_t* rows, int64_t m, float* out,
                           cudaStream_t st) {
  k_rays<kPer, kT, kStaged><<<ceil_div(ceil_div(m, kPer), kT), kT, 0, st>>>(G, rows, m, out);
}

epet_status launch_rays(const Geo& G, const int32_t* rows, int64_t m, float* out,
                        bool uniforms_only, cudaStream_t st) {
  if (m == 0) return EPET_OK;
  const int T = 128, R = G.p.nrays;
  const double per_sm = (double)m / num_sms();
  if (uniforms_only)
    k_uniforms<<<ceil_div(m, T), T, 0, st>>>(G, rows, m, out);
  else if (m > 1 && per_sm <= kRaysOnePerSm)
    launch_rays_as<1, kRaysThreadsFew, false>(G, rows, m, out, st);
  else if (per_sm <= kRaysTwoPerSm + kRaysTwoPerRay * std::min(R, 100))
    launch_rays_as<2, kRaysThreadsFew, false>(G, rows, m, out, st);
  else if (per_sm <= kRaysStagedPerSm || R < kRaysStagedRays || R * per_sm < kRaysStagedSum ||
           (R & 1) != 0 || (reinterpret_cast<uintptr_t>(out) & 15) != 0)
    launch_rays_as<4, kRaysThreads, false>(G, rows, m, out, st);
  else
    launch_rays_as<4, kRaysThreads, true>(G, rows, m, out, st);
  EPET_LAUNCHED();
  return EPET_OK;
}

// Self-test of div_cr against the correctly rounded division: n seeded
// operand pairs, a with exponents in [2^-40, 2^5), b in [2^-20, 2^5), random
// signs and mantissas; counts bitwise differences.
__device__ __forceinline__ uint64_t splitmix64(uint64_t z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

__global__ void k_selftest_div(int64_t n, uint64_t seed, unsigned long long* bad) {
  unsigned long long mine = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t r = splitmix64(seed ^ (uint64_t)i * 0x2545f4914f6cdd1dull);
    const uint32_t ea = 127 - 40 + (uint32_t)((r >> 23) % 45u);
    const uint32_t eb = 127 - 20 + (uint32_t)((r >> 46) % 25u);
    const float a = (r & 0xfffff) == 0 ? 0.f
                    : __uint_as_float(((uint32_t)(r >> 63) << 31) | (ea << 23) |
                                      ((uint32_t)r & 0x7fffffu));
    const float b = __uint_as_float(((uint32_t)(r >> 62 & 1u) << 31) | (eb << 23) |
                                    ((uint32_t)(r >> 32) & 0x7fffffu));
    if (__float_as_uint(div_cr(a, b, __frcp_rn(b))) != __float_as_uint(__fdiv_rn(a, b))) mine++;
  }
  if (mine) atomicAdd(bad, mine);
}

}  // namespace epet

using namespace epet;

// Work measure of the walk: the cells a ray crosses inside the grid, i.e. 1
// + the grid planes it passes between its entry and exit (per axis, the
// distance between the entry and exit cell indices).  Entry and exit cells
// are taken a little inside the ray's grid interval, so a ray that only
// grazes a plane counts the cells on one side of it.
__global__ void k_ray_steps(Geo G, const float* __restrict__ rays, int64_t n,
                            unsigned long long* __restrict__ total,
                            unsigned long long* __restrict__ per_row) {
  const epet_grid& g = G.p.grid;
  unsigned long long mine = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float* r = rays + 6 * i;
    float a_in = 0.f, a_out = 1.f;
    bool hit = true;
    for (int a = 0; a < 3; a++) {
      const float p0 = r[a], dp = r[a + 3] - r[a];
      const float lo = g.o[a], hi = g.o[a] + g.n[a] * g.d[a];
      if (dp == 0.f) {
        hit = hit && p0 > lo && p0 < hi;
      } else {
        const float t0 = (lo - p0) / dp, t1 = (hi - p0) / dp;
        a_in = fmaxf(a_in, fminf(t0, t1));
        a_out = fminf(a_out, fmaxf(t0, t1));
      }
    }
    if (!hit || !(a_in < a_out)) continue;
    const float span = a_out - a_in, t_in = a_in + 1e-6f * span, t_out = a_out - 1e-6f * span;
    unsigned long long st = 1;
    for (int a = 0; a < 3; a++) {
      const float dp = r[a + 3] - r[a];
      const int c0 = min(max((int)floorf((r[a] + t_in * dp - g.o[a]) / g.d[a]), 0), g.n[a] - 1);
      const int c1 = min(max((int)floorf((r[a] + t_out * dp - g.o[a]) / g.d[a]), 0), g.n[a] - 1);
      st += (unsigned long long)abs(c1 - c0);
    }
    mine += st;
    if (per_row) atomicAdd(per_row + i / G.p.nrays, st);
  }
  for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(total, mine);
}

extern "C" {

epet_status epet_build_counters(int64_t* overflow_rows_h, int64_t* exact_rows_h) {
  if (overflow_rows_h) *overflow_rows_h = overflow_rows_total();
  if (exact_rows_h) *exact_rows_h = exact_rows_total();
  return EPET_OK;
}

epet_status epet_selftest_window_error(const epet_problem* p, double* voxels_h,
                                       double* margin_h) {
  EPET_CHECK(epet_problem_validate(p));
  if (!voxels_h || !margin_h) return set_error(EPET_ERR_INVALID, "NULL output");
  *voxels_h = window_error(*p);
  *margin_h = kWinPad;
  return EPET_OK;
}

epet_status epet_selftest_division(int64_t n, uint64_t seed, int64_t* mismatches_h,
                                   epet_stream_t stream) {
  if (n < 0 || !mismatches_h) return set_error(EPET_ERR_INVALID, "bad arguments");
  cudaStream_t st = (cudaStream_t)stream;
  unsigned long long* bad = nullptr;
  EPET_CUDA(dev_alloc((void**)&bad, 8, st));
  EPET_CUDA(cudaMemsetAsync(bad, 0, 8, st));
  k_selftest_div<<<1024, 256, 0, st>>>(n, seed, bad);
  EPET_LAUNCHED();
  unsigned long long h = 0;
  EPET_CUDA(cudaMemcpyAsync(&h, bad, 8, cudaMemcpyDeviceToHost, st));
  EPET_CUDA(dev_free(bad, st));
  EPET_CUDA(cudaStreamSynchronize(st));
  *mismatches_h = (int64_t)h;
  return EPET_OK;
}

epet_status epet_ray_steps(const epet_problem* p, const int32_t* rows_d, int64_t m,
                           int64_t* row_steps_d, int64_t* steps_h, epet_stream_t stream) {
  EPET_CHECK(epet_problem_validate(p));
  if (m < 0 || (m > 0 && !rows_d) || !steps_h) return set_error(EPET_ERR_INVALID, "bad arguments");
  cudaStream_t st = (cudaStream_t)stream;
  const Geo G = make_geo(*p);
  // rays of chunks of rows (about 256 MB per chunk)
  const int64_t ch = std::max<int64_t>(1, std::min<int64_t>(m, (int64_t(256) << 20) /
                                                                   ((int64_t)p->nrays * 24)));
  Scratch scr;
  EPET_CHECK(scr.init(nullptr, 0, align256((size_t)ch * p->nrays * 24) + 256, st));
  float* rays = scr.take<float>((size_t)ch * p->nrays * 6);
  unsigned long long* tot = scr.take<unsigned long long>(1);
  if (scr.overrun) return set_error(EPET_ERR_INVALID, "internal: workspace size");
  EPET_CUDA(cudaMemsetAsync(tot, 0, 8, st));
  if (row_steps_d && m > 0) EPET_CUDA(cudaMemsetAsync(row_steps_d, 0, m * 8, st));
  for (int64_t c0 = 0; c0 < m; c0 += ch) {
    const int64_t mc = std::min(ch, m - c0);
    EPET_CHECK(launch_rays(G, rows_d + c0, mc, rays, false, st));
    const int64_t nr = mc * p->nrays;
    k_ray_steps<<<std::min<int64_t>(ceil_div(nr, 256), 8 * (int64_t)num_sms()), 256, 0, st>>>(
        G, rays, nr, tot,
        row_steps_d ? reinterpret_cast<unsigned long long*>(row_steps_d + c0) : nullptr);
    EPET_LAUNCHED();
  }
  unsigned long long h = 0;
  EPET_CUDA(cudaMemcpyAsync(&h, tot, 8, cudaMemcpyDeviceToHost, st));
  EPET_CUDA(cudaStreamSynchronize(st));
  *steps_h = (int64_t)h;
  return EPET_OK;
}

epet_status epet_trig_table(const epet_problem* p, float* sc_d,
                            epet_stream_t stream) {
  EPET_CHECK(epet_problem_validate(p));
  if (!sc_d) return set_error(EPET_ERR_INVALID, "sc_d is NULL");
  k_trig<<<ceil_div(p->setup.na, 128), 128, 0, (cudaStream_t)stream>>>(p->setup, sc_d);
  EPET_LAUNCHED();
  return EPET_OK;
}

epet_status epet_dump_uniforms(const epet_problem* p, const int32_t* rows_d,
                               int64_t m, float* out_d, epet_stream_t stream) {
  EPET_CHECK(epet_problem_validate(p));
  if (m < 0 || (m > 0 && (!rows_d || !out_d)))
    return set_error(EPET_ERR_INVALID, "bad rows/out");
  return launch_rays(make_geo(*p), rows_d, m, out_d, true, (cudaStream_t)stream);
}

epet_status epet_rays(const epet_problem* p, const int32_t* rows_d, int64_t m,
                      float* out_d, epet_stream_t stream) {
  EPET_CHECK(epet_problem_validate(p));
  if (m < 0 || (m > 0 && (!rows_d || !out_d)))
    return set_error(EPET_ERR_INVALID, "bad rows/out");
  return launch_rays(make_geo(*p), rows_d, m, out_d, false, (cudaStream_t)stream);
}

}  // extern "C"
