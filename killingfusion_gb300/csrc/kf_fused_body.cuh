// Device-side pieces of the fused float32 psi iteration, shared by the
// single-grid solver (kf_fused.cu) and the batched solver (kf_batch.cu): the
// argument block, the gradient of one band voxel (one thread with closed-form
// stencils for the interior, reference-order form for the outer shell), the
// dense passes and the band-voxel update.  Included once per translation unit (internal
// linkage).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstring>
#include <type_traits>

#include "kf_bounds.cuh"
#include "kf_internal.h"
#include "kf_ref_math.cuh"

namespace {

using namespace kfref;

constexpr int kTX = 32, kTY = 8, kThreads = kTX * kTY;
constexpr int kZSlab = 8;
// CTAs of the batch's band pass: 256 threads (chunks of 256 voxels per problem)
constexpr int kBandWarps = 8;
constexpr int kBandThreads = 32 * kBandWarps;
// CTAs of the single-grid band pass and the per-voxel schedule: 64 threads,
// 8 resident per SM (the register file at 128 registers), so that a small
// band -- a few thousand voxels taken in list order -- spreads over all the
// SMs instead of filling a few
constexpr int kLaneWarps = 2;
constexpr int kLaneThreads = 32 * kLaneWarps;
constexpr int kLaneBlocksPerSM = 8;

struct FusedArgs {
  const float *__restrict__ live;
  const float *__restrict__ can;
  const float *__restrict__ ix;
  const float *__restrict__ iy;
  const float *__restrict__ iz;
  float *__restrict__ ox;
  float *__restrict__ oy;
  float *__restrict__ oz;
  IterStats *st;
  int *rows;  // trust-region step: first failed x per row, this iteration
  int iter;
  DevParams dp;
  // float copies of the parameters
  float h, alpha, omega_k, gamma_k, omega_s, clamp, eps, voxel, oob, band_hi, band_lo;
  float inv2h, inv4hh;  // 1 / 2h and 1 / 4h^2
  int64_t row, plane;   // voxels from one to the next along y and along z
};

// Float arithmetic with every rounding spelled out: fm, fa and fsb never
// merge into a fused multiply-add, ff always is one.  The band update is
// inlined into several kernels (the single-grid band pass, the batch, the
// per-voxel schedule) whose surrounding code differs, and the compiler's
// choice of which products to fuse may follow that code; with the roundings
// explicit, a batch gives each problem the bits its own solve gives.
__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsb(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float ff(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// utils.h:6-25 in float with explicit roundings: a * (1 - t) + b * t, along
// x, then y, then z.
// u = 1 - t, t each axis's fraction.
__device__ __forceinline__ float lerp1f(float a, float b, float u, float t) { return ff(b, t, fm(a, u)); }
__device__ __forceinline__ float lerp3f(const float v[8], float x, float y, float z) {
  const float ux = fsb(1.f, x), uy = fsb(1.f, y), uz = fsb(1.f, z);
  const float s = lerp1f(lerp1f(v[0], v[1], ux, x), lerp1f(v[2], v[3], ux, x), uy, y);
  const float t = lerp1f(lerp1f(v[4], v[5], ux, x), lerp1f(v[6], v[7], ux, x), uy, y);
  return lerp1f(s, t, uz, z);
}

__device__ __forceinline__ float phi_at(const FusedArgs &a, int x, int y, int z) {
  const DevParams &d = a.dp;
  if (x < 0 || x >= d.nx || y < 0 || y >= d.ny || z < 0 || z >= d.nz) return a.oob;
  return __ldg(a.live + ((int64_t)z * d.ny + y) * d.nx + x);
}

// phi_live at grid coordinate t (SDF::getDistance after its -0.5 shift,
// SDF.cpp:503-524): truncating base, outside corners read MaxSurface+eps.
__device__ __forceinline__ float phi_tri(const FusedArgs &a, float t0, float t1, float t2) {
  const DevParams &d = a.dp;
  int b0 = (int)t0, b1 = (int)t1, b2 = (int)t2;
  float f0 = fsb(t0, (float)b0), f1 = fsb(t1, (float)b1), f2 = fsb(t2, (float)b2);
  float v[8];
  if ((unsigned)b0 < (unsigned)(d.nx - 1) && (unsigned)b1 < (unsigned)(d.ny - 1) &&
      (unsigned)b2 < (unsigned)(d.nz - 1)) {
    // all eight corners inside: one address, constant strides
    const float *p = a.live + ((int64_t)b2 * d.ny + b1) * d.nx + b0;
    const int64_t sy = d.nx, sz = (int64_t)d.nx * d.ny;
    v[0] = __ldg(p);
    v[1] = __ldg(p + 1);
    v[2] = __ldg(p + sy);
    v[3] = __ldg(p + sy + 1);
    v[4] = __ldg(p + sz);
    v[5] = __ldg(p + sz + 1);
    v[6] = __ldg(p + sz + sy);
    v[7] = __ldg(p + sz + sy + 1);
  } else {
#pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = phi_at(a, b0 + (c & 1), b1 + ((c >> 1) & 1), b2 + (c >> 2));
  }
  return lerp3f(v, f0, f1, f2);
}

// The warped value of the band test, SDF::getDistance(i, psi) (SDF.cpp:570-575).
__device__ __noinline__ float warped_value(const FusedArgs &a, int x, int y, int z, float p0, float p1,
                                           float p2) {
  return phi_tri(a, (((float)x + p0) + 0.5f) - 0.5f, (((float)y + p1) + 0.5f) - 0.5f,
                 (((float)z + p2) + 0.5f) - 0.5f);
}

// The 20 psi neighbours of the interior stencil (nb20_off): the 19-point
// Killing stencil and the far corner (1,1,1) of the cell-centre cell.
enum { N000 = 0, NXP, NXM, NYP, NYM, NZP, NZM, NXPYP, NXPYM, NXMYP, NXMYM, NXPZP, NXPZM, NXMZP,
       NXMZM, NYPZP, NYPZM, NYMZP, NYMZM, N111 };

// The stencil offsets as compile-time functions, so that a loop over them
// unrolls into constant-offset code.  off25_at: the 25 sub-voxel offsets
// (units of h) of the cell-centre samples: 0, +-e_k (gradient), +-2e_k and
// +-e_j+-e_k (Hessian).
__host__ __device__ constexpr int nb20_off(int n, int c) {
  constexpr signed char t[20][3] = {
      {0, 0, 0},  {1, 0, 0},  {-1, 0, 0}, {0, 1, 0},   {0, -1, 0}, {0, 0, 1},  {0, 0, -1},
      {1, 1, 0},  {1, -1, 0}, {-1, 1, 0}, {-1, -1, 0}, {1, 0, 1},  {1, 0, -1}, {-1, 0, 1},
      {-1, 0, -1}, {0, 1, 1}, {0, 1, -1}, {0, -1, 1},  {0, -1, -1}, {1, 1, 1}};
  return t[n][c];
}
__host__ __device__ constexpr int off25_at(int j, int c) {
  constexpr signed char t[25][3] = {
      {0, 0, 0},   {1, 0, 0},   {-1, 0, 0},  {0, 1, 0},  {0, -1, 0},  {0, 0, 1},  {0, 0, -1},
      {2, 0, 0},   {-2, 0, 0},  {0, 2, 0},   {0, -2, 0}, {0, 0, 2},   {0, 0, -2}, {1, 0, 1},
      {-1, 0, 1},  {0, 1, 1},   {0, -1, 1},  {1, 1, 0},  {-1, 1, 0},  {-1, 0, -1}, {1, 0, -1},
      {0, -1, -1}, {0, 1, -1},  {-1, -1, 0}, {1, -1, 0}};
  return t[j][c];
}

// One interior voxel (1 <= x,y,z <= n-2) by one thread: returns the step
// d = -alpha * g, the warped value s at i + psi(i), the monitored energy e
// and psi(i) in c0.  The thread loads the 20 psi neighbours of each
// component and takes all 26 samples, whose offsets are compile-time
// constants, reading the 25 cell-centre samples' corners once when they
// share one cell; the derivative stencils are the reference's
// (SDF.cpp:726-744, 867-881).  Measured against groups of lanes per voxel that shared the
// neighbours by shuffles (and so replicated the Killing stencil and the
// moments on every lane): one thread per voxel runs 112 warp instructions
// per band voxel against 291 for 4 lanes, 1.7x the band voxels/s on
// band-heavy grids, 2.3x on a 64-problem batch, 3 % faster on the dense
// 256^3 iteration; 4 lanes had been 1.32x 8 lanes and 2x 16.
// How a kernel reads psi: through the read-only path (psi not written during
// the kernel), through L2 only (ld.global.cg; the per-voxel schedule, which
// writes psi in place), or through L1 and L2 (ld.global.ca; the persistent
// passes, which write psi between iterations and order those writes with
// the fences of their grid-wide barrier -- the read-only path is outside
// that ordering, L1 is not).
enum PsiLoad { kPsiReadOnly = 0, kPsiL2 = 1, kPsiL1 = 2 };

template <int kLoad>
__device__ __forceinline__ float load_psi(const float *p) {
  if constexpr (kLoad == kPsiL2)
    return __ldcg(p);
  else if constexpr (kLoad == kPsiL1)
    return __ldca(p);
  else
    return __ldg(p);
}

template <int kLoad = kPsiReadOnly>
__device__ __forceinline__ void gradient_lane(const FusedArgs &a, int x, int y, int z, int64_t idx, float d[3],
                                              float &s_out, float &e_out, float c0[3]) {
  const DevParams &dp = a.dp;
  const int64_t sy = dp.nx, sz = (int64_t)dp.nx * dp.ny;
  const float h = a.h;
  const float *planes[3] = {a.ix, a.iy, a.iz};
  float kg[3], div[3] = {0.f, 0.f, 0.f}, m[3][7], J[3][3];
  const float two_h = fm(2.f, h), hh = fm(h, h);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float *p = planes[c] + idx;
    float v[20];
#pragma unroll
    for (int n = 0; n < 20; ++n) {
      const float *q = p + nb20_off(n, 0) + nb20_off(n, 1) * sy + nb20_off(n, 2) * sz;
      v[n] = load_psi<kLoad>(q);
    }
    const float v000 = v[N000];
    c0[c] = v000;
    // Killing second differences (DisplacementField.cpp:326-331)
    const float xx = fm(two_h, fa(fsb(v[NXP], v000), fsb(v[NXM], v000)));
    const float yy = fm(two_h, fa(fsb(v[NYP], v000), fsb(v[NYM], v000)));
    const float zz = fm(two_h, fa(fsb(v[NZP], v000), fsb(v[NZM], v000)));
    const float xy = fm(hh, fsb(fsb(v[NXPYP], v[NXPYM]), fsb(v[NXMYP], v[NXMYM])));
    const float xz = fm(hh, fsb(fsb(v[NXPZP], v[NXPZM]), fsb(v[NXMZP], v[NXMZM])));
    const float yz = fm(hh, fsb(fsb(v[NYPZP], v[NYPZM]), fsb(v[NYMZP], v[NYMZM])));
    kg[c] = fm(-2.f, fa(fa(xx, yy), zz));
    if (c == 0) { div[0] = fa(div[0], xx); div[1] = fa(div[1], xy); div[2] = fa(div[2], xz); }
    if (c == 1) { div[0] = fa(div[0], xy); div[1] = fa(div[1], yy); div[2] = fa(div[2], yz); }
    if (c == 2) { div[0] = fa(div[0], xz); div[1] = fa(div[1], yz); div[2] = fa(div[2], zz); }
    J[c][0] = fm(0.5f, fsb(v[NXP], v[NXM]));
    J[c][1] = fm(0.5f, fsb(v[NYP], v[NYM]));
    J[c][2] = fm(0.5f, fsb(v[NZP], v[NZM]));
    // moments of the cell [i, i+1]^3 (corner k_abc = psi(i + (a,b,c)))
    const float k000 = v000, k100 = v[NXP], k010 = v[NYP], k110 = v[NXPYP];
    const float k001 = v[NZP], k101 = v[NXPZP], k011 = v[NYPZP], k111 = v[N111];
    const float sx0 = fa(fa(k000, k010), fa(k001, k011)), sx1 = fa(fa(k100, k110), fa(k101, k111));
    const float sy0 = fa(fa(k000, k100), fa(k001, k101)), sy1 = fa(fa(k010, k110), fa(k011, k111));
    const float sz0 = fa(fa(k000, k100), fa(k010, k110)), sz1 = fa(fa(k001, k101), fa(k011, k111));
    m[c][0] = fm(0.125f, fa(sx0, sx1));
    m[c][1] = fm(0.25f, fsb(sx1, sx0));
    m[c][2] = fm(0.25f, fsb(sy1, sy0));
    m[c][3] = fm(0.25f, fsb(sz1, sz0));
    m[c][4] = fm(0.5f, fsb(fa(fsb(fsb(k110, k010), fsb(k100, k000)), fsb(k111, k011)), fsb(k101, k001)));
    m[c][5] = fm(0.5f, fsb(fa(fsb(fsb(k101, k001), fsb(k100, k000)), fsb(k111, k011)), fsb(k110, k010)));
    m[c][6] = fm(0.5f, fsb(fa(fsb(fsb(k011, k001), fsb(k010, k000)), fsb(k111, k101)), fsb(k110, k100)));
  }
  // Killing gradient: damped divergence term, clamp |g| to killing_clamp, /4h^2
  const float m2g = fm(-2.f, a.gamma_k);
#pragma unroll
  for (int c = 0; c < 3; ++c) kg[c] = ff(m2g, div[c], kg[c]);
  {
    const float nrm = sqrtf(ff(kg[2], kg[2], ff(kg[1], kg[1], fm(kg[0], kg[0]))));
    const float sc = nrm > a.clamp ? a.clamp / nrm : 1.f;
    const float den = fm(fm(4.f, h), h);
#pragma unroll
    for (int c = 0; c < 3; ++c) kg[c] = fm(kg[c], sc) / den;
  }
  // the 25 cell-centre samples and the warped value at i + psi(i)
  const float base[3] = {fa((float)x, 0.5f), fa((float)y, 0.5f), fa((float)z, 0.5f)};
  // Shared corner cell.  Along axis c every sample lies within
  // h * (2 + 2 (|m1| + |m2| + |m3|) + h (|m4| + |m5| + |m6|)) of the centre
  // sample base + m0: the offsets are at most 2 and the products of the
  // mixed samples' offsets are +-1.  When that interval, widened for the
  // roundings of the positions (1e-3 voxel plus 2^-20 of the coordinate,
  // several float ulps of it), has one truncated base on every axis and
  // that cell is inside the grid, the 25 samples read the same eight
  // corners: they are loaded once, and each sample interpolates them with
  // its own fractions, the arithmetic phi_tri does after loading them
  // itself.
  int cb[3];
  bool shared = true;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float m1 = fabsf(m[c][1]) + fabsf(m[c][2]) + fabsf(m[c][3]);
    const float m2 = fabsf(m[c][4]) + fabsf(m[c][5]) + fabsf(m[c][6]);
    const float ctr = fa(base[c], m[c][0]);
    const float r = h * (2.f + 2.f * m1 + h * m2) + 1e-3f + fabsf(ctr) * 0x1p-20f;
    const float lo = ctr - r, hi = ctr + r;
    const int b = (int)lo;
    const int n = c == 0 ? dp.nx : (c == 1 ? dp.ny : dp.nz);
    shared = shared && lo >= 0.f && (int)hi == b && (unsigned)b < (unsigned)(n - 1);
    cb[c] = b;
  }
  // sample j's position (SDF::getDistancef at i+0.5+h*o; the half voxel it
  // adds is removed again by getDistance): psi~ there is the cell's
  // trilinear form in its moments, terms with a zero offset dropped at
  // compile time
  auto position = [&](int j, float t[3]) {
    const int o0 = off25_at(j, 0), o1 = off25_at(j, 1), o2 = off25_at(j, 2);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float lin = 0.f, quad = 0.f;
      if (o0) lin = ff((float)o0, m[c][1], lin);
      if (o1) lin = ff((float)o1, m[c][2], lin);
      if (o2) lin = ff((float)o2, m[c][3], lin);
      if (o0 * o1) quad = ff((float)(o0 * o1), m[c][4], quad);
      if (o0 * o2) quad = ff((float)(o0 * o2), m[c][5], quad);
      if (o1 * o2) quad = ff((float)(o1 * o2), m[c][6], quad);
      const int oc = c == 0 ? o0 : (c == 1 ? o1 : o2);
      t[c] = fa(fa(base[c], fm(h, (float)oc)), ff(h, ff(h, quad, lin), m[c][0]));
    }
  };
  float f[25];
  if (shared) {
    const float *p = a.live + ((int64_t)cb[2] * dp.ny + cb[1]) * dp.nx + cb[0];
    float cell[8];
    cell[0] = __ldg(p);
    cell[1] = __ldg(p + 1);
    cell[2] = __ldg(p + sy);
    cell[3] = __ldg(p + sy + 1);
    cell[4] = __ldg(p + sz);
    cell[5] = __ldg(p + sz + 1);
    cell[6] = __ldg(p + sz + sy);
    cell[7] = __ldg(p + sz + sy + 1);
#pragma unroll
    for (int j = 0; j < 25; ++j) {
      float t[3];
      position(j, t);
      f[j] = lerp3f(cell, fsb(t[0], (float)cb[0]), fsb(t[1], (float)cb[1]), fsb(t[2], (float)cb[2]));
    }
  } else {
#pragma unroll
    for (int j = 0; j < 25; ++j) {
      float t[3];
      position(j, t);
      f[j] = phi_tri(a, t[0], t[1], t[2]);
    }
  }
  const float s = phi_tri(a, fsb(fa(fa((float)x, c0[0]), 0.5f), 0.5f), fsb(fa(fa((float)y, c0[1]), 0.5f), 0.5f),
                          fsb(fa(fa((float)z, c0[2]), 0.5f), 0.5f));
  const float cv = __ldg(a.can + idx);
  const float inv2h = a.inv2h, inv4hh = a.inv4hh;
  // SDF.cpp:726-744: (f(p + h e_k) - f(p - h e_k)) / 2h
  const float g[3] = {fm(fsb(f[1], f[2]), inv2h), fm(fsb(f[3], f[4]), inv2h), fm(fsb(f[5], f[6]), inv2h)};
  // SDF.cpp:867-881 on the same samples
  const float f02 = fm(2.f, f[0]);
  const float hxx = fm(fa(fsb(f[7], f02), f[8]), inv4hh);
  const float hyy = fm(fa(fsb(f[9], f02), f[10]), inv4hh);
  const float hzz = fm(fa(fsb(f[11], f02), f[12]), inv4hh);
  const float hxz = fm(fsb(fsb(fa(f[13], f[19]), f[20]), f[14]), inv4hh);
  const float hyz = fm(fsb(fsb(fa(f[15], f[21]), f[22]), f[16]), inv4hh);
  const float hxy = fm(fsb(fsb(fa(f[17], f[23]), f[24]), f[18]), inv4hh);

  float grad[3] = {0.f, 0.f, 0.f};
  float e = 0.f;
  if (dp.use_data) {
    const float r = fsb(s, cv) / a.voxel;
#pragma unroll
    for (int k = 0; k < 3; ++k) grad[k] = ff(r, g[k], grad[k]);
    e = ff(fm(0.5f, r), r, e);
  }
  if (dp.use_killing) {
#pragma unroll
    for (int k = 0; k < 3; ++k) grad[k] = ff(kg[k], a.omega_k, grad[k]);
    float fr = 0.f, tr = 0.f;
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        fr = ff(J[p][k], J[p][k], fr);
        tr = ff(J[p][k], J[k][p], tr);
      }
    e = ff(a.omega_k, ff(a.gamma_k, tr, fr), e);
  }
  if (dp.use_levelset) {
    const float gn = sqrtf(ff(g[2], g[2], ff(g[1], g[1], fm(g[0], g[0]))));
    const float hg0 = ff(hxz, g[2], ff(hxy, g[1], fm(hxx, g[0])));
    const float hg1 = ff(hyz, g[2], ff(hyy, g[1], fm(hxy, g[0])));
    const float hg2 = ff(hzz, g[2], ff(hyz, g[1], fm(hxz, g[0])));
    const float sc = fm(fsb(gn, 1.f) / fa(gn, a.eps), a.omega_s);
    grad[0] = ff(hg0, sc, grad[0]);
    grad[1] = ff(hg1, sc, grad[1]);
    grad[2] = ff(hg2, sc, grad[2]);
    const float r = fsb(gn / a.voxel, 1.f);
    e = ff(fm(fm(a.omega_s, 0.5f), r), r, e);
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) d[k] = fm(-a.alpha, grad[k]);
  s_out = s;
  e_out = e;
}

// ---------------------------------------------------------------------------
// A band voxel by a group of four warps
// ---------------------------------------------------------------------------
// A group takes 32 voxels at a time, one per lane of each of its warps, and
// cuts a voxel's update into parts that do not depend on one another, so that
// little is computed twice and every rounding is gradient_lane's:
//   part 1  roles 0-2 take one psi component each: its 20 neighbours, the
//           Killing second differences, the cell's moments and the corner
//           cell of the samples along that axis.  Role 3 takes the warped
//           value at i + psi(i) and phi_can(i).
//   part 2  the 25 cell-centre samples by the stencil they belong to, eight
//           or nine a warp (roles 0-2), and the Killing gradient (role 3: a
//           chain of divisions and a square root that nothing in its own warp
//           would hide).
//   part 3  one warp adds the terms up and steps psi.
// The parts hand their values over in shared memory, between two barriers of
// the group's 128 threads.
constexpr int kGroupWarps = 4;
constexpr int kGroupThreads = 32 * kGroupWarps;

struct GroupShared {
  // part 1's values of component c: {m0, m1, m2, m3}, {m4, m5, m6, the
  // samples' corner cell or -1} and {-2 (xx + yy + zz), the component's
  // shares of the divergence term}, {the row of the Jacobian, psi_c(i)}
  float4 mom[3][2][32], kil[3][2][32];
  // part 2's: {hxx, hyy, hzz, psi_0(i)}, {g, psi_1(i)}, {hxz, hxy, psi_2(i),
  // yz's last sample}, {kg, the Killing term of the monitored energy}; the
  // warped value, phi_can and yz's first samples
  float4 out[4][32];
  float more[4][32];
  float spread[25][32];  // group_samples_spread's samples
};

// psi's planes of one iteration: a.ix.. read and a.ox.. written, or (odd) the
// reverse.  Chosen where they are used, from the kernel's parameters: six
// pointers would take twelve registers through the whole iteration.
template <int kC>
__device__ __forceinline__ const float *plane_in(const FusedArgs &a, bool odd) {
  return kC == 0 ? (odd ? a.ox : a.ix) : (kC == 1 ? (odd ? a.oy : a.iy) : (odd ? a.oz : a.iz));
}
template <int kC>
__device__ __forceinline__ float *plane_out(const FusedArgs &a, bool odd) {
  return const_cast<float *>(plane_in<kC>(a, !odd));
}

// A barrier of the 128 threads of the block's group g (0..3): barrier 1 + g of
// the block, each by its number (a number in a register would reserve all 16).
__device__ __forceinline__ void group_sync(int g) {
  if (g == 0)
    asm volatile("bar.sync 1, %0;" ::"n"(kGroupThreads) : "memory");
  else if (g == 1)
    asm volatile("bar.sync 2, %0;" ::"n"(kGroupThreads) : "memory");
  else if (g == 2)
    asm volatile("bar.sync 3, %0;" ::"n"(kGroupThreads) : "memory");
  else
    asm volatile("bar.sync 4, %0;" ::"n"(kGroupThreads) : "memory");
}

// Part 1 of component c from its 20 neighbours v: the voxel's coordinate
// along axis c is xc, the grid's size there nc.  mom0, mom1, kil0, kil1: as
// GroupShared holds them.
__device__ __forceinline__ void component_values(const FusedArgs &a, int c, int xc, int nc, const float v[20],
                                                 float4 &mom0, float4 &mom1, float4 &kil0, float4 &kil1) {
  const float h = a.h, two_h = fm(2.f, h), hh = fm(h, h), v000 = v[N000];
  // moments of the cell [i, i+1]^3 (corner k_abc = psi(i + (a,b,c)))
  const float k000 = v000, k100 = v[NXP], k010 = v[NYP], k110 = v[NXPYP];
  const float k001 = v[NZP], k101 = v[NXPZP], k011 = v[NYPZP], k111 = v[N111];
  const float sx0 = fa(fa(k000, k010), fa(k001, k011)), sx1 = fa(fa(k100, k110), fa(k101, k111));
  const float sy0 = fa(fa(k000, k100), fa(k001, k101)), sy1 = fa(fa(k010, k110), fa(k011, k111));
  const float sz0 = fa(fa(k000, k100), fa(k010, k110)), sz1 = fa(fa(k001, k101), fa(k011, k111));
  float m[7];
  m[0] = fm(0.125f, fa(sx0, sx1));
  m[1] = fm(0.25f, fsb(sx1, sx0));
  m[2] = fm(0.25f, fsb(sy1, sy0));
  m[3] = fm(0.25f, fsb(sz1, sz0));
  m[4] = fm(0.5f, fsb(fa(fsb(fsb(k110, k010), fsb(k100, k000)), fsb(k111, k011)), fsb(k101, k001)));
  m[5] = fm(0.5f, fsb(fa(fsb(fsb(k101, k001), fsb(k100, k000)), fsb(k111, k011)), fsb(k110, k010)));
  m[6] = fm(0.5f, fsb(fa(fsb(fsb(k011, k001), fsb(k010, k000)), fsb(k111, k101)), fsb(k110, k100)));
  // Along axis c every sample lies within
  // h * (2 + 2 (|m1| + |m2| + |m3|) + h (|m4| + |m5| + |m6|)) of the centre
  // sample: the offsets are at most 2 and the products of the mixed samples'
  // offsets are +-1.  When that interval, widened for the roundings of the
  // positions (1e-3 voxel plus 2^-20 of the coordinate, several float ulps
  // of it), has one truncated base and that base is inside the grid, all 25
  // samples have it.
  const float m1 = fabsf(m[1]) + fabsf(m[2]) + fabsf(m[3]), m2 = fabsf(m[4]) + fabsf(m[5]) + fabsf(m[6]);
  const float ctr = fa(fa((float)xc, 0.5f), m[0]);
  const float r = h * (2.f + 2.f * m1 + h * m2) + 1e-3f + fabsf(ctr) * 0x1p-20f;
  const float lo = ctr - r, hi = ctr + r;
  const int b = (int)lo;
  const bool tight = lo >= 0.f && (int)hi == b && (unsigned)b < (unsigned)(nc - 1);
  mom0 = make_float4(m[0], m[1], m[2], m[3]);
  mom1 = make_float4(m[4], m[5], m[6], __int_as_float(tight ? b : -1));
  // Killing second differences (DisplacementField.cpp:326-331)
  const float xx = fm(two_h, fa(fsb(v[NXP], v000), fsb(v[NXM], v000)));
  const float yy = fm(two_h, fa(fsb(v[NYP], v000), fsb(v[NYM], v000)));
  const float zz = fm(two_h, fa(fsb(v[NZP], v000), fsb(v[NZM], v000)));
  const float xy = fm(hh, fsb(fsb(v[NXPYP], v[NXPYM]), fsb(v[NXMYP], v[NXMYM])));
  const float xz = fm(hh, fsb(fsb(v[NXPZP], v[NXPZM]), fsb(v[NXMZP], v[NXMZM])));
  const float yz = fm(hh, fsb(fsb(v[NYPZP], v[NYPZM]), fsb(v[NYMZP], v[NYMZM])));
  kil0 = make_float4(fm(-2.f, fa(fa(xx, yy), zz)), c == 0 ? xx : (c == 1 ? xy : xz),
                     c == 0 ? xy : (c == 1 ? yy : yz), c == 0 ? xz : (c == 1 ? yz : zz));
  kil1 = make_float4(fm(0.5f, fsb(v[NXP], v[NXM])), fm(0.5f, fsb(v[NYP], v[NYM])),
                     fm(0.5f, fsb(v[NZP], v[NZM])), v000);
}

// Part 2's inputs, read back by every warp.
struct GroupCell {
  float base[3], m[3][7];
  float b[3];       // the samples' corner cell (kTight)
  float corner[8];  // and its values
};

// The position of the cell-centre sample at offset o (SDF::getDistancef at
// i+0.5+h*o; the half voxel it adds is removed again by getDistance): psi~
// there is the cell's trilinear form in its moments, terms with a zero
// offset left out (at compile time where o is known then).
__device__ __forceinline__ void group_position(const FusedArgs &a, const GroupCell &q, int o0, int o1, int o2,
                                               float t[3]) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    float lin = 0.f, quad = 0.f;
    if (o0) lin = ff((float)o0, q.m[c][1], lin);
    if (o1) lin = ff((float)o1, q.m[c][2], lin);
    if (o2) lin = ff((float)o2, q.m[c][3], lin);
    if (o0 * o1) quad = ff((float)(o0 * o1), q.m[c][4], quad);
    if (o0 * o2) quad = ff((float)(o0 * o2), q.m[c][5], quad);
    if (o1 * o2) quad = ff((float)(o1 * o2), q.m[c][6], quad);
    const int oc = c == 0 ? o0 : (c == 1 ? o1 : o2);
    t[c] = fa(fa(q.base[c], fm(a.h, (float)oc)), ff(a.h, ff(a.h, quad, lin), q.m[c][0]));
  }
}

// The samples of role w in the order its stencils take them: the centre, the
// axes' +-2 and one of yz; the gradient's +-1 and two of yz; xz, xy and the last
// of yz.
__host__ __device__ constexpr int group_sample_id(int w, int k) {
  constexpr signed char t[3][9] = {
      {0, 7, 8, 9, 10, 11, 12, 22, -1}, {1, 2, 3, 4, 5, 6, 15, 21, -1}, {13, 19, 20, 14, 17, 23, 24, 18, 16}};
  return t[w][k];
}

// The same tables for loops that are not unrolled.
__constant__ signed char c_group_sample[3][9] = {
    {0, 7, 8, 9, 10, 11, 12, 22, -1}, {1, 2, 3, 4, 5, 6, 15, 21, -1}, {13, 19, 20, 14, 17, 23, 24, 18, 16}};
__constant__ signed char c_off25[25][3] = {
    {0, 0, 0},   {1, 0, 0},   {-1, 0, 0},  {0, 1, 0},  {0, -1, 0},  {0, 0, 1},  {0, 0, -1},
    {2, 0, 0},   {-2, 0, 0},  {0, 2, 0},   {0, -2, 0}, {0, 0, 2},   {0, 0, -2}, {1, 0, 1},
    {-1, 0, 1},  {0, 1, 1},   {0, -1, 1},  {1, 1, 0},  {-1, 1, 0},  {-1, 0, -1}, {1, 0, -1},
    {0, -1, -1}, {0, 1, -1},  {-1, -1, 0}, {1, -1, 0}};

// Role kW's samples when those of every lane lie in one cell, whose corners
// are in registers.
template <int kW>
__device__ __forceinline__ void group_samples(const FusedArgs &a, const GroupCell &q, float f[9]) {
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int j = group_sample_id(kW, k);
    if (j < 0) break;
    float t[3];
    group_position(a, q, off25_at(j, 0), off25_at(j, 1), off25_at(j, 2), t);
    f[k] = lerp3f(q.corner, fsb(t[0], q.b[0]), fsb(t[1], q.b[1]), fsb(t[2], q.b[2]));
  }
}

// The same when some lane's samples do not share a cell: each gathers its
// own corners.  A loop that is not unrolled, through shared memory, so that this rarer
// form takes no registers from the other.
__device__ __forceinline__ void group_samples_spread(const FusedArgs &a, const GroupCell &q, int w, int lane,
                                                     float (*spread)[32]) {
#pragma unroll 1
  for (int k = 0; k < 9; ++k) {
    const int j = c_group_sample[w][k];
    if (j < 0) break;
    float t[3];
    group_position(a, q, c_off25[j][0], c_off25[j][1], c_off25[j][2], t);
    spread[j][lane] = phi_tri(a, t[0], t[1], t[2]);
  }
}

// Part 2's stencils of role w from its samples (w: what goes with them in
// `out`).  SDF.cpp:726-744 (the gradient's differences over 2h) and
// SDF.cpp:867-881 (the second differences over 4h^2).
__device__ __forceinline__ float4 group_stencils(const FusedArgs &a, int w, const float f[9]) {
  const float inv2h = a.inv2h, inv4hh = a.inv4hh;
  if (w == 0) {
    const float f02 = fm(2.f, f[0]);
    return make_float4(fm(fa(fsb(f[1], f02), f[2]), inv4hh), fm(fa(fsb(f[3], f02), f[4]), inv4hh),
                       fm(fa(fsb(f[5], f02), f[6]), inv4hh), 0.f);
  }
  if (w == 1)
    return make_float4(fm(fsb(f[0], f[1]), inv2h), fm(fsb(f[2], f[3]), inv2h), fm(fsb(f[4], f[5]), inv2h), 0.f);
  return make_float4(fm(fsb(fsb(fa(f[0], f[1]), f[2]), f[3]), inv4hh),
                     fm(fsb(fsb(fa(f[4], f[5]), f[6]), f[7]), inv4hh), 0.f, f[8]);
}

// The Killing term of the monitored energy from the Jacobian's rows.
__device__ __forceinline__ float killing_energy(const FusedArgs &a, float4 j0, float4 j1, float4 j2) {
  const float J[3][3] = {{j0.x, j0.y, j0.z}, {j1.x, j1.y, j1.z}, {j2.x, j2.y, j2.z}};
  float fr = 0.f, tr = 0.f;
#pragma unroll
  for (int p = 0; p < 3; ++p)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      fr = ff(J[p][k], J[p][k], fr);
      tr = ff(J[p][k], J[k][p], tr);
    }
  return ff(a.gamma_k, tr, fr);
}

// The Killing gradient (x, y, z) and the Killing term of the monitored
// energy (w) from part 1's values: damped divergence term, clamp |g| to
// killing_clamp, /4h^2.
__device__ __forceinline__ float4 group_killing(const FusedArgs &a, const GroupShared &sh, int lane) {
  const float h = a.h, m2g = fm(-2.f, a.gamma_k);
  const float4 k0 = sh.kil[0][0][lane], k1 = sh.kil[1][0][lane], k2 = sh.kil[2][0][lane];
  float kg[3];
  kg[0] = ff(m2g, fa(fa(fa(0.f, k0.y), k1.y), k2.y), k0.x);
  kg[1] = ff(m2g, fa(fa(fa(0.f, k0.z), k1.z), k2.z), k1.x);
  kg[2] = ff(m2g, fa(fa(fa(0.f, k0.w), k1.w), k2.w), k2.x);
  const float nrm = sqrtf(ff(kg[2], kg[2], ff(kg[1], kg[1], fm(kg[0], kg[0]))));
  const float sc = nrm > a.clamp ? a.clamp / nrm : 1.f;
  const float den = fm(fm(4.f, h), h);
  return make_float4(fm(kg[0], sc) / den, fm(kg[1], sc) / den, fm(kg[2], sc) / den,
                     killing_energy(a, sh.kil[0][1][lane], sh.kil[1][1][lane], sh.kil[2][1][lane]));
}

// A group's voxel between the step and its statistics (part 3).
struct GroupStep {
  float d[3], r, gn, ke;  // the step; the terms its monitored energy is made of
  bool active;
};

// The monitored energy of the step's voxel and |d|, added to the statistics.
__device__ __forceinline__ void group_statistics(const FusedArgs &a, const GroupStep &t, float &maxd, double &energy,
                                                 unsigned &active) {
  if (!t.active) return;
  float e = 0.f;
  if (a.dp.use_data) e = ff(fm(0.5f, t.r), t.r, e);
  if (a.dp.use_killing) e = ff(a.omega_k, t.ke, e);
  if (a.dp.use_levelset) {
    const float r = fsb(t.gn / a.voxel, 1.f);
    e = ff(fm(fm(a.omega_s, 0.5f), r), r, e);
  }
  maxd = fmaxf(maxd, sqrtf(ff(t.d[2], t.d[2], ff(t.d[1], t.d[1], fm(t.d[0], t.d[0])))));
  energy += e;
  ++active;
}

__device__ __forceinline__ bool interior_voxel(const DevParams &dp, int x, int y, int z) {
  return x >= 1 && y >= 1 && z >= 1 && x <= dp.nx - 2 && y <= dp.ny - 2 && z <= dp.nz - 2;
}
__host__ __device__ inline int64_t shell_voxels(const DevParams &dp) {
  const int64_t x = dp.nx > 2 ? dp.nx - 2 : 0, y = dp.ny > 2 ? dp.ny - 2 : 0, z = dp.nz > 2 ? dp.nz - 2 : 0;
  return dp.count - x * y * z;
}

// i / d for 0 <= i < 2^31 as (umulhi(i, mul) + i) >> shift (Granlund and
// Montgomery's division by an invariant integer): 3 instructions where a
// 32-bit division by a register takes about 20.
__device__ __forceinline__ unsigned divided(unsigned i, const KfDivisor &d) {
  return (__umulhi(i, d.mul) + i) >> d.shift;
}

__device__ __forceinline__ void voxel_xyz(const DevParams &dp, int i, int &x, int &y, int &z) {
  z = (int)divided((unsigned)i, dp.by_plane);
  const unsigned r = (unsigned)i - (unsigned)z * ((unsigned)dp.nx * (unsigned)dp.ny);
  y = (int)divided(r, dp.by_row);
  x = (int)(r - (unsigned)y * (unsigned)dp.nx);
}

// Dense pass over one tile (kTX x kTY columns, kSlab planes) of block
// coordinates (bx, by, bz): stream the slab, apply the band test, append the
// band voxels to list in index order (*count counts them), but those of the
// grid's outer shell to shell_list (*shell_count).  kPassThrough (ping-pong
// buffers): copy psi of the voxels outside the band to the output buffer;
// without it (psi updated in place) they are only read.
template <bool kPassThrough, int kSlab = kZSlab>
__device__ __forceinline__ void stream_tile(const FusedArgs &a, int bx, int by, int bz,
                                            int *__restrict__ list, unsigned *count,
                                            int *__restrict__ shell_list, unsigned *shell_count) {
  static_assert(kTX == 32, "a warp is a row of the tile");
  __shared__ unsigned s_rows[kSlab * kTY];  // band voxels of each row, then of the rows before it
  __shared__ unsigned s_base;
  const DevParams &dp = a.dp;
  const int x = bx * kTX + threadIdx.x;
  const int y = by * kTY + threadIdx.y;
  const int z0 = bz * kSlab;
  const bool col = x < dp.nx && y < dp.ny;
  const int64_t sz = (int64_t)dp.nx * dp.ny;
  const int64_t base = ((int64_t)z0 * dp.ny + y) * dp.nx + x;
  float px[kSlab], py[kSlab], pz[kSlab], ph[kSlab];
#pragma unroll
  for (int j = 0; j < kSlab; ++j) {
    bool ok = col && (z0 + j) < dp.nz;
    int64_t i = base + j * sz;
    px[j] = ok ? __ldcs(a.ix + i) : 0.f;
    py[j] = ok ? __ldcs(a.iy + i) : 0.f;
    pz[j] = ok ? __ldcs(a.iz + i) : 0.f;
    ph[j] = ok ? __ldg(a.live + i) : 0.f;
  }
  // psi == 0 samples its own cell with zero weights: the warped value is
  // phi_live(i) exactly.  Voxels that have moved are tested after the
  // streamed values are dead (their trilinear gather is the rare, long path).
  unsigned moved = 0, hit = 0;
#pragma unroll
  for (int j = 0; j < kSlab; ++j) {
    int z = z0 + j;
    if (!col || z >= dp.nz) continue;
    int64_t i = base + j * sz;
    if (px[j] != 0.f || py[j] != 0.f || pz[j] != 0.f) {
      moved |= 1u << j;
    } else if (in_band(ph[j], a.band_hi, a.band_lo)) {
      hit |= 1u << j;
    } else if (kPassThrough) {
      __stcs(a.ox + i, 0.f);
      __stcs(a.oy + i, 0.f);
      __stcs(a.oz + i, 0.f);
    }
  }
  while (moved) {
    const int j = __ffs(moved) - 1;
    moved &= moved - 1;
    const int64_t i = base + j * sz;
    const float qx = a.ix[i], qy = a.iy[i], qz = a.iz[i];
    const float s = warped_value(a, x, y, z0 + j, qx, qy, qz);
    if (in_band(s, a.band_hi, a.band_lo)) {
      hit |= 1u << j;
    } else if (kPassThrough) {
      __stcs(a.ox + i, qx);
      __stcs(a.oy + i, qy);
      __stcs(a.oz + i, qz);
    }
  }
  if (hit) {
    unsigned shell = hit;  // the planes of this column that lie on the shell
    if (x >= 1 && x <= dp.nx - 2 && y >= 1 && y <= dp.ny - 2) {
      shell = z0 == 0 ? hit & 1u : 0u;
      if (z0 + kSlab >= dp.nz) shell |= hit & 1u << (dp.nz - 1 - z0);
    }
    hit &= ~shell;
    for (; shell; shell &= shell - 1) {
      const unsigned pos = atomicAdd(shell_count, 1u);
      if (KF_IN_BOUNDS(pos, dp.count, KF_SITE_STREAM_LIST)) shell_list[pos] = (int)(base + (__ffs(shell) - 1) * sz);
    }
  }
  if (!__syncthreads_or(hit != 0u)) return;
  const int lane = threadIdx.x, warp = threadIdx.y;
#pragma unroll
  for (int j = 0; j < kSlab; ++j) {
    const unsigned ball = __ballot_sync(0xffffffffu, hit >> j & 1u);
    if (lane == 0) s_rows[j * kTY + warp] = (unsigned)__popc(ball);
  }
  __syncthreads();
  if (warp == 0) {  // the rows' counts to offsets
    unsigned before = 0;
#pragma unroll
    for (int r = 0; r < kSlab * kTY; r += 32) {
      const unsigned c = s_rows[r + lane];
      unsigned incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
      }
      s_rows[r + lane] = before + incl - c;
      before += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) s_base = atomicAdd(count, before);
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kSlab; ++j) {
    const bool mine = hit >> j & 1u;
    const unsigned ball = __ballot_sync(0xffffffffu, mine);
    const unsigned pos = s_base + s_rows[j * kTY + warp] + (unsigned)__popc(ball & ((1u << lane) - 1u));
    if (mine && KF_IN_BOUNDS(pos, dp.count, KF_SITE_STREAM_LIST)) list[pos] = (int)(base + j * sz);
  }
}

// Dense pass over one run of kFlatVoxels consecutive voxels (flat index
// order): thread t streams the float4 groups t and t + kThreads of the run
// from each psi plane and from phi_live, applies the band test and appends
// the band voxels to list (*count counts them).  kPassThrough copies psi of
// all voxels to the output buffer (the band pass overwrites the band
// voxels').  The last count % 4 voxels of the grid are taken by run 0.
constexpr int kFlatGroups = 2;
constexpr int kFlatVoxels = kThreads * kFlatGroups * 4;

__device__ __forceinline__ void flat_test(const FusedArgs &a, float qx, float qy, float qz, float ph,
                                          unsigned &moved, unsigned &hit, int bit) {
  if (qx != 0.f || qy != 0.f || qz != 0.f)
    moved |= 1u << bit;
  else if (in_band(ph, a.band_hi, a.band_lo))
    hit |= 1u << bit;
}

// kCheck: the run is only tested, its band voxels are counted in *count and
// not listed (the split schedule's runs without band voxels, where a band
// voxel would break an invariant of the solver).  kPsiZero: psi is zero at
// every voxel (nothing of it is read), so the test reads phi_live alone.
// A run's voxels are listed in index order: the lanes of a band pass then
// hold neighbours along x, whose psi and phi share cache lines (in the order
// of an atomic counter, 25 lanes' loads touched about 20 lines).
// shell (or NULL): a list of the band voxels on the grid's outer shell, counted
// in *shell_count, in any order.  kShellApart: of the voxels, which are then not
// in `list`; otherwise of their positions there.
template <bool kPassThrough, bool kCheck = false, bool kPsiZero = false, bool kShellApart = false>
__device__ __forceinline__ void stream_flat(const FusedArgs &a, int64_t run, int *__restrict__ list,
                                            unsigned *count, int2 *__restrict__ range = nullptr,
                                            int *__restrict__ shell = nullptr, unsigned *shell_count = nullptr) {
  __shared__ unsigned s_warp[kThreads / 32];
  __shared__ unsigned s_base;
  const DevParams &dp = a.dp;
  const int tid = threadIdx.x;
  const int64_t n4 = dp.count >> 2;
  const float4 *ix = reinterpret_cast<const float4 *>(a.ix), *iy = reinterpret_cast<const float4 *>(a.iy),
               *iz = reinterpret_cast<const float4 *>(a.iz), *lv = reinterpret_cast<const float4 *>(a.live);
  float4 px[kFlatGroups], py[kFlatGroups], pz[kFlatGroups], ph[kFlatGroups];
  int64_t q[kFlatGroups];
#pragma unroll
  for (int g = 0; g < kFlatGroups; ++g) {
    q[g] = run * (kThreads * kFlatGroups) + g * kThreads + tid;
    const bool ok = q[g] < n4, read_psi = ok && !kPsiZero;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    px[g] = read_psi ? __ldcs(ix + q[g]) : zero;
    py[g] = read_psi ? __ldcs(iy + q[g]) : zero;
    pz[g] = read_psi ? __ldcs(iz + q[g]) : zero;
    ph[g] = ok ? __ldg(lv + q[g]) : zero;
  }
  // bit 4g + e: element e of group g has moved / is in the band
  unsigned moved = 0, hit = 0;
#pragma unroll
  for (int g = 0; g < kFlatGroups; ++g) {
    if (q[g] >= n4) continue;
    flat_test(a, px[g].x, py[g].x, pz[g].x, ph[g].x, moved, hit, 4 * g);
    flat_test(a, px[g].y, py[g].y, pz[g].y, ph[g].y, moved, hit, 4 * g + 1);
    flat_test(a, px[g].z, py[g].z, pz[g].z, ph[g].z, moved, hit, 4 * g + 2);
    flat_test(a, px[g].w, py[g].w, pz[g].w, ph[g].w, moved, hit, 4 * g + 3);
    if (kPassThrough) {
      __stcs(reinterpret_cast<float4 *>(a.ox) + q[g], px[g]);
      __stcs(reinterpret_cast<float4 *>(a.oy) + q[g], py[g]);
      __stcs(reinterpret_cast<float4 *>(a.oz) + q[g], pz[g]);
    }
  }
  // the ragged end of the grid, by run 0
  if (run == 0 && tid < (int)(dp.count & 3)) {
    const int64_t i = 4 * n4 + tid;
    const float qx = kPsiZero ? 0.f : a.ix[i], qy = kPsiZero ? 0.f : a.iy[i], qz = kPsiZero ? 0.f : a.iz[i];
    flat_test(a, qx, qy, qz, __ldg(a.live + i), moved, hit, 4 * kFlatGroups);
    if (kPassThrough) {
      a.ox[i] = qx;
      a.oy[i] = qy;
      a.oz[i] = qz;
    }
  }
  // the voxel of a thread's bit
  const auto voxel = [&](int bit) -> int64_t {
    return bit < 4 * kFlatGroups ? 4 * (run * (kThreads * kFlatGroups) + (bit >> 2) * kThreads + tid) + (bit & 3)
                                 : 4 * n4 + tid;
  };
  const bool any_moved = moved != 0u;
  // voxels that have moved: the warped value is a trilinear gather
  while (moved) {
    const int bit = __ffs(moved) - 1;
    moved &= moved - 1;
    const int64_t i = voxel(bit);
    int x, y, z;
    voxel_xyz(dp, (int)i, x, y, z);
    const float s = warped_value(a, x, y, z, a.ix[i], a.iy[i], a.iz[i]);
    if (in_band(s, a.band_hi, a.band_lo)) hit |= 1u << bit;
  }
  if (kCheck) {
    if (hit) atomicAdd(count, (unsigned)__popc(hit));
    return;
  }
  if (kShellApart) {
    for (unsigned h = hit; h; h &= h - 1) {
      const int bit = __ffs(h) - 1;
      const int64_t i = voxel(bit);
      int x, y, z;
      voxel_xyz(dp, (int)i, x, y, z);
      if (interior_voxel(dp, x, y, z)) continue;
      hit &= ~(1u << bit);
      const unsigned pos = atomicAdd(shell_count, 1u);
      if (KF_IN_BOUNDS(pos, shell_voxels(dp), KF_SITE_STREAM_LIST)) shell[pos] = (int)i;
    }
  }
  if (!__syncthreads_or(hit != 0u)) {
    if (range) {
      const bool zero = !__syncthreads_or(any_moved);
      if (tid == 0) *range = make_int2(zero ? 1 : 0, 0);  // (k_split_runs)
    }
    return;
  }
  // one scan of the three counts (group 0, group 1, ragged end), packed
  static_assert(kFlatGroups == 2, "two groups are packed");
  const unsigned mine = (unsigned)__popc(hit & 15u) | (unsigned)__popc(hit >> 4 & 15u) << 12 | (hit >> 8) << 24;
  const int lane = tid & 31, warp = tid >> 5;
  unsigned incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  unsigned before = incl - mine, total = 0;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) {
    const unsigned c = s_warp[w];
    before += w < warp ? c : 0u;
    total += c;
  }
  const unsigned n0 = total & 0xfffu, n1 = total >> 12 & 0xfffu, n = n0 + n1 + (total >> 24);
  if (tid == 0) s_base = atomicAdd(count, n);
  __syncthreads();
  const unsigned base = s_base;
  unsigned at[3] = {before & 0xfffu, n0 + (before >> 12 & 0xfffu), n0 + n1 + (before >> 24)};
#pragma unroll
  for (int g = 0; g < 3; ++g) {
    for (unsigned h = g < 2 ? hit >> (4 * g) & 15u : hit >> 8; h; h &= h - 1) {
      const unsigned pos = base + at[g]++;
      const int i = (int)voxel(4 * g + __ffs(h) - 1);
      if (KF_IN_BOUNDS(pos, dp.count, KF_SITE_STREAM_LIST)) list[pos] = i;
      if (!kShellApart && shell) {
        int x, y, z;
        voxel_xyz(dp, i, x, y, z);
        if (interior_voxel(dp, x, y, z)) continue;
        const unsigned j = atomicAdd(shell_count, 1u);
        if (KF_IN_BOUNDS(j, shell_voxels(dp), KF_SITE_STREAM_LIST)) shell[j] = (int)pos;
      }
    }
  }
  // where this run's band voxels sit in the list (for the next iteration's
  // write-back of their new psi)
  if (range && tid == 0) *range = make_int2((int)base, (int)n);
}

// Appends the voxels `next` (>= 0 on the threads that carry one) of the
// whole block to list_out (of `capacity` entries) with one atomic on
// *count, in thread order; every thread of the block calls it.
template <int kWarps>
__device__ __forceinline__ void block_append(int next, unsigned *count, int *__restrict__ list_out,
                                             int64_t capacity) {
  __shared__ unsigned s_wcnt[kWarps], s_wbase[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool has = next >= 0;
  const unsigned ball = __ballot_sync(0xffffffffu, has);
  if (lane == 0) s_wcnt[warp] = (unsigned)__popc(ball);
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned t = 0;
    for (int w = 0; w < kWarps; ++w) {
      s_wbase[w] = t;
      t += s_wcnt[w];
    }
    const unsigned b = t ? atomicAdd(count, t) : 0u;
    for (int w = 0; w < kWarps; ++w) s_wbase[w] += b;
  }
  __syncthreads();
  if (has) {
    const unsigned pos = s_wbase[warp] + (unsigned)__popc(ball & ((1u << lane) - 1u));
    if (KF_IN_BOUNDS(pos, capacity, KF_SITE_BAND_APPEND)) list_out[pos] = next;
  }
}

// The trust-region step (KillingFusion.cpp:288-314) for the float solvers:
// d = -alpha * g (float) on entry, the accepted step on return; false when
// the step size fell below 1e-7.  The search runs in double, as
// kfref::trust_step: a float position cannot resolve the steps of 1e-7 * g
// that the search reaches before it gives up (near x = 64 one float ulp is
// 7.6e-6 voxel), so in float a step that is too small to move the sample
// reads as "no worse" and the search would accept where the reference
// breaks the row.
__device__ __noinline__ bool trust_step_f(const FusedArgs &a, int x, int y, int z, int64_t i,
                                          const float c[3], float d[3]) {
  const DevParams &dp = a.dp;
  PhiView<double> lv{a.live, dp.nx, dp.ny, dp.nz, dp.oob_phi};
  const double cd[3] = {c[0], c[1], c[2]};
  const double prev = phi_sample(lv, ((double)x + cd[0]) + 0.5, ((double)y + cd[1]) + 0.5,
                                 ((double)z + cd[2]) + 0.5);
  double g[3], dd[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    g[k] = (double)d[k] / -(double)a.alpha;
    dd[k] = -dp.alpha * g[k];
  }
  const bool ok = trust_step(lv, (double)__ldg(a.can + i), prev, x, y, z, cd, g, dp.alpha, dd);
#pragma unroll
  for (int k = 0; k < 3; ++k) d[k] = (float)dd[k];
  return ok;
}

// The 20 psi neighbours of voxel i in one plane.
template <int kLoad>
__device__ __forceinline__ void group_neighbours(const FusedArgs &a, const float *plane, int i, float v[20]) {
  const float *r0 = plane + i;
  const float *yp = r0 + a.row, *ym = r0 - a.row, *zp = r0 + a.plane, *zm = r0 - a.plane;
  const float *ypzp = zp + a.row, *ymzp = zp - a.row, *ypzm = zm + a.row, *ymzm = zm - a.row;
#pragma unroll
  for (int n = 0; n < 20; ++n) {
    const int oy = nb20_off(n, 1), oz = nb20_off(n, 2);
    const float *r = oz == 0 ? (oy == 0 ? r0 : (oy > 0 ? yp : ym))
                             : (oz > 0 ? (oy == 0 ? zp : (oy > 0 ? ypzp : ymzp))
                                       : (oy == 0 ? zm : (oy > 0 ? ypzm : ymzm)));
    v[n] = load_psi<kLoad>(r + nb20_off(n, 0));
  }
}

// The warped value at x + psi (SDF::getDistance(i, psi), SDF.cpp:570-575).
__device__ __forceinline__ float group_warped(const FusedArgs &a, int x, int y, int z, float p0, float p1, float p2) {
  return phi_tri(a, fsb(fa(fa((float)x, p0), 0.5f), 0.5f), fsb(fa(fa((float)y, p1), 0.5f), 0.5f),
                 fsb(fa(fa((float)z, p2), 0.5f), 0.5f));
}

// From the group's first barrier (after part 1) to its second: part 2 of role
// w.  own: psi_w(i) on roles 0-2, the warped value on role 3; can: phi_can(i)
// (role 3).
__device__ __forceinline__ void group_middle(const FusedArgs &a, GroupShared &sh, int g, int w, int lane,
                                             bool interior, int x, int y, int z, float own, float can) {
  const DevParams &dp = a.dp;
  group_sync(g);
  // (the last round's `out` was read before this barrier)
  if (w == 3) {
    if (interior) {
      sh.more[0][lane] = own;
      sh.more[1][lane] = can;
      sh.out[3][lane] = group_killing(a, sh, lane);
    }
  } else if (__any_sync(0xffffffffu, interior)) {
    GroupCell q;
    q.base[0] = fa((float)x, 0.5f);
    q.base[1] = fa((float)y, 0.5f);
    q.base[2] = fa((float)z, 0.5f);
    int b[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float4 lo = sh.mom[c][0][lane], hi = sh.mom[c][1][lane];
      q.m[c][0] = lo.x, q.m[c][1] = lo.y, q.m[c][2] = lo.z, q.m[c][3] = lo.w;
      q.m[c][4] = hi.x, q.m[c][5] = hi.y, q.m[c][6] = hi.z;
      b[c] = __float_as_int(hi.w);
    }
    const bool tight = interior && (b[0] | b[1] | b[2]) >= 0;
    float f[9];
    // one path per warp: the samples of every interior lane in one cell, or
    // each sample its own corners (a warp with both kinds would run both)
    if (__all_sync(0xffffffffu, tight || !interior)) {
      // lanes without an interior voxel read the grid's first cell
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        b[c] = tight ? b[c] : 0;
        q.b[c] = (float)b[c];
      }
      const float *l = a.live + (((unsigned)b[2] * (unsigned)dp.ny + (unsigned)b[1]) * (unsigned)dp.nx + (unsigned)b[0]);
      const float *ly = l + a.row, *lz = l + a.plane, *lyz = lz + a.row;
      q.corner[0] = __ldg(l);
      q.corner[1] = __ldg(l + 1);
      q.corner[2] = __ldg(ly);
      q.corner[3] = __ldg(ly + 1);
      q.corner[4] = __ldg(lz);
      q.corner[5] = __ldg(lz + 1);
      q.corner[6] = __ldg(lyz);
      q.corner[7] = __ldg(lyz + 1);
      if (w == 0)
        group_samples<0>(a, q, f);
      else if (w == 1)
        group_samples<1>(a, q, f);
      else
        group_samples<2>(a, q, f);
    } else {
      if (interior) group_samples_spread(a, q, w, lane, sh.spread);
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        const int j = c_group_sample[w][k];  // (roles 0 and 1 have eight samples; only their own are read)
        f[k] = sh.spread[j < 0 ? c_group_sample[w][0] : j][lane];
      }
    }
    float4 o = group_stencils(a, w, f);
    if (w == 2)
      o.z = own;
    else
      o.w = own;
    sh.out[w][lane] = o;
    if (w == 0) sh.more[2][lane] = f[7];
    if (w == 1) sh.more[3][lane] = fa(f[6], f[7]);
  }
  group_sync(g);
}

// Part 3 of an interior voxel: its step, the terms of its monitored energy,
// psi(i) (c0) and the warped value s.
__device__ __forceinline__ void group_step(const FusedArgs &a, const GroupShared &sh, int lane, GroupStep &t,
                                           float c0[3], float &s) {
  const DevParams &dp = a.dp;
  const float4 hd = sh.out[0][lane], gr = sh.out[1][lane], ho = sh.out[2][lane], kg = sh.out[3][lane];
  c0[0] = hd.w, c0[1] = gr.w, c0[2] = ho.z;
  s = sh.more[0][lane];
  t.ke = kg.w;
  // KillingFusion.cpp:399-476
  float grad[3] = {0.f, 0.f, 0.f};
  if (dp.use_data) {
    t.r = fsb(s, sh.more[1][lane]) / a.voxel;
    grad[0] = ff(t.r, gr.x, grad[0]);
    grad[1] = ff(t.r, gr.y, grad[1]);
    grad[2] = ff(t.r, gr.z, grad[2]);
  }
  if (dp.use_killing) {
    grad[0] = ff(kg.x, a.omega_k, grad[0]);
    grad[1] = ff(kg.y, a.omega_k, grad[1]);
    grad[2] = ff(kg.z, a.omega_k, grad[2]);
  }
  if (dp.use_levelset) {
    t.gn = sqrtf(ff(gr.z, gr.z, ff(gr.y, gr.y, fm(gr.x, gr.x))));
    const float hxz = ho.x, hxy = ho.y;
    const float hyz = fm(fsb(fsb(sh.more[3][lane], sh.more[2][lane]), ho.w), a.inv4hh);
    const float hg0 = ff(hxz, gr.z, ff(hxy, gr.y, fm(hd.x, gr.x)));
    const float hg1 = ff(hyz, gr.z, ff(hd.y, gr.y, fm(hxy, gr.x)));
    const float hg2 = ff(hd.z, gr.z, ff(hyz, gr.y, fm(hxz, gr.x)));
    const float f = fm(fsb(t.gn, 1.f) / fa(t.gn, a.eps), a.omega_s);
    grad[0] = ff(hg0, f, grad[0]);
    grad[1] = ff(hg1, f, grad[1]);
    grad[2] = ff(hg2, f, grad[2]);
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) t.d[k] = fm(-a.alpha, grad[k]);
}

// Updates the voxels i (-1: none) of the lanes of group g, as
// update_interior_voxel does for one: every thread of the group calls it, in role
// w, with its lane's voxel, whose new psi goes to entry `slot` of the output
// planes.  Part 3 and its results (the voxel for the next iteration's list,
// or -1; the step for group_statistics; whether psi(i) is finite) are role
// `last`'s; the other warps return -1.
// Voxels of the outer shell are left alone (warp_shell).
template <int kLoad>
__device__ __forceinline__ int group_update(const FusedArgs &a, bool odd, int i, int slot, GroupShared &sh, int g,
                                            int w, int last, int lane, GroupStep &t, bool &diverged) {
  const DevParams &dp = a.dp;
  t.active = false;
  bool have = i >= 0;
  if (have && (!KF_IN_BOUNDS(i, dp.count, KF_SITE_BAND_LIST) || !KF_IN_BOUNDS(slot, dp.count, KF_SITE_BAND_LIST)))
    have = false;
  int x = 0, y = 0, z = 0;
  if (have) voxel_xyz(dp, i, x, y, z);
  const bool interior = have && interior_voxel(dp, x, y, z);
  float own = 0.f, can = 0.f;  // roles 0-2: psi_w(i); role 3: the warped value and phi_can(i)
  if (interior) {
    if (w < 3) {
      float v[20];
      group_neighbours<kLoad>(a, w == 0 ? plane_in<0>(a, odd) : (w == 1 ? plane_in<1>(a, odd) : plane_in<2>(a, odd)), i,
                              v);
      own = v[N000];
      component_values(a, w, w == 0 ? x : (w == 1 ? y : z), w == 0 ? dp.nx : (w == 1 ? dp.ny : dp.nz), v,
                       sh.mom[w][0][lane], sh.mom[w][1][lane], sh.kil[w][0][lane], sh.kil[w][1][lane]);
    } else {
      can = __ldg(a.can + i);
      own = group_warped(a, x, y, z, load_psi<kLoad>(plane_in<0>(a, odd) + i), load_psi<kLoad>(plane_in<1>(a, odd) + i),
                         load_psi<kLoad>(plane_in<2>(a, odd) + i));
    }
  }
  group_middle(a, sh, g, w, lane, interior, x, y, z, own, can);
  if (w != last || !interior) return -1;
  float c0[3], s;
  group_step(a, sh, lane, t, c0, s);
  t.active = in_band(s, a.band_hi, a.band_lo);
  if (t.active && (!isfinite(c0[0]) || !isfinite(c0[1]) || !isfinite(c0[2]))) diverged = true;
  // a voxel that left the band keeps psi: settle the output buffer
  plane_out<0>(a, odd)[slot] = t.active ? c0[0] + t.d[0] : c0[0];
  plane_out<1>(a, odd)[slot] = t.active ? c0[1] + t.d[1] : c0[1];
  plane_out<2>(a, odd)[slot] = t.active ? c0[2] + t.d[2] : c0[2];
  return t.active ? i : -1;
}

// A lane's statistics of an iteration, in shared memory.
struct GroupStats {
  double energy[32];
  float maxd[32];
  unsigned active[32];
};

// ---------------------------------------------------------------------------
// A voxel of the outer shell by one warp
// ---------------------------------------------------------------------------
// KillingFusion::computeEnergyGradient (KillingFusion.cpp:399-476) with the
// reference's own samples -- truncating casts, psi's linear-index wrap
// (DisplacementField.cpp:22-38), values outside the grid -- which the closed
// forms of the interior leave out.  The 25 cell-centre samples (each psi,
// then phi_live), the warped value and the 19 Killing samples are independent:
// a lane each.  One thread ran them one after the other, about 20 k
// instructions that its whole warp waited for; this takes about 500 a voxel.
// Every rounding is spelled out, so all solvers give a shell voxel the same
// bits.
struct ShellScratch {
  float f[26];      // the cell-centre samples (off25_at's order) and the warped value
  float k[19][3];   // the Killing samples, in off25_at's order of its 19 second-difference offsets
};

template <int kLoad>
__device__ __forceinline__ void shell_psi_at(const FusedArgs &a, const float *const p[3], int x, int y, int z,
                                             float out[3]) {
  const int index = z * (a.dp.nx * a.dp.ny) + y * a.dp.nx + x, total = a.dp.nx * a.dp.ny * a.dp.nz;
  const bool in = index >= 0 && index < total;
#pragma unroll
  for (int c = 0; c < 3; ++c) out[c] = in ? load_psi<kLoad>(p[c] + index) : 0.f;
}

// DisplacementField::getDisplacementAtf (DisplacementField.cpp:40-58).
template <int kLoad>
__device__ __forceinline__ void shell_psi_sample(const FusedArgs &a, const float *const p[3], const float q[3],
                                                 float out[3]) {
  const int b0 = (int)q[0], b1 = (int)q[1], b2 = (int)q[2];
  float v[3][8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    float w[3];
    shell_psi_at<kLoad>(a, p, b0 + (c & 1), b1 + ((c >> 1) & 1), b2 + (c >> 2), w);
    v[0][c] = w[0], v[1][c] = w[1], v[2][c] = w[2];
  }
#pragma unroll
  for (int k = 0; k < 3; ++k)
    out[k] = lerp3f(v[k], fsb(q[0], (float)b0), fsb(q[1], (float)b1), fsb(q[2], (float)b2));
}

// All lanes of a warp call it with the same voxel; every lane gets the step
// d = -alpha * g, the warped value s, the monitored energy e and psi(i) in
// c0.  args and sc (the warp's) in shared memory; odd: psi is in the output planes.
template <int kLoad>
__device__ __noinline__ void shell_gradient(const FusedArgs &a, bool odd, int x, int y, int z, ShellScratch &sc,
                                            float *d, float *s_out, float *e_out, float *c0) {
  const DevParams &dp = a.dp;
  const float *const p[3] = {plane_in<0>(a, odd), plane_in<1>(a, odd), plane_in<2>(a, odd)};
  const int lane = threadIdx.x & 31;
  const float h = a.h;
  __syncwarp();
  if (lane < 26) {
    float q[3] = {(float)x, (float)y, (float)z}, w[3];
    if (lane < 25) {
#pragma unroll
      for (int c = 0; c < 3; ++c) q[c] = ff(h, (float)c_off25[lane][c], fa(q[c], 0.5f));
      shell_psi_sample<kLoad>(a, p, q, w);
    } else {
      shell_psi_at<kLoad>(a, p, x, y, z, w);
    }
    sc.f[lane] = phi_tri(a, fsb(fa(fa(q[0], w[0]), 0.5f), 0.5f), fsb(fa(fa(q[1], w[1]), 0.5f), 0.5f),
                         fsb(fa(fa(q[2], w[2]), 0.5f), 0.5f));
  }
  if (lane < 19) {
    // the 19 offsets of the second differences: off25_at's 0 and 7..24
    const signed char *o = c_off25[lane == 0 ? 0 : 6 + lane];
    const float q[3] = {ff(h, (float)o[0], (float)x), ff(h, (float)o[1], (float)y), ff(h, (float)o[2], (float)z)};
    shell_psi_sample<kLoad>(a, p, q, sc.k[lane]);
  }
  __syncwarp();
  const float *f = sc.f, s = f[25];
  const float can = __ldg(a.can + ((int64_t)z * dp.ny + y) * dp.nx + x);
  const float two_h = fm(2.f, h), four_hh = fm(fm(4.f, h), h);
  const float g[3] = {fsb(f[1], f[2]) / two_h, fsb(f[3], f[4]) / two_h, fsb(f[5], f[6]) / two_h};
  float grad[3] = {0.f, 0.f, 0.f}, e = 0.f;
  if (dp.use_data) {
    const float r = fsb(s, can) / a.voxel;
#pragma unroll
    for (int k = 0; k < 3; ++k) grad[k] = ff(r, g[k], grad[k]);
    e = ff(fm(0.5f, r), r, e);
  }
  if (dp.use_killing) {
    float kg[3], div[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      // (k[n]: off25_at's sample n + 6, k[0] the centre)
      const auto v = [&](int n) { return sc.k[n][c]; };
      const float v2 = fm(2.f, v(0));
      const float xx = fa(fsb(v(1), v2), v(2)), yy = fa(fsb(v(3), v2), v(4)), zz = fa(fsb(v(5), v2), v(6));
      const float xz = fsb(fsb(fa(v(7), v(13)), v(14)), v(8)), yz = fsb(fsb(fa(v(9), v(15)), v(16)), v(10)),
                  xy = fsb(fsb(fa(v(11), v(17)), v(18)), v(12));
      kg[c] = fm(-2.f, fa(fa(xx, yy), zz));
      div[0] = fa(div[0], c == 0 ? xx : (c == 1 ? xy : xz));
      div[1] = fa(div[1], c == 0 ? xy : (c == 1 ? yy : yz));
      div[2] = fa(div[2], c == 0 ? xz : (c == 1 ? yz : zz));
    }
    const float m2g = fm(-2.f, a.gamma_k);
#pragma unroll
    for (int c = 0; c < 3; ++c) kg[c] = ff(m2g, div[c], kg[c]);
    const float nrm = sqrtf(ff(kg[2], kg[2], ff(kg[1], kg[1], fm(kg[0], kg[0]))));
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float k = nrm > a.clamp ? fm(kg[c] / nrm, a.clamp) : kg[c];
      grad[c] = ff(k / four_hh, a.omega_k, grad[c]);
    }
    // the Jacobian's clamped neighbours (kfref::monitor_energy)
    float J[3][3], fr = 0.f, tr = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int up[3] = {min(x + (k == 0), dp.nx - 1), min(y + (k == 1), dp.ny - 1), min(z + (k == 2), dp.nz - 1)};
      const int dn[3] = {max(x - (k == 0), 0), max(y - (k == 1), 0), max(z - (k == 2), 0)};
      float u[3], w[3];
      shell_psi_at<kLoad>(a, p, up[0], up[1], up[2], u);
      shell_psi_at<kLoad>(a, p, dn[0], dn[1], dn[2], w);
#pragma unroll
      for (int c = 0; c < 3; ++c) J[c][k] = fm(0.5f, fsb(u[c], w[c]));
    }
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        fr = ff(J[c][k], J[c][k], fr);
        tr = ff(J[c][k], J[k][c], tr);
      }
    e = ff(a.omega_k, ff(a.gamma_k, tr, fr), e);
  }
  if (dp.use_levelset) {
    const float f02 = fm(2.f, f[0]);
    const float hxx = fa(fsb(f[7], f02), f[8]) / four_hh, hyy = fa(fsb(f[9], f02), f[10]) / four_hh;
    const float hzz = fa(fsb(f[11], f02), f[12]) / four_hh, hxz = fsb(fsb(fa(f[13], f[19]), f[20]), f[14]) / four_hh;
    const float hyz = fsb(fsb(fa(f[15], f[21]), f[22]), f[16]) / four_hh;
    const float hxy = fsb(fsb(fa(f[17], f[23]), f[24]), f[18]) / four_hh;
    const float gn = sqrtf(ff(g[2], g[2], ff(g[1], g[1], fm(g[0], g[0]))));
    const float nm1 = fsb(gn, 1.f), np = fa(gn, a.eps);
    const float hg[3] = {ff(hxz, g[2], ff(hxy, g[1], fm(hxx, g[0]))), ff(hyz, g[2], ff(hyy, g[1], fm(hxy, g[0]))),
                         ff(hzz, g[2], ff(hyz, g[1], fm(hxz, g[0])))};
#pragma unroll
    for (int c = 0; c < 3; ++c) grad[c] = ff(fm(hg[c], nm1) / np, a.omega_s, grad[c]);
    const float r = fsb(gn / a.voxel, 1.f);
    e = ff(fm(fm(a.omega_s, 0.5f), r), r, e);
  }
  float own[3];
  shell_psi_at<kLoad>(a, p, x, y, z, own);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    d[k] = fm(-a.alpha, grad[k]);
    c0[k] = own[k];
  }
  *s_out = s;
  *e_out = e;
}

// Steps band voxel i, whose warped value is s, monitored energy en, psi c0
// and step d: writes its new psi to entry `slot` of the output planes,
// accumulates the statistics and returns the voxel for the next iteration's
// list (-1 if it left the band).
template <bool kTrust>
__device__ __forceinline__ int settle_band_voxel(const FusedArgs &a, int i, int slot, int x, int y, int z, float s,
                                                 float en, const float c0[3], float d[3], float &maxd, double &energy,
                                                 unsigned &active, bool &diverged) {
  const DevParams &dp = a.dp;
  int next = -1;
  if (in_band(s, a.band_hi, a.band_lo)) {
    if (!isfinite(c0[0]) || !isfinite(c0[1]) || !isfinite(c0[2])) diverged = true;
    if (kTrust && !trust_step_f(a, x, y, z, i, c0, d)) {
      // this voxel and the rest of its row keep psi (k_trust_fix)
      atomicMin(a.rows + (z * dp.ny + y), x);
      d[0] = d[1] = d[2] = 0.f;
    }
    a.ox[slot] = c0[0] + d[0];
    a.oy[slot] = c0[1] + d[1];
    a.oz[slot] = c0[2] + d[2];
    maxd = fmaxf(maxd, sqrtf(ff(d[2], d[2], ff(d[1], d[1], fm(d[0], d[0])))));
    energy += en;
    ++active;
    next = i;
  } else {  // left the band: its psi is final, settle the output buffer
    a.ox[slot] = c0[0];
    a.oy[slot] = c0[1];
    a.oz[slot] = c0[2];
  }
  return next;
}

// The data term alone of shell_gradient, by one thread (the trust-region step, which
// no other term goes with): 7 samples where a warp takes 45.  a: in shared memory.
__device__ __noinline__ void shell_data_gradient(const FusedArgs &a, int x, int y, int z, float *d, float *s_out,
                                                 float *e_out, float *c0) {
  const float *const p[3] = {a.ix, a.iy, a.iz};
  const float v[3] = {(float)x, (float)y, (float)z};
  const float h = a.h, two_h = fm(2.f, h);
  float g[3], own[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float f[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float q[3], w[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) q[c] = ff(h, c == k ? (e == 0 ? 1.f : -1.f) : 0.f, fa(v[c], 0.5f));
      shell_psi_sample<kPsiReadOnly>(a, p, q, w);
      f[e] = phi_tri(a, fsb(fa(fa(q[0], w[0]), 0.5f), 0.5f), fsb(fa(fa(q[1], w[1]), 0.5f), 0.5f),
                     fsb(fa(fa(q[2], w[2]), 0.5f), 0.5f));
    }
    g[k] = fsb(f[0], f[1]) / two_h;
  }
  shell_psi_at<kPsiReadOnly>(a, p, x, y, z, own);
  const float s = phi_tri(a, fsb(fa(fa(v[0], own[0]), 0.5f), 0.5f), fsb(fa(fa(v[1], own[1]), 0.5f), 0.5f),
                          fsb(fa(fa(v[2], own[2]), 0.5f), 0.5f));
  const float r = fsb(s, __ldg(a.can + ((int64_t)z * a.dp.ny + y) * a.dp.nx + x)) / a.voxel;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    d[k] = fm(-a.alpha, ff(r, g[k], 0.f));
    c0[k] = own[k];
  }
  *s_out = s;
  *e_out = ff(fm(0.5f, r), r, 0.f);
}

// Update band voxel i, which does not lie on the outer shell, and write its new
// psi to entry `slot` of the output planes (slot == i for ping-pong buffers; the
// voxel's list position for in-place updates).  The voxel is re-tested with its
// warped value: one outside the band keeps its psi (it left the band in the
// previous iteration).  Returns the voxel for the next iteration's list (-1 if
// it left the band) and accumulates the statistics.
// kTrust: the trust-region step (dp.trust set), a separate instantiation so
// that the plain band pass carries no call to it.
// kLoad: how psi is read (PsiLoad); the persistent passes, which write psi
// between iterations, read it with kPsiL1.
template <bool kTrust, int kLoad = kPsiReadOnly>
__device__ __forceinline__ int update_interior_voxel(const FusedArgs &a, int i, int slot, float &maxd, double &energy,
                                                     unsigned &active, bool &diverged) {
  if (!KF_IN_BOUNDS(i, a.dp.count, KF_SITE_BAND_LIST) || !KF_IN_BOUNDS(slot, a.dp.count, KF_SITE_BAND_LIST)) return -1;
  int x, y, z;
  voxel_xyz(a.dp, i, x, y, z);
  float d[3], s, en, c0[3];
  gradient_lane<kLoad>(a, x, y, z, i, d, s, en, c0);
  return settle_band_voxel<kTrust>(a, i, slot, x, y, z, s, en, c0, d, maxd, energy, active, diverged);
}

// ---------------------------------------------------------------------------
// An interior voxel by one warp
// ---------------------------------------------------------------------------
// A lane per sample: for few voxels, where the length of one voxel's chain
// is all that counts (a step of about 350 instructions a warp, 75 a voxel on a
// group of four warps, but without the 25 samples or the components one after
// the other, and no barrier).  The roundings are gradient_lane's.
struct WarpShared {
  float nb[3][20];    // psi at the 20 neighbours (nb20_off), per component
  float4 mom[3][2];   // as GroupShared's
  float4 kil[3][2];
  float f[26];        // the cell-centre samples and the warped value
};

__constant__ signed char c_nb20[20][3] = {
    {0, 0, 0},  {1, 0, 0},  {-1, 0, 0}, {0, 1, 0},   {0, -1, 0}, {0, 0, 1},  {0, 0, -1},
    {1, 1, 0},  {1, -1, 0}, {-1, 1, 0}, {-1, -1, 0}, {1, 0, 1},  {1, 0, -1}, {-1, 0, 1},
    {-1, 0, -1}, {0, 1, 1}, {0, 1, -1}, {0, -1, 1},  {0, -1, -1}, {1, 1, 1}};

// What a lane keeps in registers through a kernel (constant memory would serve
// a warp's different offsets one after the other): its neighbour's distance
// and its sample's offset.
struct WarpLane {
  int64_t nb;
  float o0, o1, o2;
};

__device__ __forceinline__ WarpLane warp_lane(const FusedArgs &a, int lane) {
  WarpLane l{0, 0.f, 0.f, 0.f};
  if (lane < 20) l.nb = c_nb20[lane][2] * a.plane + c_nb20[lane][1] * a.row + c_nb20[lane][0];
  if (lane < 25) l.o0 = c_off25[lane][0], l.o1 = c_off25[lane][1], l.o2 = c_off25[lane][2];
  return l;
}

// group_position with an offset of the lane's own: the terms with a zero
// offset are left out by selects.
__device__ __forceinline__ void warp_position(const FusedArgs &a, const GroupCell &q, const WarpLane &l, float t[3]) {
  const float o01 = l.o0 * l.o1, o02 = l.o0 * l.o2, o12 = l.o1 * l.o2;  // 0 or +-1
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    float lin = 0.f, quad = 0.f;
    const auto add = [](float o, float m, float &sum) {
      const float v = ff(o, m, sum);
      sum = o != 0.f ? v : sum;
    };
    add(l.o0, q.m[c][1], lin);
    add(l.o1, q.m[c][2], lin);
    add(l.o2, q.m[c][3], lin);
    add(o01, q.m[c][4], quad);
    add(o02, q.m[c][5], quad);
    add(o12, q.m[c][6], quad);
    const float oc = c == 0 ? l.o0 : (c == 1 ? l.o1 : l.o2);
    t[c] = fa(fa(q.base[c], fm(a.h, oc)), ff(a.h, ff(a.h, quad, lin), q.m[c][0]));
  }
}

// The neighbours of voxel i into sh.nb.
template <int kLoad>
__device__ __forceinline__ void warp_neighbours(const FusedArgs &a, int i, int lane, const WarpLane &l, WarpShared &sh) {
  if (lane < 20) {
    const int64_t o = i + l.nb;
    sh.nb[0][lane] = load_psi<kLoad>(a.ix + o);
    sh.nb[1][lane] = load_psi<kLoad>(a.iy + o);
    sh.nb[2][lane] = load_psi<kLoad>(a.iz + o);
  }
}

// The step of voxel (x, y, z) from sh.nb (psi(i) at entry 0): lane k < 3
// returns component k of d = -alpha * g; t holds the terms of the monitored
// energy (lane 0).  can: phi_can(i).
__device__ __forceinline__ float warp_step(const FusedArgs &a, int x, int y, int z, float can, int lane,
                                           const WarpLane &l, WarpShared &sh, GroupStep &t) {
  const DevParams &dp = a.dp;
  __syncwarp();
  if (lane < 3) {
    float v[20];
#pragma unroll
    for (int n = 0; n < 20; ++n) v[n] = sh.nb[lane][n];
    component_values(a, lane, lane == 0 ? x : (lane == 1 ? y : z), lane == 0 ? dp.nx : (lane == 1 ? dp.ny : dp.nz), v,
                     sh.mom[lane][0], sh.mom[lane][1], sh.kil[lane][0], sh.kil[lane][1]);
  }
  __syncwarp();
  if (lane < 26) {
    float p[3];
    if (lane < 25) {
      GroupCell q;
      q.base[0] = fa((float)x, 0.5f);
      q.base[1] = fa((float)y, 0.5f);
      q.base[2] = fa((float)z, 0.5f);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float4 lo = sh.mom[c][0], hi = sh.mom[c][1];
        q.m[c][0] = lo.x, q.m[c][1] = lo.y, q.m[c][2] = lo.z, q.m[c][3] = lo.w;
        q.m[c][4] = hi.x, q.m[c][5] = hi.y, q.m[c][6] = hi.z;
      }
      warp_position(a, q, l, p);
    } else {
      p[0] = fsb(fa(fa((float)x, sh.nb[0][0]), 0.5f), 0.5f);
      p[1] = fsb(fa(fa((float)y, sh.nb[1][0]), 0.5f), 0.5f);
      p[2] = fsb(fa(fa((float)z, sh.nb[2][0]), 0.5f), 0.5f);
    }
    sh.f[lane] = phi_tri(a, p[0], p[1], p[2]);
  }
  __syncwarp();
  float d = 0.f;
  if (lane < 3) {
    const float *f = sh.f, h = a.h;
    // the Killing gradient (DisplacementField.cpp:326-345), component `lane`
    const float4 k0 = sh.kil[0][0], k1 = sh.kil[1][0], k2 = sh.kil[2][0];
    const float m2g = fm(-2.f, a.gamma_k);
    const float kg[3] = {ff(m2g, fa(fa(fa(0.f, k0.y), k1.y), k2.y), k0.x),
                         ff(m2g, fa(fa(fa(0.f, k0.z), k1.z), k2.z), k1.x),
                         ff(m2g, fa(fa(fa(0.f, k0.w), k1.w), k2.w), k2.x)};
    const float nrm = sqrtf(ff(kg[2], kg[2], ff(kg[1], kg[1], fm(kg[0], kg[0]))));
    const float ksc = nrm > a.clamp ? a.clamp / nrm : 1.f;
    const float kc = fm(lane == 0 ? kg[0] : (lane == 1 ? kg[1] : kg[2]), ksc) / fm(fm(4.f, h), h);
    // SDF.cpp:726-744, 867-881
    const float g[3] = {fm(fsb(f[1], f[2]), a.inv2h), fm(fsb(f[3], f[4]), a.inv2h), fm(fsb(f[5], f[6]), a.inv2h)};
    const float gc = lane == 0 ? g[0] : (lane == 1 ? g[1] : g[2]);
    float grad = 0.f;
    if (dp.use_data) {
      t.r = fsb(f[25], can) / a.voxel;
      grad = ff(t.r, gc, grad);
    }
    if (dp.use_killing) grad = ff(kc, a.omega_k, grad);
    if (dp.use_levelset) {
      const float f02 = fm(2.f, f[0]);
      const float hd = fm(fa(fsb(f[7 + 2 * lane], f02), f[8 + 2 * lane]), a.inv4hh);
      const float hxz = fm(fsb(fsb(fa(f[13], f[19]), f[20]), f[14]), a.inv4hh);
      const float hyz = fm(fsb(fsb(fa(f[15], f[21]), f[22]), f[16]), a.inv4hh);
      const float hxy = fm(fsb(fsb(fa(f[17], f[23]), f[24]), f[18]), a.inv4hh);
      t.gn = sqrtf(ff(g[2], g[2], ff(g[1], g[1], fm(g[0], g[0]))));
      // row `lane` of the Hessian
      const float r0 = lane == 0 ? hd : (lane == 1 ? hxy : hxz);
      const float r1 = lane == 0 ? hxy : (lane == 1 ? hd : hyz);
      const float r2 = lane == 0 ? hxz : (lane == 1 ? hyz : hd);
      const float sc = fm(fsb(t.gn, 1.f) / fa(t.gn, a.eps), a.omega_s);
      grad = ff(ff(r2, g[2], ff(r1, g[1], fm(r0, g[0]))), sc, grad);
    }
    d = fm(-a.alpha, grad);
  }
  return d;
}

// The Killing term of the monitored energy of a warp's voxel, into t.
__device__ __forceinline__ void warp_energy_term(const FusedArgs &a, const WarpShared &sh, GroupStep &t) {
  t.ke = killing_energy(a, sh.kil[0][1], sh.kil[1][1], sh.kil[2][1]);
}

// Adds the step t of a lane's voxel to its statistics.
__device__ __forceinline__ void group_count(const FusedArgs &a, const GroupStep &t, GroupStats &st, int lane) {
  float maxd = st.maxd[lane];
  double energy = st.energy[lane];
  unsigned active = st.active[lane];
  group_statistics(a, t, maxd, energy, active);
  st.maxd[lane] = maxd;
  st.energy[lane] = energy;
  st.active[lane] = active;
}

// Updates voxel i of the outer shell, a warp's (all lanes the same i), and adds
// its statistics to entry `at` of st and *diverged.  True where the voxel
// stays in the band.  Out of line, and its callers keep next to nothing in
// registers across it: a value that has to survive a call is kept in memory
// for good, and after a grid barrier (whose acquire empties L1) every such
// load goes to L2.  args, sc, st and diverged: in shared memory.
template <int kLoad>
__device__ __noinline__ bool warp_shell(const FusedArgs *args, ShellScratch *sc, bool odd, int i, int at,
                                        GroupStats *st, bool *diverged) {
  if (!KF_IN_BOUNDS(i, args->dp.count, KF_SITE_BAND_LIST)) return false;
  int x, y, z;
  voxel_xyz(args->dp, i, x, y, z);
  float d[3], s, en, c0[3];
  shell_gradient<kLoad>(*args, odd, x, y, z, *sc, d, &s, &en, c0);
  const bool active = in_band(s, args->band_hi, args->band_lo);
  if ((threadIdx.x & 31) == 0) {
    if (active) {
      if (!isfinite(c0[0]) || !isfinite(c0[1]) || !isfinite(c0[2])) *diverged = true;
      st->maxd[at] = fmaxf(st->maxd[at], sqrtf(ff(d[2], d[2], ff(d[1], d[1], fm(d[0], d[0])))));
      st->energy[at] += en;
      ++st->active[at];
    }
    plane_out<0>(*args, odd)[i] = active ? c0[0] + d[0] : c0[0];
    plane_out<1>(*args, odd)[i] = active ? c0[1] + d[1] : c0[1];
    plane_out<2>(*args, odd)[i] = active ? c0[2] + d[2] : c0[2];
  }
  __syncwarp();
  return active;
}

FusedArgs make_args(kf_grid live, kf_grid can, const DevParams &dp, IterStats *st) {
  FusedArgs a;
  memset(&a, 0, sizeof(a));
  a.live = live->phi;
  a.can = can->phi;
  a.st = st;
  a.dp = dp;
  a.h = (float)dp.delta_size;
  a.row = dp.nx;
  a.plane = (int64_t)dp.nx * dp.ny;
  a.inv2h = 1.f / (2.f * a.h);
  a.inv4hh = 1.f / ((4.f * a.h) * a.h);
  a.alpha = (float)dp.alpha;
  a.omega_k = (float)dp.omega_k;
  a.gamma_k = (float)dp.gamma_k;
  a.omega_s = (float)dp.omega_s;
  a.clamp = (float)dp.killing_clamp;
  a.eps = (float)dp.epsilon;
  a.voxel = (float)dp.voxel_size;
  a.oob = dp.oob_phi_f;
  a.band_hi = dp.band_hi_f;
  a.band_lo = dp.band_lo_f;
  return a;
}

}  // namespace
