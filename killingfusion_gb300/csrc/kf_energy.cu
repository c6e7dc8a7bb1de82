// Project energy of a displacement field and its exact adjoint.
//
// The reference never evaluates an energy: its solver descends the
// Euler-Lagrange gradients of KillingFusion::computeEnergyGradient
// (KillingFusion.cpp:399-476) directly.  This file evaluates a discrete
// energy with the same three terms, written so that its gradient with respect
// to psi can be taken exactly and checked against finite differences:
//
//   E = sum over active voxels i of
//         1/2 ((phi_w(i) - phi_can(i)) / v)^2                           data
//       + w_s 1/2 (|g(i)|_e / v - 1)^2                                  level set
//       + w_k (|J(i)|^2 + gamma <J(i), J(i)^T>)                         Killing
//
//   phi_w(j) = live sampled at j + psi(j) (grid units; trilinear with the
//              reference's truncating base, SDF.cpp:503-524),
//   g(i)_k   = (phi_w(i + e_k) - phi_w(i - e_k)) / 2, neighbours clamped,
//   |g|_e    = sqrt(g.g + (v eps)^2),
//   J(i)_ak  = (psi_a(i + e_k) - psi_a(i - e_k)) / 2, neighbours clamped.
//
// Kernels:
//   k_energy       one thread per voxel of a box, FP32 or FP64 arithmetic,
//                  per-block FP64 partial sums summed in a fixed order
//                  (deterministic);
//   k_warped       phi_w (and its derivative, for the adjoint) once at every
//                  voxel that is active or a clamped neighbour of an active one,
//                  where the passes after it read it up to seven times;
//   k_energy_runs  the energy of the whole grid from phi_w, one CTA per run
//                  of kRun voxels;
//   k_ls_coef +    the adjoint as a gather: each voxel j collects the
//   k_adjoint      partial derivatives of every active voxel whose energy
//                  reads psi(j) (itself and its six clamped neighbours), so
//                  no atomics and a deterministic result;
//   k_energy_fd    central differences of the energy of the 3x3x3 window
//                  around sampled voxels with one psi component moved by
//                  +-h (the only voxels whose energy depends on it).
// Compiled without contracted multiply-add so the float64 form rounds as the
// oracle's C restatement does.
#include <cuda_runtime.h>

#include <algorithm>

#include "kf_internal.h"
#include "kf_ref_math.cuh"

namespace {

constexpr int kThreads = 256;

template <typename T>
struct EnergyTerms {
  T data, ls, killing;
};

template <typename T, typename P>
struct EArgs {
  const float *live;
  const float *can;
  const P *px, *py, *pz;
  const uint8_t *active;  // NULL: every voxel
  int nx, ny, nz;
  T v, ve, oob, omega_s, omega_k, gamma_k;
  int use_data, use_ls, use_k;
  // a virtual change of one psi entry (k_energy_fd): psi_comp(pj) += pdelta
  int64_t pj;
  int pcomp;
  T pdelta;
};

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

template <typename T, typename P>
__device__ __forceinline__ int64_t lin(const EArgs<T, P> &a, int x, int y, int z) {
  return ((int64_t)z * a.ny + y) * a.nx + x;
}

template <typename T, typename P>
__device__ __forceinline__ T psi_c(const EArgs<T, P> &a, int64_t j, int c) {
  const P *p = c == 0 ? a.px : (c == 1 ? a.py : a.pz);
  T v = (T)p[j];
  if (j == a.pj && c == a.pcomp) v = v + a.pdelta;
  return v;
}

template <typename T, typename P>
__device__ __forceinline__ T live_at(const EArgs<T, P> &a, int x, int y, int z) {
  if (x < 0 || x >= a.nx || y < 0 || y >= a.ny || z < 0 || z >= a.nz) return a.oob;
  return (T)__ldg(a.live + lin(a, x, y, z));
}

// Trilinear sample of live at t (grid units) and its derivative with
// respect to t inside the cell chosen by truncation.
template <typename T, typename P>
__device__ T sample_grad(const EArgs<T, P> &a, const T t[3], T dv[3]) {
  const int b0 = (int)t[0], b1 = (int)t[1], b2 = (int)t[2];
  T v[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) v[c] = live_at(a, b0 + (c & 1), b1 + ((c >> 1) & 1), b2 + (c >> 2));
  const T fx = t[0] - (T)b0, fy = t[1] - (T)b1, fz = t[2] - (T)b2;
  const T one = T(1);
  dv[0] = (one - fz) * ((one - fy) * (v[1] - v[0]) + fy * (v[3] - v[2])) +
          fz * ((one - fy) * (v[5] - v[4]) + fy * (v[7] - v[6]));
  dv[1] = (one - fz) * ((one - fx) * (v[2] - v[0]) + fx * (v[3] - v[1])) +
          fz * ((one - fx) * (v[6] - v[4]) + fx * (v[7] - v[5]));
  using kfref::lerp1;
  const T top = lerp1(lerp1(v[4], v[5], fx), lerp1(v[6], v[7], fx), fy);
  const T bot = lerp1(lerp1(v[0], v[1], fx), lerp1(v[2], v[3], fx), fy);
  dv[2] = top - bot;
  return lerp1(bot, top, fz);
}

template <typename T, typename P>
__device__ T warped(const EArgs<T, P> &a, int x, int y, int z, T dv[3]) {
  const int64_t j = lin(a, x, y, z);
  const T t[3] = {(T)x + psi_c(a, j, 0), (T)y + psi_c(a, j, 1), (T)z + psi_c(a, j, 2)};
  return sample_grad(a, t, dv);
}

template <typename T, typename P>
__device__ bool is_active(const EArgs<T, P> &a, int64_t i) {
  return a.active == nullptr || a.active[i] != 0;
}

// J(i)_ak = (psi_a(p_k) - psi_a(m_k)) / 2 with clamped neighbours.
template <typename T, typename P>
__device__ void jacobian(const EArgs<T, P> &a, int x, int y, int z, T J[3][3]) {
  const int c[3] = {x, y, z}, n[3] = {a.nx, a.ny, a.nz};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    int p[3] = {c[0], c[1], c[2]}, m[3] = {c[0], c[1], c[2]};
    p[k] = clampi(c[k] + 1, 0, n[k] - 1);
    m[k] = clampi(c[k] - 1, 0, n[k] - 1);
    const int64_t ip = lin(a, p[0], p[1], p[2]), im = lin(a, m[0], m[1], m[2]);
#pragma unroll
    for (int q = 0; q < 3; ++q) J[q][k] = T(0.5) * (psi_c(a, ip, q) - psi_c(a, im, q));
  }
}

// Level-set gradient g(i) (clamped central differences of phi_w).
template <typename T, typename P>
__device__ void ls_gradient(const EArgs<T, P> &a, int x, int y, int z, T g[3]) {
  const int c[3] = {x, y, z}, n[3] = {a.nx, a.ny, a.nz};
  T dv[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    int p[3] = {c[0], c[1], c[2]}, m[3] = {c[0], c[1], c[2]};
    p[k] = clampi(c[k] + 1, 0, n[k] - 1);
    m[k] = clampi(c[k] - 1, 0, n[k] - 1);
    g[k] = T(0.5) * (warped(a, p[0], p[1], p[2], dv) - warped(a, m[0], m[1], m[2], dv));
  }
}

// Energy of voxel (x,y,z), assumed active; value(j) is phi_w at voxel j,
// level(g) the level-set gradient at the voxel.
template <typename T, typename P, typename Value, typename Level>
__device__ __forceinline__ EnergyTerms<T> voxel_energy(const EArgs<T, P> &a, int x, int y, int z, Value value,
                                                       Level level) {
  EnergyTerms<T> e{T(0), T(0), T(0)};
  const int64_t i = lin(a, x, y, z);
  if (a.use_data) {
    const T r = (value(i) - (T)__ldg(a.can + i)) / a.v;
    e.data = T(0.5) * r * r;
  }
  if (a.use_ls) {
    T g[3];
    level(g);
    const T nr = sqrt(g[0] * g[0] + g[1] * g[1] + g[2] * g[2] + a.ve * a.ve);
    const T r = nr / a.v - T(1);
    e.ls = a.omega_s * T(0.5) * r * r;
  }
  if (a.use_k) {
    T J[3][3];
    jacobian(a, x, y, z, J);
    T f = T(0), s = T(0);
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        f += J[q][k] * J[q][k];
        s += J[q][k] * J[k][q];
      }
    e.killing = a.omega_k * (f + a.gamma_k * s);
  }
  return e;
}

template <typename T, typename P>
__device__ EnergyTerms<T> voxel_energy(const EArgs<T, P> &a, int x, int y, int z) {
  return voxel_energy(
      a, x, y, z,
      [&](int64_t) {
        T dv[3];
        return warped(a, x, y, z, dv);
      },
      [&](T g[3]) { ls_gradient(a, x, y, z, g); });
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Sums three doubles over the block; thread 0 gets the totals.
template <int kT>
__device__ void block_sum3(double v[3]) {
  __shared__ double red[3][kT / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    double s = warp_sum(v[k]);
    if (lane == 0) red[k][wid] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 0; k < 3; ++k) {
      double s = 0.0;
      for (int w = 0; w < kT / 32; ++w) s += red[k][w];
      v[k] = s;
    }
  }
}

template <typename T, typename P>
__global__ void __launch_bounds__(kThreads) k_energy(EArgs<T, P> a, int x0, int y0, int z0, int bx, int by,
                                                     int64_t count, double *partial) {
  double acc[3] = {0.0, 0.0, 0.0};
  for (int64_t u = (int64_t)blockIdx.x * kThreads + threadIdx.x; u < count; u += (int64_t)gridDim.x * kThreads) {
    const int x = x0 + (int)(u % bx);
    const int y = y0 + (int)((u / bx) % by);
    const int z = z0 + (int)(u / ((int64_t)bx * by));
    if (!is_active(a, lin(a, x, y, z))) continue;
    EnergyTerms<T> e = voxel_energy(a, x, y, z);
    acc[0] += (double)e.data;
    acc[1] += (double)e.ls;
    acc[2] += (double)e.killing;
  }
  block_sum3<kThreads>(acc);
  if (threadIdx.x == 0)
    for (int k = 0; k < 3; ++k) partial[3 * blockIdx.x + k] = acc[k];
}

// One block; thread t sums the partials t, t + kSumThreads, ..., then a fixed tree.
constexpr int kSumThreads = 1024;
__global__ void __launch_bounds__(kSumThreads) k_sum_partials(const double *partial, int blocks, double *out) {
  double s[3] = {0.0, 0.0, 0.0};
#pragma unroll 4
  for (int b = threadIdx.x; b < blocks; b += kSumThreads)
    for (int k = 0; k < 3; ++k) s[k] += partial[3 * (int64_t)b + k];
  block_sum3<kSumThreads>(s);
  if (threadIdx.x == 0)
    for (int k = 0; k < 3; ++k) out[k] = s[k];
}

// ---------------------------------------------------------------------------
// Passes over the whole grid
// ---------------------------------------------------------------------------
// Float64 arithmetic bounds them (two operations a cycle and SM, a warp's
// instruction at the same cost with one lane active as with 32), so each CTA
// gathers the voxels of its run that have work in shared memory, in order, and
// takes them on full warps; a small run keeps the CTAs that lie in the active
// region from being the kernel's tail.  The mapping is fixed, so the sums are.
// 121 x 128 x 115 blobs: energy 106 us (31 k_warped, 59 k_energy_runs, 16 the sum)
// and gradient 182 us (43, 20, 119), against 388 and 943 us with a thread per voxel
// of the grid that samples phi_w seven times and takes whole Jacobians.
constexpr int kRun = 256, kRunThreads = 128;

// The entries u < kRun of the run from voxel v0 on (v1: where the pass ends) for
// which pred(voxel) holds, in order, into list; their number.  Every thread of the
// block calls it.
template <typename Pred>
__device__ __forceinline__ int gather_run(int64_t v0, int64_t v1, int16_t *list, Pred pred) {
  __shared__ int s_cnt[kRun / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned ball[kRun / kRunThreads];
#pragma unroll
  for (int r = 0; r < kRun / kRunThreads; ++r) {
    const int u = r * kRunThreads + (int)threadIdx.x;
    ball[r] = __ballot_sync(0xffffffffu, v0 + u < v1 && pred(v0 + u));
    if (lane == 0) s_cnt[r * (kRunThreads / 32) + warp] = __popc(ball[r]);
  }
  __syncthreads();
  int total = 0, before[kRun / kRunThreads] = {};
#pragma unroll
  for (int k = 0; k < kRun / 32; ++k) {
#pragma unroll
    for (int r = 0; r < kRun / kRunThreads; ++r)
      if (k == r * (kRunThreads / 32) + warp) before[r] = total;
    total += s_cnt[k];
  }
#pragma unroll
  for (int r = 0; r < kRun / kRunThreads; ++r)
    if (ball[r] >> lane & 1u)
      list[before[r] + __popc(ball[r] & ((1u << lane) - 1u))] = (int16_t)(r * kRunThreads + (int)threadIdx.x);
  __syncthreads();
  return total;
}

template <typename T, typename P>
__device__ __forceinline__ void coords(const EArgs<T, P> &a, int64_t i, int &x, int &y, int &z) {
  // (grids hold fewer than 2^31 voxels)
  const unsigned plane = (unsigned)a.nx * (unsigned)a.ny, u = (unsigned)i;
  z = (int)(u / plane);
  const unsigned r = u - (unsigned)z * plane;
  y = (int)(r / (unsigned)a.nx);
  x = (int)(r - (unsigned)y * (unsigned)a.nx);
}

// Whether phi_w(i) enters some active voxel's energy.
template <typename T, typename P>
__device__ __forceinline__ bool is_needed(const EArgs<T, P> &a, int64_t i) {
  if (is_active(a, i)) return true;
  int x, y, z;
  coords(a, i, x, y, z);
  const int64_t row = a.nx, plane = (int64_t)a.nx * a.ny;
  return (x > 0 && is_active(a, i - 1)) || (x + 1 < a.nx && is_active(a, i + 1)) || (y > 0 && is_active(a, i - row)) ||
         (y + 1 < a.ny && is_active(a, i + row)) || (z > 0 && is_active(a, i - plane)) ||
         (z + 1 < a.nz && is_active(a, i + plane));
}

// The passes take the voxels [v0, v1); their buffers are indexed by the voxel
// itself (part_buffer).

// phi_w at the needed voxels, and with kGrad its derivative (dv: three planes, `step`
// apart) at those in [d0, d1).  odd (or NULL): set when live holds a value that is not
// finite.
template <typename T, typename P, bool kGrad>
__global__ void __launch_bounds__(kRunThreads) k_warped(EArgs<T, P> a, int64_t v0, int64_t v1, T *__restrict__ w,
                                                        T *__restrict__ dv, int64_t step, int64_t d0, int64_t d1,
                                                        int *__restrict__ odd) {
  __shared__ int16_t s_list[kRun];
  v0 += (int64_t)blockIdx.x * kRun;
  if (kGrad && odd) {
    bool bad = false;
    for (int u = threadIdx.x; u < kRun; u += kRunThreads) bad = bad || (v0 + u < v1 && !isfinite(__ldg(a.live + v0 + u)));
    if (bad) *odd = 1;
  }
  const int n = gather_run(v0, v1, s_list, [&](int64_t i) { return is_needed(a, i); });
  for (int k = threadIdx.x; k < n; k += kRunThreads) {
    const int64_t i = v0 + s_list[k];
    int x, y, z;
    coords(a, i, x, y, z);
    T d[3];
    w[i] = warped(a, x, y, z, d);
    if (kGrad && i >= d0 && i < d1) {
      dv[i] = d[0];
      dv[step + i] = d[1];
      dv[2 * step + i] = d[2];
    }
  }
}

// *odd = 1 where live holds a value that is not finite.
__global__ void __launch_bounds__(kThreads) k_not_finite(const float *__restrict__ live, int64_t N,
                                                         int *__restrict__ odd) {
  bool bad = false;
  for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < N; i += (int64_t)gridDim.x * kThreads)
    bad = bad || !isfinite(__ldg(live + i));
  if (bad) *odd = 1;
}

// ls_gradient from phi_w.
template <typename T, typename P>
__device__ __forceinline__ void ls_gradient_w(const EArgs<T, P> &a, const T *__restrict__ w, int64_t i, int x, int y,
                                              int z, T g[3]) {
  const int64_t row = a.nx, plane = (int64_t)a.nx * a.ny;
  const int64_t up[3] = {x + 1 < a.nx ? i + 1 : i, y + 1 < a.ny ? i + row : i, z + 1 < a.nz ? i + plane : i};
  const int64_t dn[3] = {x > 0 ? i - 1 : i, y > 0 ? i - row : i, z > 0 ? i - plane : i};
#pragma unroll
  for (int k = 0; k < 3; ++k) g[k] = T(0.5) * (w[up[k]] - w[dn[k]]);
}

// The energy of a run's active voxels (voxel_energy's terms).
template <typename T, typename P>
__global__ void __launch_bounds__(kRunThreads) k_energy_runs(EArgs<T, P> a, int64_t v0, int64_t v1,
                                                             const T *__restrict__ w, double *__restrict__ partial) {
  __shared__ int16_t s_list[kRun];
  v0 += (int64_t)blockIdx.x * kRun;
  const int n = gather_run(v0, v1, s_list, [&](int64_t i) { return is_active(a, i); });
  double acc[3] = {0.0, 0.0, 0.0};
  if (n == 0) {  // (the sums of nothing would cost the float64 unit as much as others)
    if (threadIdx.x < 3) partial[3 * (int64_t)blockIdx.x + threadIdx.x] = 0.0;
    return;
  }
  for (int k = threadIdx.x; k < n; k += kRunThreads) {
    const int64_t i = v0 + s_list[k];
    int x, y, z;
    coords(a, i, x, y, z);
    const EnergyTerms<T> e = voxel_energy(
        a, x, y, z, [&](int64_t j) { return w[j]; }, [&](T g[3]) { ls_gradient_w(a, w, i, x, y, z, g); });
    acc[0] += (double)e.data;
    acc[1] += (double)e.ls;
    acc[2] += (double)e.killing;
  }
  block_sum3<kRunThreads>(acc);
  if (threadIdx.x == 0)
    for (int k = 0; k < 3; ++k) partial[3 * (int64_t)blockIdx.x + k] = acc[k];
}

// Level-set coefficient of active voxel i: d E_ls(i) / d g_k(i) / 2, i.e. the
// weight of d phi_w(p_k(i)) (+) and d phi_w(m_k(i)) (-).
template <typename P>
__global__ void __launch_bounds__(kRunThreads) k_ls_coef(EArgs<double, P> a, int64_t v0, int64_t v1,
                                                         const double *__restrict__ w, double *__restrict__ S,
                                                         int64_t step) {
  __shared__ int16_t s_list[kRun];
  v0 += (int64_t)blockIdx.x * kRun;
  const int n = gather_run(v0, v1, s_list, [&](int64_t i) { return is_active(a, i); });
  for (int k = threadIdx.x; k < n; k += kRunThreads) {
    const int64_t i = v0 + s_list[k];
    int x, y, z;
    coords(a, i, x, y, z);
    double g[3];
    ls_gradient_w(a, w, i, x, y, z, g);
    const double nr = sqrt(g[0] * g[0] + g[1] * g[1] + g[2] * g[2] + a.ve * a.ve);
    const double coef = a.omega_s * (nr / a.v - 1.0) / (a.v * nr);
#pragma unroll
    for (int q = 0; q < 3; ++q) S[q * step + i] = coef * g[q] * 0.5;
  }
}

// d E / d psi(j) by gathering from the voxels whose energy reads psi(j): the
// voxels that no active one reads have a zero gradient (as the sum of nothing;
// where phi_w there is not finite, 0 times its derivative is kept).
template <typename P>
__global__ void __launch_bounds__(kRunThreads) k_adjoint(EArgs<double, P> a, int64_t v0, int64_t v1,
                                                         const double *__restrict__ w, const double *__restrict__ dvs,
                                                         int64_t dv_step, const double *__restrict__ S, int64_t s_step,
                                                         const int *__restrict__ odd, double *__restrict__ grad) {
  __shared__ int16_t s_list[kRun];
  v0 += (int64_t)blockIdx.x * kRun;
  const bool all = *odd != 0;
  const int n = gather_run(v0, v1, s_list, [&](int64_t i) {
    if (is_needed(a, i)) return true;
    if (a.use_ls && (all || !isfinite(a.px[i]) || !isfinite(a.py[i]) || !isfinite(a.pz[i]))) return true;
    grad[3 * i] = grad[3 * i + 1] = grad[3 * i + 2] = 0.0;
    return false;
  });
  const int64_t step[3] = {1, a.nx, (int64_t)a.nx * a.ny};
  const int size[3] = {a.nx, a.ny, a.nz};
  const P *const psi[3] = {a.px, a.py, a.pz};
  for (int k0 = threadIdx.x; k0 < n; k0 += kRunThreads) {
    const int64_t j = v0 + s_list[k0];
    int c[3];
    coords(a, j, c[0], c[1], c[2]);
    double dv[3], out[3] = {0.0, 0.0, 0.0}, wj = 0.0;
    if (is_needed(a, j)) {
      wj = w[j];
#pragma unroll
      for (int q = 0; q < 3; ++q) dv[q] = dvs[q * dv_step + j];
    } else {
      wj = warped(a, c[0], c[1], c[2], dv);
    }
    if (a.use_data && is_active(a, j)) {
      const double r = (wj - (double)__ldg(a.can + j)) / a.v;
#pragma unroll
      for (int q = 0; q < 3; ++q) out[q] += r / a.v * dv[q];
    }
    double ls = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      // the voxels i with p_k(i) == j (+) and m_k(i) == j (-); at a face j
      // reads itself as p_k (top) and/or m_k (bottom)
      const int self = (c[k] == size[k] - 1 ? 1 : 0) - (c[k] == 0 ? 1 : 0);
#pragma unroll
      for (int u = 0; u < 3; ++u) {
        if (u == 0 ? c[k] < 1 : (u == 1 ? c[k] > size[k] - 2 : self == 0)) continue;
        const int64_t i = u == 0 ? j - step[k] : (u == 1 ? j + step[k] : j);
        const int sg = u == 0 ? 1 : (u == 1 ? -1 : self);
        if (!is_active(a, i)) continue;
        if (a.use_ls) ls += sg * S[(int64_t)k * s_step + i];
        if (a.use_k) {
          // column k and row k of the Jacobian at i
          double col[3], row[3];
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            const int ck = c[q] + (q == k ? (u == 0 ? -1 : (u == 1 ? 1 : 0)) : 0);  // i's coordinate along q
            const int64_t up = ck + 1 < size[q] ? i + step[q] : i, dn = ck > 0 ? i - step[q] : i;
            row[q] = 0.5 * ((double)psi[k][up] - (double)psi[k][dn]);
          }
          const int ck = c[k] + (u == 0 ? -1 : (u == 1 ? 1 : 0));
          const int64_t up = ck + 1 < size[k] ? i + step[k] : i, dn = ck > 0 ? i - step[k] : i;
#pragma unroll
          for (int q = 0; q < 3; ++q) col[q] = q == k ? row[k] : 0.5 * ((double)psi[q][up] - (double)psi[q][dn]);
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            const double dJ = a.omega_k * (2 * col[q] + 2 * a.gamma_k * row[q]);
            out[q] += sg * (0.5 * dJ);
          }
        }
      }
    }
    if (a.use_ls)
#pragma unroll
      for (int q = 0; q < 3; ++q) out[q] += ls * dv[q];
    grad[3 * j] = out[0];
    grad[3 * j + 1] = out[1];
    grad[3 * j + 2] = out[2];
  }
}

// Central difference of the energy of the 3x3x3 window around each sampled
// voxel, one warp per (voxel, component).
template <typename P>
__global__ void k_energy_fd(EArgs<double, P> a, const int32_t *voxels, int count, double h, double *out) {
  const int pair = blockIdx.x;
  if (pair >= 3 * count) return;
  const int s = pair / 3, comp = pair % 3;
  const int jx = voxels[3 * s], jy = voxels[3 * s + 1], jz = voxels[3 * s + 2];
  if (jx < 0 || jx >= a.nx || jy < 0 || jy >= a.ny || jz < 0 || jz >= a.nz) {
    if (threadIdx.x == 0) out[3 * s + comp] = 0.0;
    return;
  }
  const int l = threadIdx.x;
  double d = 0.0;
  if (l < 27) {
    const int x = jx + l % 3 - 1, y = jy + (l / 3) % 3 - 1, z = jz + l / 9 - 1;
    if (x >= 0 && x < a.nx && y >= 0 && y < a.ny && z >= 0 && z < a.nz && is_active(a, lin(a, x, y, z))) {
      EArgs<double, P> b = a;
      b.pj = lin(a, jx, jy, jz);
      b.pcomp = comp;
      b.pdelta = h;
      EnergyTerms<double> ep = voxel_energy(b, x, y, z);
      b.pdelta = -h;
      EnergyTerms<double> em = voxel_energy(b, x, y, z);
      d = ((ep.data + ep.ls) + ep.killing) - ((em.data + em.ls) + em.killing);
    }
  }
  d = warp_sum(d);
  if (l == 0) out[3 * s + comp] = d / (2.0 * h);
}

template <typename T, typename P>
EArgs<T, P> make_args(kf_grid live, kf_grid can, kf_field psi, const DevParams &dp, const uint8_t *active) {
  EArgs<T, P> a;
  a.live = live->phi;
  a.can = can->phi;
  a.px = (const P *)psi->p[0];
  a.py = (const P *)psi->p[1];
  a.pz = (const P *)psi->p[2];
  a.active = active;
  a.nx = live->n[0];
  a.ny = live->n[1];
  a.nz = live->n[2];
  a.v = (T)dp.voxel_size;
  a.ve = (T)(dp.voxel_size * dp.epsilon);
  a.oob = (T)dp.oob_phi;
  a.omega_s = (T)dp.omega_s;
  a.omega_k = (T)dp.omega_k;
  a.gamma_k = (T)dp.gamma_k;
  a.use_data = dp.use_data;
  a.use_ls = dp.use_levelset;
  a.use_k = dp.use_killing;
  a.pj = -1;
  a.pcomp = -1;
  a.pdelta = T(0);
  return a;
}

int check_common(kf_grid live, kf_grid can, kf_field psi, const kf_params *p) {
  KF_REQUIRE(live && can && psi && p, "NULL argument");
  for (int k = 0; k < 3; ++k)
    KF_REQUIRE(live->n[k] == can->n[k] && live->n[k] == psi->n[k], "grid and field sizes differ");
  return kf_check_params(p);
}

template <typename T, typename P>
int run_energy(kf_grid live, kf_grid can, kf_field psi, const DevParams &dp, const uint8_t *active,
               const int box[6], double terms[3], cudaStream_t s) {
  const int x0 = box[0], y0 = box[1], z0 = box[2];
  const int bx = box[3] - box[0], by = box[4] - box[1], bz = box[5] - box[2];
  const int64_t count = (int64_t)bx * by * bz;
  double *buf = nullptr;
  int blocks = (int)std::min<int64_t>((count + kThreads - 1) / kThreads, (int64_t)kf_num_sms() * 8);
  if (blocks < 1) blocks = 1;
  KF_CHECK_CUDA(cudaMallocAsync((void **)&buf, sizeof(double) * (3 * (size_t)blocks + 3), s));
  EArgs<T, P> a = make_args<T, P>(live, can, psi, dp, active);
  k_energy<T, P><<<blocks, kThreads, 0, s>>>(a, x0, y0, z0, bx, by, count, buf + 3);
  k_sum_partials<<<1, kSumThreads, 0, s>>>(buf + 3, blocks, buf);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(terms, buf, 3 * sizeof(double), cudaMemcpyDeviceToHost, s);
  cudaError_t f = cudaFreeAsync(buf, s);
  if (e == cudaSuccess) e = f;
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return kf_cuda_fail(e, "kf_energy");
  return KF_OK;
}

// `doubles` float64 values of workspace (bounded, kEnergyBytes): the field's, kept with
// it (an allocation from the stream's pool is mapped anew after each
// synchronisation), or, where the stream is being captured, the graph's own
// (*own: the caller frees it on the stream).
int energy_scratch(kf_field psi, size_t doubles, cudaStream_t s, double **out, bool *own) {
  const size_t bytes = doubles * sizeof(double);
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) cudaGetLastError();
  *own = cap != cudaStreamCaptureStatusNone;
  if (*own) {
    KF_CHECK_CUDA(cudaMallocAsync((void **)out, bytes, s));
    return KF_OK;
  }
  if (psi->plain_bytes < bytes) {
    cudaFree(psi->plain_scratch);
    psi->plain_scratch = nullptr;
    psi->plain_bytes = 0;
    if (cudaMalloc(&psi->plain_scratch, bytes) != cudaSuccess) {
      cudaGetLastError();
      psi->plain_scratch = nullptr;
      return kf_fail(KF_ERR_OOM, "cudaMalloc of the energy's workspace failed");
    }
    psi->plain_bytes = bytes;
  }
  *out = (double *)psi->plain_scratch;
  return KF_OK;
}

// Above this the passes over the whole grid take it in parts (ranges of voxels, runs
// kept whole, so that the sums are the same), and that is the most a field keeps: 56 B
// a voxel for the gradient and 8 B for the energy would be 7.5 and 1 GB at 512^3.
constexpr size_t kEnergyBytes = (size_t)512 << 20;

// The voxels of a part, of `total` with `each` bytes for a voxel and `halo` bytes
// beside them.
int64_t part_voxels(int64_t total, int64_t each, int64_t halo) {
  if (total * each <= (int64_t)kEnergyBytes) return total;
  const int64_t fit = ((int64_t)kEnergyBytes - halo) / each;
  return std::max<int64_t>(fit, (int64_t)1 << 20) / kRun * kRun;
}

// A buffer of the voxels from lo on, indexed by the voxel itself.
template <typename T>
T *part_buffer(T *buf, int64_t lo) {
  return reinterpret_cast<T *>(reinterpret_cast<uintptr_t>(buf) - (uintptr_t)(lo * (int64_t)sizeof(T)));
}

unsigned run_blocks(int64_t v0, int64_t v1) { return (unsigned)((v1 - v0 + kRun - 1) / kRun); }

// run_energy over the whole grid.
template <typename T, typename P>
int run_energy_runs(kf_grid live, kf_grid can, kf_field psi, const DevParams &dp, const uint8_t *active,
                    double terms[3], cudaStream_t s) {
  const int64_t N = live->count, plane = (int64_t)live->n[0] * live->n[1];
  const int64_t part = part_voxels(N, sizeof(double), 2 * plane * (int64_t)sizeof(double));
  const unsigned blocks = run_blocks(0, N);
  double *buf = nullptr;
  bool own = false;
  int rc = energy_scratch(psi, 3 + 3 * (size_t)blocks + (size_t)std::min(part + 2 * plane, N), s, &buf, &own);
  if (rc) return rc;
  EArgs<T, P> a = make_args<T, P>(live, can, psi, dp, active);
  for (int64_t v0 = 0; v0 < N; v0 += part) {
    const int64_t v1 = std::min(v0 + part, N), lo = std::max<int64_t>(v0 - plane, 0), hi = std::min(v1 + plane, N);
    T *w = part_buffer(reinterpret_cast<T *>(buf + 3 + 3 * (size_t)blocks), lo);
    k_warped<T, P, false><<<run_blocks(lo, hi), kRunThreads, 0, s>>>(a, lo, hi, w, (T *)nullptr, 0, 0, 0, nullptr);
    k_energy_runs<T, P><<<run_blocks(v0, v1), kRunThreads, 0, s>>>(a, v0, v1, w, buf + 3 + 3 * (v0 / kRun));
  }
  k_sum_partials<<<1, kSumThreads, 0, s>>>(buf + 3, (int)blocks, buf);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(terms, buf, 3 * sizeof(double), cudaMemcpyDeviceToHost, s);
  if (own) cudaFreeAsync(buf, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return kf_cuda_fail(e, "kf_energy");
  return KF_OK;
}

template <typename P>
int run_adjoint(kf_grid live, kf_grid can, kf_field psi, const DevParams &dp, const uint8_t *active,
                double *grad, cudaStream_t s) {
  const int64_t N = live->count, plane = (int64_t)live->n[0] * live->n[1];
  EArgs<double, P> a = make_args<double, P>(live, can, psi, dp, active);
  // a flag; phi_w of a part and two planes to either side, its derivative, the
  // level-set coefficients of the part and a plane to either side
  const int64_t part = part_voxels(N, 7 * sizeof(double), 10 * plane * (int64_t)sizeof(double));
  const int64_t nw = std::min(part + 4 * plane, N), ns = std::min(part + 2 * plane, N);
  double *buf = nullptr;
  bool own = false;
  int rc = energy_scratch(psi, 1 + (size_t)nw + 3 * (size_t)part + 3 * (size_t)ns, s, &buf, &own);
  if (rc) return rc;
  int *odd = reinterpret_cast<int *>(buf);
  cudaMemsetAsync(odd, 0, sizeof(int), s);
  if (part < N) k_not_finite<<<(unsigned)kf_num_sms() * 8, kThreads, 0, s>>>(live->phi, N, odd);
  for (int64_t v0 = 0; v0 < N; v0 += part) {
    const int64_t v1 = std::min(v0 + part, N);
    const int64_t w0 = std::max<int64_t>(v0 - 2 * plane, 0), w1 = std::min(v1 + 2 * plane, N);
    const int64_t s0 = std::max<int64_t>(v0 - plane, 0), s1 = std::min(v1 + plane, N);
    double *w = part_buffer(buf + 1, w0), *dv = part_buffer(buf + 1 + nw, v0),
           *S = part_buffer(buf + 1 + nw + 3 * part, s0);
    k_warped<double, P, true><<<run_blocks(w0, w1), kRunThreads, 0, s>>>(a, w0, w1, w, dv, part, v0, v1,
                                                                         part < N ? nullptr : odd);
    if (dp.use_levelset) k_ls_coef<P><<<run_blocks(s0, s1), kRunThreads, 0, s>>>(a, s0, s1, w, S, ns);
    k_adjoint<P><<<run_blocks(v0, v1), kRunThreads, 0, s>>>(a, v0, v1, w, dv, part, S, ns, odd, grad);
  }
  cudaError_t e = cudaGetLastError();
  if (own) {
    const cudaError_t f = cudaFreeAsync(buf, s);
    if (e == cudaSuccess) e = f;
  }
  if (e != cudaSuccess) return kf_cuda_fail(e, "kf_energy_adjoint");
  return KF_OK;
}

}  // namespace

extern "C" int kf_energy(kf_grid live, kf_grid can, kf_field psi, const kf_params *p, const uint8_t *active,
                         const int box[6], kf_precision arith, double terms[3], void *stream) {
  int rc = check_common(live, can, psi, p);
  if (rc) return rc;
  KF_REQUIRE(terms, "NULL terms");
  KF_REQUIRE(arith == KF_F32 || arith == KF_F64, "bad arithmetic precision");
  int b[6] = {0, 0, 0, live->n[0], live->n[1], live->n[2]};
  if (box) {
    for (int k = 0; k < 3; ++k) {
      KF_REQUIRE(box[k] >= 0 && box[k] <= box[k + 3] && box[k + 3] <= live->n[k], "box outside the grid");
      b[k] = box[k];
      b[k + 3] = box[k + 3];
    }
  }
  DevParams dp = kf_make_dev_params(live->n, p);
  cudaStream_t s = kf_stream(stream);
  if (b[3] == b[0] || b[4] == b[1] || b[5] == b[2]) {
    terms[0] = terms[1] = terms[2] = 0.0;
    return KF_OK;
  }
  if (b[0] == 0 && b[1] == 0 && b[2] == 0 && b[3] == live->n[0] && b[4] == live->n[1] && b[5] == live->n[2]) {
    if (psi->prec == KF_F32)
      return arith == KF_F64 ? run_energy_runs<double, float>(live, can, psi, dp, active, terms, s)
                             : run_energy_runs<float, float>(live, can, psi, dp, active, terms, s);
    return arith == KF_F64 ? run_energy_runs<double, double>(live, can, psi, dp, active, terms, s)
                           : run_energy_runs<float, double>(live, can, psi, dp, active, terms, s);
  }
  if (psi->prec == KF_F32)
    return arith == KF_F64 ? run_energy<double, float>(live, can, psi, dp, active, b, terms, s)
                           : run_energy<float, float>(live, can, psi, dp, active, b, terms, s);
  return arith == KF_F64 ? run_energy<double, double>(live, can, psi, dp, active, b, terms, s)
                         : run_energy<float, double>(live, can, psi, dp, active, b, terms, s);
}

extern "C" int kf_energy_adjoint(kf_grid live, kf_grid can, kf_field psi, const kf_params *p,
                                 const uint8_t *active, double *grad, void *stream) {
  int rc = check_common(live, can, psi, p);
  if (rc) return rc;
  KF_REQUIRE(grad, "NULL grad");
  DevParams dp = kf_make_dev_params(live->n, p);
  cudaStream_t s = kf_stream(stream);
  return psi->prec == KF_F32 ? run_adjoint<float>(live, can, psi, dp, active, grad, s)
                             : run_adjoint<double>(live, can, psi, dp, active, grad, s);
}

extern "C" int kf_energy_fd(kf_grid live, kf_grid can, kf_field psi, const kf_params *p,
                            const uint8_t *active, const int32_t *voxels, int count, double h, double *out,
                            void *stream) {
  int rc = check_common(live, can, psi, p);
  if (rc) return rc;
  KF_REQUIRE(count >= 0 && (count == 0 || (voxels && out)), "bad voxel list");
  KF_REQUIRE(h > 0.0, "h must be positive");
  if (count == 0) return KF_OK;
  KF_REQUIRE((int64_t)count * 3 <= 0x7fffffff, "too many voxels");
  DevParams dp = kf_make_dev_params(live->n, p);
  cudaStream_t s = kf_stream(stream);
  if (psi->prec == KF_F32) {
    k_energy_fd<float><<<3 * count, 32, 0, s>>>(make_args<double, float>(live, can, psi, dp, active), voxels,
                                                 count, h, out);
  } else {
    k_energy_fd<double><<<3 * count, 32, 0, s>>>(make_args<double, double>(live, can, psi, dp, active), voxels,
                                                  count, h, out);
  }
  KF_CHECK_LAUNCH("kf_energy_fd");
  return KF_OK;
}
