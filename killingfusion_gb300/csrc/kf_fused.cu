// Fused float32 psi update (KillingFusion::computeDisplacementField,
// KillingFusion.cpp:248-352, with the gradient of
// KillingFusion::computeEnergyGradient, :399-476) and the CUDA-graph capture
// of the fixed-iteration loop.
//
// KF_SOLVER_FUSED on small grids (persistent_test_blocks) is the band-only
// solver's persistent launch with warps that test the voxels outside the band.
// On the others an iteration is two passes over psi held in place, the first
// one split after the first iteration (k_split_runs):
//   k_fused_stream (dense)  reads psi and phi_live and applies the band test
//     of KillingFusion.cpp:272-274.  The warped value phi_live(i + psi(i)) is
//     phi_live(i) itself when psi(i) == 0 (zero interpolation weights), so only
//     voxels that have moved gather their 8 corners.  A voxel outside the
//     band keeps its psi, which therefore need not be written; the voxels
//     inside are compacted into a list.  16 bytes per voxel, 4 where psi is
//     known to be zero.
//   k_fused_band  evaluates the full gradient of every listed voxel, one
//     thread per voxel: the thread loads the 20 psi neighbours
//     of the stencil per component, takes the 25 warped-SDF samples of the
//     gradient and Hessian at compile-time offsets plus the warped value (26
//     independent trilinear gathers), and applies the reference's difference
//     stencils.  The new psi goes to a side buffer indexed by list position,
//     so every voxel still reads its neighbours' old values (Jacobi).
//   The next iteration's dense pass writes the band voxels' new psi back,
//     each run of voxels its own (k_fused_scatter after the last iteration).
// The band-only solver (KF_SOLVER_BAND) runs the dense pass once.  A voxel
// outside the band keeps psi, so its band test keeps failing and the band can
// only shrink: each band pass hands the voxels it updated to the next
// iteration, which re-tests them with the warped value it samples anyway and
// copies the ones that left the band into its output buffer (ping-pong
// buffers).  Both solvers produce the same psi.
//
// In the interior the psi samples that the reference takes at sub-voxel offsets
// are closed-form linear combinations of the 3x3x3 neighbourhood:
//   Killing (at i + h*o):  second differences 2h*(psi(+1) - 2psi(0) + psi(-1))
//     on the axes and h^2*(psi(++) - psi(+-) - psi(-+) + psi(--)) on the
//     diagonals;
//   cell centre (at i + 0.5 + h*o):  m0 + h*(o.m1) + h^2*(pairwise o o.m2)
//     from eight moments of the cell [i, i+1]^3.
// Voxels on the grid's outer shell take the reference-order path (truncating
// casts, linear-index wrap, outside values), a warp per voxel.
#include <algorithm>
#include <type_traits>

#include "kf_fused_body.cuh"
#include "kf_grid_sync.cuh"

namespace {

// Dense pass: stream the slab, list the band voxels (st[iter].list counts
// them); kPassThrough copies psi of the other voxels to the output buffer.
// In place (runs != NULL): the run first writes back the new psi that the
// previous iteration's band pass left for its own band voxels -- the entries
// runs[run] of prev_list and of the second planes (a.ox..a.oz) -- and then
// streams; it records where its band voxels land in `list`.
template <bool kPassThrough>
__global__ void __launch_bounds__(kThreads) k_fused_stream(FusedArgs a, int *__restrict__ list,
                                                          const int *__restrict__ prev_list,
                                                          int2 *__restrict__ runs, int *__restrict__ shell) {
  if (runs && a.iter > 0 && !a.st[a.iter - 1].skipped) {
    const int2 r = runs[blockIdx.x];
    float *px = const_cast<float *>(a.ix), *py = const_cast<float *>(a.iy), *pz = const_cast<float *>(a.iz);
    for (int j = threadIdx.x; j < r.y; j += kThreads) {
      const int slot = r.x + j;
      if (!KF_IN_BOUNDS(slot, a.dp.count, KF_SITE_WRITE_BACK)) continue;
      const int v = prev_list[slot];
      if (!KF_IN_BOUNDS(v, a.dp.count, KF_SITE_WRITE_BACK)) continue;
      px[v] = a.ox[slot];
      py[v] = a.oy[slot];
      pz[v] = a.oz[slot];
    }
    __syncthreads();
  }
  if (iteration_gated(a.st, a.iter, a.dp)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) a.st[a.iter].skipped = 1;
    return;
  }
  stream_flat<kPassThrough>(a, blockIdx.x, list, &a.st[a.iter].list, runs ? runs + blockIdx.x : nullptr, shell,
                            &a.st[a.iter].shell);
}

// The band-only solver's first band test when both psi buffers are zero at
// every voxel: psi(i) = 0 samples voxel i's own cell with zero weights, so
// the test reads phi_live alone (4 B a voxel, against 16 B read and 12 B
// copied by k_fused_stream<true>), and the second buffer already holds
// every voxel's psi.  The same list as k_fused_stream<true> gives.
__global__ void __launch_bounds__(kThreads) k_band_first_zero(FusedArgs a, int *__restrict__ list, int *__restrict__ shell) {
  stream_flat<false, false, true, true>(a, blockIdx.x, list, &a.st[0].list, nullptr, shell, &a.st[1].list);
}

// The same where psi may be anything: k_fused_stream<true> with the band's
// voxels of the outer shell in a list of their own.
__global__ void __launch_bounds__(kThreads) k_band_first(FusedArgs a, int *__restrict__ list, int *__restrict__ shell) {
  stream_flat<true, false, false, true>(a, blockIdx.x, list, &a.st[0].list, nullptr, shell, &a.st[1].list);
}

// Split dense schedule (grids above persistent_test_blocks' limit).  After the
// first iteration's dense pass, k_split_runs sorts the runs into those that
// listed band voxels ("hot") and the others ("cold"), each in run order.  A
// voxel outside the band keeps its psi and phi_live does not change, so the
// band tests of a cold run give the first iteration's result again: a cold
// run has no psi to write back and no band voxel, and no band pass reads
// anything a cold pass writes.  Every later iteration streams its hot runs
// (write-back, test, list) on the solve's stream, before its band pass, and
// its cold runs (test only) on a second stream, beside the band pass of the
// iteration before.  A band voxel found in a cold run is counted in
// IterStats::cold and fails the solve.
// Memory bounds the cold passes (16 B a voxel).  Where psi is zero at every
// voxel of a cold run, as the first iteration found and as it stays, a voxel
// warps to itself and its test reads phi_live alone (4 B; such a run's entry is
// ~run).  That is all of them when psi starts at zero: an iteration at 256^3
// with 14.7 k band voxels went from 38.3 to 20.0 us, where hot pass and band
// pass, one after the other, bound it; 384^3 with 615 k from 183 to 107 us.
constexpr int kSplitThreads = 1024;
constexpr int kColdRuns = 4;        // runs a cold block takes
// resident CTAs of the hot passes (48 registers).  256^3 with 14.7 k band voxels, 200
// iterations, with 5, 6 and 8: 4037, 4240 and 4231 us.
constexpr int kHotBlocksPerSM = 5;

__global__ void __launch_bounds__(kSplitThreads) k_split_runs(const int2 *__restrict__ runs, int nruns,
                                                             int *__restrict__ hot, int *__restrict__ cold,
                                                             unsigned *__restrict__ counts) {
  __shared__ int s_warp[kSplitThreads / 32];
  __shared__ int s_total;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // thread t takes the runs [r0, r1)
  const int per = (nruns + kSplitThreads - 1) / kSplitThreads;
  const int r0 = min(tid * per, nruns), r1 = min(r0 + per, nruns);
  int mine = 0;
  for (int r = r0; r < r1; ++r) mine += runs[r].y > 0;
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const int w = s_warp[lane];
    int wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += v;
    }
    s_warp[lane] = wi - w;
    if (lane == 31) s_total = wi;
  }
  __syncthreads();
  int h = s_warp[warp] + incl - mine;  // hot runs before r0
  int c = r0 - h;                       // cold runs before r0
  for (int r = r0; r < r1; ++r) {
    if (runs[r].y > 0) {
      if (KF_IN_BOUNDS(h, nruns, KF_SITE_RUNS)) hot[h] = r;
      ++h;
    } else {
      if (KF_IN_BOUNDS(c, nruns, KF_SITE_RUNS)) cold[c] = runs[r].x ? ~r : r;
      ++c;
    }
  }
  if (tid == 0) {
    counts[0] = (unsigned)s_total;
    counts[1] = (unsigned)(nruns - s_total);
  }
}

// The band test of kColdRuns cold runs (entries ~run) whose psi is zero, all their
// loads in flight together.
__device__ __forceinline__ void test_zero_runs(const FusedArgs &a, const int entry[kColdRuns], int runs_in_grid) {
  const DevParams &dp = a.dp;
  const int n4 = (int)(dp.count >> 2), tid = threadIdx.x;
  const float4 *lv = reinterpret_cast<const float4 *>(a.live);
  float4 ph[kColdRuns][kFlatGroups];
#pragma unroll
  for (int j = 0; j < kColdRuns; ++j) {
    const bool known = KF_IN_BOUNDS(~entry[j], runs_in_grid, KF_SITE_RUNS);
#pragma unroll
    for (int g = 0; g < kFlatGroups; ++g) {
      const int q = ~entry[j] * (kThreads * kFlatGroups) + g * kThreads + tid;
      // (one past the grid's end: outside any band)
      const float far = __int_as_float(0x7f800000);
      ph[j][g] = known && q < n4 ? __ldg(lv + q) : make_float4(far, far, far, far);
    }
  }
  unsigned hits = 0;
#pragma unroll
  for (int j = 0; j < kColdRuns; ++j) {
#pragma unroll
    for (int g = 0; g < kFlatGroups; ++g)
      hits += in_band(ph[j][g].x, a.band_hi, a.band_lo) + in_band(ph[j][g].y, a.band_hi, a.band_lo) +
              in_band(ph[j][g].z, a.band_hi, a.band_lo) + in_band(ph[j][g].w, a.band_hi, a.band_lo);
    // the ragged end, run 0's
    if (entry[j] == ~0 && tid < (int)(dp.count & 3)) hits += in_band(__ldg(a.live + 4 * n4 + tid), a.band_hi, a.band_lo);
  }
  if (hits) atomicAdd(&a.st[a.iter].cold, hits);
}

// Dense pass of iteration a.iter >= 1 over the listed runs (counts[0] hot
// runs, counts[1] cold runs), a run per loop step.  Hot: each run writes
// back its band voxels' new psi from the iteration before (as
// k_fused_stream), then streams and lists.  Cold (kCold): the runs are
// tested only; their band voxels, never expected, are counted in
// st[iter].cold.  A cold pass stops once the iteration before it was
// skipped (the statistics of that iteration's band pass may still be in
// flight when it runs, so it may run once after convergence, to no effect).
// A block whose kColdRuns runs all have zero psi loads them at once
// (test_zero_runs), the others take one run after the other, whose moved voxels'
// gathers want the registers (five CTAs per SM): 512^3 frames from zero 66.5 ms
// against 68.9 ms with eight CTAs of 32 registers and a run at a time (80.5 and 85.7
// ms with six and five of those); 128^3 from random psi, 60 iterations, 2.85 ms
// against 3.00 ms, from a smooth one 2.32 against 2.55 ms, 256^3 11.0 against 10.7.
template <bool kCold>
__global__ void __launch_bounds__(kThreads, 5) k_fused_stream_runs(FusedArgs a, const int *__restrict__ run_list,
                                                               const unsigned *__restrict__ counts,
                                                               int *__restrict__ list,
                                                               const int *__restrict__ prev_list,
                                                               int2 *__restrict__ runs, int *__restrict__ shell) {
  const unsigned n = counts[kCold ? 1 : 0];
  if (kCold) {
    if (a.st[a.iter - 1].skipped) return;
    const int runs_in_grid = (int)max((a.dp.count / 4 + kFlatVoxels / 4 - 1) / (kFlatVoxels / 4), (int64_t)1);
    for (unsigned k0 = blockIdx.x; k0 < n; k0 += gridDim.x * kColdRuns) {
      int entry[kColdRuns];
      bool all_zero = k0 + (kColdRuns - 1) * gridDim.x < n;
#pragma unroll
      for (int j = 0; j < kColdRuns; ++j) {
        entry[j] = k0 + j * gridDim.x < n ? run_list[k0 + j * gridDim.x] : 0;
        all_zero = all_zero && entry[j] < 0;
      }
      if (all_zero) {
        test_zero_runs(a, entry, runs_in_grid);
        continue;
      }
#pragma unroll 1
      for (unsigned k = k0; k < n && k < k0 + kColdRuns * gridDim.x; k += gridDim.x) {
        const int e = run_list[k], r = e < 0 ? ~e : e;
        if (!KF_IN_BOUNDS(r, runs_in_grid, KF_SITE_RUNS)) continue;
        if (e < 0)
          stream_flat<false, true, true>(a, r, nullptr, &a.st[a.iter].cold);
        else
          stream_flat<false, true>(a, r, nullptr, &a.st[a.iter].cold);
      }
    }
    return;
  }
  const bool write_back = !a.st[a.iter - 1].skipped;
  const bool gated = iteration_gated(a.st, a.iter, a.dp);
  if (gated && blockIdx.x == 0 && threadIdx.x == 0) a.st[a.iter].skipped = 1;
  float *px = const_cast<float *>(a.ix), *py = const_cast<float *>(a.iy), *pz = const_cast<float *>(a.iz);
  for (unsigned idx = blockIdx.x; idx < n; idx += gridDim.x) {
    const int r = run_list[idx];
    if (!KF_IN_BOUNDS(r, max((a.dp.count / 4 + kThreads * kFlatGroups - 1) / (kThreads * kFlatGroups), (int64_t)1),
                      KF_SITE_RUNS))
      continue;
    if (write_back) {
      const int2 rr = runs[r];
      for (int j = threadIdx.x; j < rr.y; j += kThreads) {
        const int slot = rr.x + j;
        if (!KF_IN_BOUNDS(slot, a.dp.count, KF_SITE_WRITE_BACK)) continue;
        const int v = prev_list[slot];
        if (!KF_IN_BOUNDS(v, a.dp.count, KF_SITE_WRITE_BACK)) continue;
        px[v] = a.ox[slot];
        py[v] = a.oy[slot];
        pz[v] = a.oz[slot];
      }
      __syncthreads();
    }
    if (!gated)
      stream_flat<false>(a, r, list, &a.st[a.iter].list, runs + r, shell, &a.st[a.iter].shell);
    __syncthreads();
  }
}

// Band pass: one thread per listed voxel, launched as one resident
// wave that loops over the list.  kCarry (band-only solver): the voxels
// updated here form the next iteration's list (list_out, counted in
// st[iter+1].list).  kInPlace: the new psi of list entry k goes to entry k
// of the output planes, for k_fused_scatter to write back.  kTrust: the
// trust-region step (dp.trust), followed by k_trust_fix.
// Voxels of the outer shell (shell: their positions in list_in) follow, a
// warp each (shell_gradient), dealt out over the whole launch: they lie next to
// one another in index order, up to 2048 of them in a run along a z face.  Bands
// cut by the face z = 0, 100 iterations at 112^3 (99 k band voxels), 160^3 (201 k)
// and 256^3 (510 k): 3.4, 4.4 and 10.0 ms; 11.2, 13.4 and 17.1 ms where the warp
// that met them took them one after the other, 5.9, 7.6 and 15.7 ms with a thread
// per shell voxel.  With the trust-region step, which takes the data term alone, they
// stay on their lanes (shell_data_gradient): its search is the longer part, and a
// warp runs it once for both kinds.  A block's two warps then take entries apart
// (voxels whose search is long lie together): bands with a face, 40 iterations at 48^3
// and 100^3: 5.4 and 12.5 ms, band-only 4.3 and 6.5 ms; 5.4, 13.0, 4.3 and 7.5 ms with
// the warps' entries together, 9.0, 17.9, 6.1 and 13.3 ms with a warp per shell voxel
// (5.7, 12.0, 4.6 and 8.3 ms with a thread each in the order of an atomic counter).
// The dense solver runs it beside the cold passes, which live on L1 and
// occupancy, so it takes no shared memory to speak of: with the groups of four
// warps of the band-only solver (13 KB a group) the 256^3 iteration took 42.7 us
// against 41.6 us, and 53 us where their carveout was half the SM's (measured while
// every cold run read psi; not since).
template <bool kCarry, bool kInPlace, bool kTrust = false>
__global__ void __launch_bounds__(kLaneThreads, kLaneBlocksPerSM) k_fused_band(FusedArgs a, const int *__restrict__ list_in,
                                                             int *__restrict__ list_out,
                                                             const int *__restrict__ shell) {
  if (iteration_gated(a.st, a.iter, a.dp)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) a.st[a.iter].skipped = 1;
    return;
  }
  __shared__ FusedArgs s_args;
  __shared__ ShellScratch s_shell[kLaneWarps];
  const int nq = (int)a.st[a.iter].list;
  const int total_threads = gridDim.x * kLaneThreads;
  const int rounds = (nq + total_threads - 1) / total_threads;
  float maxd = 0.f;
  double energy = 0.0;  // this thread's voxels, summed in float64 as the block and grid sums
  unsigned active = 0;
  bool diverged = false;
  if (kTrust) {
    if (threadIdx.x == 0) s_args = a;
    __syncthreads();
  }
  for (int r = 0; r < rounds; ++r) {
    const int k = kTrust ? ((r * kLaneWarps + (int)(threadIdx.x >> 5)) * (int)gridDim.x + (int)blockIdx.x) * 32 +
                               (int)(threadIdx.x & 31)
                         : (r * gridDim.x + blockIdx.x) * kLaneThreads + threadIdx.x;
    const int v = k < nq ? list_in[k] : -1;
    int x, y, z, next = -1;  // next: the voxel this thread hands to the next iteration
    const int slot = kInPlace ? k : v;
    if (v >= 0) {
      voxel_xyz(a.dp, v, x, y, z);
      const bool interior = interior_voxel(a.dp, x, y, z);
      if (kTrust) {
        // (one call for both kinds: a warp with both searches once)
        if (KF_IN_BOUNDS(v, a.dp.count, KF_SITE_BAND_LIST) && KF_IN_BOUNDS(slot, a.dp.count, KF_SITE_BAND_LIST)) {
          float d[3], s, en, c0[3];
          if (interior)
            gradient_lane<kPsiReadOnly>(a, x, y, z, v, d, s, en, c0);
          else
            shell_data_gradient(s_args, x, y, z, d, &s, &en, c0);
          next = settle_band_voxel<true>(a, v, slot, x, y, z, s, en, c0, d, maxd, energy, active, diverged);
        }
      } else if (interior) {
        next = update_interior_voxel<false>(a, v, slot, maxd, energy, active, diverged);
      }
    }
    if (kCarry) block_append<kLaneWarps>(next, &a.st[a.iter + 1].list, list_out, a.dp.count);
  }
  const unsigned nshell = kTrust ? 0u : a.st[a.iter].shell;
  if (blockIdx.x < nshell) {
    if (threadIdx.x == 0) s_args = a;
    __syncthreads();
    const unsigned warp = threadIdx.x >> 5;
    for (unsigned j = warp * gridDim.x + blockIdx.x; j < nshell; j += kLaneWarps * gridDim.x) {
      const int k = shell[j];
      if (!KF_IN_BOUNDS(k, a.dp.count, KF_SITE_BAND_LIST)) continue;
      const int v = list_in[k];
      if (!KF_IN_BOUNDS(v, a.dp.count, KF_SITE_BAND_LIST)) continue;
      int x, y, z;
      voxel_xyz(a.dp, v, x, y, z);
      if (interior_voxel(a.dp, x, y, z)) continue;  // (the bounds-check build's unwritten entries)
      float d[3], s, en, c0[3];
      shell_gradient<kPsiReadOnly>(s_args, false, x, y, z, s_shell[warp], d, &s, &en, c0);
      if ((threadIdx.x & 31) == 0)
        settle_band_voxel<false>(a, v, kInPlace ? k : v, x, y, z, s, en, c0, d, maxd, energy, active, diverged);
    }
    __syncwarp();
  }
  reduce_iter_stats<kLaneThreads>(a.st + a.iter, active, maxd, energy, diverged);
}

// Band-only solver, every iteration in one cooperative launch.  One band pass
// per iteration (ping-pong buffers, the updated voxels carried to the next
// iteration's list), then a grid-wide barrier (kf_grid_sync.cuh) instead of
// a kernel boundary.
// - Each group of four warps (group_update) takes an equal contiguous slice
//   of the first band list and keeps its own voxels from then on: the band
//   can only shrink, so a group's carried voxels are compacted into its own
//   slice of the other list by a ballot of its warp 0, with no atomic and no
//   block-wide step.  Neighbouring band voxels (which share psi neighbours)
//   stay in one SM's L1.
// - Voxels of the outer shell have a list of their own (k_band_first), in place.
// - psi is read through L1 and L2 (kPsiL1: the blocks write it between
//   iterations, ordered by the barrier's fences), the SDFs through the
//   read-only path.  A gated iteration (converged, diverged) ends the kernel
//   in every block alike: the barrier brings each block the same verdict
//   (grid_verdict), so no block reads the statistics after it, and a
//   group's first round of voxels comes from shared memory: the psi loads
//   of the next iteration start as soon as the barrier lets a block go.
// - Before the barrier a group only votes on the two facts that the verdict
//   carries; its statistics are summed while the block waits and committed
//   after it.
//
// What bounds it: the latency of an iteration's chain -- psi loads from L2
// (the barrier's acquire empties L1), the parts of group_update, the barrier.
// Four groups per SM: 128 voxels a round, the bench's band (14.7 k voxels, 97
// per SM) in one round.  104 registers a thread: fewer spill loop state, which
// costs a trip to L2 after every barrier, more leave the SM's L1 less
// (sequences at 256^3 with 80, 88, 96, 104, 112, 128: 5258, 5297, 5210, 4913,
// 5017, 5025 us for four frames).
// Measured at 256^3 (14.7 k band voxels, 200 iterations): 4.7 us an iteration
// against 8.9 us with one thread per voxel in 96-thread blocks, where 97 voxels
// took two rounds; 64^3 (1.7 k band voxels): 3.4 us against 6.0 us.
// Voxels of the outer shell take about 4 us each (a warp's lanes share the 45
// samples of one), so they are not in the groups' slices, which lie along a
// face where one is in the band, but dealt out to all warps.  48^3 with 87 k
// band voxels, 10 k of them on the shell, 100 iterations: 3.0 ms against 57 ms
// with the shell's voxels in their groups and 22.9 ms with a thread per voxel;
// 64^3 with all 236 k: 6.6 ms against 154 and 52 ms.
// Blocks: a band of few voxels uses fewer, one per kPersistPerBlock voxels (a
// barrier of fewer blocks is shorter, a block of fewer voxels no faster).
// Whole 64^3 frames with 24, 32, 48, 64, 96 and 128 voxels a block: 1788, 1783,
// 1807, 1849, 2003 and 2129 us for three.
constexpr int kPersistGroups = 4;
constexpr int kPersistThreads = kGroupThreads * kPersistGroups;
constexpr unsigned kPersistPerBlock = 32;
// Where the grid has blocks to spare, or has them without one more round of the
// groups, they take the shell's voxels beside the groups' round, which else
// come after it: 24^3 with 3.5 k band voxels, 100 iterations: 853 us with none,
// 670, 604 and 561 us with one per 16, 8 and 4 shell voxels.
constexpr unsigned kShellPerBlock = 4;

// The dense solver of a small grid (persistent_test_blocks) is the same
// kernel with four more warps a block, which test every voxel outside the
// band in every iteration, beside the band pass (96 registers a thread: 20
// warps of 104 do not fit the four register files).  One launch per solve and
// the voxels' tests hidden, against three launches an iteration of which each
// waits for the one before: 64^3 with 17.3 k band voxels 5.4 us an iteration
// against 15.6, 100^3 with 41.8 k 11 against 20.5.
constexpr int kTestThreads = 128;
constexpr int kTestChunks = 16;    // most groups of four voxels a test thread takes
constexpr int kTestFlight = 2;     // voxels whose corners a lane loads at a time (test_moved)
constexpr int kTestChunksMin = 4;  // the fewest worth a block

struct PersistShared {
  GroupShared group[kPersistGroups];
  int first[kPersistGroups][32];   // the next iteration's first round
  unsigned k0[kPersistGroups];     // each group's slice of the lists: [k0, k0 + per)
  unsigned n[kPersistGroups];      // voxels each group carries
  unsigned carried[kPersistGroups];
  bool fail[kPersistGroups], open[kPersistGroups];
  GroupStats stats[kPersistGroups];
  BlockStats part[kPersistGroups];
  FusedArgs args;                  // for warp_shell
  ShellScratch scratch[kPersistGroups * kGroupWarps];
  GroupStats shell;                // entry w: warp w's voxels of the grid's outer shell
  unsigned nshell;                 // the grid's list of those
  unsigned band_blocks;            // the blocks that carry band voxels in their groups
  bool shell_open[kPersistGroups * kGroupWarps];  // warp w's: some step above the threshold
  bool shell_fail;
  bool ok, any_open, any_fail;     // the barrier's verdict
  unsigned long long seen[2];      // grid_verdict's record of the two barrier words
};
struct DensePersistShared : PersistShared {
  unsigned char first[kTestChunks][kTestThreads];    // test_outside_band
};

template <bool kDense>
using PersistSharedOf = std::conditional_t<kDense, DensePersistShared, PersistShared>;

// Compacts a warp's carried voxels `next` (-1: none) into the group's slice of
// `out`, after those already there.
__device__ __forceinline__ void group_carry(int next, int lane, int *__restrict__ out, unsigned per, PersistShared &sh,
                                            int g) {
  const unsigned ball = __ballot_sync(0xffffffffu, next >= 0), carried = sh.carried[g];
  if (next >= 0) {
    const unsigned pos = carried + (unsigned)__popc(ball & ((1u << lane) - 1u));
    if (KF_IN_BOUNDS(pos, per, KF_SITE_BAND_APPEND)) out[sh.k0[g] + pos] = next;
    if (pos < 32u) sh.first[g][pos] = next;
  }
  __syncwarp();
  if (lane == 0) sh.carried[g] = carried + (unsigned)__popc(ball);
  __syncwarp();
}

// The band test of moved voxels by a whole warp, for voxels i0 .. i0 + 127: lane l's
// `moved` names those of i0 + 4 l .. + 3 to test, its result those of them that are
// in the band (warped_value).  A lane takes every 32nd voxel, so that the lanes'
// gathers touch neighbouring cells, kTestFlight of them at a time.
// What bounds it, and the dense solver where psi is non-zero everywhere: the
// instructions of the four test warps, one on each scheduler.  60 iterations at
// 64^3, 100^3 and 104^3 from a smooth psi: 0.75, 1.76 and 2.23 ms, from random
// vectors of 0.4 voxel 0.78, 1.95 and 2.36 ms; 1.07, 4.23 and 5.25 ms, 1.93, 5.07 and
// 6.80 ms where each lane gathered its own four voxels one after the other; four at
// a time 0.81, 1.77 and 2.45 ms, 0.82, 2.19 and 2.88 ms (spills).  On the split
// schedule's two passes an iteration: 1.34, 1.67 and 2.46 ms, 1.79, 2.18 and 2.50 ms.
__device__ __forceinline__ unsigned test_moved(const FusedArgs &a, const float *px, const float *py, const float *pz,
                                               int i0, unsigned moved) {
  const DevParams &dp = a.dp;
  const int lane = threadIdx.x & 31;
  unsigned hit = 0;
#pragma unroll 1
  for (int e0 = 0; e0 < 4; e0 += kTestFlight) {
    float t[kTestFlight][3], v[kTestFlight][8];
    bool test[kTestFlight], in[kTestFlight], any = false;
#pragma unroll
    for (int e = 0; e < kTestFlight; ++e) {
      test[e] = __shfl_sync(0xffffffffu, moved, 8 * (e0 + e) + (lane >> 2)) >> (lane & 3) & 1u;
      any = any || test[e];
    }
    if (!__any_sync(0xffffffffu, any)) continue;
#pragma unroll
    for (int e = 0; e < kTestFlight; ++e) {
      const int i = test[e] ? i0 + 32 * (e0 + e) + lane : 0;
      t[e][0] = __ldcg(px + i);
      t[e][1] = __ldcg(py + i);
      t[e][2] = __ldcg(pz + i);
    }
#pragma unroll
    for (int e = 0; e < kTestFlight; ++e) {
      int x, y, z;
      voxel_xyz(dp, test[e] ? i0 + 32 * (e0 + e) + lane : 0, x, y, z);
      t[e][0] = fsb(fa(fa((float)x, t[e][0]), 0.5f), 0.5f);
      t[e][1] = fsb(fa(fa((float)y, t[e][1]), 0.5f), 0.5f);
      t[e][2] = fsb(fa(fa((float)z, t[e][2]), 0.5f), 0.5f);
      const int b0 = (int)t[e][0], b1 = (int)t[e][1], b2 = (int)t[e][2];
      in[e] = (unsigned)b0 < (unsigned)(dp.nx - 1) && (unsigned)b1 < (unsigned)(dp.ny - 1) &&
              (unsigned)b2 < (unsigned)(dp.nz - 1);
      const bool load = test[e] && in[e];
      const float *p = a.live + (load ? (b2 * dp.ny + b1) * dp.nx + b0 : 0);
      const int one = load ? 1 : 0, row = load ? dp.nx : 0, plane = load ? dp.nx * dp.ny : 0;
      v[e][0] = __ldg(p);
      v[e][1] = __ldg(p + one);
      v[e][2] = __ldg(p + row);
      v[e][3] = __ldg(p + row + one);
      v[e][4] = __ldg(p + plane);
      v[e][5] = __ldg(p + plane + one);
      v[e][6] = __ldg(p + plane + row);
      v[e][7] = __ldg(p + plane + row + one);
    }
#pragma unroll
    for (int e = 0; e < kTestFlight; ++e) {
      float s = lerp3f(v[e], fsb(t[e][0], (float)(int)t[e][0]), fsb(t[e][1], (float)(int)t[e][1]),
                       fsb(t[e][2], (float)(int)t[e][2]));
      if (test[e] && !in[e]) s = phi_tri(a, t[e][0], t[e][1], t[e][2]);  // some corners lie outside the grid
      const unsigned ball = __ballot_sync(0xffffffffu, test[e] && in_band(s, a.band_hi, a.band_lo));
      if (lane >> 3 == e0 + e) hit = ball >> (4 * (lane & 7)) & 15u;
    }
  }
  return hit;
}

// A test warp's iteration.  Thread t of the grid's test threads takes the
// groups of four voxels t, t + threads, ...; `first` keeps the four bits of each,
// the voxels in the band at iteration 0.  Those are in the band list, whose
// pass tests them, until they leave it, which sets their bit of `dropped`;
// every other voxel is tested here, on the psi that the iteration reads.  A
// voxel that passes was never in the band or had left it: none may, as psi
// changes in the band alone.  Returns how many did.
__device__ __forceinline__ unsigned test_outside_band(const FusedArgs &a, int it, unsigned nblocks,
                                                      const unsigned *dropped,
                                                      unsigned char (*first)[kTestThreads]) {
  const DevParams &dp = a.dp;
  const bool odd = it & 1;
  const int n = (int)dp.count, n4 = (n + 3) >> 2;
  const int threads = (int)nblocks * kTestThreads;
  const float *px = plane_in<0>(a, odd), *py = plane_in<1>(a, odd), *pz = plane_in<2>(a, odd);
  unsigned entered = 0;
  unsigned long long todo = 0;  // bits 4c .. 4c + 3: the moved voxels of the c-th group
  const int t = (int)threadIdx.x - kPersistThreads;
  int c = 0;
#pragma unroll 2
  for (int q = (int)blockIdx.x * kTestThreads + t; q < n4 && c < kTestChunks; q += threads, ++c) {
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x, z = x, ph = x;
    unsigned valid = 15u;
    if (4 * q + 4 <= n) {
      x = __ldcg(reinterpret_cast<const float4 *>(px) + q);
      y = __ldcg(reinterpret_cast<const float4 *>(py) + q);
      z = __ldcg(reinterpret_cast<const float4 *>(pz) + q);
      ph = __ldg(reinterpret_cast<const float4 *>(a.live) + q);
    } else {  // the ragged end of the grid
      valid = (1u << (n & 3)) - 1u;
      float e[4][4] = {};
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (valid >> k & 1u) {
          e[0][k] = __ldcg(px + 4 * q + k);
          e[1][k] = __ldcg(py + 4 * q + k);
          e[2][k] = __ldcg(pz + 4 * q + k);
          e[3][k] = __ldg(a.live + 4 * q + k);
        }
      x = make_float4(e[0][0], e[0][1], e[0][2], 0.f);
      y = make_float4(e[1][0], e[1][1], e[1][2], 0.f);
      z = make_float4(e[2][0], e[2][1], e[2][2], 0.f);
      ph = make_float4(e[3][0], e[3][1], e[3][2], 0.f);
    }
    unsigned moved = 0, hit = 0;
    flat_test(a, x.x, y.x, z.x, ph.x, moved, hit, 0);
    flat_test(a, x.y, y.y, z.y, ph.y, moved, hit, 1);
    flat_test(a, x.z, y.z, z.z, ph.z, moved, hit, 2);
    flat_test(a, x.w, y.w, z.w, ph.w, moved, hit, 3);
    if (it > 0) {
      const unsigned was = first[c][t];
      const unsigned left = was ? was & __ldcg(dropped + (q >> 3)) >> (4 * (q & 7)) : 0u;
      hit &= ~was;
      moved = (moved & ~was) | left;  // (one that left is tested as the band pass did)
    }
    hit &= valid;
    todo |= (unsigned long long)(moved & valid) << (4 * c);
    if (it == 0)
      first[c][t] = (unsigned char)hit;
    else
      entered += (unsigned)__popc(hit);
  }
  // The voxels that have moved, in a pass of their own: where there are none, as
  // outside the band with psi from zero, the loop above is all there is.
  if (!__any_sync(0xffffffffu, todo != 0ull)) return entered;
  int q0 = (int)blockIdx.x * kTestThreads + (t & ~31);
  for (c = 0; q0 < n4 && c < kTestChunks; q0 += threads, ++c) {
    const unsigned moved = (unsigned)(todo >> (4 * c)) & 15u;
    if (!__any_sync(0xffffffffu, moved != 0u)) continue;
    const unsigned hit = test_moved(a, px, py, pz, 4 * q0, moved);
    if (it == 0)
      first[c][t] |= (unsigned char)hit;
    else
      entered += (unsigned)__popc(hit);
  }
  return entered;
}

// Voxel v has left the band (test_outside_band tests it from the next
// iteration on).  shell: of which list it was; a voxel of the other list (the
// bounds-check build's unwritten entries) has not left.
__device__ __forceinline__ void note_dropped(const DevParams &dp, unsigned *dropped, int v, bool shell) {
  if (!KF_IN_BOUNDS(v, dp.count, KF_SITE_BAND_LIST)) return;
  int x, y, z;
  voxel_xyz(dp, v, x, y, z);
  if (interior_voxel(dp, x, y, z) != shell) atomicOr(dropped + (v >> 5), 1u << (v & 31));
}

// The first entry of the shell's list that is warp `warp`'s of this block; every
// `nblocks` times a block's warps on is its next one.  The blocks without band
// voxels (from band_blocks on) come first.
__device__ __forceinline__ unsigned shell_entry(unsigned warp, unsigned band_blocks, unsigned nblocks) {
  const unsigned extra = nblocks - band_blocks;
  return blockIdx.x >= band_blocks ? warp * extra + blockIdx.x - band_blocks
                                   : kPersistGroups * kGroupWarps * extra + warp * band_blocks + blockIdx.x;
}

// A warp's share of the shell's list.  An entry turns -1 when its voxel leaves
// the band.
template <bool kDense>
__device__ __forceinline__ void shell_round(bool odd, unsigned nblocks, int *shell, unsigned *dropped,
                                            PersistShared &sh) {
  const unsigned warp = threadIdx.x >> 5, stride = kPersistGroups * kGroupWarps * nblocks;
  for (unsigned j = shell_entry(warp, sh.band_blocks, nblocks); j < sh.nshell; j += stride) {
    const int v = __ldcg(shell + j);
    if (v < 0) continue;
    if (!warp_shell<kPsiL1>(&sh.args, &sh.scratch[warp], odd, v, (int)warp, &sh.shell, &sh.shell_fail) &&
        (threadIdx.x & 31) == 0) {
      __stcg(shell + j, -1);
      if (kDense) note_dropped(sh.args.dp, dropped, v, true);
    }
    __syncwarp();
  }
}

// Iteration `it` of the group's voxels, the entries [k0, k0 + n) of lst0 (lst1
// in odd iterations); carried ones go to the other list.  False when the
// kernel must end (the iteration was the last, a barrier wait gave up, or the
// next iteration is gated).  The first 32 entries are read from first[] (from
// lst0 at it == 0).  What a group keeps from one round to the next is in shared
// memory, not in registers (warp_shell).  The voxels of the outer shell, which are
// in no group's slice, are dealt out to all warps of all blocks, one at a time each.
template <bool kDense>
__device__ __forceinline__ bool persistent_band_iteration(const FusedArgs &a, int it, bool last, int *lst0, int *lst1, int *shell,
                                                          unsigned nshell, unsigned per, GridSync *sync, unsigned nblocks,
                                                          unsigned long long limit_ns, unsigned *dropped,
                                                          PersistShared &sh) {
  // group g on warps 4g..4g+3, its roles rotated by g so that every scheduler
  // has each role once; part 3 is on a warp of another scheduler in each group
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = warp / kGroupWarps, w = (warp + g) % kGroupWarps, last_role = (2 * g) % kGroupWarps;
  const bool odd = it & 1;
  if (kDense && g == kPersistGroups) {  // a test warp
    DensePersistShared &d = static_cast<DensePersistShared &>(sh);
    const unsigned entered = __reduce_add_sync(0xffffffffu, test_outside_band(a, it, nblocks, dropped, d.first));
    if (lane == 0 && entered) atomicAdd(&a.st[it].cold, entered);
    __syncthreads();
    __syncthreads();
    return !last && sh.ok && !sh.any_fail && (!a.dp.early_exit || sh.any_open);
  }
  GroupStep t;
  t.active = false;
  bool diverged = false;
  int v = (unsigned)lane < sh.n[g] ? (it == 0 ? __ldcg(lst0 + sh.k0[g] + lane) : sh.first[g][lane]) : -1;
  for (unsigned k = 0; k < sh.n[g]; k += 32) {
    if (w == last_role && k > 0) group_count(a, t, sh.stats[g], lane);  // the round before
    const int next = group_update<kPsiL1>(a, odd, v, v, sh.group[g], g, w, last_role, lane, t, diverged);
    if (kDense && w == last_role && v >= 0 && next < 0) note_dropped(a.dp, dropped, v, false);
    v = k + 32 + lane < sh.n[g] ? __ldcg((odd ? lst1 : lst0) + sh.k0[g] + k + 32 + lane) : -1;
    if (w == last_role) group_carry(next, lane, odd ? lst0 : lst1, per, sh, g);
  }
  if (w == last_role) {
    const bool fail = __any_sync(0xffffffffu, diverged);
    if (lane == 0) sh.fail[g] = fail;
    __syncwarp();
    if (nshell || a.dp.early_exit) {
      group_count(a, t, sh.stats[g], lane);
      t.active = false;
    }
    // (the verdict needs the largest step only then)
    const bool open = a.dp.early_exit && __any_sync(0xffffffffu, sh.stats[g].maxd[lane] > (float)a.dp.threshold);
    if (lane == 0) sh.open[g] = open;
  }
  if (nshell) {
    shell_round<kDense>(odd, nblocks, shell, dropped, sh);
    // (noted here: sh.shell is summed and cleared while the verdict is formed)
    if (lane == 0) sh.shell_open[warp] = a.dp.early_exit && sh.shell.maxd[warp] > (float)a.dp.threshold;
  }
  __syncthreads();
  if (threadIdx.x == 96 && !last) {
    bool open = false, fail = nshell && sh.shell_fail;
    for (int k = 0; a.dp.early_exit && nshell && k < kPersistGroups * kGroupWarps; ++k) open |= sh.shell_open[k];
#pragma unroll
    for (int k = 0; k < kPersistGroups; ++k) {
      open |= sh.open[k];
      fail |= sh.fail[k];
    }
    // the gate of iteration it + 1 (iteration_gated): no block diverged, and
    // with early_exit some block moved psi by more than the threshold
    sh.ok = grid_verdict(sync, nblocks, limit_ns, it, open, fail, sh.seen[it & 1], sh.any_open, sh.any_fail);
  }
  if (w == last_role) {  // while the polling thread (of another warp) waits
    group_count(a, t, sh.stats[g], lane);
    float maxd = sh.stats[g].maxd[lane];
    double energy = sh.stats[g].energy[lane];
    unsigned active = sh.stats[g].active[lane];
    sh.stats[g].maxd[lane] = 0.f;
    sh.stats[g].energy[lane] = 0.0;
    sh.stats[g].active[lane] = 0u;
    if (nshell && g == 0) {
      energy += sh.shell.energy[lane];
      maxd = fmaxf(maxd, sh.shell.maxd[lane]);
      active += sh.shell.active[lane];
      sh.shell.energy[lane] = 0.0;
      sh.shell.maxd[lane] = 0.f;
      sh.shell.active[lane] = 0u;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      energy += __shfl_xor_sync(0xffffffffu, energy, o);
      maxd = fmaxf(maxd, __shfl_xor_sync(0xffffffffu, maxd, o));
      active += __shfl_xor_sync(0xffffffffu, active, o);
    }
    if (lane == 0) {
      sh.part[g] = BlockStats{energy, active, maxd, sh.fail[g] || (nshell && g == 0 && sh.shell_fail)};
      sh.n[g] = sh.carried[g];
      sh.carried[g] = 0u;
    }
  }
  __syncthreads();
  if (threadIdx.x == 64) {
    BlockStats b = sh.part[0];
#pragma unroll
    for (int k = 1; k < kPersistGroups; ++k) {
      b.energy += sh.part[k].energy;
      b.active += sh.part[k].active;
      b.max_delta = fmaxf(b.max_delta, sh.part[k].max_delta);
      b.diverged |= sh.part[k].diverged;
    }
    commit_iter_stats(a.st + it, b);
  }
  if (last) return false;
  if (!sh.ok) {
    if (threadIdx.x == 0) a.st[0].timeout = 1;
    return false;
  }
  if (sh.any_fail || (a.dp.early_exit && !sh.any_open)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) a.st[it + 1].skipped = 1;
    return false;
  }
  return true;
}

// a: psi in the primary planes, out to the second (iteration 0, then every
// other one; the others read the second planes and write the primary ones).
// The band list of the dense first pass is lst0[0, st[0].list).  touched
// (or NULL): a copy of that list and its length, the only voxels whose psi
// the solve can change (the iterations overwrite lst0).  per_block: the
// fewest band voxels worth a block; a smaller band leaves the last blocks
// without any, and they end at once.  kDense (kTestThreads more threads): the
// dense solver; least_blocks: the blocks that its test warps need, dropped: a
// zeroed bit per voxel (test_outside_band).
template <bool kDense>
__global__ void __maxnreg__(kDense ? 96 : 104)
    k_band_persistent(FusedArgs a, int *lst0, int *lst1, int *shell, int iterations, GridSync *sync,
                      unsigned long long limit_ns, int *touched, unsigned *touched_n, unsigned per_block,
                      unsigned least_blocks, unsigned *dropped) {
  extern __shared__ __align__(16) unsigned char smem[];
  PersistShared &sh = *reinterpret_cast<PersistSharedOf<kDense> *>(smem);
  const unsigned nq = __ldcg(&a.st[0].list), nshell = __ldcg(&a.st[1].list);
  // blocks for the groups' voxels and, where that takes the groups no more
  // rounds, blocks for the shell's beside them
  constexpr unsigned kWarps = kPersistGroups * kGroupWarps, kRound = 32 * kPersistGroups;
  const unsigned most = gridDim.x, wanted = min(most, (nq + per_block - 1) / per_block);
  const unsigned rounds = (nq + most * kRound - 1) / (most * kRound);
  const unsigned least = rounds ? (nq + rounds * kRound - 1) / (rounds * kRound) : 0u;
  const unsigned shell_blocks = min(most, (nshell + kShellPerBlock - 1) / kShellPerBlock);
  const unsigned band_blocks = max(min(wanted, max(least, most - shell_blocks)), 1u);
  const unsigned nblocks = min(most, max(band_blocks + shell_blocks, least_blocks));
  if (blockIdx.x >= nblocks) return;
  const unsigned groups = band_blocks * kPersistGroups;
  const unsigned per = (nq + groups - 1) / groups;  // a group's slice
  if (threadIdx.x == 0) {
    sh.args = a;
    sh.seen[0] = sh.seen[1] = 0;
    sh.nshell = nshell;
    sh.band_blocks = band_blocks;
    sh.shell_fail = false;
  }
  if (threadIdx.x < kPersistGroups) {
    const unsigned k0 = min((blockIdx.x * kPersistGroups + threadIdx.x) * per, nq);
    sh.k0[threadIdx.x] = k0;
    sh.n[threadIdx.x] = min(k0 + per, nq) - k0;
    sh.carried[threadIdx.x] = 0u;
  }
  if (threadIdx.x < 32 * kPersistGroups) {
    GroupStats &st = sh.stats[threadIdx.x / 32];
    st.energy[threadIdx.x % 32] = 0.0;
    st.maxd[threadIdx.x % 32] = 0.f;
    st.active[threadIdx.x % 32] = 0u;
  } else if (threadIdx.x < 32 * kPersistGroups + 32) {
    sh.shell.energy[threadIdx.x % 32] = 0.0;
    sh.shell.maxd[threadIdx.x % 32] = 0.f;
    sh.shell.active[threadIdx.x % 32] = 0u;
  }
  __syncthreads();
  if (touched) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *touched_n = nq + nshell;
    for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < nq; k += nblocks * blockDim.x)
      touched[k] = __ldcg(lst0 + k);
    // (a warp's own: iteration 0 already overwrites entries of this list)
    const unsigned warp = threadIdx.x >> 5, stride = kWarps * nblocks;
    if (warp < kWarps) {
      for (unsigned j = shell_entry(warp, band_blocks, nblocks) + (threadIdx.x & 31) * stride; j < nshell;
           j += 32 * stride)
        touched[nq + j] = __ldcg(shell + j);
      __syncwarp();
    }
  }
  for (int it = 0; it < iterations; ++it)
    if (!persistent_band_iteration<kDense>(a, it, it + 1 == iterations, lst0, lst1, shell, nshell, per, sync, nblocks, limit_ns,
                                           dropped, sh)) {
      if (kDense && blockIdx.x == 0 && threadIdx.x == 0) a.st[0].executed = it + 1;
      return;
    }
}

// Dense solver: psi stays in the primary planes.  After an odd number of
// iterations the result is in the second ones, which differ at the voxels of
// the first band list alone.
__global__ void __launch_bounds__(kThreads) k_dense_settle(FusedArgs a, const int *__restrict__ touched,
                                                          const unsigned *touched_n) {
  if (!(a.st[0].executed & 1)) return;
  float *px = const_cast<float *>(a.ix), *py = const_cast<float *>(a.iy), *pz = const_cast<float *>(a.iz);
  const unsigned n = *touched_n;
  for (unsigned k = blockIdx.x * kThreads + threadIdx.x; k < n; k += gridDim.x * kThreads) {
    const int v = touched[k];
    if (!KF_IN_BOUNDS(v, a.dp.count, KF_SITE_WRITE_BACK)) continue;
    px[v] = a.ox[v];
    py[v] = a.oy[v];
    pz[v] = a.oz[v];
  }
}

// In-place update after the last iteration: psi(list[k]) = entry k of the
// band pass's output planes (the dense passes write back the others).
__global__ void __launch_bounds__(kThreads) k_fused_scatter(FusedArgs a, const int *__restrict__ list,
                                                           float *__restrict__ px, float *__restrict__ py,
                                                           float *__restrict__ pz) {
  if (iteration_gated(a.st, a.iter, a.dp)) return;
  const int nq = (int)a.st[a.iter].list;
  for (int k = blockIdx.x * kThreads + threadIdx.x; k < nq; k += gridDim.x * kThreads) {
    const int v = list[k];
    if (!KF_IN_BOUNDS(k, a.dp.count, KF_SITE_WRITE_BACK) || !KF_IN_BOUNDS(v, a.dp.count, KF_SITE_WRITE_BACK))
      continue;
    px[v] = a.ox[k];
    py[v] = a.oy[k];
    pz[v] = a.oz[k];
  }
}

// Trust-region step, after the band pass of iteration a.iter: the reference
// breaks out of a row's x loop at the first voxel whose step failed
// (KillingFusion.cpp:312-313), so listed voxels at or after that x (a.rows)
// get their old psi back in the output planes (entry k in place, voxel v
// ping-pong).  Also clears next_rows, the table of the next band pass.
__global__ void __launch_bounds__(kThreads) k_trust_fix(FusedArgs a, const int *__restrict__ list, bool in_place,
                                                       int *__restrict__ next_rows) {
  const int nrows = a.dp.ny * a.dp.nz;
  const int stride = gridDim.x * kThreads;
  const int t0 = blockIdx.x * kThreads + threadIdx.x;
  for (int r = t0; r < nrows; r += stride) next_rows[r] = kRowClear;
  if (a.st[a.iter].skipped) return;
  const int nq = (int)a.st[a.iter].list;
  for (int k = t0; k < nq; k += stride) {
    const int v = list[k];
    if (!KF_IN_BOUNDS(v, a.dp.count, KF_SITE_BAND_LIST)) continue;
    int x, y, z;
    voxel_xyz(a.dp, v, x, y, z);
    if (x >= a.rows[z * a.dp.ny + y]) {
      const int slot = in_place ? k : v;
      a.ox[slot] = a.ix[v];
      a.oy[slot] = a.iy[v];
      a.oz[slot] = a.iz[v];
    }
  }
}

// KillingFusion::computeDisplacementField, default per-voxel schedule
// (KillingFusion.cpp:353-396), in eight colours (x&1) | (y&1)<<1 | (z&1)<<2.
// The listed voxels of a colour (inside the symmetric band) step their psi in
// place -- a.ix and a.ox are the same planes -- until the step or the
// gradient is at most the threshold or max_iters steps were taken.  A
// voxel's gradient reads psi only in its 3x3x3 neighbourhood, where no other
// voxel has its colour, so its neighbours stay fixed while it iterates, as
// in the reference's sequential loop, and the result does not depend on
// scheduling.

// The dense pass's list sorted by colour: the voxels inside from the front of the
// colour's part of `out` (counts[c]), those on the grid's outer shell from its back
// (counts[8 + c]).  The part of a colour, [start[c], start[c + 1]), has room for
// all the grid's voxels of it.
struct ColourParts {
  unsigned start[9];
};
constexpr int kColourCounts = 16;

static ColourParts colour_parts(const DevParams &dp) {
  ColourParts p;
  p.start[0] = 0;
  for (int c = 0; c < 8; ++c) {
    const unsigned x = c & 1 ? dp.nx / 2 : (dp.nx + 1) / 2, y = c & 2 ? dp.ny / 2 : (dp.ny + 1) / 2,
                   z = c & 4 ? dp.nz / 2 : (dp.nz + 1) / 2;
    p.start[c + 1] = p.start[c] + x * y * z;
  }
  return p;
}

__global__ void __launch_bounds__(kThreads) k_colour_lists(FusedArgs a, const int *__restrict__ list,
                                                          unsigned *__restrict__ counts, ColourParts parts,
                                                          int *__restrict__ out) {
  const unsigned nq = a.st[0].list;
  const unsigned lane = threadIdx.x & 31;
  // whole warps loop together
  for (unsigned k = blockIdx.x * kThreads + threadIdx.x; k - lane < nq; k += gridDim.x * kThreads) {
    int v = k < nq ? list[k] : -1;
    if (v >= 0 && !KF_IN_BOUNDS(v, a.dp.count, KF_SITE_BAND_LIST)) v = -1;
    int x = 0, y = 0, z = 0;
    if (v >= 0) voxel_xyz(a.dp, v, x, y, z);
    const int colour = (x & 1) | (y & 1) << 1 | (z & 1) << 2;
    const bool inside = interior_voxel(a.dp, x, y, z);
    const int which = v < 0 ? kColourCounts : colour + (inside ? 0 : 8);
    const unsigned same = __match_any_sync(0xffffffffu, which);
    if (v < 0) continue;
    const int leader = __ffs(same) - 1;
    unsigned at = 0;
    if ((int)lane == leader) at = atomicAdd(counts + which, (unsigned)__popc(same));
    at = __shfl_sync(same, at, leader) + (unsigned)__popc(same & ((1u << lane) - 1u));
    const unsigned pos = inside ? parts.start[colour] + at : parts.start[colour + 1] - 1u - at;
    if (KF_IN_BOUNDS(pos, a.dp.count, KF_SITE_BAND_APPEND)) out[pos] = v;
  }
}

// Whether the step d of a voxel, its iter-th before it, was its last
// (KillingFusion.cpp:374-394); n: its new psi, which *diverged reports when it
// is not finite.
__device__ __forceinline__ bool pervoxel_done(const FusedArgs &a, float dn, const float n[3], int max_iters, int &iter,
                                              bool &diverged) {
  const float thr = (float)a.dp.threshold;
  if (dn <= thr) return true;
  if (!isfinite(n[0]) || !isfinite(n[1]) || !isfinite(n[2])) {
    diverged = true;
    return true;
  }
  ++iter;
  // |gradient| = |step| / alpha
  return !(dn / a.alpha > thr) || iter >= max_iters;
}

// The voxels of one colour.  Few of them take a warp each (warp_step): a voxel's
// neighbours are loaded once and its psi stays on chip until the last step, so a
// step costs no trip to memory beyond the samples' corners (L1).  Many take a
// thread each (gradient_lane, the same roundings).  Voxels of the outer shell take a
// warp each (shell_gradient).
// Statistics: record 0 voxels (list, from the dense pass), last step, last
// monitored energy, divergence; record 1 voxels that hit the cap (active) and
// the most steps of one voxel (list).
// What bounds it: the chain of a step times the steps of the slowest voxel, and with
// a warp each, above a voxel or so per resident warp, the instructions (350 a warp
// and step against 62 a voxel as lanes of full warps).  60 steps from zero with 5.3 k,
// 17 k, 27 k, 42 k and 107 k band voxels: a warp each 640, 818, 1345, 1954 and 4259 us, a
// thread each 1110, 1157, 1158, 1166 and 1210 us.  Samples that do not share a cell
// slow the threads alone (10 steps from a smooth psi, 20 k voxels: 299 us a warp each,
// 640 us a thread each), so the line lies a little above one voxel per resident
// warp.  One or two steps do not earn back the warps' start: 2 steps with 5.3 k, 10 k,
// 14 k and 17 k voxels take 97, 111, 129 and 146 us a warp each, 111, 107, 104 and 109
// us a thread each.
// (A thread per voxel of the unsorted list, most lanes of another colour: 60 steps
// 1170, 1184, 1441, 1607 and 2982 us.)
constexpr int kPervoxelWarps = 4;
constexpr int kPervoxelBlocksPerSM = 4;
constexpr int kPervoxelFewSteps = 2;

__global__ void __launch_bounds__(32 * kPervoxelWarps, kPervoxelBlocksPerSM)
    k_pervoxel(FusedArgs a, const int *__restrict__ list, const unsigned *__restrict__ counts, unsigned first,
               unsigned end, int max_iters, int colour) {
  __shared__ WarpShared s_warp[kPervoxelWarps];
  __shared__ ShellScratch s_shell[kPervoxelWarps];
  __shared__ FusedArgs s_args;
  const DevParams &dp = a.dp;
  // (more than the colour's part holds: the bounds-check build's unwritten entries,
  // which may name one voxel many times)
  const unsigned ni = min(counts[colour], end - first), ns = min(counts[8 + colour], end - first);
  if (blockIdx.x * kPervoxelWarps >= max(ni, ns)) return;
  if (threadIdx.x == 0) s_args = a;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned warps = gridDim.x * kPervoxelWarps, w0 = blockIdx.x * kPervoxelWarps + warp;
  // the same on every lane but where noted
  float maxd = 0.f;
  double energy = 0.0;  // lane 0: float64 from the per-voxel terms up
  unsigned capped = 0, most = 0;
  bool diverged = false;
  for (unsigned k = w0; k < ns; k += warps) {
    const int i = list[end - 1u - k];
    if (!KF_IN_BOUNDS(i, dp.count, KF_SITE_BAND_LIST)) continue;
    int x, y, z, iter = 0;
    unsigned steps = 0;
    float dn = 0.f, en = 0.f;
    voxel_xyz(dp, i, x, y, z);
    while (true) {
      float d[3], s, c0[3];
      shell_gradient<kPsiL2>(s_args, false, x, y, z, s_shell[warp], d, &s, &en, c0);
      const float n[3] = {c0[0] + d[0], c0[1] + d[1], c0[2] + d[2]};
      __syncwarp();  // every lane has read psi
      if (lane == 0) {
        a.ox[i] = n[0];
        a.oy[i] = n[1];
        a.oz[i] = n[2];
      }
      __syncwarp();
      ++steps;
      dn = sqrtf(ff(d[2], d[2], ff(d[1], d[1], fm(d[0], d[0]))));
      if (pervoxel_done(a, dn, n, max_iters, iter, diverged)) break;
    }
    if (lane == 0) energy += en;
    maxd = fmaxf(maxd, dn);
    capped += iter >= max_iters;
    most = max(most, steps);
  }
  __syncwarp();
  if (ni <= (max_iters > kPervoxelFewSteps ? warps + warps / 8 : warps / 2)) {
    WarpShared &sh = s_warp[warp];
    const WarpLane wl = warp_lane(a, lane);
    for (unsigned k = w0; k < ni; k += warps) {
      const int i = list[first + k];
      if (!KF_IN_BOUNDS(i, dp.count, KF_SITE_BAND_LIST)) continue;
      int x, y, z, iter = 0;
      unsigned steps = 0;
      float dn = 0.f;
      voxel_xyz(dp, i, x, y, z);
      if (!interior_voxel(dp, x, y, z)) continue;  // (the bounds-check build's unwritten entries)
      const float can = __ldg(a.can + i);
      __syncwarp();
      warp_neighbours<kPsiL2>(a, i, lane, wl, sh);
      GroupStep t;
      float n[3];
      while (true) {
        const float d = warp_step(a, x, y, z, can, lane, wl, sh, t);
        if (lane < 3) sh.nb[lane][0] = sh.nb[lane][0] + d;
#pragma unroll
        for (int c = 0; c < 3; ++c) t.d[c] = __shfl_sync(0xffffffffu, d, c);
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 3; ++c) n[c] = sh.nb[c][0];
        ++steps;
        dn = sqrtf(ff(t.d[2], t.d[2], ff(t.d[1], t.d[1], fm(t.d[0], t.d[0]))));
        if (pervoxel_done(a, dn, n, max_iters, iter, diverged)) break;
      }
      if (lane == 0) {
        // DisplacementField::update (DisplacementField.cpp:65-71): the other
        // colours read psi in later launches only
        a.ox[i] = n[0];
        a.oy[i] = n[1];
        a.oz[i] = n[2];
        t.active = true;
        warp_energy_term(a, sh, t);
        float m = 0.f;
        double e = 0.0;
        unsigned one = 0;
        group_statistics(a, t, m, e, one);
        energy += e;
      }
      maxd = fmaxf(maxd, dn);
      capped += iter >= max_iters;
      most = max(most, steps);
    }
  } else {
    float lane_maxd = 0.f;
    double lane_energy = 0.0;
    unsigned lane_capped = 0, lane_most = 0;
    bool lane_diverged = false;
    for (unsigned k = 32 * w0 + lane; k < ni; k += 32 * warps) {
      const int i = list[first + k];
      if (!KF_IN_BOUNDS(i, dp.count, KF_SITE_BAND_LIST)) continue;
      int x, y, z, iter = 0;
      unsigned steps = 0;
      float dn, en;
      voxel_xyz(dp, i, x, y, z);
      if (!interior_voxel(dp, x, y, z)) continue;
      while (true) {
        float d[3], s, c0[3];
        gradient_lane<kPsiL2>(a, x, y, z, i, d, s, en, c0);
        const float n[3] = {c0[0] + d[0], c0[1] + d[1], c0[2] + d[2]};
        a.ox[i] = n[0];
        a.oy[i] = n[1];
        a.oz[i] = n[2];
        ++steps;
        dn = sqrtf(ff(d[2], d[2], ff(d[1], d[1], fm(d[0], d[0]))));
        if (pervoxel_done(a, dn, n, max_iters, iter, lane_diverged)) break;
      }
      lane_energy += en;
      lane_maxd = fmaxf(lane_maxd, dn);
      lane_capped += iter >= max_iters;
      lane_most = max(lane_most, steps);
    }
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) lane_energy += __shfl_xor_sync(0xffffffffu, lane_energy, o);
    energy += lane_energy;
    maxd = fmaxf(maxd, __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(lane_maxd))));
    capped += __reduce_add_sync(0xffffffffu, lane_capped);
    most = max(most, __reduce_max_sync(0xffffffffu, lane_most));
    diverged = __any_sync(0xffffffffu, lane_diverged) || diverged;
  }
  if (lane == 0) {
    commit_iter_stats(a.st, BlockStats{energy, 0u, maxd, diverged});
    if (capped) atomicAdd(&a.st[1].active, capped);
    if (most) atomicMax(&a.st[1].list, most);
  }
}

}  // namespace

// A captured iteration loop, valid for one set of buffers and parameters.
struct FusedGraph {
  cudaGraphExec_t exec = nullptr;
  cudaStream_t capture = nullptr;
  cudaStream_t cold = nullptr;                     // cold passes of the split schedule
  cudaEvent_t fork = nullptr, join = nullptr;
  const void *key_ptr[12] = {};
  int iterations = 0;
  bool band_only = false;
  DevParams dp;
};

void kf_fused_graph_destroy(FusedGraph *g) {
  if (!g) return;
  if (g->exec) cudaGraphExecDestroy(g->exec);
  if (g->capture) cudaStreamDestroy(g->capture);
  if (g->cold) cudaStreamDestroy(g->cold);
  if (g->fork) cudaEventDestroy(g->fork);
  if (g->join) cudaEventDestroy(g->join);
  delete g;
}

static int64_t num_runs(const DevParams &dp) {
  return std::max<int64_t>((dp.count / 4 + kThreads * kFlatGroups - 1) / (kThreads * kFlatGroups), 1);
}

static bool split_schedule(const DevParams &dp, bool band_only) {
  return !band_only && !dp.trust;
}

// A launch whose graph node carries a priority: the hot chain of the split
// schedule (hot pass, band pass) goes ahead of the cold passes' CTAs.
template <typename... KArgs, typename... Args>
static void launch_prio(void (*kernel)(KArgs...), unsigned grid, unsigned block, cudaStream_t s, int prio,
                        Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributePriority;
  attr[0].val.priority = prio;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Whether the grid is small enough for the dense solver in one persistent launch
// (persistent_test_blocks).
static bool persistent_size(const DevParams &dp) {
  return (dp.count + 3) / 4 <= (int64_t)kf_num_sms() * kTestThreads * kTestChunks;
}

// The split schedule's lists after the run table: hot runs, cold runs (one
// int per run each) and their two counts.  On small grids the same memory
// also holds the persistent kernel's bit per voxel.
static size_t runs_table_bytes(const DevParams &dp) {
  const size_t nruns = (size_t)num_runs(dp);
  const size_t table = nruns * sizeof(int2) + (2 * nruns + 4) * sizeof(int);
  const size_t bits = persistent_size(dp) ? (size_t)((dp.count + 31) / 32) * sizeof(unsigned) : 0;
  return std::max(table, bits);
}

// The dense fused iterations on the split schedule (see k_split_runs).
static void launch_split_iterations(FusedArgs a, kf_field psi, const DevParams &dp, int iterations,
                                    int *lists, int2 *runs, cudaStream_t s, cudaStream_t cold_s,
                                    cudaEvent_t fork, cudaEvent_t join) {
  int lo = 0, hi = 0;
  cudaDeviceGetStreamPriorityRange(&lo, &hi);
  // the cold passes rank between the hot chain and default-priority work
  // that a caller runs beside the solve (the next frame's integration,
  // meshes), where the device has more than two priority levels
  const int mid = hi < lo - 1 ? (lo + hi) / 2 : lo;
  const unsigned band_blocks = (unsigned)kf_num_sms() * kLaneBlocksPerSM;
  const int64_t nruns = num_runs(dp);
  const unsigned grid = (unsigned)nruns;
  const unsigned hot_grid = (unsigned)std::min<int64_t>(nruns, (int64_t)kf_num_sms() * kHotBlocksPerSM);
  const unsigned cold_grid = (unsigned)((nruns + kColdRuns - 1) / kColdRuns);
  int *hot = reinterpret_cast<int *>(runs + nruns), *cold = hot + nruns;
  unsigned *counts = reinterpret_cast<unsigned *>(cold + nruns);
  int *lst[2] = {lists, lists + dp.count}, *shell = lists + 2 * dp.count;
  a.ix = (const float *)psi->p[0];
  a.iy = (const float *)psi->p[1];
  a.iz = (const float *)psi->p[2];
  a.ox = (float *)psi->q[0];
  a.oy = (float *)psi->q[1];
  a.oz = (float *)psi->q[2];
  for (int it = 0; it < iterations; ++it) {
    a.iter = it;
    if (it == 0) {
      launch_prio(k_fused_stream<false>, grid, kThreads, s, hi, a, lst[0], lst[1], runs, shell);
      if (iterations > 1)
        launch_prio(k_split_runs, 1, kSplitThreads, s, hi, (const int2 *)runs, (int)nruns, hot, cold, counts);
    } else {
      // cold runs beside the band pass of the iteration before
      cudaStreamWaitEvent(cold_s, fork, 0);
      launch_prio(k_fused_stream_runs<true>, cold_grid, kThreads, cold_s, mid, a, (const int *)cold,
                  (const unsigned *)counts, (int *)nullptr, (const int *)nullptr, (int2 *)nullptr,
                  (int *)nullptr);
      launch_prio(k_fused_stream_runs<false>, hot_grid, kThreads, s, hi, a, (const int *)hot,
                  (const unsigned *)counts, lst[it & 1], (const int *)lst[(it + 1) & 1], runs, shell);
    }
    if (it + 1 < iterations) cudaEventRecord(fork, s);
    launch_prio(k_fused_band<false, true>, band_blocks, kLaneThreads, s, hi, a, (const int *)lst[it & 1],
                (int *)nullptr, (const int *)shell);
    if (it == iterations - 1)
      launch_prio(k_fused_scatter, band_blocks, kThreads, s, hi, a, (const int *)lst[it & 1],
                  (float *)psi->p[0], (float *)psi->p[1], (float *)psi->p[2]);
  }
  if (iterations > 1) {
    cudaEventRecord(join, cold_s);
    cudaStreamWaitEvent(s, join, 0);
  }
}

static void launch_iterations(kf_grid live, kf_grid can, kf_field psi, const DevParams &dp,
                              int iterations, IterStats *st, int *lists, int2 *runs, int *rows,
                              bool band_only, cudaStream_t s) {
  const unsigned band_blocks = (unsigned)kf_num_sms() * kLaneBlocksPerSM;  // one resident wave
  const unsigned grid = (unsigned)std::max<int64_t>((dp.count / 4 + kThreads * kFlatGroups - 1) /
                                                        (kThreads * kFlatGroups), 1);
  const unsigned block = kThreads;
  FusedArgs a = make_args(live, can, dp, st);
  void *buf[2][3] = {{psi->p[0], psi->p[1], psi->p[2]}, {psi->q[0], psi->q[1], psi->q[2]}};
  int *lst[2] = {lists, lists + dp.count};
  const int nrows = dp.ny * dp.nz;
  if (dp.trust) cudaMemsetAsync(rows, 0x7f, (size_t)nrows * sizeof(int), s);
  for (int it = 0; it < iterations; ++it) {
    // dense: psi stays in the primary planes, the second planes hold the
    // band voxels' new values by list position; band-only: ping-pong
    void **in = band_only ? buf[it & 1] : buf[0], **out = band_only ? buf[(it + 1) & 1] : buf[1];
    a.ix = (const float *)in[0];
    a.iy = (const float *)in[1];
    a.iz = (const float *)in[2];
    a.ox = (float *)out[0];
    a.oy = (float *)out[1];
    a.oz = (float *)out[2];
    a.iter = it;
    a.rows = dp.trust ? rows + (it & 1) * nrows : nullptr;
    int *next_rows = dp.trust ? rows + ((it + 1) & 1) * nrows : nullptr;
    if (!band_only) {
      // lists alternate so that a run can still read the previous iteration's
      k_fused_stream<false><<<grid, block, 0, s>>>(a, lst[it & 1], lst[(it + 1) & 1], runs, nullptr);
      k_fused_band<false, true, true><<<band_blocks, kLaneThreads, 0, s>>>(a, lst[it & 1], nullptr, nullptr);
      k_trust_fix<<<band_blocks, kThreads, 0, s>>>(a, lst[it & 1], true, next_rows);
      if (it == iterations - 1)
        k_fused_scatter<<<band_blocks, kThreads, 0, s>>>(a, lst[it & 1], (float *)in[0], (float *)in[1],
                                                        (float *)in[2]);
    } else {
      if (it == 0) k_fused_stream<true><<<grid, block, 0, s>>>(a, lst[0], nullptr, nullptr, nullptr);
      // (with the trust-region step; without it the solver is k_band_persistent)
      k_fused_band<true, false, true><<<band_blocks, kLaneThreads, 0, s>>>(a, lst[it & 1], lst[(it + 1) & 1],
                                                                         nullptr);
      k_trust_fix<<<band_blocks, kThreads, 0, s>>>(a, lst[it & 1], false, next_rows);
    }
  }
}

// Resident blocks per SM of k_band_persistent on the current device (at most
// one): the cooperative launch must fit on the GPU at once.
// Its shared-memory carveout is kBesideSolveCarveout (kf_internal.h), the
// one of the kernels that run beside it.
template <bool kDense>
static int persistent_blocks_per_sm() {
  static int cached[64] = {};
  static bool carveout[64] = {};
  const void *kernel = (const void *)k_band_persistent<kDense>;
  kf_prefer_carveout(kernel, kBesideSolveCarveout, carveout);
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (!cached[dev]) {
    int n = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PersistSharedOf<kDense>)) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kPersistThreads + (kDense ? kTestThreads : 0),
                                                      sizeof(PersistSharedOf<kDense>)) != cudaSuccess)
      return 0;
    cached[dev] = std::min(n, 1);
  }
  return cached[dev];
}

// The blocks that the dense solver's test warps need in the persistent kernel;
// 0: it takes another schedule.  That is for large grids (above 1.2 M voxels,
// kTestChunks: their bands take the groups of the persistent kernel many
// rounds.  100 iterations at 104^3 with 45 k, 506 k and 1.1 M band voxels: 1.1,
// 7.9 and 28.7 ms against 2.0, 16.6 and 49.6 on the split schedule; 128^3 with
// 68 k and 341 k: 2.0 and 4.7 ms against 2.2 and 4.1), a single iteration, which
// its three launches and two clears outweigh (64^3 and 100^3: 26 and 36 us against 16 and 17), a wait limit
// below the default (the other schedules wait for nothing, so no limit makes
// them fail) and a stream that is being captured (which refuses the others'
// graph).
static unsigned persistent_test_blocks(const DevParams &dp, int iterations, cudaStream_t s) {
  if (dp.trust || iterations < 2 || kf_wait_limit_ns() < kDefaultWaitLimitNs) return 0;
  const int64_t groups = (dp.count + 3) / 4, sms = kf_num_sms();
  if (!persistent_size(dp) || persistent_blocks_per_sm<true>() < 1) return 0;
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusActive;
  if (cudaStreamIsCapturing(s, &capturing) != cudaSuccess || capturing != cudaStreamCaptureStatusNone) return 0;
  return (unsigned)std::min((groups + kTestThreads * kTestChunksMin - 1) / (kTestThreads * kTestChunksMin), sms);
}

// KF_SOLVER_BAND without the trust-region step: the dense first pass (on
// phi_live alone when both buffers are zero), then every band pass in one
// cooperative launch (k_band_persistent).  Iteration k reads buffer k % 2
// and writes (k + 1) % 2, as the per-iteration form.  From a zero p the
// first pass leaves both buffers zero outside its list (it copies p to q),
// and the solve records the list: the field's buffers are then zero outside
// its records (kf_field_zero clears just those).
// kDense: the dense solver (psi ends in the primary planes; nothing is
// recorded of what the field's planes hold) with its persistent_test_blocks.
template <bool kDense>
static int launch_band_persistent(kf_grid live, kf_grid can, kf_field psi, const DevParams &dp,
                                  int iterations, IterStats *st, bool p_zero, bool q_zero, unsigned least_blocks,
                                  cudaStream_t s) {
  void *sync = nullptr;
  int rc = kf_field_sync(psi, &sync);
  if (rc) return rc;
  const int bps = persistent_blocks_per_sm<kDense>();
  if (bps < 1) return kf_fail(KF_ERR_CUDA, "the persistent band pass does not fit on an SM");
  KF_CHECK_CUDA(cudaMemsetAsync(sync, 0, sizeof(GridSync), s));
  FusedArgs even = make_args(live, can, dp, st);
  even.ix = (const float *)psi->p[0];
  even.iy = (const float *)psi->p[1];
  even.iz = (const float *)psi->p[2];
  even.ox = (float *)psi->q[0];
  even.oy = (float *)psi->q[1];
  even.oz = (float *)psi->q[2];
  int *lst0 = psi->band, *lst1 = psi->band + dp.count, *shell = lst1 + dp.count;
  int *touched = nullptr;
  unsigned *touched_n = nullptr, *dropped = nullptr;
  if (p_zero || kDense) {
    KfRecords r;
    rc = kf_field_records(psi, s, &r);
    if (rc) return rc;
    KF_CHECK_CUDA(cudaMemsetAsync(r.side_n, 0, sizeof(unsigned), s));
    touched = r.touched;
    touched_n = r.touched_n;
  }
  if (kDense) {
    dropped = reinterpret_cast<unsigned *>(psi->runs);
    KF_CHECK_CUDA(cudaMemsetAsync(dropped, 0, (size_t)((dp.count + 31) / 32) * sizeof(unsigned), s));
  }
  if (p_zero && q_zero)
    k_band_first_zero<<<(unsigned)num_runs(dp), kThreads, 0, s>>>(even, lst0, shell);
  else
    k_band_first<<<(unsigned)num_runs(dp), kThreads, 0, s>>>(even, lst0, shell);
  KF_CHECK_LAUNCH("dense first pass of the persistent solver");
  GridSync *gs = static_cast<GridSync *>(sync);
  unsigned long long limit = kf_wait_limit_ns();
  int iters = iterations;
  unsigned per_block = kPersistPerBlock;
  void *args[] = {&even, &lst0, &lst1, &shell, &iters, &gs, &limit, &touched, &touched_n, &per_block,
                  &least_blocks, &dropped};
  KF_CHECK_CUDA(cudaLaunchCooperativeKernel(
      (const void *)k_band_persistent<kDense>, dim3((unsigned)(kf_num_sms() * bps)),
      dim3(kPersistThreads + (kDense ? kTestThreads : 0)), args, sizeof(PersistSharedOf<kDense>), s));
  if (kDense) {
    k_dense_settle<<<(unsigned)kf_num_sms(), kThreads, 0, s>>>(even, touched, touched_n);
    KF_CHECK_LAUNCH("k_dense_settle");
  } else if (p_zero) {
    psi->p_state = psi->q_state = kPsiRecorded;
    psi->side_recorded = false;
  }
  return KF_OK;
}

int kf_solve_fused(kf_grid live, kf_grid can, kf_field psi, const DevParams &dp, int iterations,
                   IterStats *st, bool band_only, bool p_zero, bool q_zero, cudaStream_t s) {
  int rc = kf_field_ensure_pair(psi);
  if (rc) return rc;
  rc = kf_field_band_list(psi, &psi->band);
  if (rc) return rc;
  const int64_t nruns = num_runs(dp);
  if (psi->runs_cap < nruns) {
    cudaFree(psi->runs);
    psi->runs = nullptr;
    psi->runs_cap = 0;
    if (cudaMalloc(&psi->runs, runs_table_bytes(dp)) != cudaSuccess) {
      cudaGetLastError();
      return kf_fail(KF_ERR_OOM, "cudaMalloc of the dense pass's run table failed");
    }
    psi->runs_cap = nruns;
  }
  if (band_only && !dp.trust)
    return launch_band_persistent<false>(live, can, psi, dp, iterations, st, p_zero, q_zero, 1u, s);
  if (const unsigned test_blocks = band_only ? 0u : persistent_test_blocks(dp, iterations, s))
    return launch_band_persistent<true>(live, can, psi, dp, iterations, st, p_zero, q_zero, test_blocks, s);
  int *rows = nullptr;
  if (dp.trust) {
    rc = kf_field_trust_rows(psi, &rows);
    if (rc) return rc;
  }
  const void *key[12] = {live->phi, can->phi, psi->p[0], psi->p[1], psi->p[2],
                         psi->q[0], psi->q[1], psi->q[2], st, psi->band, psi->runs, rows};
  FusedGraph *g = psi->graph;
  bool hit = g && g->iterations == iterations && g->band_only == band_only &&
             memcmp(g->key_ptr, key, sizeof(key)) == 0 && memcmp(&g->dp, &dp, sizeof(dp)) == 0;
  if (!hit) {
    kf_fused_graph_destroy(psi->graph);
    psi->graph = g = new FusedGraph();
    KF_CHECK_CUDA(cudaStreamCreateWithFlags(&g->capture, cudaStreamNonBlocking));
    const bool split = split_schedule(dp, band_only);
    if (split) {
      KF_CHECK_CUDA(cudaStreamCreateWithFlags(&g->cold, cudaStreamNonBlocking));
      KF_CHECK_CUDA(cudaEventCreateWithFlags(&g->fork, cudaEventDisableTiming));
      KF_CHECK_CUDA(cudaEventCreateWithFlags(&g->join, cudaEventDisableTiming));
    }
    cudaGraph_t graph;
    KF_CHECK_CUDA(cudaStreamBeginCapture(g->capture, cudaStreamCaptureModeThreadLocal));
    if (split)
      launch_split_iterations(make_args(live, can, dp, st), psi, dp, iterations, psi->band, psi->runs,
                              g->capture, g->cold, g->fork, g->join);
    else
      launch_iterations(live, can, psi, dp, iterations, st, psi->band, psi->runs, rows, band_only,
                        g->capture);
    cudaError_t le = cudaGetLastError();
    KF_CHECK_CUDA(cudaStreamEndCapture(g->capture, &graph));
    if (le != cudaSuccess) {
      cudaGraphDestroy(graph);
      return kf_cuda_fail(le, "fused kernel launch during capture");
    }
    cudaError_t ie = cudaGraphInstantiateWithFlags(&g->exec, graph, cudaGraphInstantiateFlagUseNodePriority);
    cudaGraphDestroy(graph);
    if (ie != cudaSuccess) return kf_cuda_fail(ie, "cudaGraphInstantiate");
    g->iterations = iterations;
    g->band_only = band_only;
    memcpy(g->key_ptr, key, sizeof(key));
    g->dp = dp;
  }
  KF_CHECK_CUDA(cudaGraphLaunch(g->exec, s));
  return KF_OK;
}

int kf_solve_pervoxel(kf_grid live, kf_grid can, kf_field psi, const DevParams &dp, int max_iters,
                      IterStats *st, cudaStream_t s) {
  int rc = kf_field_band_list(psi, &psi->band);
  if (rc) return rc;
  // the symmetric band of KillingFusion.cpp:369 and psi read and written in
  // place
  DevParams pd = dp;
  pd.early_exit = 0;
  pd.trust = 0;  // the per-voxel schedule has no trust-region step
  FusedArgs a = make_args(live, can, pd, st);
  a.band_lo = dp.pv_lo_f;
  a.ix = (const float *)psi->p[0];
  a.iy = (const float *)psi->p[1];
  a.iz = (const float *)psi->p[2];
  a.ox = (float *)psi->p[0];
  a.oy = (float *)psi->p[1];
  a.oz = (float *)psi->p[2];
  a.iter = 0;
  const unsigned grid = (unsigned)std::max<int64_t>((dp.count / 4 + kThreads * kFlatGroups - 1) /
                                                        (kThreads * kFlatGroups), 1);
  k_fused_stream<false><<<grid, kThreads, 0, s>>>(a, psi->band, nullptr, nullptr, nullptr);
  // the colours' counts, and their lists in the second band list
  void *sync = nullptr;
  rc = kf_field_sync(psi, &sync);
  if (rc) return rc;
  unsigned *counts = static_cast<unsigned *>(sync);
  KF_CHECK_CUDA(cudaMemsetAsync(counts, 0, kColourCounts * sizeof(unsigned), s));
  int *lists = psi->band + dp.count;
  const unsigned spread = (unsigned)kf_num_sms() * 4;
  const ColourParts parts = colour_parts(dp);
  k_colour_lists<<<spread, kThreads, 0, s>>>(a, psi->band, counts, parts, lists);
  for (int colour = 0; colour < 8; ++colour)
    k_pervoxel<<<(unsigned)kf_num_sms() * kPervoxelBlocksPerSM, 32 * kPervoxelWarps, 0, s>>>(
        a, lists, counts, parts.start[colour], parts.start[colour + 1], max_iters, colour);
  KF_CHECK_LAUNCH("per-voxel solve");
  return KF_OK;
}


KF_BOUNDS_TU_API(fused)
