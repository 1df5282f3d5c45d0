// sp_analysis.cu -- configuration analysis of sample-packed jobs: plane
// overlaps of replica pairs and their correlation functions along the tube.
//
// The reference ships no analysis code; its data description (DATA/README.md)
// names the ingredients: correlation functions built from basis functions
// f, g in {x, x^3, sign x} of the overlap, computed with r = 2, 4, 6, 8
// replicas, and the 3 x 3 (and 2 x 2) matrices of those correlations per
// distance.  The definition used here:
//
//   plane overlap   q_z = (1/L^2) sum over the plane z of s^a s^c, for the
//                   replica pairs (a, c) = (0,1), (2,3), ... among the first
//                   r replicas, at each temperature slot (the configuration
//                   the slot holds);
//   correlation     C_fg(d) = < f(q_z) g(q_{z+d}) >, averaged over the pairs
//                   and the planes z (z + d taken modulo Lz under PBC; only
//                   z + d < Lz under open boundaries).
//
// Two kernels: bit-sliced counts of the differing spins of each (word, pair,
// slot, plane) for the 64 samples of a word, and from them the basis values x
// and x^3; then the nine products summed in a fixed order (FP64) by one lane
// per (sample, slot, distance).
#include <cstdint>

#include "host.hpp"
#include "kernels_dev.cuh"
#include "sp.cuh"

namespace eagb {

void set_last_error(const char *msg);  // api.cu

constexpr int kPlanePlanes = 12;  // bit planes of a plane's count: L^2 < 4096

constexpr int kDiffThreads = 256;
// Lane groups of a block: every group's bit planes are summed by a few lanes, so
// a small plane has one group for 4 sites (3667 planes of 3 x 3 sites, 2 slots:
// ea_sp_plane_overlaps took 232 us with all 128 groups, 135 with 3; 4 x 10, 2
// slots, one word 37 and 29).
__host__ __device__ inline int plane_groups(int NB, int L2) {
  const int most = kDiffThreads / NB, few = (L2 + 3) / 4;
  return few < most ? few : most;
}

// Spins that differ between the pair's two replicas on plane z, for every slot
// and sample: one block per (word, pair, plane), lane groups of one lane per
// slot over the plane's sites, the groups' bit planes added through SMEM (one
// thread a plane and slot was a chain of L^2 loads on few SMs: 63 us on 12 x 12
// x 48, 24 slots, 2 pairs, now 14).  Writes the counts to diff [w][sample]
// [pair][slot][z] or, when xs is given, x = 1 - 2 diff / L^2 and x^3 to
// xs [2][w][pair][slot][z][sample].
__global__ void __launch_bounds__(kDiffThreads) k_sp_plane_diff(const __grid_constant__ SpDev d, int npairs,
                                                                int32_t *diff, double *xs) {
  extern __shared__ u64 pl[];  // [group][bit plane][slot]
  const int NB = d.NB, NR = d.NR, G = NR * NB, Lz = d.Lz, L2 = d.L * d.L;
  const int z = blockIdx.x % Lz, k = (blockIdx.x / Lz) % npairs, w = blockIdx.x / (Lz * npairs);
  const int groups = plane_groups(NB, L2), g = threadIdx.x / NB, b = threadIdx.x - g * NB;
  if (g < groups) {
    const u64 *Sa = d.S + ((size_t)w * d.V + (size_t)z * L2) * G + (size_t)(2 * k) * NB + b;
    u64 P[kPlanePlanes];
#pragma unroll
    for (int q = 0; q < kPlanePlanes; ++q) P[q] = 0;
#pragma unroll 4
    for (int i = g; i < L2; i += groups) {
      u64 c = __ldg(Sa + (size_t)i * G) ^ __ldg(Sa + (size_t)i * G + NB);
#pragma unroll
      for (int q = 0; q < kPlanePlanes; ++q) {
        const u64 h = P[q] & c;
        P[q] ^= c;
        c = h;
      }
    }
#pragma unroll
    for (int q = 0; q < kPlanePlanes; ++q) pl[(g * kPlanePlanes + q) * NB + b] = P[q];
  }
  __syncthreads();
  const double inv = 1.0 / (double)L2;
  const size_t tab = (size_t)d.nw * npairs * NB * Lz * 64;
  // a task: samples s, s + 16, s + 32, s + 48 of a slot as 16-bit fields
  for (int t = threadIdx.x; t < NB * 16; t += kDiffThreads) {
    const int slot = t >> 4, s = t & 15;
    u64 acc = 0;
    for (int q = 0; q < groups; ++q)
#pragma unroll
      for (int p = 0; p < kPlanePlanes; ++p)
        acc += ((pl[(q * kPlanePlanes + p) * NB + slot] >> s) & 0x0001000100010001ull) << p;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int n = (int)((acc >> (16 * q)) & 0xFFFFu), smp = s + 16 * q;
      if (xs) {
        // 0 where half of the plane differs: 2/L^2 times L^2/2 may round to
        // less than 1 (L = 14), and sign(x) is read from x
        const double x = 2 * n == L2 ? 0.0 : __dsub_rn(1.0, __dmul_rn(2.0 * inv, (double)n));
        const size_t o = ((((size_t)w * npairs + k) * NB + slot) * Lz + z) * 64 + smp;
        xs[o] = x;
        xs[tab + o] = __dmul_rn(__dmul_rn(x, x), x);
      } else {
        diff[((((size_t)w * 64 + smp) * npairs + k) * NB + slot) * Lz + z] = n;
      }
    }
  }
}

// C[w*64 + sample][slot][d][3][3] = the correlation matrix at distance d
// (sums over pairs and planes in a fixed order, then divided by their count).
// A warp takes one distance of (word, slot) and 32 samples, so its lanes make
// equally many steps and read neighbouring words.  Bound by the FP64 pipe: a
// step takes 4 products and 8 sums; products with a sign are sign flips, the
// signs' own product is counted in integers (both exact).  Thread per
// (sample, slot, distance), the basis made from the counts at every step:
// 457 us on 12 x 12 x 48, 24 slots, 2 pairs, 48 distances; now 134 (of which the pipe needs some 75).
__global__ void __launch_bounds__(256) k_sp_plane_corr(const __grid_constant__ SpDev d, int npairs, int dmax,
                                                       const double *xs, double *C) {
  const int NB = d.NB, Lz = d.Lz, nd = dmax + 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int ngrp = (nd + nwarp - 1) / nwarp;
  const int dg = blockIdx.x % ngrp, half = (blockIdx.x / ngrp) & 1, wb = blockIdx.x / (2 * ngrp);
  const int dd = dg + warp * ngrp, b = wb % NB, w = wb / NB, smp = half * 32 + lane;
  if (dd >= nd) return;
  const bool pbc = d.bc == EA_PBC;
  const size_t tab = (size_t)d.nw * npairs * NB * Lz * 64;
  const int zmax = pbc ? Lz : Lz - dd;
  double acc[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) acc[q] = 0.0;
  long long ss = 0;
  // the value times sign(x): v with its sign flipped, or 0; sign(x) itself.
  // In integers: FP64 comparisons would take the same pipe as the sums.
  auto times = [](double v, double x) {
    const long long xb = __double_as_longlong(x);
    return __longlong_as_double((xb << 1) == 0 ? 0ll : __double_as_longlong(v) ^ (xb & (1ll << 63)));
  };
  auto sgn = [](double x) {
    const long long xb = __double_as_longlong(x);
    return (xb << 1) == 0 ? 0 : (xb < 0 ? -1 : 1);
  };
  for (int k = 0; k < npairs; ++k) {
    const double *X = xs + (((size_t)w * npairs + k) * NB + b) * Lz * 64 + smp;
#pragma unroll 2
    for (int z = 0; z < zmax; ++z) {
      int z2 = z + dd;
      if (z2 >= Lz) z2 -= Lz;
      const double f0 = __ldg(X + (size_t)z * 64), f1 = __ldg(X + tab + (size_t)z * 64);
      const double g0 = __ldg(X + (size_t)z2 * 64), g1 = __ldg(X + tab + (size_t)z2 * 64);
      acc[0] = __dadd_rn(acc[0], __dmul_rn(f0, g0));
      acc[1] = __dadd_rn(acc[1], __dmul_rn(f0, g1));
      acc[2] = __dadd_rn(acc[2], times(f0, g0));
      acc[3] = __dadd_rn(acc[3], __dmul_rn(f1, g0));
      acc[4] = __dadd_rn(acc[4], __dmul_rn(f1, g1));
      acc[5] = __dadd_rn(acc[5], times(f1, g0));
      acc[6] = __dadd_rn(acc[6], times(g0, f0));
      acc[7] = __dadd_rn(acc[7], times(g1, f0));
      ss += sgn(f0) * sgn(g0);
    }
  }
  const long long n = (long long)npairs * zmax;
  double *o = C + (((size_t)w * 64 + smp) * NB + b) * nd * 9 + (size_t)dd * 9;
#pragma unroll
  for (int q = 0; q < 8; ++q) o[q] = n ? acc[q] / (double)n : 0.0;
  o[8] = n ? (double)ss / (double)n : 0.0;
}

}  // namespace eagb

using namespace eagb;

extern "C" {

// Defined in sp.cu: the job's device view and stream.
int ea_sp_device_view(ea_sp *job, SpDev *d, cudaStream_t *st);

static void launch_plane_diff(const SpDev &d, int npairs, int32_t *diff, double *xs, cudaStream_t st) {
  const size_t sm = (size_t)plane_groups(d.NB, d.L * d.L) * d.NB * kPlanePlanes * 8;
  k_sp_plane_diff<<<(unsigned)((size_t)d.nw * npairs * d.Lz), kDiffThreads, sm, st>>>(d, npairs, diff, xs);
}

static int an_fail(const char *m) {
  set_last_error(m);
  return EA_ERR_ARG;
}

static int an_cuda_fail(cudaError_t e) {
  set_last_error(cudaGetErrorString(e));
  (void)cudaGetLastError();  // reported here, not by the next launch
  return EA_ERR_CUDA;
}

int ea_sp_plane_overlaps(ea_sp *job, int32_t nrep, int32_t *diff) {
  SpDev d;
  cudaStream_t st;
  int rc = ea_sp_device_view(job, &d, &st);
  if (rc) return rc;
  if (!diff || nrep < 2 || (nrep & 1) || nrep > d.NR) return an_fail("nrep: an even number of replicas, 2..NR");
  if (d.L * d.L >= (1 << kPlanePlanes)) return an_fail("planes of at most 4095 sites");
  const int npairs = nrep / 2;
  const size_t n = (size_t)d.nw * 64 * npairs * d.NB * d.Lz;
  int32_t *dd = nullptr;
  cudaError_t e = cudaMalloc((void **)&dd, n * 4);
  if (e == cudaSuccess) {
    launch_plane_diff(d, npairs, dd, nullptr, st);
    e = cudaGetLastError();
  }
  prefault(diff, n * 4);
  if (e == cudaSuccess) e = cudaMemcpyAsync(diff, dd, n * 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (dd) cudaFree(dd);
  return e == cudaSuccess ? EA_OK : an_cuda_fail(e);
}

int ea_sp_plane_correlations(ea_sp *job, int32_t nrep, int32_t dmax, double *C) {
  SpDev d;
  cudaStream_t st;
  int rc = ea_sp_device_view(job, &d, &st);
  if (rc) return rc;
  if (!C || nrep < 2 || (nrep & 1) || nrep > d.NR) return an_fail("nrep: an even number of replicas, 2..NR");
  if (dmax < 0 || dmax >= d.Lz) return an_fail("dmax: 0..Lz-1");
  if (d.L * d.L >= (1 << kPlanePlanes)) return an_fail("planes of at most 4095 sites");
  const int npairs = nrep / 2;
  const size_t nx = 2 * (size_t)d.nw * 64 * npairs * d.NB * d.Lz, nc = (size_t)d.nw * 64 * d.NB * (dmax + 1) * 9;
  double *dx = nullptr, *dc = nullptr;
  cudaError_t e = cudaMalloc((void **)&dx, nx * 8);
  if (e == cudaSuccess) e = cudaMalloc((void **)&dc, nc * 8);
  if (e == cudaSuccess) {
    launch_plane_diff(d, npairs, nullptr, dx, st);
    const int ngrp = (dmax + 1 + 7) / 8;
    k_sp_plane_corr<<<(unsigned)((size_t)d.nw * d.NB * 2 * ngrp), 256, 0, st>>>(d, npairs, dmax, dx, dc);
    e = cudaGetLastError();
  }
  prefault(C, nc * 8);
  if (e == cudaSuccess) e = cudaMemcpyAsync(C, dc, nc * 8, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (dx) cudaFree(dx);
  if (dc) cudaFree(dc);
  return e == cudaSuccess ? EA_OK : an_cuda_fail(e);
}

}  // extern "C"
