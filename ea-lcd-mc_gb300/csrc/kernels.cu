// kernels.cu -- the one-job kernels of the EA-LCD-MC hot path (bodies in
// kernels_dev.cuh) and their launchers.
#include "kernels_dev.cuh"

#include <algorithm>
#include <cstdio>

namespace eagb {

// SMEM of a slab's labelling: three CTAs an SM when slabs of a fair number of
// planes still fit (fewer planes leave more faces to the union across slabs).
constexpr size_t kSlabSmem = 74 * 1024;
constexpr size_t kRunMax = 224 * 1024;

static int cc_threads(const RunShape &r) {
  const int passes = (r.nseg + 1023) / 1024;
  return std::min(1024, ((r.nseg + passes - 1) / passes + 31) / 32 * 32);
}

CcShape cc_shape(const JobDev &j) {
  CcShape c{};
  const int S = j.L * j.L;
  const size_t q = (size_t)j.V / 8;
  // whole: label indices in 16 bits, the overlap words beside the labels
  if (j.V <= 65536 && run_label_smem(run_shape(j.L, j.Lz)) + q <= kRunMax) {
    const RunShape r = run_shape(j.L, j.Lz);
    c.whole = true;
    c.planes = j.Lz;
    c.nslab = 1;
    c.threads = cc_threads(r);
    c.smem = run_label_smem(r) + q;
    return c;
  }
  if (S > kSlabPlane) return c;
  size_t lim = kSlabSmem;
  auto most = [&](size_t smem) {
    int D = 0;
    while (D < j.Lz && S * (D + 1) <= 65536 && run_label_smem(run_shape(j.L, D + 1)) <= smem) ++D;
    return D;
  };
  int D = most(lim);
  if (D < 8) D = most(lim = kRunMax);
  if (D < 1) return c;
  c.nslab = (j.Lz + D - 1) / D;
  c.planes = (j.Lz + c.nslab - 1) / c.nslab;  // slabs of equal height
  c.nslab = (j.Lz + c.planes - 1) / c.planes;
  const RunShape r = run_shape(j.L, c.planes);
  c.threads = cc_threads(r);
  c.smem = run_label_smem(r);
  return c;
}

void set_dividers(JobDev &j) {
  j.fd_L.set(j.L); j.fd_S.set(j.L * j.L); j.fd_ml.set(j.msc_l); j.fd_mlz.set(j.msc_lz);
  j.fd_hl.set(j.msc_l / 2); j.fd_nclust.set(j.nclust > 0 ? j.nclust : 1);
  const CcShape c = cc_shape(j);
  j.cc_D = c.planes;
  j.cc_nslab = c.nslab;
}

__global__ void k_ctr_chain(const __grid_constant__ JobDev j, int npass) {
  extern __shared__ __align__(16) unsigned char smem[];
  ctr_chain_body(j.prc, j.xo, j.iter, j.jobid, j.NR, npass, j.ctrs, j.ctr, smem, [](int p, long long) { return p & 1; });
}

template <int NR, int KT, bool UPDATE>
__global__ void __launch_bounds__(512, 2) k_sweep(const __grid_constant__ JobDev j, int pass, int parity, int energy) {
  extern __shared__ __align__(16) unsigned char smem[];
  sweep_body<NR, KT, UPDATE>(j, j.ctrs + (size_t)pass * NR, blockIdx.x, parity, energy, smem);
}

__global__ void __launch_bounds__(256) k_pt(const __grid_constant__ JobDev j) {
  __shared__ PtShared sh;
  pt_body(j, blockIdx.x, blockIdx.y, sh);
}

__global__ void k_measure(const __grid_constant__ JobDev j, int itm) {
  measure_body(j, blockIdx.x * blockDim.x + threadIdx.x, itm);
}

__global__ void k_hou_overlap(const __grid_constant__ JobDev j, int g) {
  overlap_body(j, g, blockIdx.x * blockDim.x + threadIdx.x, blockIdx.y);
}

__global__ void __launch_bounds__(1024) k_cc_slab(const __grid_constant__ JobDev j) {
  extern __shared__ __align__(16) unsigned char smem[];
  cc_slab_body(j, j.cc_D, blockIdx.x, blockIdx.y, smem);
}

__global__ void __launch_bounds__(1024) k_hou_move(const __grid_constant__ JobDev j) {
  extern __shared__ __align__(16) unsigned char smem[];
  move_body(j, blockIdx.y, blockIdx.x, smem);
}

__global__ void k_cc_merge(const __grid_constant__ JobDev j, int D, int nslab) {
  cc_merge_body(j, D, nslab, blockIdx.x * blockDim.x + threadIdx.x, blockIdx.y);
}

__global__ void k_cc_compress(const __grid_constant__ JobDev j, int D, int nslab) {
  cc_compress_body(j, D, nslab, blockIdx.x * blockDim.x + threadIdx.x, blockIdx.y);
}

__global__ void __launch_bounds__(512) k_hou_flip(const __grid_constant__ JobDev j, int g) {
  extern __shared__ uint32_t s_flip[];
  flip_body(j, g, blockIdx.x, s_flip + 64, reinterpret_cast<int *>(s_flip));
}

size_t flip_smem_bytes(const JobDev &j) { return 256 + (size_t)j.V / 8; }

__global__ void __launch_bounds__(256) k_hou_select(const __grid_constant__ JobDev j, int g) {
  select_body(j, g, blockIdx.x * blockDim.x + threadIdx.x, blockIdx.y);
}

__global__ void __launch_bounds__(256) k_hou_apply(const __grid_constant__ JobDev j, int g) {
  __shared__ unsigned s_sel[8];
  apply_body(j, g, blockIdx.x, blockIdx.y, s_sel);
}

// Bonds between equal-overlap neighbours towards -x, -y (periodic) and -z
// (periodic under PBC, none across z = 0 under OBC); the initial label is the
// smallest bonded index (HoudayerXEA.cu:77-121).
__global__ void k_cc_init(JobDev j) {
  const size_t n = (size_t)j.ns * j.nclust * j.V;
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const size_t lat = t / j.V;
  const int i = (int)(t % j.V), L = j.L, S = L * L;
  const int x = i % L, y = (i / L) % L, z = i / S;
  const u64 *Q = j.Q + lat * 2 * j.half;
  const int q = q_bit(j, Q, x, y, z);
  uint32_t m = (uint32_t)i;
  const int xm = x == 0 ? L - 1 : x - 1, ym = y == 0 ? L - 1 : y - 1;
  if (q_bit(j, Q, xm, y, z) == q) m = min(m, (uint32_t)(xm + L * y + S * z));
  if (q_bit(j, Q, x, ym, z) == q) m = min(m, (uint32_t)(x + L * ym + S * z));
  if (z > 0 || j.bc == EA_PBC) {
    const int zm = z == 0 ? j.Lz - 1 : z - 1;
    if (q_bit(j, Q, x, y, zm) == q) m = min(m, (uint32_t)(x + L * y + S * zm));
  }
  j.label[t] = m;
}

// Label reduction of Komura (HoudayerXEA.cu:254-331): every bond that is not
// the initial tree edge is merged with atomicMin, so each root ends as the
// smallest site index of its cluster.
__global__ void k_cc_union(JobDev j) {
  const size_t n = (size_t)j.ns * j.nclust * j.V;
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const size_t lat = t / j.V;
  const int i = (int)(t % j.V), L = j.L, S = L * L;
  const int x = i % L, y = (i / L) % L, z = i / S;
  const u64 *Q = j.Q + lat * 2 * j.half;
  uint32_t *lab = j.label + lat * j.V;
  const int q = q_bit(j, Q, x, y, z);
  const int xm = x == 0 ? L - 1 : x - 1, ym = y == 0 ? L - 1 : y - 1;
  // site 0 tests its x-wrap bond against x = cc_xq (see JobDev::cc_xq)
  const int xt = i == 0 ? j.cc_xq : xm;
  if (q_bit(j, Q, xt, y, z) == q) cc_unite(lab, (uint32_t)i, (uint32_t)(xm + L * y + S * z));
  if (q_bit(j, Q, x, ym, z) == q) cc_unite(lab, (uint32_t)i, (uint32_t)(x + L * ym + S * z));
  if (z == 0 && j.bc == EA_PBC && q_bit(j, Q, x, y, j.Lz - 1) == q)
    cc_unite(lab, (uint32_t)i, (uint32_t)(x + L * y + S * (j.Lz - 1)));
}

__global__ void k_cc_flatten(JobDev j) {
  const size_t n = (size_t)j.ns * j.nclust * j.V;
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const size_t lat = t / j.V;
  uint32_t *lab = j.label + lat * j.V;
  j.label[t] = cc_find(lab, (uint32_t)(t % j.V));
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
int sweep_kt(const JobDev &j) { return j.kt; }

size_t sweep_smem_bytes(const JobDev &j) { return sweep_smem_for(j.NB, j.NR, j.kt); }

template <int NR, int KT>
static cudaError_t launch_sweep_t(const JobDev &j, int pass, int parity, int energy, bool update, cudaStream_t st) {
  if (update) {
    const size_t sm = sweep_smem_bytes(j);
    static bool attr = false;
    if (!attr) {
      cudaFuncSetAttribute(k_sweep<NR, KT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSweepMax);
      attr = true;
    }
    k_sweep<NR, KT, true><<<j.ntiles * j.nsplit, 512, sm, st>>>(j, pass, parity, energy);
  } else {
    k_sweep<NR, KT, false><<<j.ntiles * j.nsplit, 512, (size_t)KT * 8 * 4, st>>>(j, pass, parity, energy);
  }
  return cudaGetLastError();
}

static cudaError_t dispatch_sweep(const JobDev &j, int pass, int parity, int energy, bool update, cudaStream_t st) {
  switch (j.NR * 100 + j.kt) {
    case 801: return launch_sweep_t<8, 1>(j, pass, parity, energy, update, st);
    case 802: return launch_sweep_t<8, 2>(j, pass, parity, energy, update, st);
    case 804: return launch_sweep_t<8, 4>(j, pass, parity, energy, update, st);
    case 402: return launch_sweep_t<4, 2>(j, pass, parity, energy, update, st);
    case 404: return launch_sweep_t<4, 4>(j, pass, parity, energy, update, st);
    case 408: return launch_sweep_t<4, 8>(j, pass, parity, energy, update, st);
    case 204: return launch_sweep_t<2, 4>(j, pass, parity, energy, update, st);
    case 208: return launch_sweep_t<2, 8>(j, pass, parity, energy, update, st);
    case 216: return launch_sweep_t<2, 16>(j, pass, parity, energy, update, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_ctr_chain(const JobDev &j, int npass, cudaStream_t st) {
  k_ctr_chain<<<1, kCtrThreads, ctr_smem(j.NR), st>>>(j, npass);
  return cudaGetLastError();
}

cudaError_t launch_sweep(const JobDev &j, int pass, int parity, int energy, cudaStream_t st) {
  return dispatch_sweep(j, pass, parity, energy, true, st);
}

cudaError_t launch_energy(const JobDev &j, cudaStream_t st) {
  const cudaError_t e = cudaMemsetAsync(j.E, 0, sizeof(int32_t) * (size_t)j.ns * j.NB * j.NR, st);
  return e != cudaSuccess ? e : dispatch_sweep(j, 0, 0, kEnergyAdd, false, st);
}

cudaError_t launch_pt(const JobDev &j, cudaStream_t st) {
  dim3 grid(j.ns, (j.NR + 7) / 8);
  k_pt<<<grid, 256, 0, st>>>(j);
  return cudaGetLastError();
}

cudaError_t launch_measure(const JobDev &j, int itm, cudaStream_t st) {
  const int n = j.ns * j.NB * j.NR;
  k_measure<<<(n + 255) / 256, 256, 0, st>>>(j, itm);
  return cudaGetLastError();
}

cudaError_t houdayer_setup() {
  cudaError_t e = cudaFuncSetAttribute(k_cc_slab, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRunMax);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_hou_move, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRunMax);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_hou_flip, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFlipMaxSmem);
  return e;
}

cudaError_t launch_houdayer(const JobDev &j, cudaStream_t st) {
  const CcShape cc = cc_shape(j);
  if (cc.whole) {
    k_hou_move<<<dim3((unsigned)(j.ns * j.nclust), 2), cc.threads, cc.smem, st>>>(j);
    return cudaGetLastError();
  }
  cudaError_t e = cudaSuccess;
  for (int g = 0; g < 2 && e == cudaSuccess; ++g) e = launch_houdayer_group(j, g, st);
  return e;
}

cudaError_t launch_houdayer_group(const JobDev &j, int g, cudaStream_t st) {
  const size_t ns = (size_t)j.ns * j.nclust * j.V;
  const unsigned bs = (unsigned)((ns + 255) / 256);
  const unsigned nlat = (unsigned)(j.ns * j.nclust);
  k_hou_overlap<<<dim3((2 * j.half + 255) / 256, nlat), 256, 0, st>>>(j, g);
  const CcShape cc = cc_shape(j);
  if (cc.planes > 0) {
    const int D = cc.planes, nslab = cc.nslab;
    k_cc_slab<<<dim3(nslab, nlat), cc.threads, cc.smem, st>>>(j);
    k_cc_merge<<<dim3((nslab * j.L * j.L + 255) / 256, nlat), 256, 0, st>>>(j, D, nslab);
    k_cc_compress<<<dim3((nslab * j.L * j.L + 255) / 256, nlat), 256, 0, st>>>(j, D, nslab);
    const size_t sm = flip_smem_bytes(j);
    if (sm <= kFlipMaxSmem) {
      k_hou_flip<<<nlat, 512, sm, st>>>(j, g);
      return cudaGetLastError();
    }
  } else {
    // planes too large for SMEM: Komura's passes on global labels
    k_cc_init<<<bs, 256, 0, st>>>(j);
    k_cc_flatten<<<bs, 256, 0, st>>>(j);
    k_cc_union<<<bs, 256, 0, st>>>(j);
  }
  k_hou_select<<<dim3((j.V + 255) / 256, nlat), 256, 0, st>>>(j, g);
  k_hou_apply<<<dim3((2 * j.half + 3) / 4, nlat), 256, 0, st>>>(j, g);
  return cudaGetLastError();
}

}  // namespace eagb
