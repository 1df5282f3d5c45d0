// sp_resident.cu -- resident bin kernel of small sample-packed jobs.
//
// A job too small to fill the GPU spends a per-phase launch on every colour
// pass, energy count, tempering step and permute, and each of those phases
// is a short latency-bound chain.  A job whose words fit in the shared memory
// of one thread-block cluster runs instead as four launches per chunk of
// sweeps (with cluster moves, per block of sweeps between two):
//
//   k_sp_ctr_chain  the Philox counters of every colour pass of the chunk: one
//                   thread per replica steps its xoshiro256++ and
//                   Parisi-Rapuano generators (the counters never depend on
//                   the spins), the states staged in SMEM;
//   k_sp_draw       the random words of every (pass, site, replica, slot) at
//                   once on the whole GPU -- the integer-heavy part of a
//                   sweep, now fully parallel;
//   k_sp_pt_draw    the tempering draws of every (step, pair, chain);
//   k_sp_resident   a cluster of up to 16 CTAs for each unit -- a (word,
//                   replica), whose chain of temperatures meets no other
//                   between two moves -- holds its spin and coupling words in
//                   distributed shared memory (CTA c owns a run of sites) and
//                   runs every sweep, energy count, tempering step, permute
//                   and measurement of the chunk, phases separated by cluster
//                   barriers; neighbour words on other CTAs are read through
//                   DSMEM.
//
// What bounds the resident kernel is latency.  A step (a sweep, a count, a
// tempering step) of the 6^2 x 24 tube with 12 temperatures, 2 replicas and 64
// samples takes 7 us: 3 cluster barriers of 1600 cycles, most of it the fence
// of cluster scope, two colour passes of 1600, the count's sum and the stores
// to the other CTAs 2700, the tempering walk 2800.  One cluster for the whole
// job (three in four of its neighbour words on other CTAs), four barriers, a
// tempering step in one CTA with a table look-up a pair and two items' code
// unrolled side by side took 13.8 us (a bin of 64 steps with its draws 1011 us,
// now 687); a bin of 32 sweeps and 4 moves of a 7^2 x 21 tube with 13
// temperatures, 3 words and 3 replicas, 9 units, took 1952 us, now 955.
//
// Every phase computes what the per-phase kernels of sp.cu compute (same
// random words, update rule, bit-sliced counts, FP64 tempering rule and
// Philox uniforms, same order of the floating-point additions), so a job's
// words, energies, swaps and averages are identical either way.
#include <cooperative_groups.h>

#include <algorithm>

#include "host.hpp"
#include "kernels_dev.cuh"
#include "sp.cuh"

namespace cg = cooperative_groups;

namespace eagb {

constexpr int kResThreads = 512;
constexpr size_t kResSmem = 227 * 1024 - 256;  // dynamic, less the static part
// bit planes of the per-sample counts summed over a warp: a CTA holds at most
// (2^15 - 1) / 6 sites
constexpr int kResPlanes = 15;
constexpr int kResMaxSites = ((1 << kResPlanes) - 1) / 6;

// ---------------------------------------------------------------------------
// Counters of npass consecutive colour passes (ctr_chain_body): pass p uses
// time counter iter0 + p and its parity.  Every path but the persistent
// kernel's draws its passes' counters this way.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void sp_ctr_chain_body(const SpDev &d, int npass, uint4 *ctrs, unsigned char *sm) {
  ctr_chain_body(d.prc, d.xo, d.iter, d.jobid, d.NR, npass, ctrs, d.ctr, sm,
                 [](int, long long it) { return (int)(it & 1); });
}

__global__ void k_sp_ctr_chain(const __grid_constant__ SpDev d, int npass, uint4 *ctrs) {
  extern __shared__ __align__(16) unsigned char sm[];
  sp_ctr_chain_body(d, npass, ctrs, sm);
}
// A block per job of a batch, nsweep sweeps of its colours.
__global__ void kb_sp_ctr_chain(const __grid_constant__ SpBatchDev b, int nsweep) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ SpDev d;
  if (threadIdx.x == 0) d = b.jobs[blockIdx.x];
  __syncthreads();
  sp_ctr_chain_body(d, nsweep * d.ncol, d.ctrs, sm);
}

cudaError_t sp_launch_ctr_chain(const SpDev &d, int npass, uint4 *ctrs, cudaStream_t st) {
  k_sp_ctr_chain<<<1, kCtrThreads, ctr_smem(d.NR), st>>>(d, npass, ctrs);
  return cudaGetLastError();
}

cudaError_t sp_batch_ctr_setup() {
  return cudaFuncSetAttribute(kb_sp_ctr_chain, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ctr_smem(64));
}

cudaError_t sp_batch_ctr_chain(const SpBatchDev &b, int nsweep, cudaStream_t st) {
  kb_sp_ctr_chain<<<b.njobs, kCtrThreads, ctr_smem(b.nrep), st>>>(b, nsweep);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Random words of nsweep sweeps: every (sweep, colour, site of the colour,
// replica, slot) as the two words of its flip mask (draw_ids of the words
// sp_pass_body draws; thresholds and pre-search through the read-only cache).
// Per sweep the colours follow each other; colour k's block holds 2 planes of
// NR * NB * n_k words, item (r, b, kk) at (r * NB + b) * n_k + kk of each plane
// (the site fastest, as the resident kernel's lanes read them).  A CTA draws
// kDrawItems of them.  (All six words of every item, an 8-bit pre-search and
// three planes: 13 thousand items a us of the 6^2 x 24 tube, now 24.)
// ---------------------------------------------------------------------------
constexpr int kDrawItems = 768, kDrawThreads = 256;
__global__ void __launch_bounds__(kDrawThreads) k_sp_draw(const __grid_constant__ SpDev d, int nsweep, const uint4 *ctrs,
                                                          u64 *R) {
  __shared__ u64 id1[kDrawItems], id2[kDrawItems];
  __shared__ uint16_t queue[4 * kDrawItems];
  __shared__ int cnt[2];
  const int NB = d.NB, NR = d.NR, G = NR * NB, V = d.V, ncol = d.ncol, per = V * G;
  const long long t0 = (long long)blockIdx.x * kDrawItems, left = (long long)per * nsweep - t0;
  const int n = left < kDrawItems ? (int)left : kDrawItems, s0 = (int)(t0 / per), e0 = (int)(t0 - (long long)s0 * per);
  // item t of the CTA: its sweep, colour and place e in the colour's block
  auto place = [&](int t, int &s, int &k, int &nk, int &e) {
    e = e0 + t;
    s = s0;
    while (e >= per) e -= per, ++s;
    k = 0;
    while (k + 1 < ncol && e >= d.col_off[k + 1] * G) ++k;
    nk = d.col_off[k + 1] - d.col_off[k];
    e -= d.col_off[k] * G;
  };
  draw_ids(
      n,
      [&](int t, uint4 &c, uint32_t &key, uint32_t &tp, int &b) {
        int s, k, nk, e;
        place(t, s, k, nk, e);
        const int col = e / nk, r = col / NB, site = __ldg(d.col_sites + d.col_off[k] + e - col * nk);
        b = col - r * NB;
        c = ctrs[((size_t)s * ncol + k) * NR + r];
        key = __ldg(d.keys + r);
        tp = (uint32_t)(((size_t)b * V + site) * NR + r);
        return true;
      },
      [&](int b, uint32_t hi, uint32_t lo) {
        return lut_byte11(hi, lo, d.cum + b * 256, d.pre11 + (size_t)b * kPre11Stride);
      },
      id1, id2, queue, cnt);
  for (int t = threadIdx.x; t < n; t += blockDim.x) {
    int s, k, nk, e;
    place(t, s, k, nk, e);
    u64 *o = R + (size_t)s * 2 * per + (size_t)2 * d.col_off[k] * G + e;
    o[0] = id1[t];
    o[(size_t)nk * G] = id2[t];
  }
}

// ---------------------------------------------------------------------------
// Tempering draws of npt steps (sp_pt_body's): u of Philox4x32-10 of (step,
// pair, chain) keyed by the tempering seed, x = FNORM * u in FP64 (an exact
// scaling of u rounded to 53 bits), and from it the largest m = -dE / 2 the
// pair's exchange is still accepted at: the table's exp(pt(m)), m = 1, 2, ...,
// decrease (sp_res_ok), so x < exp(pt(m)) holds up to some m.  INT_MAX: at
// every m (x = 0, or betas that are equal); INT_MIN: at none (betas the other
// way round).  Off the resident kernel's serial chain, where a look-up of the
// table a pair took 510 cycles with all around it.
// X: [step][word x replica][pair][sample].
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_sp_pt_draw(const __grid_constant__ SpDev d, int npt, int32_t *X) {
  const int NR = d.NR, NP = d.NB - 1, nunits = d.nw * NR;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)npt * nunits * NP * 64) return;
  const int lane = (int)(t & 63);
  long long rest = t >> 6;
  const int pi = (int)(rest % NP);
  rest /= NP;
  const int u = (int)(rest % nunits), j = (int)(rest / nunits);
  const int w = u / NR, r = u - w * NR;
  const unsigned long long step = *d.ptstep + (unsigned long long)j;
  const uint32_t chain = (uint32_t)(((size_t)w * 64 + lane) * NR + r);
  uint32_t v0 = (uint32_t)step, v1 = (uint32_t)(step >> 32), v2 = (uint32_t)pi, v3 = chain;
  philox10(v0, v1, v2, v3, (uint32_t)d.pt_seed, (uint32_t)(d.pt_seed >> 32));
  const double FNORM = 5.4210108624275218e-20;
  const double x = __dmul_rn(FNORM, __ull2double_rn(((u64)v0 << 32) | v1));
  const double f = -__dsub_rn(d.betas[pi + 1], d.betas[pi]);
  int m = 0x7FFFFFFF;
  if (x != 0.0 && f != 0.0) {
    if (f < 0.0) m = (int)0x80000000;
    else {
      const double *tab = d.exptab + d.expoff[pi];
      int lo = 0, hi = d.expoff[pi + 1] - d.expoff[pi];
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (x < __ldg(tab + mid)) lo = mid + 1; else hi = mid;
      }
      m = lo;
    }
  }
  X[t] = m;
}

// ---------------------------------------------------------------------------
// The resident kernel's phases, of one chain of temperatures (unit = (word,
// replica)) in a cluster.  Site i of the lattice lives in CTA i / nslm at local
// index i % nslm.  SMEM arrays keep the site (or the sample) as the fastest
// index, so that the lanes of a warp -- consecutive sites of one slot, or
// consecutive samples -- touch consecutive words:
//   S   [NB][nslm]  spin words                J    [6][nslm] coupling words
//   nbl [6][nslm]   SMEM address of each bond slot's neighbour in slot 0, mapped
//                   into its CTA, bit 0 set if that is another one
//   lst [nsl]       the CTA's sites, colour by colour
//   Pt  [ncta][NB][64]  every CTA's counts of its sites
// and the unit's tempering state, the same in every CTA:
//   U2s, Es, Av, Ps [NB][64]    As, Xs [NB-1][64]    Ms [NB-1]
// ---------------------------------------------------------------------------
struct ResCta {
  int rank, unit, w, r, site_lo, nsl;
};

struct ResShared {
  int32_t *Xs;   // the step's draws (k_sp_pt_draw)
  uint16_t *Pt;
  u64 *S, *J;
  u64 *Ms;       // lanes that swapped, per pair
  long long *Av; // the bin's energy sums (integers: exactly the double sums, all below 2^53)
  int32_t *U2s;  // counts of the whole lattice
  int32_t *Es;
  uint32_t *As;
  uint32_t *nbl;
  int32_t *SG;   // [NB-1] sign of -(beta[i+1] - beta[i])
  uint16_t *lst;
  uint8_t *Ps;
};

// parts: CTAs that leave their counts in Pt (0: added to U2s by atomics, for
// ladders whose Pt would not fit)
__host__ __device__ inline size_t res_smem_bytes(int nslm, int NB, int parts) {
  const size_t NP = NB - 1;
  const size_t b = 8 * ((size_t)nslm * NB + (size_t)nslm * 6 + NP + 64 * NB) +
                   4 * (2 * 64 * NB + 2 * 64 * NP + (size_t)nslm * 6 + NP) + 2 * ((size_t)nslm + parts * 64 * NB) + 64 * NB;
  return (b + 15) & ~(size_t)15;
}

__device__ __forceinline__ ResShared res_carve(unsigned char *smem, const SpResDev &p) {
  const size_t NB = p.d.NB, NP = NB - 1;
  ResShared s;
  s.Xs = reinterpret_cast<int32_t *>(smem);
  s.Pt = reinterpret_cast<uint16_t *>(s.Xs + 64 * NP);
  s.S = reinterpret_cast<u64 *>(s.Pt + p.parts * 64 * NB);
  s.J = s.S + p.nslm * NB;
  s.Ms = s.J + (size_t)p.nslm * 6;
  s.Av = reinterpret_cast<long long *>(s.Ms + NP);
  s.U2s = reinterpret_cast<int32_t *>(s.Av + 64 * NB);
  s.Es = s.U2s + 64 * NB;
  s.As = reinterpret_cast<uint32_t *>(s.Es + 64 * NB);
  s.nbl = s.As + 64 * NP;
  s.SG = reinterpret_cast<int32_t *>(s.nbl + (size_t)p.nslm * 6);
  s.lst = reinterpret_cast<uint16_t *>(s.SG + NP);
  s.Ps = reinterpret_cast<uint8_t *>(s.lst + p.nslm);
  return s;
}

// Cluster barrier in two halves.  The release is one warp's, behind a barrier
// of the CTA that orders the other warps' writes before it: a fence of cluster
// scope by each of 16 warps took 1750 cycles, by one 1600, and the others are
// free meanwhile.
__device__ __forceinline__ void cluster_arrive() {
  __syncthreads();
  if (threadIdx.x < 32) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  else asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Addresses in the cluster's shared memory.
__device__ __forceinline__ uint32_t smem_addr(const void *q) { return (uint32_t)__cvta_generic_to_shared(q); }
__device__ __forceinline__ uint32_t mapa(uint32_t a, int rank) {
  uint32_t o;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"(a), "r"(rank));
  return o;
}
// The neighbour word a (an nbl entry) of the column `off` bytes behind column
// 0: one of two predicated loads, so that a site's six are in flight together
// (branches between them took one round trip after another).
__device__ __forceinline__ u64 res_word(uint32_t a, uint32_t off) {
  u64 v;
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.u32 p, %2, 0;\n@p ld.shared::cluster.u64 %0, [%1];\n@!p ld.shared.u64 %0, [%1];\n}"
      : "=l"(v)
      : "r"((a & ~7u) + off), "r"(a & 1u)
      : "memory");
  return v;
}

// A colour's share of the CTA: the colour's sites, the CTA's of them, the
// first of those in the colour's list and in lst.
struct ResColour {
  int nk, nkc, kb, loff;
  uint32_t mul;  // ceil(2^32 / nkc): i / nkc = umulhi(i, mul) for the items' i, i nkc < 2^32 (SMEM bounds i)
};
__device__ __forceinline__ int res_slot(const ResColour &q, int i) {
  return q.nkc == 1 ? i : (int)__umulhi((uint32_t)i, q.mul);
}
// The random words of item (slot b, site kl) of a colour pass: planes pl apart.
struct ResPass {
  const u64 *R;
  size_t pl;
};
__device__ __forceinline__ ResPass res_pass_at(const SpResDev &p, const ResCta &me, const ResColour &q, int sweep, int k) {
  const size_t G = (size_t)p.d.NR * p.d.NB;
  return {p.R + ((size_t)sweep * p.d.V + p.d.col_off[k]) * 2 * G + (size_t)me.r * p.d.NB * q.nk + q.kb, q.nk * G};
}
__device__ __forceinline__ void res_fetch(const ResPass &a, const ResColour &q, int b, int kl, bool on, u64 r[2]) {
  if (!on) return;
  const u64 *g = a.R + b * q.nk + kl;
  r[0] = __ldg(g);
  r[1] = __ldg(g + a.pl);
}
// Whether the energy is counted in pass k of sweep sw of a tempering step.
__device__ __forceinline__ bool res_counts(const SpResDev &p, int sw, int k) {
  return p.pair_energy && k == p.d.ncol - 1 && sw == p.ptfr - 1;
}
// The random words of a thread's first item of a pass, read while the barrier
// before it is waited for (the read from L2 is about as long as the rest of a
// pass of a small job).  A pass that counts has a warp per slot, lanes over the
// colour's sites, the others their (slot, site) items over all threads.
__device__ __forceinline__ void res_prefetch(const SpResDev &p, const ResCta &me, const ResColour *col, int sweep, int k,
                                             bool counts, u64 r[2]) {
  if (sweep >= p.nsweep) return;
  const ResColour q = col[k];
  if (q.nkc <= 0) return;
  const int b = counts ? (int)threadIdx.x >> 5 : res_slot(q, threadIdx.x);
  const int kl = counts ? (int)threadIdx.x & 31 : (int)threadIdx.x - b * q.nkc;
  res_fetch(res_pass_at(p, me, q, sweep, k), q, b, kl, b < p.d.NB && kl < q.nkc, r);
}

// sv ^ J ^ neighbour of the six bond slots of a site (sp_pass_body's f).
__device__ __forceinline__ void res_bonds(const SpResDev &p, const ResShared &s, int b, int local, u64 sv, u64 f[6]) {
  const int nslm = p.nslm;
  const u64 *J = s.J + local;
  const uint32_t off = (uint32_t)(b * nslm) * 8u;
#pragma unroll
  for (int q = 0; q < 6; ++q) f[q] = res_word(s.nbl[q * nslm + local], off);
#pragma unroll
  for (int q = 0; q < 6; ++q) f[q] ^= sv ^ J[q * nslm];
}

// One colour pass over the CTA's sites of colour k (sp_pass_body's update), the
// random words of a thread's first item in r, the next one's read before an
// item is worked on.
__device__ __forceinline__ void res_pass(const SpResDev &p, const ResCta &me, const ResShared &s, const ResColour &q,
                                         int sweep, int k, u64 r[2]) {
  if (q.nkc <= 0) return;
  const ResPass a = res_pass_at(p, me, q, sweep, k);
  const int n = p.d.NB * q.nkc, nth = blockDim.x;
  int i = threadIdx.x, b = res_slot(q, i), kl = i - b * q.nkc;
#pragma unroll 1
  while (i < n) {
    const int ni = i + nth, nb = res_slot(q, ni), nkl = ni - nb * q.nkc;
    u64 x[2] = {0, 0}, f[6];
    res_fetch(a, q, nb, nkl, ni < n, x);
    const int local = s.lst[q.loff + kl];
    u64 *S = s.S + b * p.nslm + local;
    const u64 sv = *S;
    res_bonds(p, s, b, local, sv, f);
    *S = sv ^ flip_mask_id(f, r[0], r[1]);
    i = ni;
    b = nb;
    kl = nkl;
#pragma unroll
    for (int j = 0; j < 2; ++j) r[j] = x[j];
  }
}

// Asynchronous 16-byte global-to-SMEM copies (cp.async); a thread waits for
// all of its copies with cp_async_wait_all (a hardware wait) before the
// barrier that publishes them.
__device__ __forceinline__ void cp_async16(void *smem, const void *g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(smem)), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Draws of the unit for tempering step ptj into Xs.
__device__ __forceinline__ void res_stage_x(const SpResDev &p, const ResCta &me, const ResShared &s, int ptj) {
  const int NP = p.d.NB - 1;
  const int32_t *g = p.X + ((size_t)ptj * p.d.nw * p.d.NR + me.unit) * NP * 64;
  for (int t = threadIdx.x; t < NP * 16; t += blockDim.x) cp_async16(s.Xs + 4 * t, g + 4 * t);
  cp_async_commit();
}

__device__ __forceinline__ void res_count_add(u64 *P, int npl, const u64 f[6]) {
  const u64 x1 = f[0] ^ f[1] ^ f[2], y1 = (f[0] & f[1]) | (f[2] & (f[0] ^ f[1]));
  const u64 x2 = f[3] ^ f[4] ^ f[5], y2 = (f[3] & f[4]) | (f[5] & (f[3] ^ f[4]));
  const u64 z0 = x1 ^ x2, c0 = x1 & x2;
  const u64 z1 = y1 ^ y2 ^ c0, z2 = (y1 & y2) | (c0 & (y1 ^ y2));
  u64 cy = P[0] & z0;
  P[0] ^= z0;
  u64 t = P[1] ^ z1 ^ cy;
  cy = (P[1] & z1) | (cy & (P[1] ^ z1));
  P[1] = t;
  t = P[2] ^ z2 ^ cy;
  cy = (P[2] & z2) | (cy & (P[2] ^ z2));
  P[2] = t;
#pragma unroll
  for (int q = 3; q < npl; ++q) {
    const u64 h = P[q] & cy;
    P[q] ^= cy;
    cy = h;
  }
}

// A warp (one slot) sums its bit-sliced counters: in each round a lane keeps
// half of its samples and gives the other half's planes to its partner, so that
// lane l ends with samples 2 l and 2 l + 1.  Their counts go into this CTA's
// part of every CTA's Pt, or, on ladders whose Pt would not fit (61 temperatures
// in 16 CTAs), are added to the U2s of the slot's CTA, b mod ncta, where
// res_tempering fetches the sums.  (Added to every CTA's U2s, 16 times the
// atomics, 8 sweeps of the 6^2 x 30 tube with 61 temperatures and one replica
// took 530 us, now 308.)  Loops are kept rolled: the kernel runs through all its
// code once a step, and what is unrolled comes from the instruction cache again
// each time.
template <int NPL, bool PARTS>
__device__ __forceinline__ void res_count_flush(const SpResDev &p, const ResCta &me, const ResShared &s, const u64 *P,
                                                int b, int scale) {
  const int lane = threadIdx.x & 31;
  uint32_t H[NPL];
  {
    const bool up = lane & 16;
    uint32_t cy = 0;
#pragma unroll
    for (int q = 0; q < NPL; ++q) {
      const uint32_t lo = (uint32_t)P[q], hi = (uint32_t)(P[q] >> 32), a = up ? hi : lo;
      const uint32_t o = __shfl_xor_sync(0xffffffffu, up ? lo : hi, 16);
      H[q] = a ^ o ^ cy;
      cy = (a & o) | (cy & (a ^ o));
    }
  }
#pragma unroll 1
  for (int m = 8; m >= 1; m >>= 1) {  // 2 m samples kept; the bits above them are no longer used
    const int keep = lane & m ? 2 * m : 0, give = 2 * m - keep;
    uint32_t cy = 0;
#pragma unroll
    for (int q = 0; q < NPL; ++q) {
      const uint32_t a = H[q] >> keep, o = __shfl_xor_sync(0xffffffffu, H[q] >> give, m);
      H[q] = a ^ o ^ cy;
      cy = (a & o) | (cy & (a ^ o));
    }
  }
  uint32_t v = 0;
#pragma unroll
  for (int q = 0; q < NPL; ++q) v |= ((H[q] & 1u) | (H[q] & 2u) << 15) << q;
  if (!PARTS) {
    const uint32_t to = mapa(smem_addr(s.U2s + b * 64 + 2 * lane), b % p.ncta);
    for (int j = 0; j < 2; ++j)
      asm volatile("red.relaxed.cluster.shared::cluster.add.u32 [%0], %1;" ::"r"(to + 4 * j),
                   "r"(scale * (j ? v >> 16 : v & 0xFFFFu))
                   : "memory");
    return;
  }
  const uint32_t own = smem_addr(s.Pt + ((size_t)me.rank * p.d.NB + b) * 64 + 2 * lane);
#pragma unroll 2
  for (int c = 0; c < p.ncta; ++c)
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(mapa(own, c)), "r"(v) : "memory");
}

// The last colour pass of a sweep on a two-colour lattice with the energy
// counted on the way (sp.cu's update, then sp_energy_body's count): every bond
// joins a colour-0 site to a colour-1 site and both ends hold its coupling,
// so U2 is twice the unsatisfied half-edges of the colour-1 sites, all final
// once their pass has flipped them (f ^= flip).  A warp per (word, column),
// lanes over the colour's sites.
template <int NPL, bool PARTS>
__device__ __forceinline__ void res_pass_count(const SpResDev &p, const ResCta &me, const ResShared &s,
                                               const ResColour &q, int sweep, int k, u64 r[2]) {
  const ResPass a = res_pass_at(p, me, q, sweep, k);
  const int NB = p.d.NB, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
#pragma unroll 1
  for (int b = threadIdx.x >> 5; b < NB; b += nwarp) {
    u64 P[NPL];
#pragma unroll
    for (int j = 0; j < NPL; ++j) P[j] = 0;
#pragma unroll 1
    for (int kl = lane; kl < q.nkc; kl += 32) {
      u64 x[2] = {0, 0}, f[6];
      res_fetch(a, q, b, kl + 32, kl + 32 < q.nkc, x);
      const int local = s.lst[q.loff + kl];
      u64 *S = s.S + b * p.nslm + local;
      const u64 sv = *S;
      res_bonds(p, s, b, local, sv, f);
      const u64 m = flip_mask_id(f, r[0], r[1]);
      *S = sv ^ m;
#pragma unroll
      for (int e = 0; e < 6; ++e) f[e] ^= m;
      res_count_add(P, NPL, f);
#pragma unroll
      for (int j = 0; j < 2; ++j) r[j] = x[j];
    }
    res_fetch(a, q, b + nwarp, lane, b + nwarp < NB && lane < q.nkc, r);
    res_count_flush<NPL, PARTS>(p, me, s, P, b, 2);
  }
}

// Unsatisfied half-edges per (sample, slot) of the CTA's sites
// (sp_energy_body's count).
template <int NPL, bool PARTS>
__device__ __forceinline__ void res_energy(const SpResDev &p, const ResCta &me, const ResShared &s) {
  const int NB = p.d.NB, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
#pragma unroll 1
  for (int b = threadIdx.x >> 5; b < NB; b += nwarp) {
    u64 P[NPL];
#pragma unroll
    for (int q = 0; q < NPL; ++q) P[q] = 0;
#pragma unroll 1
    for (int i = lane; i < me.nsl; i += 32) {
      u64 f[6];
      res_bonds(p, s, b, i, s.S[b * p.nslm + i], f);
      res_count_add(P, NPL, f);
    }
    res_count_flush<NPL, PARTS>(p, me, s, P, b, 1);
  }
}

// One tempering step of the unit (sp_pt_body's rule and draws), by every CTA
// for itself: what it costs is one chain of NB - 1 decisions, and another
// CTA's would be a barrier away.  The counts are first summed from the CTAs'
// parts.  pt = -(beta[i+1] - beta[i]) * dE is >= 0 exactly when dE has the
// sign of -(beta[i+1] - beta[i]) (or that factor is zero); below, the exchange
// is accepted up to the m = -dE / 2 that k_sp_pt_draw found.  The walk finds the
// lanes that swap and nothing more; res_permute applies them.  `last`: the
// counts are handed back.
template <bool PARTS>
__device__ __forceinline__ void res_tempering(const SpResDev &p, const ResCta &me, const ResShared &s, bool last) {
  const SpDev &d = p.d;
  const int NB = d.NB, NP = NB - 1, ncta = p.ncta;
  const int n2 = NB * 32, scale = p.pair_energy ? 2 : 1;
  const uint32_t *Pw = reinterpret_cast<const uint32_t *>(s.Pt);
  for (int i = threadIdx.x; i < n2; i += blockDim.x) {
    int2 &U2 = reinterpret_cast<int2 *>(s.U2s)[i];
    if (PARTS) {
      int lo = 0, hi = 0;
#pragma unroll 4
      for (int c = 0; c < ncta; ++c) {
        const uint32_t v = Pw[c * n2 + i];
        lo += (int)(v & 0xFFFFu);
        hi += (int)(v >> 16);
      }
      U2 = make_int2(scale * lo, scale * hi);
    } else if (const int own = (i >> 5) % ncta; own != me.rank) {  // the others stay as they are
      int x, y;
      asm volatile("ld.shared::cluster.v2.s32 {%0, %1}, [%2];" : "=r"(x), "=r"(y) : "r"(mapa(smem_addr(&U2), own)) : "memory");
      U2 = make_int2(x, y);
    }
    if (last && me.rank == 0) {
      const int smp = 2 * (i & 31), b = i >> 5;
      int32_t *U = d.U2 + ((size_t)me.w * 64 + smp) * d.NR * NB + (size_t)me.r * NB + b;
      U[0] = U2.x;
      U[(size_t)d.NR * NB] = U2.y;
    }
  }
  __syncthreads();
  if (threadIdx.x < 64) {
    const int lane = threadIdx.x;
    const int32_t *Uo = s.U2s + lane, *xo = s.Xs + lane;
    uint32_t *Mh = reinterpret_cast<uint32_t *>(s.Ms) + (lane >> 5);
    // what does not depend on the carried configuration is read a pair ahead
    int carry = Uo[0], u1 = Uo[64], x = xo[0], sg = s.SG[0];
#pragma unroll 1
    for (int i = 0; i < NP; ++i) {
      const int n = min(i + 1, NP - 1), u1n = Uo[(n + 1) * 64], xn = xo[n * 64], sgn = s.SG[n];
      const int dE = carry - u1, m = (-dE) >> 1;  // energies are 3 V - U2
      const bool change = (sg < 0 ? dE <= 0 : dE >= 0) || (m <= x && (m != 0 || x == 0x7FFFFFFF));
      const uint32_t lanes = __ballot_sync(0xffffffffu, change);
      if ((lane & 31) == 0) Mh[2 * i] = lanes;
      carry = change ? carry : u1;
      u1 = u1n;
      x = xn;
      sg = sgn;
    }
  }
  __syncthreads();
}

// The swaps applied to the unit's acceptances, and by the last two warps, a lane
// a sample, to its energies and slot ids; with `measure`, the slots' energies
// are added to the bin's sums (sp_measure_u2_body after a tempering step).
// Needed by the next tempering step only, so it runs while the barrier behind
// the permute is waited for.
__device__ __forceinline__ void res_state(const SpResDev &p, const ResShared &s, bool measure) {
  const int NP = p.d.NB - 1, nth = blockDim.x, nt = 3 * p.d.V;
  if (threadIdx.x < nth - 64) {
    for (int i = threadIdx.x; i < NP * 64; i += nth - 64) s.As[i] += (uint32_t)(s.Ms[i >> 6] >> (i & 63)) & 1u;
    return;
  }
  const int lane = threadIdx.x & 63;
  int carry_e = nt - s.U2s[lane], e1 = nt - s.U2s[64 + lane];
  uint32_t carry_p = s.Ps[lane], p1 = s.Ps[64 + lane];
#pragma unroll 1
  for (int i = 0; i < NP; ++i) {
    const int o = i * 64 + lane, n = min(i + 2, NP) * 64 + lane, e1n = nt - s.U2s[n];
    const uint32_t p1n = s.Ps[n];
    const bool change = (s.Ms[i] >> lane) & 1ull;
    const int e = change ? e1 : carry_e;
    s.Es[o] = e;
    s.Ps[o] = (uint8_t)(change ? p1 : carry_p);
    if (measure) s.Av[o] += e;
    carry_e = change ? carry_e : e1;
    carry_p = change ? carry_p : p1;
    e1 = e1n;
    p1 = p1n;
  }
  s.Es[NP * 64 + lane] = carry_e;
  s.Ps[NP * 64 + lane] = (uint8_t)carry_p;
  if (measure) s.Av[NP * 64 + lane] += carry_e;
}

// The sums of this CTA's slots cleared, when every CTA has fetched them (behind
// the barrier of the permute).  The next counts come after another barrier: two
// colours, or the energy's own phase.
__device__ __forceinline__ void res_clear(const SpResDev &p, const ResCta &me, const ResShared &s) {
  for (int i = threadIdx.x; i < p.d.NB * 64; i += blockDim.x)
    if ((i >> 6) % p.ncta == me.rank) s.U2s[i] = 0;
}

// The accepted swaps applied to the CTA's sites (sp_permute_body), four slots
// read ahead of the chain through them.
__device__ __forceinline__ void res_permute(const SpResDev &p, const ResCta &me, const ResShared &s) {
  const int NP = p.d.NB - 1, nslm = p.nslm, nth = blockDim.x;
  for (int t = threadIdx.x; t < me.nsl; t += nth) {
    u64 *row = s.S + t;
    u64 cur = row[0];
#pragma unroll 1
    for (int b0 = 0; b0 < NP; b0 += 4) {
      u64 m[4], nxt[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int b = min(b0 + j, NP - 1);
        m[j] = s.Ms[b];
        nxt[j] = row[(b + 1) * nslm];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (b0 + j >= NP) break;
        const u64 x = (cur ^ nxt[j]) & m[j];
        row[(b0 + j) * nslm] = cur ^ x;
        cur = nxt[j] ^ x;
      }
    }
    row[NP * nslm] = cur;
  }
}

// NPL: bit planes of a warp's per-sample count, 6 * nslm < 2^NPL.
template <int NPL, bool PARTS>
__global__ void __launch_bounds__(kResThreads, 1) k_sp_resident(const __grid_constant__ SpResDev p) {
  const cg::cluster_group cl = cg::this_cluster();
  const SpDev &d = p.d;
  const int NB = d.NB, NR = d.NR, G = NR * NB, NP = NB - 1, V = d.V, ncol = d.ncol;
  const int nslm = p.nslm;
  ResCta me;
  me.rank = (int)cl.block_rank();
  me.unit = (int)(blockIdx.x / (unsigned)p.ncta);
  me.w = me.unit / NR;
  me.r = me.unit - me.w * NR;
  me.site_lo = me.rank * nslm;
  me.nsl = min(nslm, V - me.site_lo);
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ ResColour col[kResMaxColours];
  const ResShared s = res_carve(smem, p);
  const int tid = threadIdx.x, nth = blockDim.x;

  // the CTA's words and neighbour table, its sites by colour, and the unit's
  // signs, energies, slot ids, acceptances and sums
  if (tid < ncol) {
    ResColour q;
    q.nk = d.col_off[tid + 1] - d.col_off[tid];
    q.kb = p.kr[me.rank][tid];
    q.nkc = p.kr[me.rank + 1][tid] - q.kb;
    q.loff = 0;
    for (int c = 0; c < tid; ++c) q.loff += p.kr[me.rank + 1][c] - p.kr[me.rank][c];
    q.mul = q.nkc > 1 ? (uint32_t)(0xFFFFFFFFu / (uint32_t)q.nkc) + 1u : 0u;
    col[tid] = q;
  }
  const int nS = me.nsl * NB, nJ = me.nsl * 6;
  u64 *gS = d.S + ((size_t)me.w * V + me.site_lo) * G + (size_t)me.r * NB;
  for (int i = tid; i < nS; i += nth) {
    const int si = i / NB, b = i - si * NB;
    s.S[b * nslm + si] = gS[(size_t)si * G + b];
  }
  for (int i = tid; i < nJ; i += nth) {
    const int q = i % 6, si = i / 6;
    s.J[q * nslm + si] = d.J[((size_t)me.w * V + me.site_lo) * 6 + i];
    const int nbs = __ldg(d.nb + (size_t)me.site_lo * 6 + i), own = nbs / nslm;
    const uint32_t a = smem_addr(s.S + (nbs - own * nslm));
    s.nbl[q * nslm + si] = own == me.rank ? a : mapa(a, own) | 1u;
  }
  for (int k = 0, loff = 0; k < ncol; ++k) {
    const int kb = p.kr[me.rank][k], nkc = p.kr[me.rank + 1][k] - kb, off = d.col_off[k];
    for (int j = tid; j < nkc; j += nth) s.lst[loff + j] = (uint16_t)(__ldg(d.col_sites + off + kb + j) - me.site_lo);
    loff += nkc;
  }
  for (int i = tid; i < NP; i += nth) {
    const double f = -__dsub_rn(d.betas[i + 1], d.betas[i]);
    s.SG[i] = f > 0.0 ? 1 : (f < 0.0 ? -1 : 0);
  }
  const size_t row0 = (size_t)me.w * 64 * NR + me.r;  // of sample 0; samples NR rows apart
  for (int i = tid; i < 64 * NB; i += nth) {
    const size_t o = (row0 + (size_t)(i & 63) * NR) * NB + (i >> 6);
    s.Es[i] = d.E[o];
    s.Ps[i] = d.perm[o];
    s.Av[i] = (long long)d.avgE[o];
  }
  for (int i = tid; i < 64 * NB; i += nth) s.U2s[i] = 0;
  for (int i = tid; i < 64 * NP; i += nth) s.As[i] = d.acc[(row0 + (size_t)(i & 63) * NR) * NP + (i >> 6)];
  cl.sync();

  int sweep = 0, ptj = 0;
  u64 words[2] = {};
  res_prefetch(p, me, col, 0, 0, res_counts(p, 0, 0), words);
  for (int it = 0; it < p.nit; ++it)
    for (int im = 0; im < p.mesfr; ++im)
      for (int ih = 0; ih < p.houfr; ++ih) {
        res_stage_x(p, me, s, ptj);
        for (int sw = 0; sw < p.ptfr; ++sw, ++sweep)
          for (int k = 0; k < ncol; ++k) {
            if (res_counts(p, sw, k)) res_pass_count<NPL, PARTS>(p, me, s, col[k], sweep, k, words);
            else res_pass(p, me, s, col[k], sweep, k, words);
            const bool wrap = k == ncol - 1;
            if (wrap && sw == p.ptfr - 1) cp_async_wait_all();  // the step's draws
            cluster_arrive();  // before the reads: its fence would wait for them
            const int sw1 = wrap ? (sw + 1 == p.ptfr ? 0 : sw + 1) : sw, k1 = wrap ? 0 : k + 1;
            res_prefetch(p, me, col, sweep + wrap, k1, res_counts(p, sw1, k1), words);
            cluster_wait();
          }
        if (!p.pair_energy) {
          res_energy<NPL, PARTS>(p, me, s);
          cluster_arrive();
          cluster_wait();
        }
        const bool lastpt = im == p.mesfr - 1 && ih == p.houfr - 1;
        res_tempering<PARTS>(p, me, s, lastpt && it == p.nit - 1);
        res_permute(p, me, s);
        cluster_arrive();
        res_state(p, s, p.measure && lastpt);
        cluster_wait();
        if (!PARTS) {
          __syncthreads();  // res_state's reads
          res_clear(p, me, s);
        }
        ++ptj;
      }

  __syncthreads();  // res_state's writes

  // back to global memory
  for (int i = tid; i < nS; i += nth) {
    const int si = i / NB, b = i - si * NB;
    gS[(size_t)si * G + b] = s.S[b * nslm + si];
  }
  if (me.rank != 0) return;
  for (int i = tid; i < 64 * NB; i += nth) {
    const size_t o = (row0 + (size_t)(i & 63) * NR) * NB + (i >> 6);
    d.E[o] = s.Es[i];
    d.perm[o] = s.Ps[i];
    d.avgE[o] = (double)s.Av[i];
  }
  for (int i = tid; i < 64 * NP; i += nth) d.acc[(row0 + (size_t)(i & 63) * NR) * NP + (i >> 6)] = s.As[i];
  for (int i = tid; i < NP; i += nth) d.M[(size_t)me.unit * NP + i] = s.Ms[i];
  if (blockIdx.x == 0 && tid == 0) *d.ptstep += (unsigned long long)ptj;
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
// Counter planes of the energy phase's warp sums: 6 * nslm < 2^NPL.
static int res_npl(int nslm) { return 6 * nslm < (1 << 10) ? 10 : kResPlanes; }

using ResKernel = void (*)(SpResDev);
static ResKernel res_kernel(int npl, bool parts) {
  if (npl == 10) return parts ? k_sp_resident<10, true> : k_sp_resident<10, false>;
  return parts ? k_sp_resident<kResPlanes, true> : k_sp_resident<kResPlanes, false>;
}

cudaError_t sp_res_setup() {
  cudaError_t e = cudaSuccess;
  for (int npl : {10, kResPlanes})
    for (bool parts : {false, true}) {
      const ResKernel k = res_kernel(npl, parts);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResSmem);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_sp_ctr_chain, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             64 * (int)(sizeof(ea_hq) + sizeof(ea_xoshiro)));
  return e;
}

static cudaLaunchConfig_t res_config(int ncta, int units, size_t smem, cudaStream_t st, cudaLaunchAttribute *at) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(ncta * units));
  cfg.blockDim = dim3(kResThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = (unsigned)ncta;
  at->val.clusterDim.y = 1;
  at->val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

// Whether a unit's share of the widest split (sites split evenly over 16 CTAs)
// fits one CTA's shared memory, and the job's words those of kResMaxCta.
bool sp_res_fits(int L, int Lz, int nw, int NR, int NB) {
  if (NB < 2 || L < 1 || Lz < 1) return false;
  const long long V = (long long)L * L * Lz, nslm = (V + kResMaxCta - 1) / kResMaxCta;
  if (nslm > kResMaxSites || 8 * V * nw * NR * NB > (long long)kResMaxCta * 227 * 1024) return false;
  return res_smem_bytes((int)nslm, NB, 0) <= kResSmem;
}

// The CTAs of a unit's cluster (sites split into equal runs, at most 16): the
// most whose clusters the GPU can hold at once for all units, else the fewest
// whose share fits; none when no share does.  (Steps of the 6^2 x 24 tube, two
// units: 16, 12, 8 CTAs a unit 701, 729, 759 us a bin of 64, 6 and 4 856 and
// 977 before the last changes to the kernel.)
bool sp_res_plan(const SpDev &d, const int32_t *col_sites, SpResPlan &pl) {
  if (d.ncol < 1 || d.ncol > kResMaxColours || !sp_res_fits(d.L, d.Lz, d.nw, d.NR, d.NB)) return false;
  const int units = d.nw * d.NR;
  int last = 0;
  bool found = false;
  for (int want = std::min(kResMaxCta, d.V); want >= 1; --want) {
    const int nslm = (d.V + want - 1) / want, ncta = (d.V + nslm - 1) / nslm;
    if (ncta == last) continue;
    last = ncta;
    int parts = ncta;
    size_t smem = res_smem_bytes(nslm, d.NB, parts);
    if (smem > kResSmem) smem = res_smem_bytes(nslm, d.NB, parts = 0);
    if (nslm > kResMaxSites || smem > kResSmem) break;
    const int npl = res_npl(nslm);
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = res_config(ncta, units, smem, nullptr, &at);
    int nclusters = 0;
    const cudaError_t e = cudaOccupancyMaxActiveClusters(&nclusters, res_kernel(npl, parts > 0), &cfg);
    if (e != cudaSuccess) {
      cudaGetLastError();
      continue;
    }
    if (nclusters < 1) continue;
    found = true;
    for (int c = 0; c <= ncta; ++c)
      for (int k = 0; k < d.ncol; ++k) {
        const int32_t *b = col_sites + d.col_off[k], *e2 = col_sites + d.col_off[k + 1];
        pl.kr[c][k] = (int)(std::lower_bound(b, e2, c * nslm) - b);
      }
    pl.ncta = ncta;
    pl.nslm = nslm;
    pl.parts = parts;
    pl.npl = npl;
    pl.smem = smem;
    if (nclusters >= units) break;
  }
  return found;
}

size_t sp_res_launch_sweeps(size_t V, size_t G, const ea_cadence *cad) {
  const size_t spi = (size_t)cad->mesfr * cad->houfr * cad->ptfr, bytes_sweep = 16 * V * G;
  if (cad->cluster) {
    // one launch per block of houfr x ptfr sweeps between two cluster moves
    const size_t blk = (size_t)cad->houfr * cad->ptfr;
    return blk >= (size_t)kResMinBlock && blk * bytes_sweep <= ((size_t)256 << 20) ? blk : 0;
  }
  if (spi * bytes_sweep > ((size_t)256 << 20)) return 0;
  const size_t its = std::max<size_t>(1, ((size_t)16 << 20) / (bytes_sweep * spi));
  return std::min(its, (size_t)std::max(cad->itmax, 1)) * spi;
}

cudaError_t sp_res_chunk(const SpResDev &p, const SpResPlan &pl, int npass, uint4 *ctrs, cudaStream_t st) {
  const SpDev &d = p.d;
  cudaError_t e = sp_launch_ctr_chain(d, npass, ctrs, st);
  if (e != cudaSuccess) return e;
  const int nsweep = npass / d.ncol;
  const long long n = (long long)nsweep * d.V * d.NR * d.NB;
  k_sp_draw<<<(unsigned)((n + kDrawItems - 1) / kDrawItems), kDrawThreads, 0, st>>>(d, nsweep, ctrs, const_cast<u64 *>(p.R));
  const int npt = p.nit * p.mesfr * p.houfr;
  const long long nx = (long long)npt * d.nw * d.NR * (d.NB - 1) * 64;
  if (nx > 0) k_sp_pt_draw<<<(unsigned)((nx + 255) / 256), 256, 0, st>>>(d, npt, const_cast<int32_t *>(p.X));
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute at;
  const cudaLaunchConfig_t cfg = res_config(pl.ncta, d.nw * d.NR, pl.smem, st, &at);
  return cudaLaunchKernelEx(&cfg, res_kernel(pl.npl, pl.parts > 0), p);
}

}  // namespace eagb
