// kernels.cuh -- device-side job descriptor and kernel launchers.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "eagb.h"

namespace eagb {

// Division by a value fixed at set-up, exact for every 32-bit numerator: one
// multiply-high, an add and two shifts (the round-up method for unsigned
// division by invariant integers, Granlund & Montgomery, PLDI 1994).
struct FastDiv {
  uint32_t d = 1, m = 1, s1 = 0, s2 = 0;
  void set(uint32_t dd) {
    d = dd ? dd : 1;
    int l = 0;
    while ((1ull << l) < d) ++l;
    m = (uint32_t)((((1ull << 32) * ((1ull << l) - d)) / d) + 1);
    s1 = l < 1 ? l : 1;
    s2 = l > 1 ? l - 1 : 0;
  }
#ifdef __CUDACC__
  __device__ __forceinline__ uint32_t div(uint32_t n) const {
    const uint32_t t = __umulhi(m, n);
    return (t + ((n - t) >> s1)) >> s2;
  }
  __device__ __forceinline__ uint32_t mod(uint32_t n) const { return n - div(n) * d; }
#endif
};

// Everything a kernel needs about one job, by value (kernel parameter).
// All arrays live in device memory, in the reference's layouts.
struct JobDev {
  int NB, NR, ns, half, msc_l, msc_s, msc_lz, L, Lz, V, bc;
  unsigned long long *spins;        // [s][parity][clone][half][rep]
  const unsigned long long *J;      // [s][parity][dir][half]
  const int32_t *nbidx;             // [parity][dir][half]
  const uint8_t *nbflag;            // [parity][half]
  const unsigned long long *cum;    // [NB][256] thresholds
  const uint8_t *pre;               // [NB][pre_stride(pre_bits)] pre-search
  int pre_bits;
  uint8_t *wctb, *wbtc;             // [s][rep][NB]
  uint4 *ctr;                       // [NR] Philox counters of the last half-sweep
  uint4 *ctrs;                      // [kCtrPasses][NR] those of the half-sweeps drawn ahead
  const uint32_t *keys;             // [NR]
  ea_hq *prc;                       // [NR]
  ea_xoshiro *xo;                   // [NR]
  long long *iter;                  // half-sweep counter (device scalar)
  uint32_t jobid;
  int ntiles, kt;
  int nsplit;                       // CTAs that share a tile of the half-sweep
  int32_t *E;                       // energies: s NR NB + rep e_r + clone e_c
  int e_r, e_c;                     // (1, NR): a tile's sums of the replicas of a clone are neighbours
  // parallel tempering
  ea_hq *pt;                        // [s][rep]
  const double *betas;              // [NB]
  const double *exptab;             // glibc exp table
  const int32_t *expoff;            // [NB]
  double *acc, *att, *accraw;       // [s][rep][NB-1]
  unsigned long long *inexact;      // decisions decided outside the table (u == 0)
  // measurements
  double *avgE;                     // [s][rep][NB]
  uint8_t *hist;                    // [s][rep][maxit][NB]
  int maxit_trw;
  // Houdayer
  ea_hq *rc;
  int32_t *pairs;                   // [2 groups][2]
  unsigned long long *Q;            // [s][nclust][2][half] overlap words
  uint32_t *label;                  // [s][nclust][V] natural order
  uint32_t *sel;                    // [s][nclust][V / 32] cluster selection bits, natural order
  int nclust;
  // cluster coins (xorwow.cuh): [U < 0.5] of the move's uniforms, both groups
  uint32_t *xw_bits;                // bit (xw_pos[0] mod 32) + i: coin i of the move
  uint32_t *xw_state;               // [segment][d, v0..v4][4096] generator states at the next move's rows
  const uint32_t *xw_jump;          // advances a state from its segment's end to the next move's segment
  unsigned long long *xw_pos;       // first position of this move, of the next; blocks of its start that are done
  unsigned long long xw_n;          // coins of a move: 2 groups x [s][NB][V]
  int xw_seg, xw_w;                 // segments, rows of a segment
  // x coordinate against which site 0 tests its periodic -x bond.  The
  // reference computes (ltid-1+nx)%nx with a 32-bit ltid (HoudayerXEA.cu:96),
  // i.e. (2^32-1+L) mod L, which differs from L-1 unless L is a power of two;
  // the union itself still joins sites 0 and L-1 (HoudayerXEA.cu:288).
  int cc_xq;
  // dividers of the site <-> multispin-word maps
  FastDiv fd_L, fd_S, fd_ml, fd_mlz, fd_hl, fd_nclust;
  int cc_D, cc_nslab;               // planes of a slab, slabs (see CcShape)
};

// Half-sweeps (colour passes) whose counters are drawn by one launch.
constexpr int kCtrPasses = 512;
// Planes of up to this many sites are labelled in SMEM.
constexpr int kSlabPlane = 8192;

// Shared memory of the one-CTA-per-lattice selection and flip (V/8 bytes of
// selection bits + the 64 bit offsets); larger lattices take the two-kernel
// path (global selection bits).
constexpr size_t kFlipMaxSmem = 200 * 1024;
size_t flip_smem_bytes(const JobDev &j);

// How a move labels a job's lattices: whole (a CTA a lattice does the whole
// move), in slabs of `planes` z planes, or (planes = 0) in global memory.
struct CcShape {
  bool whole;
  int planes, nslab;
  int threads;
  size_t smem;
};
CcShape cc_shape(const JobDev &j);

// Fills the dividers of j from its sizes (nclust included).
void set_dividers(JobDev &j);

// Tile width (half-sites per CTA) of the fused sweep kernel.
int sweep_kt(const JobDev &j);
size_t sweep_smem_bytes(const JobDev &j);
constexpr size_t kSweepMax = 227 * 1024 - 64;  // less the kernel's static SMEM
// Bits of the pre-search tables, so that two CTAs of a half-sweep fit an SM:
// the more, the fewer threshold searches (0.22 steps a byte with 8 bits, 0.04
// with 11, on a ladder of 32 temperatures from 0.7 to 1.6: a half-sweep of the
// 24^2 x 192 tube takes 104, 100, 96, 93 us with 8, 9, 10, 11 bits, of 8^2 x 16
// 12.5, 11.1, 10.4, 9.5).
inline int sweep_pre_bits(int NB) { return NB <= 40 ? 11 : NB <= 72 ? 10 : NB <= 128 ? 9 : 8; }
// Dynamic SMEM of a fused half-sweep CTA: the flip mask's two words of every
// triple of the tile and the queues of their halves, the pre-search tables
// and the tile's neighbour records (KT x 8 ints).
inline size_t sweep_smem_for(int NB, int NR, int KT) {
  return (size_t)NB * KT * NR * (16 + 8) + (size_t)NB * (((1 << sweep_pre_bits(NB)) + 16) & ~15) + (size_t)KT * 8 * 4;
}

// Counters of npass half-sweeps (even, odd, even, ...) into j.ctrs.
cudaError_t launch_ctr_chain(const JobDev &j, int npass, cudaStream_t st);
// Half-sweep `pass` of the counters drawn last.  energy: kEnergyZero clears the
// energies (before the odd half-sweep that adds them up), kEnergyAdd adds.
enum { kEnergyNone = 0, kEnergyAdd = 1, kEnergyZero = 2 };
cudaError_t launch_sweep(const JobDev &j, int pass, int parity, int energy, cudaStream_t st);
cudaError_t launch_energy(const JobDev &j, cudaStream_t st);
cudaError_t launch_pt(const JobDev &j, cudaStream_t st);
cudaError_t launch_measure(const JobDev &j, int itm, cudaStream_t st);
// The move's kernels of both groups, after launch_move_start.
cudaError_t launch_houdayer(const JobDev &j, cudaStream_t st);
// Those of one group of a job that is not labelled whole.
cudaError_t launch_houdayer_group(const JobDev &j, int group, cudaStream_t st);
cudaError_t houdayer_setup();

}  // namespace eagb
