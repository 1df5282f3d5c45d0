// kernels_dev.cuh -- device code of the hot path: helpers and the body of each
// kernel as a function of (job, block coordinates).  The one-job kernels
// (kernels.cu) and the persistent batched kernels (batch.cu) both call these
// bodies, so a job gives the same words alone and in a batch.
//
// The work is integer bit-slicing, so tensor cores play no part; the kernels
// are bound by the integer pipes (Philox + threshold search) and by HBM/L2
// traffic on the spin words.  Reference behaviour is cited per kernel (paths
// relative to the reference project).
#pragma once
#include "kernels.cuh"
#include "runs.cuh"
#include "xorwow.cuh"

namespace eagb {

typedef unsigned long long u64;

// ---------------------------------------------------------------------------
// Philox counter of a half-sweep (fill_bits.h:47-68): advance the replica's
// xoshiro256++ and Parisi-Rapuano generators once and place 52 entropy bits
// around the time counter and the job id.  One thread per replica.
// ---------------------------------------------------------------------------
__device__ __forceinline__ u64 d_rotl(u64 x, int k) { return (x << k) | (x >> (64 - k)); }

__device__ __forceinline__ u64 d_hq_next(ea_hq *h) {
  const uint8_t ip = h->ip, ip1 = h->ip1, ip2 = h->ip2, ip3 = h->ip3;
  const u64 a = h->ira[ip1] + h->ira[ip2];
  h->ira[ip] = a;
  h->PR = a ^ h->ira[ip3];
  h->zseed = h->zseed * 3202034522624059733ULL + 1;
  h->final = h->zseed + h->PR;
  h->ip = ip + 1; h->ip1 = ip1 + 1; h->ip2 = ip2 + 1; h->ip3 = ip3 + 1;
  return h->final;
}

// One step of a replica's two generators and the counter it gives for time
// counter `iter` (the state may live in global or shared memory).
__device__ __forceinline__ uint4 next_counter(ea_xoshiro *x, ea_hq *h, long long iter, int parity, uint32_t jobid) {
  u64 s0 = x->s[0], s1 = x->s[1], s2 = x->s[2], s3 = x->s[3];
  const u64 xf = d_rotl(s0 + s3, 23) + s0;
  const u64 t = s1 << 17;
  s2 ^= s0; s3 ^= s1; s1 ^= s2; s0 ^= s3; s2 ^= t; s3 = d_rotl(s3, 45);
  x->s[0] = s0; x->s[1] = s1; x->s[2] = s2; x->s[3] = s3; x->t = t; x->final = xf;
  const u64 pf = d_hq_next(h);
  u64 e = (pf + xf) >> 12;
  uint4 c;
  c.y = (uint32_t)((u64)iter >> 15);
  c.x = (uint32_t)((((u64)iter & 32767ULL) << 3) | ((u64)(parity & 1) << 2));
  c.x |= (uint32_t)((e & 0x3FFFULL) << 18); e >>= 14;
  c.y |= (uint32_t)((e & 0x7FULL) << 25); e >>= 7;
  c.z = (uint32_t)((e & 0x1FFFULL) << 19); e >>= 13;
  c.w = ((uint32_t)(e << 14)) | jobid;
  return c;
}

// Counters of npass consecutive half-sweeps (colour passes), one thread per
// replica with the states staged in SMEM: a launch of one step alone is a 4 us
// link in a small job's chain of kernels, a step here takes half a
// microsecond (a block of 256 threads: 32 took 30 us to stage 8 replicas).
// parity(pass, time counter) is the counter's parity bit.
// sm: NR x (sizeof(ea_hq) + sizeof(ea_xoshiro)) bytes.
template <class Parity>
__device__ __forceinline__ void ctr_chain_body(ea_hq *prc, ea_xoshiro *xo, long long *iter, uint32_t jobid, int NR,
                                               int npass, uint4 *ctrs, uint4 *last, unsigned char *sm, Parity parity) {
  ea_hq *hs = reinterpret_cast<ea_hq *>(sm);
  ea_xoshiro *xs = reinterpret_cast<ea_xoshiro *>(hs + NR);
  const int nh = NR * (int)(sizeof(ea_hq) / 8), nx = NR * (int)(sizeof(ea_xoshiro) / 8);
  u64 *h64 = reinterpret_cast<u64 *>(hs), *x64 = reinterpret_cast<u64 *>(xs);
  u64 *hg = reinterpret_cast<u64 *>(prc), *xg = reinterpret_cast<u64 *>(xo);
#pragma unroll 8
  for (int i = threadIdx.x; i < nh; i += blockDim.x) h64[i] = hg[i];
  for (int i = threadIdx.x; i < nx; i += blockDim.x) x64[i] = xg[i];
  const long long iter0 = *iter;
  __syncthreads();
  const int r = threadIdx.x;
  if (r < NR) {
    uint4 c = make_uint4(0u, 0u, 0u, 0u);
    for (int p = 0; p < npass; ++p) {
      c = next_counter(xs + r, hs + r, iter0 + p, parity(p, iter0 + p), jobid);
      ctrs[(size_t)p * NR + r] = c;
    }
    if (npass > 0) last[r] = c;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nh; i += blockDim.x) hg[i] = h64[i];
  for (int i = threadIdx.x; i < nx; i += blockDim.x) xg[i] = x64[i];
  if (threadIdx.x == 0) *iter = iter0 + npass;
}
inline size_t ctr_smem(int NR) { return (size_t)NR * (sizeof(ea_hq) + sizeof(ea_xoshiro)); }
constexpr int kCtrThreads = 256;

__device__ __forceinline__ void fill_bits_body(const JobDev &j, int parity) {
  const int r = threadIdx.x;
  const long long iter = *j.iter;
  __syncthreads();
  if (r < j.NR) j.ctr[r] = next_counter(j.xo + r, j.prc + r, iter, parity, j.jobid);
  if (r == 0) *j.iter = iter + 1;
}

// ---------------------------------------------------------------------------
// Random words: Philox4x32-10 (main.cu:996-1043), the post-mix of
// main.cu:1045-1060, and for each of the four 64-bit keys the first byte n with
// R < cum[n] (the heat-bath thresholds); this is the function the reference's
// pre-search + bisection computes (main.cu:1063-1078).  Here the pre-search is
// indexed by the top 8 to 11 bits, so that every temperature's table fits in
// SMEM.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void philox10(uint32_t &v0, uint32_t &v1, uint32_t &v2, uint32_t &v3, uint32_t k0,
                                         uint32_t k1) {
#pragma unroll
  for (int i = 0; i < 10; ++i) {
    if (i) { k0 += 0x9E3779B9u; k1 += 0xBB67AE85u; }
    const u64 p0 = (u64)0xD2511F53u * v0;
    const u64 p1 = (u64)0xCD9E8D57u * v2;
    const uint32_t n0 = (uint32_t)(p1 >> 32) ^ v1 ^ k0;
    const uint32_t n2 = (uint32_t)(p0 >> 32) ^ v3 ^ k1;
    v1 = (uint32_t)p1; v3 = (uint32_t)p0; v0 = n0; v2 = n2;
  }
}

// Threshold search of a random byte with the pre-search of presearch
// (host.cpp): a key in bucket t = hi >> shift (shift = 32 - bits) has its byte
// in [pre[t], pre[t+1]]; thresholds through the read-only cache.  Narrower
// buckets leave a bisection to fewer keys: 0.04 steps a byte on the benchmark
// sets with 11 bits against 0.22 with 8, and a warp waits for its slowest lane
// at each search.
__device__ __forceinline__ uint32_t lut_byte_pre(uint32_t hi, uint32_t lo, const u64 *cum, const uint8_t *pre, int shift) {
  const u64 R = ((u64)hi << 32) | lo;
  const uint32_t t = hi >> shift;
  uint32_t a = pre[t], b = pre[t + 1];
  while (a < b) {
    const uint32_t m = (a + b) >> 1;
    if (R < __ldg(cum + m)) b = m; else a = m + 1;
  }
  return a;
}
__device__ __forceinline__ uint32_t lut_byte11(uint32_t hi, uint32_t lo, const u64 *cum, const uint8_t *pre) {
  return lut_byte_pre(hi, lo, cum, pre, 21);
}

// One random word from a Philox counter: the four keys' bytes by `byte`
// (a threshold search), rotated as the post-mix says.
template <class Byte>
__device__ __forceinline__ uint32_t rnd_word_by(uint32_t cx, uint32_t cy, uint32_t cz, uint32_t cw, uint32_t key,
                                                uint32_t tid, Byte byte) {
  uint32_t v0 = cx, v1 = cy, v2 = cz, v3 = cw;
  philox10(v0, v1, v2, v3, tid, key);
  const uint32_t h = v0 ^ v2, l = v1 ^ v3;
  const uint32_t s0 = __funnelshift_l(v0, v1, 17) ^ h ^ __funnelshift_l(l, h, 21);
  const uint32_t s1 = __funnelshift_l(v1, v0, 17) ^ l ^ (l << 21);
  const uint32_t s2 = __funnelshift_l(l, h, 28);
  const uint32_t s3 = __funnelshift_l(h, l, 28);
  const uint32_t rot = (s0 + v1 + s2 + v3) >> 27;
  const uint32_t bb = byte(v0, s0) | (byte(v1, s1) << 8) | (byte(v2, s2) << 16) | (byte(v3, s3) << 24);
  return __funnelshift_l(bb, bb, rot);  // rotate left; rot 0 leaves the word as it is
}

// ---------------------------------------------------------------------------
// Multispin neighbour words: bit rotation across the sub-block wrap
// (main.cu:1154-1190) and the OBC fake bond patch (main.cu:1460-1472).
// ---------------------------------------------------------------------------
__device__ __forceinline__ u64 rot_dir(int d, u64 o) {
  switch (d) {
    case 0: return (o & 0x1111111111111111ull) << 3 | (o & ~0x1111111111111111ull) >> 1;
    case 1: return (o & 0x000F000F000F000Full) << 12 | (o & ~0x000F000F000F000Full) >> 4;
    case 2: return (o & 0x000000000000FFFFull) << 48 | (o & ~0x000000000000FFFFull) >> 16;
    case 3: return (o & 0x8888888888888888ull) >> 3 | (o & ~0x8888888888888888ull) << 1;
    case 4: return (o & 0xF000F000F000F000ull) >> 12 | (o & ~0xF000F000F000F000ull) << 4;
    default: return (o & 0xFFFF000000000000ull) >> 48 | (o & ~0xFFFF000000000000ull) << 16;
  }
}
#define MASK_TOP (~0xFFFF000000000000ull)  // keeps bz < 3 (main.cu:1207)
#define MASK_BOT (~0x000000000000FFFFull)  // keeps bz > 0 (main.cu:1206)

__device__ __forceinline__ void gather6(const u64 *oth, const int *nb, int flags, int parity, bool obc, int NR,
                                        u64 n[6]) {
#pragma unroll
  for (int d = 0; d < 6; ++d) {
    u64 w = oth[(size_t)nb[d] * NR];
    if ((flags >> d) & 1) w = rot_dir(d, w);
    n[d] = w;
  }
  if (obc) {
    const u64 aux = parity == 0 ? n[1] : n[4];
    if (flags & 0x40) n[2] = (n[2] & MASK_TOP) | (aux & ~MASK_TOP);
    if (flags & 0x80) n[5] = (n[5] & MASK_BOT) | (aux & ~MASK_BOT);
  }
}

// Bit-sliced local field and Metropolis flip mask (main.cu:1474-1506): flip with
// probability min(1, p^(3-c)) where c counts satisfied-minus-unsatisfied pairs.
// From the random words b0, b1, b2 it takes id2 = b0 & b1 and id1 = (b0 ^ id2)
// | (id2 & b2).
__device__ __forceinline__ u64 flip_mask_id(const u64 f[6], u64 id1, u64 id2) {
  u64 k1 = f[0] ^ f[1], k2 = f[0] & f[1];
  const u64 j1 = k1 ^ f[2], j2 = k2 ^ (k1 & f[2]);
  k1 = f[3] ^ f[4]; k2 = f[3] & f[4];
  const u64 j3 = k1 ^ f[5], j4 = k2 ^ (k1 & f[5]);
  const u64 j24 = j2 | j4;
  return (j1 & j3 & id1) | ((j24 | id2) & (j1 | j3 | id1)) | ((j2 & j4) | (j24 & id2));
}
// ---------------------------------------------------------------------------
// The flip mask's two words (flip_mask_id) of ntrip random triples, drawn by a
// CTA: id1 = (b0 ^ id2) | (id2 & b2), id2 = b0 & b1.  Where a 32-bit half of b0
// is 0 that half of b1 and b2 does not matter, nor that of b2 where b0 & b1 is
// 0, and b0's bits are rare on a tempering ladder (exp(-4 beta)): the halves
// that need a draw are queued and drawn by whichever threads are free, 3.2 to
// 3.3 draws a triple instead of 6 (counter-based: the ones made are the same).
// item(t, c, key, tp, b): the Philox counter, key and index of triple t and its
// temperature, false if it has none; byte(b, hi, lo): the threshold search.
// queue: 4 ntrip entries, ntrip <= 2^14; cnt: 2.  All in SMEM; ends with a
// barrier.
template <class Item, class Byte>
__device__ __forceinline__ void draw_ids(int ntrip, Item &&item, Byte &&byte, u64 *id1, u64 *id2, uint16_t *queue, int *cnt) {
  uint32_t *i1 = reinterpret_cast<uint32_t *>(id1), *i2 = reinterpret_cast<uint32_t *>(id2);
  uint16_t *qa = queue, *qb = queue + 2 * ntrip;
  const int lane = threadIdx.x & 31, i00 = threadIdx.x - lane;
  const unsigned below = (1u << lane) - 1u;
  if (threadIdx.x == 0) cnt[0] = cnt[1] = 0;
  __syncthreads();
  auto word = [&](int q, int t) -> uint32_t {
    uint4 c;
    uint32_t key, tp;
    int b;
    if (!item(t, c, key, tp, b)) return 0u;
    return rnd_word_by(c.x + q, c.y, c.z + tp, c.w, key, tp, [&](uint32_t hi, uint32_t lo) { return byte(b, hi, lo); });
  };
  auto push = [&](uint16_t *qu, int *n, bool on, int i) {
    const unsigned m = __ballot_sync(0xffffffffu, on);
    int base = 0;
    if (lane == 0 && m) base = atomicAdd(n, __popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (on) qu[base + __popc(m & below)] = (uint16_t)i;
  };
  // i = 2 t + h: half h (0: the high one) of triple t
#pragma unroll 1
  for (int i0 = i00; i0 < 2 * ntrip; i0 += blockDim.x) {
    const int i = i0 + lane;
    uint32_t w = 0;
    if (i < 2 * ntrip) {
      w = word(i & 1, i >> 1);
      i1[i ^ 1] = w;
      i2[i ^ 1] = 0;
    }
    push(qa, cnt, w != 0, i);
  }
  __syncthreads();
  const int n1 = cnt[0];
#pragma unroll 1
  for (int i0 = i00; i0 < n1; i0 += blockDim.x) {
    const bool on = i0 + lane < n1;
    const int i = on ? qa[i0 + lane] : 0;
    uint32_t a = 0;
    if (on) {
      const uint32_t b0 = i1[i ^ 1];
      a = b0 & word(2 + (i & 1), i >> 1);
      i2[i ^ 1] = a;
      i1[i ^ 1] = b0 ^ a;
    }
    push(qb, cnt + 1, a != 0, i);
  }
  __syncthreads();
  const int n2 = cnt[1];
#pragma unroll 1
  for (int q = threadIdx.x; q < n2; q += blockDim.x) {
    const int i = qb[q];
    i1[i ^ 1] |= i2[i ^ 1] & word(4 + (i & 1), i >> 1);
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// Fused half-sweep.  A CTA owns KT half-sites of one parity.  It stages every
// temperature's pre-search in SMEM -- the thresholds
// themselves, rarely needed past the pre-search, are read through the
// read-only cache, which keeps a CTA's SMEM small -- draws the random words
// of each (beta, half-site, replica) once -- they are shared by all samples, as
// the reference's random buffer has no sample axis (main.cu:1430) -- and then
// updates every (sample, clone, half-site, replica) word of its tile, picking
// the words of the clone's current temperature.  What bounds it is issue and
// latency (ALU pipe 60 % busy, 41 % of the warps); the draws were about half of
// a CTA's time.  Six words a thread one after another through an
// 8-bit pre-search, a chain of threshold reads behind most of them, took 104 us
// a half-sweep of the 24^2 x 192 tube (32 temperatures, 8 replicas, 31
// samples), draw_ids and 11 bits take 93; 16^2 x 48 with 40 temperatures
// 27 -> 21 us, 16^2 x 64 with 24 17.4 -> 13.1, 8^2 x 16 11.9 -> 9.6.
// The random word indices
// depend only on (beta, half-site, replica, counter), never on the launch
// shape.  A tile of a job too small to fill the GPU is shared by nsplit CTAs,
// each drawing the words and updating its share of the (sample, clone) pairs
// (`part` of nsplit).
// With energy = kEnergyAdd it also adds, per (sample, clone, replica),
// the energy of the updated words (each bond has exactly one end on each
// parity) to E, one atomic addition per tile (integers: the order does not
// matter); kEnergyZero clears E, which the half-sweep before that one does.
// Per-tile partial sums and a reduction kernel took 34 us a sweep on the large
// tube and a link of 3 to 10 us in a small job's chain.
// ---------------------------------------------------------------------------
// stage = false: the pre-search tables of this job are already in SMEM (the
// block's previous tile was of the same job).
template <int NR, int KT, bool UPDATE>
__device__ __forceinline__ void sweep_body(const JobDev &j, const uint4 *ctr, int blk, int parity, int energy,
                                           unsigned char *smem, bool stage = true) {
  const int tile = blk / j.nsplit, part = blk - tile * j.nsplit;
  const int NB = j.NB, half = j.half;
  const int ntrip = UPDATE ? NB * KT * NR : 0, stride = UPDATE ? (((1 << j.pre_bits) + 16) & ~15) : 0;
  u64 *s_id1 = reinterpret_cast<u64 *>(smem), *s_id2 = s_id1 + ntrip;
  uint16_t *s_queue = reinterpret_cast<uint16_t *>(s_id2 + ntrip);
  uint8_t *s_pre = reinterpret_cast<uint8_t *>(s_queue + 4 * ntrip);
  int *s_nb = reinterpret_cast<int *>(s_pre + (size_t)NB * stride);
  __shared__ int s_cnt[2];
  const int k0 = tile * KT;
  const int tid = threadIdx.x, nth = blockDim.x;

  if (energy == kEnergyZero)
    for (int i = blk * nth + tid; i < j.ns * NB * NR; i += j.ntiles * j.nsplit * nth) j.E[i] = 0;
  if (UPDATE && stage) {
    const uint4 *ps = reinterpret_cast<const uint4 *>(j.pre);
    uint4 *pd = reinterpret_cast<uint4 *>(s_pre);
    for (int i = tid; i < NB * (stride / 16); i += nth) pd[i] = ps[i];
  }
  if (tid < KT * 8) {
    const int kk = tid >> 3, f = tid & 7, k = k0 + kk;
    int v = 0;
    if (k < half) v = f < 6 ? j.nbidx[(parity * 6 + f) * half + k] : (f == 6 ? (int)j.nbflag[parity * half + k] : 0);
    s_nb[tid] = v;
  }
  __syncthreads();

  if (UPDATE) {
    draw_ids(
        ntrip,
        [&](int t, uint4 &c, uint32_t &key, uint32_t &tp, int &b) {
          const int r = t % NR, kk = (t / NR) % KT, k = k0 + kk;
          b = t / (NR * KT);
          tp = (uint32_t)((b * half + k) * NR + r);
          c = ctr[r];
          key = j.keys[r];
          return k < half;
        },
        [&](int b, uint32_t hi, uint32_t lo) {
          return lut_byte_pre(hi, lo, j.cum + b * 256, s_pre + b * stride, 32 - j.pre_bits);
        },
        s_id1, s_id2, s_queue, s_cnt);
  }

  // Update phase.  Lanes form groups of G = KT*NR; a lane keeps its
  // (half-site, replica) and its neighbour record for the whole loop, and a
  // group walks a contiguous run of (sample, clone) pairs, clone fastest, so
  // the G lanes of a group touch G consecutive words of one clone array and a
  // lane loads the six coupling words of its (sample, half-site) once per
  // sample rather than once per word.
  constexpr int G = KT * NR;
  const size_t wpc = (size_t)half * NR, wpp = wpc * NB;
  const int lg = tid % G, grp = tid / G, ngrp = nth / G;
  const int r = lg % NR, kk = lg / NR, k = k0 + kk;
  const bool kvalid = k < half;
  const bool obc = j.bc != EA_PBC;
  int nb[6];
#pragma unroll
  for (int d = 0; d < 6; ++d) nb[d] = s_nb[kk * 8 + d];
  const int nflags = s_nb[kk * 8 + 6];
  const int all = j.ns * NB, share = (all + j.nsplit - 1) / j.nsplit;
  const int nsc = min(all, (part + 1) * share), iters = (share + ngrp - 1) / ngrp;
  const int sc0 = part * share + grp * iters;
  int s = sc0 / NB, c = sc0 - s * NB, js = -1;
  u64 jw[6];
  for (int it = 0, sc = sc0; it < iters; ++it, ++sc) {
    const bool valid = kvalid && sc < nsc;
    int e = 0;
    if (valid) {
      u64 *base = j.spins + (size_t)s * 2 * wpp + (size_t)c * wpc;
      u64 *tgt = base + (size_t)parity * wpp + (size_t)k * NR + r;
      const u64 *oth = base + (size_t)(1 - parity) * wpp + r;
      if (s != js) {
        const u64 *Jp = j.J + ((size_t)s * 2 + parity) * 6 * half + k;
#pragma unroll
        for (int d = 0; d < 6; ++d) jw[d] = __ldg(Jp + (size_t)d * half);
        js = s;
      }
      const u64 sv = *tgt;
      u64 n[6];
      gather6(oth, nb, nflags, parity, obc, NR, n);
      u64 f[6];
#pragma unroll
      for (int d = 0; d < 6; ++d) f[d] = sv ^ jw[d] ^ n[d];
      u64 fl = 0;
      if (UPDATE) {
        const int beta = j.wbtc[(s * NR + r) * NB + c];
        const int o = (beta * KT + kk) * NR + r;
        fl = flip_mask_id(f, s_id1[o], s_id2[o]);
        *tgt = sv ^ fl;
      }
      if (energy == kEnergyAdd) {
        int le = 0;
#pragma unroll
        for (int d = 0; d < 6; ++d) le += __popcll(f[d] ^ fl);
        e = 6 * 64 - 2 * le;
      }
    }
    if (energy == kEnergyAdd) {
#pragma unroll
      for (int m = NR; m < G; m <<= 1) e += __shfl_xor_sync(0xffffffffu, e, m);
      if (valid && kk == 0) atomicAdd(j.E + (size_t)s * NR * NB + r * j.e_r + c * j.e_c, e);
    }
    if (++c == NB) { c = 0; ++s; }
  }
}

// ---------------------------------------------------------------------------
// Parallel tempering (upd.c:3-48), one warp per (sample, replica) chain.
//
// The decisions are a serial chain over the pairs; all else is done by the
// warp's lanes side by side.  The chain's draws do not depend on the
// decisions: the Parisi-Rapuano generator adds words at least 24 places back,
// so 24 draws at a time are made by 24 lanes (the LCG part jumps by its powers,
// composed over the lanes).  Energies and draws wait in SMEM; the walk takes
// each decision by a single-precision exp(pt) when the draw is not within
// 1e-4 of it (its error is below 2e-5, see sp_pt_body) and by the host-libm
// table otherwise, so it is exact.  The acceptance sums, which take the
// table's value or exp(pt) of every pair, follow in parallel, one addition
// per pair and step in FP64 as on the host.  One lane walking everything took
// 34 us at 32 temperatures and 41 us at 40; this takes 12 and 14.
// ---------------------------------------------------------------------------
struct PtWarp {
  u64 ira[256];
  u64 x[256];       // FNORM * draw, as bits
  int es[256];      // energies in beta order, then each pair's dE
  uint8_t wc[256];
};
struct PtShared {
  PtWarp w[8];
  float db[256];    // b[i] - b[i+1]
  int eo[256];      // exp table offsets
};

__device__ __forceinline__ void pt_body(const JobDev &j, int s, int ry, PtShared &sh) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = ry * 8 + w, NB = j.NB, NP = NB - 1;
  for (int i = threadIdx.x; i < NB; i += blockDim.x) {
    sh.eo[i] = j.expoff[i];
    // betas descend; a difference too small for single precision stays positive
    const double f = i < NP ? -__dsub_rn(j.betas[i + 1], j.betas[i]) : 0.0;
    sh.db[i] = f > 0.0 ? fmaxf((float)f, 1e-30f) : (float)f;
  }
  __syncthreads();
  if (r >= j.NR) return;
  PtWarp &q = sh.w[w];
  const size_t o = (size_t)s * j.NR + r;
  ea_hq *h = j.pt + o;
  const int32_t *E = j.E + (size_t)s * j.NR * NB + (size_t)r * j.e_r;
#pragma unroll
  for (int i = 0; i < 8; ++i) q.ira[i * 32 + lane] = h->ira[i * 32 + lane];
  for (int i = lane; i < NB; i += 32) {
    const uint8_t c = j.wctb[o * NB + i];
    q.wc[i] = c;
    q.es[i] = E[c * j.e_c];
  }
  const uint8_t ip = h->ip, ip1 = h->ip1, ip2 = h->ip2, ip3 = h->ip3;
  u64 zseed = h->zseed, PR = h->PR, fin = h->final;
  // draws a batch can make at once: no word of it may be read by a later draw,
  // nor (ip3, read when all are written) by an earlier one
  auto lag = [](uint8_t d) { return d ? (int)d : 256; };
  const int most = min(min(min(32, lag((uint8_t)(ip - ip1))), min(lag((uint8_t)(ip - ip2)), lag((uint8_t)(ip - ip3)))),
                       lag((uint8_t)(ip3 - ip)));
  // lane k: k + 1 steps of z -> a z + 1
  u64 A = 3202034522624059733ULL, C = 1;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const u64 pa = __shfl_up_sync(0xffffffffu, A, d), pc = __shfl_up_sync(0xffffffffu, C, d);
    if (lane >= d) { C += A * pc; A *= pa; }
  }
  const double FNORM = 5.4210108624275218e-20;
  __syncwarp();
  for (int i0 = 0; i0 < NP; i0 += most) {
    const int n = min(most, NP - i0);
    const bool on = lane < n;
    const u64 a = on ? q.ira[(uint8_t)(ip1 + i0 + lane)] + q.ira[(uint8_t)(ip2 + i0 + lane)] : 0;
    __syncwarp();
    if (on) q.ira[(uint8_t)(ip + i0 + lane)] = a;
    __syncwarp();
    u64 z = 0, p = 0;
    if (on) {
      p = a ^ q.ira[(uint8_t)(ip3 + i0 + lane)];
      z = A * zseed + C;
      q.x[i0 + lane] = (u64)__double_as_longlong(__dmul_rn(FNORM, __ull2double_rn(z + p)));
    }
    zseed = __shfl_sync(0xffffffffu, z, n - 1);
    PR = __shfl_sync(0xffffffffu, p, n - 1);
    fin = zseed + PR;
    __syncwarp();
  }
  // the walk, every lane alike (slot i + 1 still holds its own clone when pair
  // i is decided, slot i the one carried up from below)
  const u64 *tab = reinterpret_cast<const u64 *>(j.exptab);
  uint32_t chg = 0;  // pairs i = lane mod 32 that changed, bit i / 32
  int ce = q.es[0];
  uint8_t cc = q.wc[0];
#pragma unroll 2
  for (int i = 0; i < NP; ++i) {
    const int e1 = q.es[i + 1];
    const uint8_t c1 = q.wc[i + 1];
    const u64 x = q.x[i];
    const int base = sh.eo[i], nx = sh.eo[i + 1] - base;
    const int dE = e1 - ce, m = (-dE) >> 1;
    const float pt = sh.db[i] * (float)dE, ex = __expf(pt), xf = (float)__longlong_as_double((long long)x);
    bool change = pt >= 0.f;
    if (!change) {
      change = xf < ex;
      if ((dE & 1) || m < 1 || m > nx)  // outside the table: exp(pt) < 2^-72 (or an odd dE, never seen)
        change = __longlong_as_double((long long)x) <
                 exp(__dmul_rn(-__dsub_rn(j.betas[i + 1], j.betas[i]), (double)dE));
      else if (fabsf(xf - ex) <= 1e-4f * ex)
        change = x < __ldg(tab + base + m - 1);
    }
    __syncwarp();
    if (lane == 0) {
      q.es[i] = dE;
      q.wc[i] = change ? c1 : cc;
    }
    if ((i & 31) == lane && change) chg |= 1u << (i >> 5);
    ce = change ? ce : e1;
    cc = change ? cc : c1;
  }
  if (lane == 0) q.wc[NP] = cc;
  __syncwarp();
  double *acc = j.acc + o * NP, *att = j.att + o * NP, *accraw = j.accraw + o * NP;
  for (int i = lane; i < NP; i += 32) {
    att[i] += 1.0;
    const int dE = q.es[i];
    const double pt = __dmul_rn(-__dsub_rn(j.betas[i + 1], j.betas[i]), (double)dE);
    double a = 1.0;
    if (!(pt >= 0.0)) {
      const int base = sh.eo[i], n = sh.eo[i + 1] - base, m = (-dE) >> 1;
      if (!(dE & 1) && m >= 1 && m <= n) {
        a = j.exptab[base + m - 1];
      } else {
        a = exp(pt);
        if (q.x[i] == 0 || (dE & 1)) atomicAdd(j.inexact, 1ULL);  // decided by a draw of 0
      }
    }
    acc[i] += a;
    if ((chg >> (i >> 5)) & 1u) accraw[i] += 1.0;
    h->ira[(uint8_t)(ip + i)] = q.ira[(uint8_t)(ip + i)];
  }
  if (lane == 0) {
    h->ip = (uint8_t)(ip + NP); h->ip1 = (uint8_t)(ip1 + NP); h->ip2 = (uint8_t)(ip2 + NP); h->ip3 = (uint8_t)(ip3 + NP);
    h->zseed = zseed; h->PR = PR; h->final = fin;
  }
  for (int i = lane; i < NB; i += 32) {
    const uint8_t c = q.wc[i];
    j.wctb[o * NB + i] = c;
    j.wbtc[o * NB + c] = (uint8_t)i;
  }
}

// Energy average in beta order and temperature history (main.cu:208-228).
__device__ __forceinline__ void measure_body(const JobDev &j, int i, int itm) {
  const int n = j.ns * j.NR * j.NB;
  if (i >= n) return;
  const size_t o = i / j.NB;
  const int b = i % j.NB, s = (int)o / j.NR, r = (int)o - s * j.NR;
  j.avgE[i] += (double)j.E[(size_t)s * j.NR * j.NB + r * j.e_r + j.wctb[o * j.NB + b] * j.e_c];
  if (itm >= 0) j.hist[(o * j.maxit_trw + itm) * j.NB + b] = j.wbtc[o * j.NB + b];
}

// ---------------------------------------------------------------------------
// Houdayer move.
// ---------------------------------------------------------------------------
// Replica pairs of both groups with random_c (main.cu:409-421).
__device__ __forceinline__ void pairs_body(const JobDev &j) {
  const int h = j.NR / 2;
  for (int g = 0; g < 2; ++g) {
    int idx[32];
    for (int k = 0; k < h; ++k) idx[k] = k + g * h;
    for (int k = 0; k < h - 1; ++k) {
      const u64 f = d_hq_next(j.rc);
      const int q = k + (int)(((uint32_t)(f >> 32)) % (uint32_t)(h - k));
      const int t = idx[k]; idx[k] = idx[q]; idx[q] = t;
    }
    j.pairs[2 * g] = idx[0];
    j.pairs[2 * g + 1] = idx[1];
  }
}

// q = s_r1 ^ s_r2 per (sample, beta < nclust, parity, half) (main.cu:889-936).
__device__ __forceinline__ void overlap_body(const JobDev &j, int g, int w, size_t lat) {
  if (w >= 2 * j.half) return;
  const size_t i = lat * 2 * j.half + w;
  const int p = w >= j.half, k = w - p * j.half;
  const int s = j.fd_nclust.div((uint32_t)lat), b = (int)lat - s * j.nclust;
  const int r1 = j.pairs[2 * g], r2 = j.pairs[2 * g + 1];
  const int c1 = j.wctb[((size_t)s * j.NR + r1) * j.NB + b], c2 = j.wctb[((size_t)s * j.NR + r2) * j.NB + b];
  const size_t wpc = (size_t)j.half * j.NR, wpp = wpc * j.NB;
  const u64 *base = j.spins + (size_t)s * 2 * wpp + (size_t)p * wpp + (size_t)k * j.NR;
  j.Q[i] = base[(size_t)c1 * wpc + r1] ^ base[(size_t)c2 * wpc + r2];
}

// Overlap bit of a site in natural order (x + L y + L^2 z): parity, half index
// and bit of the multispin word (ini.c:355-375).
__device__ __forceinline__ int q_bit(const JobDev &j, const u64 *Q, int x, int y, int z) {
  const int bx = j.fd_ml.div(x), gx = x - bx * j.msc_l, by = j.fd_ml.div(y), gy = y - by * j.msc_l;
  const int bz = j.fd_mlz.div(z), gz = z - bz * j.msc_lz;
  const int m = gx + j.msc_l * gy + j.msc_s * gz, p = (x ^ y ^ z) & 1;
  return (int)((Q[(size_t)p * j.half + (m >> 1)] >> (bx + 4 * by + 16 * bz)) & 1);
}

__device__ __forceinline__ uint32_t cc_find(const uint32_t *lab, uint32_t i) {
  uint32_t l = lab[i];
  while (l != i) { i = l; l = lab[i]; }
  return l;
}

// Lock-free union: the larger of the two roots is hung below the smaller one
// with atomicMin; when another thread got there first the walk continues from
// the value it left.  Labels only decrease, so every chain ends at the
// smallest index of its cluster.  Works on global and shared memory.
__device__ __forceinline__ void cc_unite(uint32_t *lab, uint32_t a, uint32_t b) {
  uint32_t l1 = cc_find(lab, a), l2 = cc_find(lab, b);
  if (l1 == l2) return;
  if (l1 < l2) { const uint32_t t = l1; l1 = l2; l2 = t; }
  for (;;) {
    const uint32_t l3 = atomicMin(&lab[l1], l2);
    if (l3 == l2 || l3 == l1) return;  // already joined, or l1 was a root and now hangs below l2
    if (l3 > l2) { l1 = l3; }
    else { l1 = l2; l2 = l3; }
  }
}

// Labelling by runs (runs.cuh) of one lattice in SMEM, whole or D consecutive z
// planes of it.  Local index order is natural order shifted by z0 L^2, so a
// root is the smallest global index of its (piece of a) cluster.  The bonds are
// those of the union-find of the reference (HoudayerXEA.cu:77-121): x and y
// periodic, z inside the planes, the z wrap under PBC when the lattice is
// whole; site 0 tests its x-wrap bond against x = cc_xq (see JobDev::cc_xq).
// A thread takes a column of a chunk of planes: neighbouring lanes take
// neighbouring columns, whose label slots lie in distinct banks but for pairs.

// Planes bonded along x of a column, with site 0's test put right: the contact
// of column L - 1 (y = 0) with column 0 on the first plane.
__device__ __forceinline__ uint32_t cc_bonds(const JobDev &j, const RunLab<1> &rl, int z0, int ch, int col, uint32_t eq) {
  if (z0 == 0 && ch == 0 && col == j.L - 1)
    eq = (eq & ~1u) | (uint32_t)(((rl.qm[0] ^ rl.qm[j.cc_xq]) & 1u) == 0);
  return eq;
}

// The q words of the planes [z0, z0 + nz) from the lattice's overlap words
// (word(index): the 64 bits of a (parity, half) word).
template <class Word>
__device__ __forceinline__ void cc_columns(const JobDev &j, const RunLab<1> &rl, int z0, Word &&word) {
  const RunShape &r = rl.r;
  rl.columns();
  rl.items([&](int it, int ch, int col) {
    const int y = j.fd_L.div(col), x = col - y * j.L, bx = j.fd_ml.div(x), by = j.fd_ml.div(y);
    const int mxy = (x - bx * j.msc_l) + j.msc_l * (y - by * j.msc_l), sxy = bx + 4 * by;
    int z = z0 + ch * r.H, bz = j.fd_mlz.div(z), gz = z - bz * j.msc_lz, p = (x ^ y ^ z) & 1;
    const int hc = min(r.H, r.nz - ch * r.H);
    uint32_t m = 0;
    for (int k = 0; k < hc; ++k) {
      m |= (uint32_t)((word(p * j.half + ((mxy + j.msc_s * gz) >> 1)) >> (sxy + 16 * bz)) & 1ull) << k;
      p ^= 1;
      if (++gz == j.msc_lz) { gz = 0; ++bz; }
    }
    rl.qm[it] = m;
  });
}

// Planes [slab D, ...) of lattice lat, labels written as global indices.
// Threads: any number; SMEM: slab_smem.
__device__ __forceinline__ void cc_slab_body(const JobDev &j, int D, int slab, size_t lat, unsigned char *sm) {
  const int z0 = slab * D, nz = min(D, j.Lz - z0);
  const u64 *Q = j.Q + lat * 2 * j.half;
  const RunLab<1> rl(sm, j.L, nz);
  const RunShape &r = rl.r;
  cc_columns(j, rl, z0, [&](int i) { return __ldg(Q + i); });
  rl.label(false, false, [&](int ch, int col, uint32_t eq) { return cc_bonds(j, rl, z0, ch, col, eq); });
  rl.jump([](uint16_t *, int, uint32_t) {});
  __syncthreads();
  const uint32_t off = (uint32_t)z0 * r.S;
  uint32_t *glab = j.label + lat * j.V + off;
  for (int i = threadIdx.x; i < nz * r.S; i += blockDim.x) {
    const int z = j.fd_S.div(i), col = i - z * r.S, ch = z / r.H;
    const uint32_t st = run_starts(rl.qm[ch * r.S + col], (2u << (z - ch * r.H)) - 1u);
    glab[i] = off + rl.lab[(ch * r.H + 31 - __clz(st)) * r.S + col];
  }
}

// The whole move of group g on lattice lat in one CTA, for lattices that fit
// SMEM (whole_smem): overlap words, labels, selection and the flip of both
// replicas (main.cu:776-991; HoudayerXEA.cu:54-374).
__device__ __forceinline__ void move_body(const JobDev &j, int g, size_t lat, unsigned char *sm) {
  const RunLab<1> rl(sm, j.L, j.Lz);
  const RunShape &r = rl.r;
  u64 *Q = reinterpret_cast<u64 *>(sm + run_label_smem(r));
  const int s = j.fd_nclust.div((uint32_t)lat), b = (int)lat - s * j.nclust;
  const int r1 = j.pairs[2 * g], r2 = j.pairs[2 * g + 1];
  const int c1 = j.wctb[((size_t)s * j.NR + r1) * j.NB + b], c2 = j.wctb[((size_t)s * j.NR + r2) * j.NB + b];
  const size_t wpc = (size_t)j.half * j.NR, wpp = wpc * j.NB;
  u64 *S1 = j.spins + (size_t)s * 2 * wpp + (size_t)c1 * wpc + r1;
  u64 *S2 = j.spins + (size_t)s * 2 * wpp + (size_t)c2 * wpc + r2;
  for (int w = threadIdx.x; w < 2 * j.half; w += blockDim.x) {
    const size_t o = (w >= j.half ? wpp : 0) + (size_t)(w >= j.half ? w - j.half : w) * j.NR;
    Q[w] = S1[o] ^ S2[o];
  }
  __syncthreads();
  cc_columns(j, rl, 0, [&](int i) { return Q[i]; });
  rl.label(j.bc == EA_PBC, false, [&](int ch, int col, uint32_t eq) { return cc_bonds(j, rl, 0, ch, col, eq); });
  __syncthreads();
  const u64 ub = xw_base(j, g) + ((u64)s * j.NB + b) * (u64)j.V;
  const uint32_t *u = j.xw_bits + (ub >> 5), us = (uint32_t)ub & 31u;
  uint32_t *Q32 = reinterpret_cast<uint32_t *>(Q);
  rl.items([&](int it, int ch, int col) {
    const uint16_t *l = rl.slot(ch, col);
    const uint32_t mask = run_mask(r, ch);
    // coins at the run starts as changes from run to run, then summed upwards
    uint32_t f = 0, prev = 0;
    for (uint32_t st = run_starts(rl.qm[it], mask); st; st &= st - 1u) {
      const uint32_t bit = st & (0u - st);
      const uint32_t c = xw_coin(u, us + (uint32_t)rl.root(l[(31 - __clz(bit)) * r.S]));
      if (c != prev) f |= bit;
      prev = c;
    }
    f ^= f << 1; f ^= f << 2; f ^= f << 4; f ^= f << 8; f ^= f << 16;
    const int y = j.fd_L.div(col), x = col - y * j.L, bx = j.fd_ml.div(x), by = j.fd_ml.div(y);
    const int mxy = (x - bx * j.msc_l) + j.msc_l * (y - by * j.msc_l), sxy = bx + 4 * by;
    for (f &= mask; f; f &= f - 1u) {
      const int z = ch * r.H + 31 - __clz(f & (0u - f)), bz = j.fd_mlz.div(z), gz = z - bz * j.msc_lz;
      const int w = ((x ^ y ^ z) & 1) * j.half + ((mxy + j.msc_s * gz) >> 1), bit = sxy + 16 * bz;
      atomicXor(Q32 + 2 * w + (bit >> 5), 1u << (bit & 31));  // q' = q xor [selected]
    }
  });
  __syncthreads();
  for (int w = threadIdx.x; w < 2 * j.half; w += blockDim.x) {
    const size_t o = (w >= j.half ? wpp : 0) + (size_t)(w >= j.half ? w - j.half : w) * j.NR;
    const u64 q = Q[w];
    S1[o] ^= q;
    S2[o] ^= q;
  }
}

// Bonds across slab faces (z = f D with z - 1), and the z wrap under PBC,
// merged into the global labels.
__device__ __forceinline__ void cc_merge_body(const JobDev &j, int D, int nslab, int r, size_t lat) {
  const int L = j.L, S = L * L;
  if (r >= nslab * S) return;
  const int f = j.fd_S.div(r), xy = r - f * S;
  int z, zm;
  if (f == 0) {
    if (j.bc != EA_PBC) return;
    z = 0; zm = j.Lz - 1;
  } else {
    z = f * D; zm = z - 1;
  }
  const int y = j.fd_L.div(xy), x = xy - y * L;
  const u64 *Q = j.Q + lat * 2 * j.half;
  if (q_bit(j, Q, x, y, z) == q_bit(j, Q, x, y, zm))
    cc_unite(j.label + lat * j.V, (uint32_t)(xy + S * z), (uint32_t)(xy + S * zm));
}

// After the merge, every slab root whose piece was joined across a face is
// re-pointed straight at its cluster's root; all such pieces touch a face, so
// walking once from each face site reaches them.  Afterwards any site finds
// its root in at most three loads (site -> slab root -> root).  Plain stores:
// every value written is the final root of the same cluster.
__device__ __forceinline__ void cc_compress_body(const JobDev &j, int D, int nslab, int r, size_t lat) {
  const int L = j.L, S = L * L;
  if (r >= nslab * S) return;
  const int f = j.fd_S.div(r), xy = r - f * S;
  int z, zm;
  if (f == 0) {
    if (j.bc != EA_PBC) return;
    z = 0; zm = j.Lz - 1;
  } else {
    z = f * D; zm = z - 1;
  }
  uint32_t *lab = j.label + lat * j.V;
  const uint32_t a = lab[xy + S * z], b = lab[xy + S * zm];
  const uint32_t ra = cc_find(lab, a), rb = cc_find(lab, b);
  if (ra != a) lab[a] = ra;
  if (rb != b) lab[b] = rb;
}

// Offsets, in natural site index, of the 64 sites of a multispin word from
// its bit-0 site: bit = bx + 4 by + 16 bz.
__device__ __forceinline__ int word_bit_offset(const JobDev &j, int bit) {
  return (bit & 3) * j.msc_l + ((bit >> 2) & 3) * j.msc_l * j.L + (bit >> 4) * j.msc_lz * j.L * j.L;
}

// Natural index of the bit-0 site of word (p, k).
__device__ __forceinline__ int word_site0(const JobDev &j, int p, int k) {
  const int hl = j.msc_l >> 1;
  const int row = j.fd_hl.div(k), gz = j.fd_ml.div(row), gy = row - gz * j.msc_l;
  const int gx = 2 * (k - row * hl) + ((gy + gz + p) & 1);
  return gx + j.L * gy + j.L * j.L * gz;
}

// Selection and flip of one lattice in one CTA (HoudayerXEA.cu:54-75,358-374;
// main.cu:776-832,938-991): bit i of s_bits is [U(root(i)) < 0.5], built in
// natural order (coalesced label reads, one ballot per 32 sites); then each
// word gathers its 64 bits from SMEM, q' = q xor sel, and s_r1 ^= q',
// s_r2 ^= q'.  s_bits holds V/32 words, s_off 64.  What bounds it is the chain
// of reads behind a site's label, two to three of 64 (24^2 x 192 sites, 496
// lattices: 185 us with a site a thread at a time, 131 with 4, 126 with 8 or 12).
constexpr int kFlipSites = 8;
__device__ __forceinline__ void flip_body(const JobDev &j, int g, size_t lat, uint32_t *s_bits,
                                          int *s_off) {
  const int t = threadIdx.x, nth = blockDim.x;
  const int s = j.fd_nclust.div((uint32_t)lat), b = (int)lat - s * j.nclust;
  const uint32_t *lab = j.label + lat * j.V;
  const u64 ub = xw_base(j, g) + ((u64)s * j.NB + b) * (u64)j.V;
  const uint32_t *u = j.xw_bits + (ub >> 5);
  const uint32_t us = (uint32_t)ub & 31u;
  if (t < 64) s_off[t] = word_bit_offset(j, t);
  for (int base = t; base - t < j.V; base += kFlipSites * nth) {
    uint32_t l[kFlipSites];
#pragma unroll
    for (int i = 0; i < kFlipSites; ++i) l[i] = base + i * nth < j.V ? lab[base + i * nth] : 0u;
    bool more;
    do {  // cc_find of all of them
      uint32_t n[kFlipSites];
      more = false;
#pragma unroll
      for (int i = 0; i < kFlipSites; ++i) n[i] = lab[l[i]];
#pragma unroll
      for (int i = 0; i < kFlipSites; ++i) {
        more = more || n[i] != l[i];
        l[i] = n[i];
      }
    } while (more);
    bool sel[kFlipSites];
#pragma unroll
    for (int i = 0; i < kFlipSites; ++i) sel[i] = xw_coin(u, us + l[i]);
#pragma unroll
    for (int i = 0; i < kFlipSites; ++i) {
      const int site = base + i * nth;
      const unsigned ball = __ballot_sync(0xffffffffu, sel[i]);
      if ((t & 31) == 0 && site < j.V) s_bits[site >> 5] = ball;
    }
  }
  __syncthreads();
  const int r1 = j.pairs[2 * g], r2 = j.pairs[2 * g + 1];
  const int c1 = j.wctb[((size_t)s * j.NR + r1) * j.NB + b], c2 = j.wctb[((size_t)s * j.NR + r2) * j.NB + b];
  const size_t wpc = (size_t)j.half * j.NR, wpp = wpc * j.NB;
  const u64 *Q = j.Q + lat * 2 * j.half;
  for (int w = t; w < 2 * j.half; w += nth) {
    const int p = w >= j.half, k = w - p * j.half;
    const int s0 = word_site0(j, p, k);
    u64 mask = 0;
#pragma unroll 16
    for (int bit = 0; bit < 64; ++bit) {
      const int site = s0 + s_off[bit];
      mask |= (u64)((s_bits[site >> 5] >> (site & 31)) & 1u) << bit;
    }
    const u64 qn = Q[w] ^ mask;
    u64 *base = j.spins + (size_t)s * 2 * wpp + (size_t)p * wpp + (size_t)k * j.NR;
    base[(size_t)c1 * wpc + r1] ^= qn;
    base[(size_t)c2 * wpc + r2] ^= qn;
  }
}

// Cluster selection, natural order: bit i of sel[lat][i / 32] is
// [U(root(i)) < 0.5] for site i (HoudayerXEA.cu:358-374).  Consecutive lanes
// take consecutive sites, so the label reads are coalesced; the decisions of
// a lattice (V / 8 bytes) then stay in cache for the word-order flip.
__device__ __forceinline__ void select_body(const JobDev &j, int g, int site, size_t lat) {
  const int s = j.fd_nclust.div((uint32_t)lat), b = (int)lat - s * j.nclust;
  bool sel = false;
  if (site < j.V) {
    const uint32_t root = cc_find(j.label + lat * j.V, (uint32_t)site);
    const u64 ub = xw_base(j, g) + ((u64)s * j.NB + b) * (u64)j.V;
    sel = xw_coin(j.xw_bits + (ub >> 5), ((uint32_t)ub & 31u) + root);
  }
  const unsigned ball = __ballot_sync(0xffffffffu, sel);
  if ((threadIdx.x & 31) == 0 && site < j.V) j.sel[lat * (j.V >> 5) + (site >> 5)] = ball;
}

// q' = q xor [selected] packed back into words, then s_r1 ^= q', s_r2 ^= q'
// (HoudayerXEA.cu:54-75; main.cu:776-832,938-991).  Two warps per word, one
// lane per bit.
__device__ __forceinline__ void apply_body(const JobDev &j, int g, int bx, size_t lat, unsigned *s_sel) {
  const int t = threadIdx.x, wl = t >> 6, bit = t & 63;
  const int w = bx * 4 + wl;            // word of this lattice: parity * half + k
  const size_t i = lat * 2 * j.half + w;
  const bool valid = w < 2 * j.half;
  const int p = w >= j.half, k = w - p * j.half;
  const int s = j.fd_nclust.div((uint32_t)lat), b = (int)lat - s * j.nclust;
  bool sel = false;
  if (valid) {
    const int hl = j.msc_l >> 1;
    const int row = j.fd_hl.div(k), gz = j.fd_ml.div(row), gy = row - gz * j.msc_l;
    const int gx = 2 * (k - row * hl) + ((gy + gz + p) & 1);
    const int x = gx + (bit & 3) * j.msc_l, y = gy + ((bit >> 2) & 3) * j.msc_l, z = gz + (bit >> 4) * j.msc_lz;
    const uint32_t site = (uint32_t)(x + j.L * y + j.L * j.L * z);
    sel = (__ldg(j.sel + lat * (j.V >> 5) + (site >> 5)) >> (site & 31)) & 1u;
  }
  const unsigned ball = __ballot_sync(0xffffffffu, sel);
  if ((t & 31) == 0) s_sel[t >> 5] = ball;
  __syncthreads();
  if (!valid || bit != 0) return;
  const u64 qn = j.Q[i] ^ ((u64)s_sel[2 * wl] | ((u64)s_sel[2 * wl + 1] << 32));
  const int r1 = j.pairs[2 * g], r2 = j.pairs[2 * g + 1];
  const int c1 = j.wctb[((size_t)s * j.NR + r1) * j.NB + b], c2 = j.wctb[((size_t)s * j.NR + r2) * j.NB + b];
  const size_t wpc = (size_t)j.half * j.NR, wpp = wpc * j.NB;
  u64 *base = j.spins + (size_t)s * 2 * wpp + (size_t)p * wpp + (size_t)k * j.NR;
  base[(size_t)c1 * wpc + r1] ^= qn;
  base[(size_t)c2 * wpc + r2] ^= qn;
}

}  // namespace eagb
