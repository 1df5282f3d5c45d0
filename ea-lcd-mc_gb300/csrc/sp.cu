// sp.cu -- kernels of the sample-packed layout (64 samples per word) and its
// C ABI (ea_sp_*).  See sp.cuh for the layout.
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "host.hpp"
#include "kernels_dev.cuh"
#include "runs.cuh"
#include "sp.cuh"

namespace eagb {

void set_last_error(const char *msg);  // api.cu

// ---------------------------------------------------------------------------
// Philox counters of a colour pass: the reference's fill_bits step per
// replica (fill_bits.h:47-68) with the pass counter in place of the
// half-sweep counter (its parity bit = the counter's lowest bit, as for
// half-sweeps), so every pass of every sweep has its own counters.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void sp_fill_body(const SpDev &d) {
  JobDev j{};
  j.NR = d.NR; j.xo = d.xo; j.prc = d.prc; j.ctr = d.ctr; j.iter = d.iter; j.jobid = d.jobid;
  const int parity = (int)(*d.iter & 1);
  fill_bits_body(j, parity);
}

// ---------------------------------------------------------------------------
// One colour pass.  A CTA owns kt sites of the colour: it stages every
// temperature's pre-search in SMEM (the thresholds, rarely read past it, come
// through the read-only cache), draws the random words of each (slot, site,
// replica) once -- shared by the nw sample words, as the reference shares them
// across samples (main.cu:1430) -- and updates all (word, site, replica, slot)
// words of its tile in memory order, so that consecutive lanes touch
// consecutive words of a site.  The Philox thread index of (slot b, site i,
// replica r) is (b*V + i)*NR + r.  The draws (draw_ids) are most of a pass of
// few sample words: six words a thread, an 8-bit pre-search and the thresholds
// in SMEM took 77 us a
// sweep of the 12^2 x 48 tube (24 temperatures, 4 replicas) with 128 samples,
// 55 now, with 4096 313 and 258.  (A CTA that kept the tables for its next tile
// spilled registers: 4 % slower.)
// ---------------------------------------------------------------------------
__device__ __forceinline__ void sp_pass_body(const SpDev &d, const uint4 *ctr, int off, int n, int tile,
                                             unsigned char *smem) {
  const int NB = d.NB, NR = d.NR, kt = d.kt, V = d.V;
  const int plane = NB * kt * NR;
  uint8_t *s_pre = smem;
  u64 *s_id1 = reinterpret_cast<u64 *>(s_pre + (size_t)NB * kPre11Stride), *s_id2 = s_id1 + plane;
  uint16_t *s_queue = reinterpret_cast<uint16_t *>(s_id2 + plane);
  int *s_nb = reinterpret_cast<int *>(s_queue + 4 * plane);  // [kt][7]: site, 6 neighbours
  __shared__ int s_cnt[2];
  const int tid = threadIdx.x, nth = blockDim.x;
  const int k0 = tile * kt;
  {
    const uint4 *ps = reinterpret_cast<const uint4 *>(d.pre11);
    uint4 *pd = reinterpret_cast<uint4 *>(s_pre);
    for (int i = tid; i < NB * (kPre11Stride / 16); i += nth) pd[i] = ps[i];
  }
  for (int i = tid; i < kt * 7; i += nth) {
    const int kk = i / 7, f = i % 7, k = k0 + kk;
    int v = -1;
    if (k < n) {
      const int site = d.col_sites[off + k];
      v = f == 0 ? site : d.nb[(size_t)site * 6 + f - 1];
    }
    s_nb[i] = v;
  }
  __syncthreads();
  // random words at [site of the tile][replica][slot]: the update phase's
  // consecutive lanes (consecutive slots) then read consecutive words
  const uint32_t mB = 0xFFFFFFFFu / (uint32_t)NB + 1u, mR = NR > 1 ? 0xFFFFFFFFu / (uint32_t)NR + 1u : 0u;
  draw_ids(
      plane,
      [&](int t, uint4 &c, uint32_t &key, uint32_t &tp, int &b) {
        const int q = (int)__umulhi((uint32_t)t, mB);  // t / NB, exact: t NB < 2^32
        const int kk = NR > 1 ? (int)__umulhi((uint32_t)q, mR) : q, r = q - kk * NR;
        b = t - q * NB;
        tp = (uint32_t)(((size_t)b * V + s_nb[kk * 7]) * NR + r);
        c = ctr[r];
        key = d.keys[r];
        return k0 + kk < n;
      },
      [&](int b, uint32_t hi, uint32_t lo) { return lut_byte11(hi, lo, d.cum + b * 256, s_pre + b * kPre11Stride); },
      s_id1, s_id2, s_queue, s_cnt);
  // Update phase.  A thread keeps one (replica, slot) column (lg) for the
  // whole loop -- its random words stay in registers per site -- and
  // walks (site of the tile, sample word) with a stride of nth/G groups, so
  // the G lanes of a group touch the G consecutive words of one site.
  const int G = NR * NB;
  const size_t wps = (size_t)V * G;  // words per sample word
  const int nk = min(kt, n - k0), nidx = nk * d.nw;
  if ((NB & 1) == 0) {
    // even NB: a lane takes two adjacent slots of a (replica, site) with
    // 16-byte loads and stores (every word offset here is even)
    const int G2 = G >> 1, NB2 = NB >> 1;
    const size_t wps2 = wps >> 1;
    for (int lg = tid % G2, grp = tid / G2, ngrp = max(1, nth / G2); lg < G2; lg += (nth >= G2 ? G2 : nth)) {
      if (nth >= G2 && grp >= ngrp) break;
      const int b = 2 * (lg % NB2), r = lg / NB2;
      ulonglong2 *Sc = reinterpret_cast<ulonglong2 *>(d.S + r * NB + b);
      const int step = nth >= G2 ? ngrp : 1;
      int idx = nth >= G2 ? grp : 0, kk = idx % nk, w = idx / nk;
      for (; idx < nidx; idx += step) {
        const int *sn = s_nb + kk * 7;
        const int site = sn[0];
        ulonglong2 *Sw = Sc + (size_t)w * wps2;
        const u64 *Jp = d.J + ((size_t)w * V + site) * 6;
        const ulonglong2 sv = Sw[(size_t)site * G2];
        u64 f0[6], f1[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) {
          const u64 jq = __ldg(Jp + q);
          const ulonglong2 nq = Sw[(size_t)sn[q + 1] * G2];
          f0[q] = sv.x ^ jq ^ nq.x;
          f1[q] = sv.y ^ jq ^ nq.y;
        }
        const int o = (kk * NR + r) * NB + b;
        const ulonglong2 i1 = *reinterpret_cast<const ulonglong2 *>(s_id1 + o);
        const ulonglong2 i2 = *reinterpret_cast<const ulonglong2 *>(s_id2 + o);
        ulonglong2 out;
        out.x = sv.x ^ flip_mask_id(f0, i1.x, i2.x);
        out.y = sv.y ^ flip_mask_id(f1, i1.y, i2.y);
        Sw[(size_t)site * G2] = out;
        for (kk += step; kk >= nk; kk -= nk) ++w;
      }
    }
    return;
  }
  for (int lg = tid % G, grp = tid / G, ngrp = max(1, nth / G); lg < G; lg += (nth >= G ? G : nth)) {
    if (nth >= G && grp >= ngrp) break;
    const int b = lg % NB, r = lg / NB;
    u64 *Sc = d.S + lg;
    const int step = nth >= G ? ngrp : 1;
    int idx = nth >= G ? grp : 0, kk = idx % nk, w = idx / nk;
    for (; idx < nidx; idx += step) {
      const int *sn = s_nb + kk * 7;
      const int site = sn[0];
      u64 *Sw = Sc + (size_t)w * wps;
      const u64 *Jp = d.J + ((size_t)w * V + site) * 6;
      const u64 sv = Sw[(size_t)site * G];
      u64 f[6];
#pragma unroll
      for (int q = 0; q < 6; ++q) f[q] = sv ^ __ldg(Jp + q) ^ Sw[(size_t)sn[q + 1] * G];
      const int o = (kk * NR + r) * NB + b;
      Sw[(size_t)site * G] = sv ^ flip_mask_id(f, s_id1[o], s_id2[o]);
      for (kk += step; kk >= nk; kk -= nk) ++w;
    }
  }
}

// The per-item form of a colour pass.  A thread takes (site, replica, slot)
// items of the colour in turn -- consecutive lanes on consecutive slots, so a
// warp's loads and stores cover consecutive words -- draws the item's random
// words and updates the item's word in each sample word.  The block stages the
// 11-bit pre-search tables once (the thresholds, rarely read past them, come
// through the read-only cache); no barrier separates drawing from updating.
// The words are those of the tiles (same random words per (slot, site,
// replica), same flip mask).  This form suits jobs with few sample words,
// whose tiles spend their time on barriers and SMEM traffic for random words
// used once.
//
// The flip mask uses the three random words as b0, b0 & b1 and b0 & b1 & b2
// only, and a bit of b0 is set with probability exp(-4 beta): where a 32-bit
// half of b0 is 0 that half of b1 and b2 does not matter, nor that of b2 where
// b0 & b1 is 0.  So a warp draws b0 for kItemsRound items a lane, collects the
// halves that need b1 in a queue, draws those -- a full warp at a time, each
// lane one half of any lane's item -- and the same for b2: 3.2 to 3.3 of an
// item's 6 words on T in [0.6, 1.6] and [0.7, 1.6] (the draws are
// counter-based, so the ones made are the same).  The loops stay rolled: the
// three copies of a draw are most of the code, and unrolled by item they
// missed the instruction cache.  The pass is bound by instruction issue (67 % of
// the slots), mostly of these draws: 24 x 24 x 192, 32 temperatures, 4
// replicas, one word: 760 -> 559 us a sweep; 12 x 12 x 48, 24 temperatures: 62
// -> 55.
// The thread takes items t0, t0 + stride, ... below tend of the colour's
// n x NR x NB (the block's threads take consecutive t0): one job runs it on
// a grid of resident CTAs (k_sp_pass_items), a batch on kItemsPerThread x 512
// items a block (sp_pass_any).
constexpr int kItemsRound = 3;
constexpr int kItemsThreads = 1024;  // one job: one table copy for an SM's 32 warps
// A warp's SMEM: the flip mask's two words in the making by (item, half,
// lane), the items' Philox index and column, and the queue.
struct ItemsWarp {
  uint32_t id1[kItemsRound][2][32];  // b0, then (b0 ^ id2) | b0 & b1 & b2
  uint32_t id2[kItemsRound][2][32];  // b0 & b1
  uint32_t tp[kItemsRound][32];
  uint16_t col[kItemsRound][32];
  uint16_t queue[kItemsRound * 64];
};

__device__ __forceinline__ void sp_pass_items_body(const SpDev &d, const uint4 *ctr, int off, int n, long long t0,
                                                   long long tend, long long stride, unsigned char *smem) {
  const int NB = d.NB, NR = d.NR, G = NR * NB, V = d.V, lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const uint8_t *s_pre = smem;
  ItemsWarp &sw = reinterpret_cast<ItemsWarp *>(smem + (size_t)NB * kPre11Stride)[threadIdx.x >> 5];
  {
    const uint4 *ps = reinterpret_cast<const uint4 *>(d.pre11);
    uint4 *pd = reinterpret_cast<uint4 *>(smem);
    for (int i = threadIdx.x; i < NB * (kPre11Stride / 16); i += blockDim.x) pd[i] = ps[i];
  }
  __syncthreads();
  const long long t1 = min(tend, (long long)n * G);
  const size_t wps = (size_t)V * G;  // words per sample word
  // the item's site index k and column g, stepped without divisions
  int k = (int)(t0 / G), g = (int)(t0 - (long long)k * G);
  const int sk = (int)(stride / G), sg = (int)(stride - (long long)sk * G);
  for (long long t = t0; t - lane < t1;) {
    int site[kItemsRound], col[kItemsRound];
#pragma unroll
    for (int it = 0; it < kItemsRound; ++it, t += stride, k += sk, g += sg) {
      if (g >= G) { g -= G; ++k; }
      site[it] = t < t1 ? __ldg(d.col_sites + off + k) : -1;
      col[it] = g;
      const int r = (int)d.fd_NB.div((uint32_t)g), b = g - r * NB;
      sw.tp[it][lane] = (uint32_t)(((size_t)b * V + site[it]) * NR + r);
      sw.col[it][lane] = t < t1 ? (uint16_t)g : 0xFFFFu;
    }
    int nq = 0;
#pragma unroll 1
    for (int it = 0; it < kItemsRound; ++it) {
      const uint32_t cg = sw.col[it][lane], tp = sw.tp[it][lane];
      uint32_t w0 = 0, w1 = 0;
      if (cg != 0xFFFFu) {
        const int r = (int)d.fd_NB.div(cg), b = (int)cg - r * NB;
        const uint4 c = ctr[r];
        const uint32_t key = __ldg(d.keys + r);
        const u64 *cum = d.cum + b * 256;
        const uint8_t *pre = s_pre + b * kPre11Stride;
        auto byte = [&](uint32_t hi, uint32_t lo) { return lut_byte11(hi, lo, cum, pre); };
        w0 = rnd_word_by(c.x, c.y, c.z + tp, c.w, key, tp, byte);
        w1 = rnd_word_by(c.x + 1, c.y, c.z + tp, c.w, key, tp, byte);
      }
      sw.id1[it][0][lane] = w0;
      sw.id1[it][1][lane] = w1;
      sw.id2[it][0][lane] = sw.id2[it][1][lane] = 0;
      unsigned m = __ballot_sync(0xffffffffu, w0 != 0);
      if (w0) sw.queue[nq + __popc(m & below)] = (uint16_t)(it << 6 | lane);
      nq += __popc(m);
      m = __ballot_sync(0xffffffffu, w1 != 0);
      if (w1) sw.queue[nq + __popc(m & below)] = (uint16_t)(it << 6 | 32 | lane);
      nq += __popc(m);
    }
#pragma unroll 1
    for (int q = 2; q < 6 && nq; q += 2) {
      __syncwarp();
      int next = 0;  // the next queue, in place: it never runs ahead of the reads
      for (int i0 = 0; i0 < nq; i0 += 32) {
        const bool on = i0 + lane < nq;
        const int e = on ? sw.queue[i0 + lane] : 0, it = e >> 6, h = (e >> 5) & 1, l = e & 31;
        uint32_t a = 0;
        if (on) {
          const uint32_t cg = sw.col[it][l], tp = sw.tp[it][l];
          const int r = (int)d.fd_NB.div(cg), b = (int)cg - r * NB;
          const uint4 c = ctr[r];
          const u64 *cum = d.cum + b * 256;
          const uint8_t *pre = s_pre + b * kPre11Stride;
          a = rnd_word_by(c.x + q + h, c.y, c.z + tp, c.w, __ldg(d.keys + r), tp,
                          [&](uint32_t hi, uint32_t lo) { return lut_byte11(hi, lo, cum, pre); });
          if (q == 2) {
            const uint32_t b0 = sw.id1[it][h][l];
            a &= b0;
            sw.id2[it][h][l] = a;
            sw.id1[it][h][l] = b0 ^ a;
          } else {
            sw.id1[it][h][l] |= a & sw.id2[it][h][l];
          }
        }
        if (q == 2) {
          const unsigned m = __ballot_sync(0xffffffffu, a != 0);
          if (a) sw.queue[next + __popc(m & below)] = (uint16_t)e;
          next += __popc(m);
        }
      }
      nq = next;
    }
    __syncwarp();
#pragma unroll
    for (int it = 0; it < kItemsRound; ++it) {
      if (site[it] < 0) continue;
      const u64 id1 = ((u64)sw.id1[it][0][lane] << 32) | sw.id1[it][1][lane];
      const u64 id2 = ((u64)sw.id2[it][0][lane] << 32) | sw.id2[it][1][lane];
      int nbr[6];
#pragma unroll
      for (int q = 0; q < 6; ++q) nbr[q] = __ldg(d.nb + (size_t)site[it] * 6 + q);
      u64 *Sc = d.S + col[it];
      for (int ww = 0; ww < d.nw; ++ww) {
        u64 *Sw = Sc + (size_t)ww * wps;
        const u64 *Jp = d.J + ((size_t)ww * V + site[it]) * 6;
        const u64 sv = Sw[(size_t)site[it] * G];
        u64 f[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) f[q] = sv ^ __ldg(Jp + q) ^ Sw[(size_t)nbr[q] * G];
        Sw[(size_t)site[it] * G] = sv ^ flip_mask_id(f, id1, id2);
      }
    }
    __syncwarp();
  }
}

// A job's colour pass by its form; blk counts the job's blocks of the pass
// (tiles, or kItemsPerThread x blockDim.x items of the per-item form).
// One round: a second one with an item or two a lane costs a batch of small
// jobs 3 to 10 %; two full rounds suit 24 tubes of L 8..12 (9.2 against 9.6 ms a
// bin) but not 16 of L 6 and 9 (7.7 against 6.3).
constexpr int kItemsPerThread = kItemsRound;
__device__ __forceinline__ void sp_pass_any(const SpDev &d, const uint4 *ctr, int colour, int blk, unsigned char *smem) {
  const int off = d.col_off[colour], n = d.col_off[colour + 1] - off;
  if (d.pgrid) {
    const long long t0 = (long long)blk * blockDim.x * kItemsPerThread;
    sp_pass_items_body(d, ctr, off, n, t0 + threadIdx.x, t0 + (long long)blockDim.x * kItemsPerThread, blockDim.x,
                       smem);
  } else {
    sp_pass_body(d, ctr, off, n, blk, smem);
  }
}

// ---------------------------------------------------------------------------
// Energy: per (word, sample, replica, slot) the number of unsatisfied
// half-edges U2 (each bond counted from both ends), so E = 3V - U2
// (main.cu:1379).  A block owns a tile of sites of one word: the sites'
// neighbours and couplings are staged in SMEM once, lane groups of one lane
// per (replica, slot) column walk the tile's sites in turn, counting the
// unsatisfied slots of all 64 samples in bit-sliced counters (one bit plane
// per power of two), the groups' counts are added up through SMEM, and the
// block adds one total per (column, sample) to U2.
// With epair (two colours, both ends of every bond holding its coupling word:
// checked on the host when the couplings are set) every bond has exactly one
// colour-1 end, so the count walks the colour-1 sites only and doubles them.
//
// Bound by issue and the latency of the neighbours' loads; the words come from
// DRAM once (340 MB on 64 words of 12 x 12 x 48, 24 temperatures, 4 replicas:
// 50 us at the copy rate).  One thread a column and run of sites, each ending
// in 64 global atomic additions, took 257 us there (190 instructions a word)
// and 28 us on one word; this form 160 and 12.  Two columns a lane (16-byte loads)
// took 181 us: 115 registers leave 16 warps an SM.
// ---------------------------------------------------------------------------
constexpr int kEnPlanes = 8;
constexpr int kEnSites = 42;      // sites a lane counts: 6 * 42 < 2^8
constexpr int kEnMaxThreads = 288;
constexpr size_t kEnSiteBytes = 80;      // 6 coupling words and 8 indices of a staged site
constexpr size_t kEnSmem = 64 * 1024;    // of a block, in every form of the count

// Fills the count's launch shape (d.en) for `chunk` sites a lane, fewer where
// the lane groups of a few columns would stage more sites than kEnSmem holds.
static void en_threads(const SpDev &d, EnShape &e) {
  const int G = d.NR * d.NB;
  e.nslice = (G + kEnMaxThreads - 1) / kEnMaxThreads;
  e.lanes = (G + e.nslice - 1) / e.nslice;
  e.threads = (e.lanes + 31) / 32 * 32;
  for (int t = e.threads; t <= kEnMaxThreads; t += 32)  // the multiple of 32 that lane groups fill best
    if (t / e.lanes * e.lanes * e.threads >= e.threads / e.lanes * e.lanes * t) e.threads = t;
}
void sp_energy_shape(SpDev &d, int chunk) {
  EnShape &e = d.en;
  en_threads(d, e);
  d.echunk = chunk;
  e.tile = std::min({e.threads / e.lanes * chunk, d.esites, (int)(kEnSmem / kEnSiteBytes)});
  e.ntile = (d.esites + e.tile - 1) / e.tile;
}
inline size_t en_blocks(const SpDev &d) { return (size_t)d.nw * d.en.ntile * d.en.nslice; }
// The staged sites; then, in the same bytes, the groups' planes.  `threads` of
// the launch's blocks.
inline size_t en_smem(const SpDev &d, int threads) {
  return std::max((size_t)d.en.tile * kEnSiteBytes, (size_t)(threads / d.en.lanes) * d.en.lanes * kEnPlanes * 8);
}

// Sites per lane of the energy count, a multiple of the 4 that the counters take
// at a time, at most what they hold.  A block ends with an atomic addition a (column,
// sample), so n sites a lane cost a / n in additions (a = 64 columns x sites /
// lane groups, some 2 us a million) and about half a microsecond each: the sum
// is least at sqrt(4e-6 a).  us a count with the sites of three waves of blocks
// / with these, and of the form without blocks: 12^2 x 48, 96 columns, 64
// words 175 / 160, 262; 24^2 x 192, 128 columns 84 / 74, 123; 10^2 x 80, 240
// columns, 3 words 80 / 33, 62; 18^2 x 55, 189 columns 99 / 43, 68.
int sp_energy_chunk(const SpDev &d) {
  EnShape e{};
  en_threads(d, e);
  const double a = 64.0 * d.nw * d.esites * d.NR * d.NB / (e.threads / e.lanes);
  const double n = std::sqrt(4e-6 * a);
  return n >= kEnSites ? kEnSites : std::max(4, 4 * (int)std::lround(n / 4));
}

// Bit-sliced counters of 64 samples.  site() takes a site's six unsatisfied
// bits and returns its carry of weight 8; carries are added in pairs and
// rippled once every 4 sites.
struct EnCount {
  u64 P[kEnPlanes];
  static __device__ __forceinline__ u64 maj(u64 a, u64 b, u64 c) { return (a & b) | (c & (a ^ b)); }
  __device__ __forceinline__ u64 site(const u64 f[6]) {
    // six bits -> a 3-bit count per sample (two full adders and a merge)
    const u64 x1 = f[0] ^ f[1] ^ f[2], y1 = maj(f[0], f[1], f[2]);
    const u64 x2 = f[3] ^ f[4] ^ f[5], y2 = maj(f[3], f[4], f[5]);
    const u64 z0 = x1 ^ x2, c0 = x1 & x2, z1 = y1 ^ y2 ^ c0, z2 = maj(y1, y2, c0);
    u64 c = P[0] & z0;
    P[0] ^= z0;
    const u64 t = P[1] ^ z1 ^ c;
    c = maj(P[1], z1, c);
    P[1] = t;
    const u64 s = P[2] ^ z2 ^ c;
    c = maj(P[2], z2, c);
    P[2] = s;
    return c;
  }
  __device__ __forceinline__ u64 pair(u64 a, u64 b) {
    const u64 c = maj(P[3], a, b);
    P[3] ^= a ^ b;
    return c;
  }
  __device__ __forceinline__ void ripple(u64 a, u64 b) {
    u64 c = maj(P[4], a, b);
    P[4] ^= a ^ b;
#pragma unroll
    for (int p = 5; p < kEnPlanes; ++p) {
      const u64 h = P[p] & c;
      P[p] ^= c;
      c = h;
    }
  }
};

__device__ __forceinline__ void sp_energy_body(const SpDev &d, int blk, unsigned char *sm) {
  const EnShape &e = d.en;
  const int G = d.NR * d.NB, V = d.V;
  const int part = blk / e.nslice, sl = blk - part * e.nslice, w = part / e.ntile, tl = part - w * e.ntile;
  const int s0 = tl * e.tile, ns = min(e.tile, d.esites - s0);
  u64 *sJ = reinterpret_cast<u64 *>(sm);                                   // [tile][6]
  uint32_t *sN = reinterpret_cast<uint32_t *>(sJ + (size_t)6 * e.tile);    // [tile][8]: the 6 neighbours and the site
  const int32_t *c1 = d.col_sites + d.col_off[1];
  const u64 *Jw = d.J + (size_t)w * V * 6;
  for (int i = threadIdx.x; i < ns * 8; i += blockDim.x) {
    const int k = i >> 3, f = i & 7, site = d.epair ? __ldg(c1 + s0 + k) : s0 + k;
    if (f < 6) sJ[k * 6 + f] = __ldg(Jw + (size_t)site * 6 + f);
    if (f < 7) sN[i] = (uint32_t)(f < 6 ? __ldg(d.nb + (size_t)site * 6 + f) : site);
  }
  __syncthreads();
  const int groups = blockDim.x / e.lanes, g = threadIdx.x / e.lanes, ln = threadIdx.x - g * e.lanes;
  const int col = sl * e.lanes + ln;
  EnCount n;
#pragma unroll
  for (int p = 0; p < kEnPlanes; ++p) n.P[p] = 0;
  if (g < groups && col < G) {
    // a site's words G apart: the product in 64 bits (2^32 words are 34 GB)
    const char *Sc = reinterpret_cast<const char *>(d.S + (size_t)w * V * G + col);
    const uint32_t gb = (uint32_t)G * 8u;
    auto word = [&](uint32_t i) { return *reinterpret_cast<const u64 *>(Sc + (u64)i * gb); };
    auto site = [&](int k) -> u64 {
      const uint4 *nb = reinterpret_cast<const uint4 *>(sN + k * 8);
      const ulonglong2 *J = reinterpret_cast<const ulonglong2 *>(sJ + k * 6);
      const uint4 na = nb[0], nc = nb[1];
      const u64 sv = word(nc.z);
      u64 f[6];
      f[0] = word(na.x); f[1] = word(na.y); f[2] = word(na.z);
      f[3] = word(na.w); f[4] = word(nc.x); f[5] = word(nc.y);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const ulonglong2 j = J[q];
        f[2 * q] ^= sv ^ j.x;
        f[2 * q + 1] ^= sv ^ j.y;
      }
      return n.site(f);
    };
    int k = g;
    for (; k + 3 * groups < ns; k += 4 * groups) {
      u64 a = site(k), b = site(k + groups);
      const u64 p = n.pair(a, b);
      a = site(k + 2 * groups);
      b = site(k + 3 * groups);
      n.ripple(p, n.pair(a, b));
    }
    for (; k < ns; k += groups) n.ripple(n.pair(site(k), 0), 0);
  }
  __syncthreads();
  u64 *pl = reinterpret_cast<u64 *>(sm);  // [group][plane][lane]
  if (g < groups) {
#pragma unroll
    for (int p = 0; p < kEnPlanes; ++p) pl[(g * kEnPlanes + p) * e.lanes + ln] = n.P[p];
  }
  __syncthreads();
  // totals: a task takes 8 samples of a column -- byte j of the 8 planes, an
  // 8 x 8 bit matrix whose transpose holds the 8 samples' counts -- from every
  // group, added as 16-bit fields
  const int cols = min(e.lanes, G - sl * e.lanes);
  int32_t *U = d.U2 + (size_t)w * 64 * G + sl * e.lanes;
  for (int t = threadIdx.x; t < cols * 8; t += blockDim.x) {
    const int j = t / cols, c = t - j * cols;
    const uint8_t *P = reinterpret_cast<const uint8_t *>(pl + c) + j;
    u64 even = 0, odd = 0;
    for (int q = 0; q < groups; ++q, P += (size_t)kEnPlanes * e.lanes * 8) {
      u64 x = 0;
#pragma unroll
      for (int p = 0; p < kEnPlanes; ++p) x |= (u64)P[(size_t)p * e.lanes * 8] << (8 * p);
      x = transpose8(x);
      even += x & 0x00FF00FF00FF00FFull;
      odd += (x >> 8) & 0x00FF00FF00FF00FFull;
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int cnt = (int)(((q & 1 ? odd : even) >> (16 * (q >> 1))) & 0xFFFFu);
      if (cnt) atomicAdd(U + (size_t)(8 * j + q) * G + c, cnt << d.epair);
    }
  }
}

// ---------------------------------------------------------------------------
// Tempering: one block per (word, replica), one lane per sample's chain; the
// rule of upd.c:3-48 over the slot pairs in order (pt = -(b[i+1]-b[i]) * dE,
// accept when pt >= 0 or FNORM * u < exp(pt), exp from the host's libm table;
// beyond the table exp(pt) < 2^-72 and only u = 0 accepts).  The 64-bit
// uniform u of (step, pair, chain) is Philox4x32-10 keyed by the job's
// tempering seed -- the reference draws it from a per-chain Parisi-Rapuano
// generator; sample-packed jobs have 64 chains per word, so a counter-based
// draw replaces the 2 KB of state per chain.
//
// The walk over the pairs is a serial chain, so everything that does not
// depend on the carried configuration is put in SMEM by the whole block first:
// energies, slot ids and the uniforms as FNORM * u.  The chain needs no FP64
// (pt >= 0 exactly when dE has the sign of -(b[i+1]-b[i]), and non-negative
// doubles order as their bit patterns), and it reads the table only when a
// single-precision exp(pt) cannot tell: that is within 2e-5 of the true value
// (pt in [-50, 0) has a relative error of 3 * 2^-24, so its exponential 9e-6;
// __expf adds 2 + 1.16 |x| ulp, 7e-6), so a uniform more than 1e-4 away from
// it decides alone, and one draw in some 10^4 looks at the table.
// A warp's accepted swaps of pair i form half of the lane mask M[i].
// Bound by latency.  24 temperatures, one word: 31 us with every operand read
// from global memory on the way, 23 staged with a table read a pair, 12 so.
// ---------------------------------------------------------------------------
constexpr int kPtThreads = 256;
// SMEM: uniforms [NB-1][64] u64, masks [NB-1] u64, energies [NB][65] i32, table
// offsets [NB], b[i]-b[i+1] [NB] f32, slot ids [NB][64] u8
__host__ __device__ inline size_t pt_smem(int NB) { return (size_t)8 * 65 * (NB - 1) + 4 * 67 * NB + 64 * NB; }

__device__ __forceinline__ void sp_pt_body(const SpDev &d, int wr, unsigned char *sm) {
  const int NB = d.NB, NP = NB - 1, NR = d.NR, G = NR * NB;
  const int w = wr / NR, r = wr % NR, nt = 3 * d.V;
  u64 *xs = reinterpret_cast<u64 *>(sm), *Ms = xs + 64 * NP;
  int *es = reinterpret_cast<int *>(Ms + NP), *eo = es + 65 * NB;
  float *db = reinterpret_cast<float *>(eo + NB);
  uint8_t *ps = reinterpret_cast<uint8_t *>(db + NB);
  const size_t row = (size_t)w * 64 * G + (size_t)r * NB;
#pragma unroll 8
  for (int t = threadIdx.x; t < 64 * NB; t += blockDim.x) {
    const int lane = t / NB, b = t - lane * NB;
    const size_t o = row + (size_t)lane * G + b;
    es[b * 65 + lane] = nt - d.U2[o];
    ps[b * 64 + lane] = d.perm[o];
  }
  for (int i = threadIdx.x; i < NB; i += blockDim.x) {
    eo[i] = __ldg(d.expoff + i);
    // betas descend; a difference too small for single precision stays
    // positive (exp(pt) is then within 1e-4 of 1 and the table decides)
    const double f = i < NP ? -__dsub_rn(__ldg(d.betas + i + 1), __ldg(d.betas + i)) : 0.0;
    db[i] = f > 0.0 ? fmaxf((float)f, 1e-30f) : (float)f;
  }
  const unsigned long long step = *d.ptstep;
  const double FNORM = 5.4210108624275218e-20;
  for (int t = threadIdx.x; t < 64 * NP; t += blockDim.x) {
    uint32_t v0 = (uint32_t)step, v1 = (uint32_t)(step >> 32), v2 = (uint32_t)(t >> 6);
    uint32_t v3 = (uint32_t)(((size_t)w * 64 + (t & 63)) * NR + r);
    philox10(v0, v1, v2, v3, (uint32_t)d.pt_seed, (uint32_t)(d.pt_seed >> 32));
    xs[t] = (u64)__double_as_longlong(__dmul_rn(FNORM, __ull2double_rn(((u64)v0 << 32) | v1)));
  }
  __syncthreads();
  if (threadIdx.x < 64) {
    // The pairs in order: slot i+1 still holds its own configuration when pair
    // i is decided, slot i holds the one carried up from below (a swap at i
    // moves it on to i+1); slot i's final values are written as soon as pair i
    // is decided.
    const int lane = threadIdx.x;
    uint32_t *Mh = reinterpret_cast<uint32_t *>(Ms) + (lane >> 5);
    const u64 *tab = reinterpret_cast<const u64 *>(d.exptab);
    int carry_e = es[lane];
    uint8_t carry_p = ps[lane];
#pragma unroll 4
    for (int i = 0; i < NP; ++i) {
      const int e1 = es[(i + 1) * 65 + lane];
      const uint8_t p1 = ps[(i + 1) * 64 + lane];
      const u64 x = xs[i * 64 + lane];
      const float f = db[i], xf = (float)__longlong_as_double((long long)x);
      const int base = eo[i], nx = eo[i + 1] - base;
      const int dE = e1 - carry_e, m = (-dE) >> 1;
      const float pt = f * (float)dE, ex = __expf(pt);
      bool change = pt >= 0.f;
      if (!change) {
        change = xf < ex;
        if (m < 1 || m > nx) change = x == 0;                 // beyond the table: exp(pt) < 2^-72
        else if (fabsf(xf - ex) <= 1e-4f * ex) change = x < __ldg(tab + base + m - 1);
      }
      es[i * 65 + lane] = change ? e1 : carry_e;
      ps[i * 64 + lane] = change ? p1 : carry_p;
      carry_e = change ? carry_e : e1;
      carry_p = change ? carry_p : p1;
      const unsigned mask = __ballot_sync(0xffffffffu, change);
      if ((lane & 31) == 0) Mh[2 * i] = mask;
    }
    es[NP * 65 + lane] = carry_e;
    ps[NP * 64 + lane] = carry_p;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < 64 * NB; t += blockDim.x) {
    const int lane = t / NB, b = t - lane * NB;
    const size_t o = row + (size_t)lane * G + b;
    d.E[o] = es[b * 65 + lane];
    d.perm[o] = ps[b * 64 + lane];
  }
  uint32_t *acc = d.acc + ((size_t)w * 64 * NR + r) * NP;
  for (int t = threadIdx.x; t < 64 * NP; t += blockDim.x) {
    const int lane = t / NP, i = t - lane * NP;
    if ((Ms[i] >> lane) & 1ull) atomicAdd(acc + (size_t)lane * NR * NP + i, 1u);  // no wait for the old value
  }
  for (int i = threadIdx.x; i < NP; i += blockDim.x) d.M[((size_t)w * NR + r) * NP + i] = Ms[i];
}

// The accepted swaps of the last tempering step, applied to the words in
// pair order: slot i exchanges the masked samples with slot i+1, and is final
// after that (one carry word).  A block takes kPermRows consecutive (word,
// site, replica) rows of NB words, a thread one row.
// NB a multiple of 4: rows are whole 32-byte sectors, so a thread streams its
// row through registers with 32-byte loads and stores, the next four words
// in flight while four are exchanged.  Other NB: the block stages its rows in
// SMEM so that loads and stores are coalesced.  Both move the words once each
// way (2 x 340 MB on 64 words of 12 x 12 x 48: 100 us at the copy rate); the
// staged form took 219 us there, the streamed one 115 (0.87 of the copy rate).
constexpr int kPermRows = 128;

__device__ __forceinline__ void ld32(u64 v[4], const u64 *p) {
  asm volatile("ld.global.v4.u64 {%0, %1, %2, %3}, [%4];"
               : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]) : "l"(p));
}
__device__ __forceinline__ void st32(u64 *p, const u64 v[4]) {
  asm volatile("st.global.v4.u64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(v[0]), "l"(v[1]), "l"(v[2]), "l"(v[3]));
}

inline size_t perm_smem(int NB) { return NB & 3 ? (size_t)kPermRows * (NB | 1) * 8 : 0; }

__device__ __forceinline__ void sp_permute_body(const SpDev &d, int blk, u64 *rows) {
  const int NB = d.NB, NR = d.NR;
  const long long nrows = (long long)d.nw * d.V * NR;
  const long long r0 = (long long)blk * kPermRows;
  if (blk == 0 && threadIdx.x == 0) *d.ptstep += 1ull;
  const int nr = (int)min((long long)kPermRows, nrows - r0);
  const long long t = r0 + threadIdx.x;
  const int r = (int)(t % NR), w = (int)(t / ((long long)NR * d.V));
  const u64 *M = d.M + ((size_t)w * NR + r) * (NB - 1);
  u64 *g = d.S + (size_t)r0 * NB;
  if ((NB & 3) == 0) {
    if (threadIdx.x >= nr) return;
    u64 *p = g + (size_t)threadIdx.x * NB;
    u64 v[4], n[4];
    ld32(v, p);
    u64 cur = v[0];
    for (int i = 0; i < NB; i += 4) {
      u64 o[4];
      const bool more = i + 4 < NB;
      if (more) ld32(n, p + i + 4);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const u64 x = (cur ^ v[q + 1]) & M[i + q];
        o[q] = cur ^ x;
        cur = v[q + 1] ^ x;
      }
      o[3] = cur;
      if (more) {
        const u64 x = (cur ^ n[0]) & M[i + 3];
        o[3] = cur ^ x;
        cur = n[0] ^ x;
      }
      st32(p + i, o);
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = n[q];
    }
    return;
  }
  // rows sit in SMEM with an odd stride (in words): the threads' scans then
  // hit distinct banks (an even stride such as NB = 22 is a many-way conflict)
  const int rs = NB | 1;
  for (int k = threadIdx.x; k < nr * NB; k += blockDim.x) {
    const int row = k / NB;
    rows[row * rs + (k - row * NB)] = g[k];
  }
  __syncthreads();
  if (threadIdx.x < nr) {
    u64 *p = rows + (size_t)threadIdx.x * rs;
    u64 cur = p[0];
    for (int i = 0; i < NB - 1; ++i) {
      const u64 m = M[i];
      const u64 nxt = p[i + 1];
      const u64 x = (cur ^ nxt) & m;
      p[i] = cur ^ x;
      cur = nxt ^ x;
    }
    p[NB - 1] = cur;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < nr * NB; k += blockDim.x) {
    const int row = k / NB;
    g[k] = rows[row * rs + (k - row * NB)];
  }
}


// ---------------------------------------------------------------------------
// Houdayer move (main.cu:351-453, HoudayerXEA.cu:54-374), per sample.
// Replica pairs: as the reference picks them (main.cu:408-421) from random_c,
// in two groups of NR/2 replicas (one group of NR when NR < 4).  For each
// group and each slot b < nclust, the overlap q = s_r1 ^ s_r2 of every sample
// is split into maximal clusters of equal q along all six bond slots (the
// fake bonds of open planes included, so every move conserves E(r1)+E(r2)
// for any L; for even L the fake bonds duplicate y bonds and the clusters
// are the reference's); a cluster's root is its smallest site index, as in
// the reference, and each cluster flips in both replicas with probability
// 1/2.  The coin of a cluster is the lowest bit of Philox4x32-10 of (move,
// root, sample, slot, group) -- the reference compares a cuRAND uniform per
// (sample, beta, root) with 0.5 (HoudayerXEA.cu:373); a counter-based bit
// needs no V*NB uniforms per sample.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void sp_pairs_body(const SpDev &d) {
  *d.move += 1ull;
  const int ng = d.NR >= 4 ? 2 : 1, h = d.NR / ng;
  for (int g = 0; g < ng; ++g) {
    int idx[64];
    for (int k = 0; k < h; ++k) idx[k] = k + g * h;
    for (int k = 0; k < h - 1; ++k) {
      const u64 f = d_hq_next(d.rc);
      const int q = k + (int)(((uint32_t)(f >> 32)) % (uint32_t)(h - k));
      const int t = idx[k]; idx[k] = idx[q]; idx[q] = t;
    }
    d.pairs[2 * g] = idx[0];
    d.pairs[2 * g + 1] = idx[1];
  }
}

__device__ __forceinline__ void sp_overlap_body(const SpDev &d, int g, long long t) {  // t = (w, b, site)
  const int V = d.V, nc = d.nclust;
  if (t >= (long long)d.nw * nc * V) return;
  const int i = (int)(t % V), b = (int)((t / V) % nc), w = (int)(t / ((long long)V * nc));
  const int r1 = d.pairs[2 * g], r2 = d.pairs[2 * g + 1];
  const u64 *p = d.S + (((size_t)w * V + i) * d.NR) * d.NB + b;
  d.Q[t] = p[(size_t)r1 * d.NB] ^ p[(size_t)r2 * d.NB];
}

// The labelling of lattices that the runs (runs.cuh) do not take: wide flat
// ones, whose run words pass the SMEM, and in batches and the persistent kernel
// those above kSpClusterMaxV sites.  One CTA per (word, slot, group of 8
// samples): the CTA reads its byte of every site's overlap word into SMEM and
// labels the 8 samples' lattices one after the other with lock-step rounds --
// each site hooks the labels of its
// equal-q neighbours of smaller index with atomicMin, then labels are
// pointer-jumped until stable, until a round hooks nothing.  Labels only
// decrease and stay inside the cluster, so each cluster ends labelled by its
// smallest site.  The roots' coins give the samples' flip bits, gathered per
// site in a byte that replaces the CTA's byte of the overlap word (the 8
// groups of a word own disjoint bytes, so no atomics); k_sp_flip then applies
// the flip words to both replicas.
// Lattices above kSpClusterMaxV sites keep the same arrays in a global
// scratch region of the CTA (L2-resident) instead of SMEM.
// Key of the cluster coins of a job: its tempering seed, offset.
__host__ __device__ inline unsigned long long sp_cluster_key(const SpDev &d) { return d.pt_seed ^ 0xC2B2AE3585EBCA6BULL; }

__device__ __forceinline__ void sp_cluster_body(const SpDev &d, int g, int blk, uint32_t *sm) {
  const unsigned long long key = sp_cluster_key(d);
  const int V = d.V, nc = d.nclust;
  uint32_t *base = V <= kSpClusterMaxV ? sm : d.cscratch + (size_t)blk * sp_cluster_words(V);
  uint32_t *lab = base;                                              // [V]
  uint8_t *qb = reinterpret_cast<uint8_t *>(lab + V);                // [V] q bits of the 8 samples
  uint8_t *fb = qb + V;                                              // [V] flip bits of the 8 samples
  uint8_t *bond = fb + V;                                            // [V] equal-q slots to smaller sites
  const int grp = blk & 7, lat = blk >> 3;                           // lat = w * nc + b
  const int b = lat % nc, w = lat / nc;
  uint8_t *Qb = reinterpret_cast<uint8_t *>(d.Q + (size_t)lat * V) + grp;
  for (int i = threadIdx.x; i < V; i += blockDim.x) {
    qb[i] = Qb[(size_t)i * 8];
    fb[i] = 0;
  }
  __syncthreads();
  const unsigned long long mv = *d.move;
  for (int l = 0; l < 8; ++l) {
    for (int i = threadIdx.x; i < V; i += blockDim.x) {
      const unsigned qi = (qb[i] >> l) & 1u;
      unsigned m = 0;
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        const int p = __ldg(d.nb + (size_t)i * 6 + q);
        if (p < i && ((qb[p] >> l) & 1u) == qi) m |= 1u << q;
      }
      bond[i] = (uint8_t)m;
      lab[i] = (uint32_t)i;
    }
    __syncthreads();
    for (;;) {
      int hooked = 0;
      for (int i = threadIdx.x; i < V; i += blockDim.x) {
        const unsigned m = bond[i];
        if (!m) continue;
        const uint32_t li = lab[i];
#pragma unroll
        for (int q = 0; q < 6; ++q)
          if ((m >> q) & 1u) {
            const uint32_t lj = lab[__ldg(d.nb + (size_t)i * 6 + q)];
            if (lj != li) { atomicMin(&lab[max(li, lj)], min(li, lj)); hooked = 1; }
          }
      }
      if (!__syncthreads_or(hooked)) break;
      for (;;) {
        int moved = 0;
        for (int i = threadIdx.x; i < V; i += blockDim.x) {
          const uint32_t x = lab[i], y = lab[x];
          if (y != x) { lab[i] = y; moved = 1; }
        }
        if (!__syncthreads_or(moved)) break;
      }
    }
    // coins of the roots, kept in the roots' bond bytes (no longer needed)
    const int lane = grp * 8 + l;
    const uint32_t tag = (((uint32_t)(w * 64 + lane) << 6 | (uint32_t)b) << 1) | (uint32_t)g;
    for (int i = threadIdx.x; i < V; i += blockDim.x) {
      if (lab[i] != (uint32_t)i) continue;
      uint32_t v0 = (uint32_t)mv, v1 = (uint32_t)(mv >> 32), v2 = (uint32_t)i, v3 = tag;
      philox10(v0, v1, v2, v3, (uint32_t)key, (uint32_t)(key >> 32));
      bond[i] = (uint8_t)(v0 & 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < V; i += blockDim.x) fb[i] |= (uint8_t)(bond[lab[i]] << l);
    __syncthreads();
  }
  __syncthreads();
  for (int i = threadIdx.x; i < V; i += blockDim.x) Qb[(size_t)i * 8] = fb[i];
}

// Samples at a time for a whole lattice in SMEM; 0: it does not fit.
__host__ __device__ inline int run_samples(int L, int Lz) {
  if (L * L * Lz > kSpClusterMaxV) return 0;
  const RunShape r = run_shape(L, Lz);
  for (int ns = 8; ns >= 1; ns >>= 1)
    if (run_smem(r, ns) <= kRunSmem) return ns;
  return 0;
}

// One (word, slot, 8 samples) of the move: labels by runs, a coin per root
// (bit 15 of the root's label: labels are below 2^15), and the flip bytes in
// place of the overlap bytes.
template <int NS>
__device__ __forceinline__ void sp_cluster_runs(const SpDev &d, int g, int blk, unsigned char *sm) {
  const unsigned long long key = sp_cluster_key(d);
  const int V = d.V, nc = d.nclust, grp = blk & 7, lat = blk >> 3;
  const int b = lat % nc, w = lat / nc;
  uint8_t *Qb = reinterpret_cast<uint8_t *>(d.Q + (size_t)lat * V) + grp;
  const RunLab<NS> rl(sm, d.L, d.Lz);
  const RunShape &r = rl.r;
  const int zs = r.S * NS;
  rl.load(Qb);
  const unsigned long long mv = *d.move;
  for (int h = 0; h < 8 / NS; ++h) {
    rl.words(h);
    rl.label(d.bc == EA_PBC, (d.L & 1) != 0, [](int, int, uint32_t eq) { return eq; });
    const int lane = grp * 8 + h * NS + (int)(threadIdx.x % NS);
    const uint32_t tag = (((uint32_t)(w * 64 + lane) << 6 | (uint32_t)b) << 1) | (uint32_t)g;
    // roots are collected before their coins are drawn: the coins then take as
    // many steps as the lane with most roots, not one for every run
    rl.template jump<0x7FFF>([&](uint16_t *l, int id, uint32_t roots) {
      for (; roots; roots &= roots - 1u) {
        const int z = 31 - __clz(roots & (0u - roots));
        uint32_t v0 = (uint32_t)mv, v1 = (uint32_t)(mv >> 32), v2 = (uint32_t)(id + z * r.S), v3 = tag;
        philox10(v0, v1, v2, v3, (uint32_t)key, (uint32_t)(key >> 32));
        l[z * zs] = (uint16_t)((uint32_t)(id + z * r.S) | ((v0 & 1u) << 15));
      }
    });
    __syncthreads();
    rl.items([&](int it, int ch, int col) {
      const uint16_t *l = rl.slot(ch, col), *ln = rl.lab + threadIdx.x % NS;
      const uint32_t mask = run_mask(r, ch), s0 = run_starts(rl.qm[it], mask);
      // the coins' changes from run to run, then summed upwards
      uint32_t f = 0, prev = 0;
      for (uint32_t st = s0; st; st &= st - 1u) {
        const uint32_t bit = st & (0u - st);
        const uint32_t c = ln[(l[(31 - __clz(bit)) * zs] & 0x7FFF) * NS] >> 15;
        if (c != prev) f |= bit;
        prev = c;
      }
      f ^= f << 1; f ^= f << 2; f ^= f << 4; f ^= f << 8; f ^= f << 16;
      rl.cx[it] = f & mask;
    });
    __syncthreads();
    rl.bytes([&](int j, int sg, int ch, int col, int n) {
      const uint8_t *f = reinterpret_cast<const uint8_t *>(rl.cx + (size_t)sg * NS) + j;
      u64 x = 0;
#pragma unroll
      for (int l = 0; l < NS; ++l) x |= (u64)f[4 * l] << (8 * l);
      x = transpose8(x) << (NS * h);
      const int i0 = (ch * r.H + 8 * j) * r.S + col;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (k >= n) break;
        const int i = i0 + k * r.S;
        const uint8_t byte = (uint8_t)(x >> (8 * k));
        if (NS == 8) Qb[(size_t)i * 8] = byte;
        else if (h == 0) rl.fb[i] = byte;
        else if (h < 8 / NS - 1) rl.fb[i] |= byte;
        else Qb[(size_t)i * 8] = rl.fb[i] | byte;
      }
    });
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Lattices above kSpClusterMaxV sites, one-job path: slabs of slabD z planes
// labelled by runs in SMEM, slabNS samples at a time, each site's label written
// as a global site index into slab_lab [unit = lattice * 8 + group][8][V];
// then the bonds between slabs joined by the lock-free union of the
// multispin path (cc_unite: a root hung below the smaller one with
// atomicMin), the roots' coins drawn (slab_coin [unit][V], one bit a sample),
// and the flip bytes written in place of the overlap bytes.  Labels only decrease and never drop below
// the smallest site of their cluster, so the roots -- and the coins and
// flips -- are those of the one-CTA labelling.
// ---------------------------------------------------------------------------
template <int NS>
__device__ __forceinline__ void sp_slab_body(const SpDev &d, int unit, int sl, unsigned char *sm) {
  const int V = d.V, L2 = d.L * d.L, z0 = sl * d.slabD, nz = min(d.slabD, d.Lz - z0);
  const int base = z0 * L2, Vs = nz * L2;
  const int grp = unit & 7, lat = unit >> 3;
  const uint8_t *Qb = reinterpret_cast<const uint8_t *>(d.Q + (size_t)lat * V) + grp;
  const RunLab<NS> rl(sm, d.L, nz);
  const RunShape &r = rl.r;
  rl.load(Qb + (size_t)base * 8);
  uint32_t *Lu = d.slab_lab + (size_t)unit * 8 * V + base;
  for (int h = 0; h < 8 / NS; ++h) {
    rl.words(h);
    rl.label(false, false, [](int, int, uint32_t eq) { return eq; });
    rl.jump([](uint16_t *, int, uint32_t) {});
    __syncthreads();
    for (int i = threadIdx.x; i < Vs; i += blockDim.x) {
      const int z = i / L2, col = i - z * L2, ch = z / r.H;
      const uint32_t low = (2u << (z - ch * r.H)) - 1u;
      const uint32_t *m = rl.qm + (size_t)(ch * L2 + col) * NS;
      const uint16_t *l = rl.lab + ((size_t)ch * r.H * L2 + col) * NS;
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const int zr = 31 - __clz(run_starts(m[s], low));
        Lu[(size_t)(h * NS + s) * V + i] = (uint32_t)(base + l[(size_t)zr * L2 * NS + s]);
      }
    }
    __syncthreads();
  }
}

// Bonds between slabs, each once, from its larger end, which is in a slab's
// first plane or (the z wrap and the corner bonds between the open planes) in
// the lattice's last: sp_face_planes of them a unit.  (Over all sites it took
// 190 us at 24^2 x 192, 128 units, over 13 of its 192 planes 68.)
__host__ __device__ inline int sp_face_planes(int Lz, int D) { return (Lz + D - 1) / D; }
__device__ __forceinline__ void sp_slab_merge_body(const SpDev &d, long long t) {
  const int V = d.V, L2 = d.L * d.L, nf = sp_face_planes(d.Lz, d.slabD), per = nf * L2;
  if (t >= (long long)d.nw * d.nclust * 8 * per) return;
  const int unit = (int)(t / per), e = (int)(t - (long long)unit * per), f = e / L2;
  // planes D, 2 D, ... and the last one, which may be one of them
  const int z = f + 1 < nf ? (f + 1) * d.slabD : d.Lz - 1;
  if (f + 1 == nf && nf > 1 && z == (nf - 1) * d.slabD) return;
  const int gi = z * L2 + e - f * L2;
  const int grp = unit & 7, lat = unit >> 3;
  const uint8_t *Qb = reinterpret_cast<const uint8_t *>(d.Q + (size_t)lat * V) + grp;
  const int s1 = gi / L2 / d.slabD;
  const uint32_t qi = Qb[(size_t)gi * 8];
  uint32_t *Lu = d.slab_lab + (size_t)unit * 8 * V;
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    const int p = __ldg(d.nb + (size_t)gi * 6 + q);
    if (p >= gi || p / L2 / d.slabD == s1) continue;
    const uint32_t eq = ~(qi ^ Qb[(size_t)p * 8]) & 0xFFu;
    for (int l = 0; l < 8; ++l)
      if ((eq >> l) & 1u) cc_unite(Lu + (size_t)l * V, (uint32_t)gi, (uint32_t)p);
  }
}

// Coins of the roots, the sites that are their own label: t = unit * V + site.
__device__ __forceinline__ void sp_slab_coins_body(const SpDev &d, int g, long long t) {
  const int V = d.V, nc = d.nclust;
  if (t >= (long long)d.nw * nc * 8 * V) return;
  const int unit = (int)(t / V), gi = (int)(t - (long long)unit * V);
  const int grp = unit & 7, lat = unit >> 3, b = lat % nc, w = lat / nc;
  const uint32_t *Lu = d.slab_lab + (size_t)unit * 8 * V + gi;
  uint32_t roots = 0, coins = 0;
#pragma unroll
  for (int l = 0; l < 8; ++l) roots |= (uint32_t)(Lu[(size_t)l * V] == (uint32_t)gi) << l;
  if (!roots) return;
  const unsigned long long key = sp_cluster_key(d), mv = *d.move;
#pragma unroll 1
  for (uint32_t m = roots; m; m &= m - 1) {
    const int l = __ffs(m) - 1, lane = grp * 8 + l;
    const uint32_t tag = (((uint32_t)(w * 64 + lane) << 6 | (uint32_t)b) << 1) | (uint32_t)g;
    uint32_t v0 = (uint32_t)mv, v1 = (uint32_t)(mv >> 32), v2 = (uint32_t)gi, v3 = tag;
    philox10(v0, v1, v2, v3, (uint32_t)key, (uint32_t)(key >> 32));
    coins |= (v0 & 1u) << l;
  }
  d.slab_coin[(size_t)unit * V + gi] = (uint8_t)coins;
}

// Flip bytes from the roots' coins, in place of the overlap bytes: the eight
// samples' chains of labels followed together.  What bounds it and the coins
// is the reads of the labels (2 x 453 MB at 24^2 x 192, 16 slots, one word: 133
// us at the copy rate).  Writing every site's root back first, one chain after
// another, took 389 us and the flip bytes 93; coins and flip bytes take
// 101 and 191.
__device__ __forceinline__ void sp_slab_flip_body(const SpDev &d, long long t) {
  const int V = d.V;
  if (t >= (long long)d.nw * d.nclust * 8 * V) return;
  const int unit = (int)(t / V), gi = (int)(t - (long long)unit * V);
  const int grp = unit & 7, lat = unit >> 3;
  const uint32_t *Lu = d.slab_lab + (size_t)unit * 8 * V;
  const uint8_t *Cu = d.slab_coin + (size_t)unit * V;
  uint32_t x[8], f = 0;
#pragma unroll
  for (int l = 0; l < 8; ++l) x[l] = Lu[(size_t)l * V + gi];
  bool more;
  do {
    uint32_t y[8];
    more = false;
#pragma unroll
    for (int l = 0; l < 8; ++l) y[l] = Lu[(size_t)l * V + x[l]];
#pragma unroll
    for (int l = 0; l < 8; ++l) {
      more = more || y[l] != x[l];
      x[l] = y[l];
    }
  } while (more);
#pragma unroll
  for (int l = 0; l < 8; ++l) f |= (uint32_t)((Cu[x[l]] >> l) & 1u) << l;
  reinterpret_cast<uint8_t *>(d.Q + (size_t)lat * V)[(size_t)gi * 8 + grp] = (uint8_t)f;
}

// Labelling of one CTA's (word, slot, 8 samples) by lattice size.
__device__ __forceinline__ void sp_cluster_any(const SpDev &d, int g, int blk, unsigned char *sm) {
  switch (run_samples(d.L, d.Lz)) {
    case 8: sp_cluster_runs<8>(d, g, blk, sm); break;
    case 4: sp_cluster_runs<4>(d, g, blk, sm); break;
    case 2: sp_cluster_runs<2>(d, g, blk, sm); break;
    case 1: sp_cluster_runs<1>(d, g, blk, sm); break;
    default: sp_cluster_body(d, g, blk, reinterpret_cast<uint32_t *>(sm));  // wide flat lattices; global scratch
  }
}

// Both replicas of the group take the flip words: thread per (word, site, slot).
__device__ __forceinline__ void sp_flip_body(const SpDev &d, int g, long long t) {
  const int V = d.V, nc = d.nclust;
  if (t >= (long long)d.nw * V * nc) return;
  const int b = (int)(t % nc), i = (int)((t / nc) % V), w = (int)(t / ((long long)nc * V));
  const u64 F = d.Q[((size_t)w * nc + b) * V + i];
  if (!F) return;
  const int r1 = d.pairs[2 * g], r2 = d.pairs[2 * g + 1];
  u64 *p = d.S + (((size_t)w * V + i) * d.NR) * d.NB + b;
  p[(size_t)r1 * d.NB] ^= F;
  p[(size_t)r2 * d.NB] ^= F;
}

// Energy measurement of a bin's iteration: avgE += 3V - U2 (slot order).
// from_e: the measurement follows a tempering step directly (no cluster
// move in between), whose E already holds the energy of the configuration
// now at each slot (energies move with their configurations): no recount.
__device__ __forceinline__ void sp_measure_u2_body(const SpDev &d, long long i, int from_e) {
  if (i < (long long)d.nw * 64 * d.NR * d.NB) d.avgE[i] += from_e ? (double)d.E[i] : (double)(3 * d.V - d.U2[i]);
}

// ---------------------------------------------------------------------------
// Exact enumeration: for every sample of every word, the number of spin
// configurations at each energy E = 3V - U2 among the 2^(V-1) with spin 0 up
// (E is even under the global flip, so the full counts are twice these; the
// averages do not change).  Block row y = sample.  A thread walks 2^12
// configurations in Gray-code order from a prefix of the higher spins:
// flipping spin k changes U2 by 2 (6 - 2 n_k), n_k = unsatisfied slots at k.
// Counts go to a per-block SMEM histogram, then to the 64-bit global one.
// ---------------------------------------------------------------------------
constexpr int kDosLow = 12;

__global__ void __launch_bounds__(256) k_sp_dos(const __grid_constant__ SpDev d, int nprefix_bits) {
  __shared__ uint32_t h[6 * 32 + 1];
  const int V = d.V, nbins = 6 * V + 1;
  const int sample = blockIdx.y, w = sample / 64, lane = sample % 64;
  __shared__ int s_nb[32 * 6];
  __shared__ uint8_t s_j[32 * 6];
  for (int i = threadIdx.x; i < nbins; i += blockDim.x) h[i] = 0;
  for (int i = threadIdx.x; i < V * 6; i += blockDim.x) {
    s_nb[i] = d.nb[i];
    s_j[i] = (uint8_t)((d.J[(size_t)w * V * 6 + i] >> lane) & 1ull);
  }
  __syncthreads();
  const int nlow = min(kDosLow, V - 1);
  const uint64_t prefix = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (prefix < (1ull << nprefix_bits)) {
    // configuration bits: spin 0 up (bit 0 = 0), spins 1..nlow by Gray code,
    // the rest from the prefix
    uint32_t s = (uint32_t)(prefix << (nlow + 1));
    auto unsat = [&](int k) {
      int n = 0;
      const int sk = (s >> k) & 1;
#pragma unroll
      for (int q = 0; q < 6; ++q) n += sk ^ (int)((s >> s_nb[k * 6 + q]) & 1u) ^ s_j[k * 6 + q];
      return n;
    };
    int U2 = 0;
    for (int k = 0; k < V; ++k) U2 += unsat(k);
    atomicAdd(&h[3 * V - U2 + 3 * V], 1u);
    for (uint32_t g = 1; g < (1u << nlow); ++g) {
      const int k = __ffs(g);  // Gray step g flips spin 1 + (trailing zeros of g)
      const int nk = unsat(k);
      U2 += 2 * (6 - 2 * nk);
      s ^= 1u << k;
      atomicAdd(&h[3 * V - U2 + 3 * V], 1u);
    }
  }
  __syncthreads();
  unsigned long long *out = d.dos + (size_t)sample * nbins;
  for (int i = threadIdx.x; i < nbins; i += blockDim.x)
    if (h[i]) atomicAdd(out + i, (unsigned long long)h[i]);
}

// <E>(beta) of each sample from its density of states, in FP64: weights
// g(E) exp(beta (E - Emax)) over the bins.
__global__ void k_sp_exact(const __grid_constant__ SpDev d, const double *betas, int nbeta, double *meanE) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int V = d.V, nbins = 6 * V + 1;
  if (t >= d.nw * 64 * nbeta) return;
  const int sample = t / nbeta, k = t % nbeta;
  const unsigned long long *g = d.dos + (size_t)sample * nbins;
  int emax = -3 * V;
  for (int i = 0; i < nbins; ++i)
    if (g[i]) emax = i - 3 * V;
  double Z = 0, ZE = 0;
  for (int i = 0; i < nbins; ++i) {
    if (!g[i]) continue;
    const int E = i - 3 * V;
    const double wgt = (double)g[i] * exp(betas[k] * (double)(E - emax));
    Z += wgt;
    ZE += wgt * (double)E;
  }
  meanE[t] = ZE / Z;
}

// ---------------------------------------------------------------------------
// Batched kernels: block b works for job j with pre[j] <= b < pre[j+1], on the
// job's block b - pre[j]; the bodies are the one-job kernels', so a job's
// words are the same alone and in a batch.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int spb_job(const uint32_t *pre, int n, uint32_t v) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(pre + mid) <= v) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// The block's job descriptor is copied to SMEM once (SMEM cannot alias the
// job's global arrays, and a per-thread copy would go to the stack).
#define SPB_ITEM(KIND)                                        \
  __shared__ SpDev s_job;                                     \
  const uint32_t *pre_ = b.pre[KIND];                         \
  const int jb = spb_job(pre_, b.njobs, blockIdx.x);          \
  if (threadIdx.x == 0) s_job = b.jobs[jb];                   \
  __syncthreads();                                            \
  const SpDev &d = s_job;                                     \
  const int blk = (int)(blockIdx.x - __ldg(pre_ + jb));

__global__ void __launch_bounds__(512, 2) kb_sp_pass(const __grid_constant__ SpBatchDev b, int sweep, int colour) {
  extern __shared__ __align__(16) unsigned char smem[];
  SPB_ITEM(SPB_PASS0 + colour)
  sp_pass_any(d, d.ctrs + (size_t)(sweep * d.ncol + colour) * d.NR, colour, blk, smem);
}
__global__ void kb_sp_zero(const __grid_constant__ SpBatchDev b) {
  SPB_ITEM(SPB_ZERO)
  const long long i = (long long)blk * blockDim.x + threadIdx.x;
  if (i < (long long)d.nw * 64 * d.NR * d.NB) d.U2[i] = 0;
}
__global__ void __launch_bounds__(kEnMaxThreads, 4) kb_sp_energy(const __grid_constant__ SpBatchDev b) {
  extern __shared__ __align__(16) unsigned char smem[];
  SPB_ITEM(SPB_ENERGY)
  sp_energy_body(d, blk, smem);
}
__global__ void __launch_bounds__(kPtThreads) kb_sp_pt(const __grid_constant__ SpBatchDev b) {
  extern __shared__ __align__(16) unsigned char smem[];
  SPB_ITEM(SPB_PT)
  sp_pt_body(d, blk, smem);
}
__global__ void __launch_bounds__(kPermRows) kb_sp_permute(const __grid_constant__ SpBatchDev b) {
  extern __shared__ u64 rows[];
  SPB_ITEM(SPB_PERMUTE)
  sp_permute_body(d, blk, rows);
}
__global__ void kb_sp_measure(const __grid_constant__ SpBatchDev b, int from_e) {
  SPB_ITEM(SPB_MEASURE)
  sp_measure_u2_body(d, (long long)blk * blockDim.x + threadIdx.x, from_e);
}
__global__ void kb_sp_pairs(const __grid_constant__ SpBatchDev b) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < b.njobs && b.jobs[j].nclust > 0) sp_pairs_body(b.jobs[j]);
}
__global__ void kb_sp_overlap(const __grid_constant__ SpBatchDev b, int g) {
  SPB_ITEM(SPB_OVL0 + g)
  sp_overlap_body(d, g, (long long)blk * blockDim.x + threadIdx.x);
}
__global__ void __launch_bounds__(1024, 1) kb_sp_cluster(const __grid_constant__ SpBatchDev b, int g) {
  extern __shared__ __align__(16) uint32_t sm[];
  SPB_ITEM(SPB_CL0 + g)
  sp_cluster_any(d, g, blk, reinterpret_cast<unsigned char *>(sm));
}
__global__ void kb_sp_flip(const __grid_constant__ SpBatchDev b, int g) {
  SPB_ITEM(SPB_FL0 + g)
  sp_flip_body(d, g, (long long)blk * blockDim.x + threadIdx.x);
}

size_t sp_cluster_smem(int L, int Lz);

// Blocks of job d for each batched kernel kind (the one-job launch geometry).
void sp_batch_blocks(const SpDev &d, bool cluster, uint32_t out[SPB_COUNT]) {
  const long long G = (long long)d.NR * d.NB, nw = d.nw;
  for (int k = 0; k < SPB_COUNT; ++k) out[k] = 0;
  for (int c = 0; c < kSpBatchMaxColours && c < d.ncol; ++c) {
    const long long n = d.col_off[c + 1] - d.col_off[c];
    out[SPB_PASS0 + c] = d.pgrid ? (uint32_t)((n * G + 512LL * kItemsPerThread - 1) / (512LL * kItemsPerThread))
                                 : (uint32_t)((n + d.kt - 1) / d.kt);
  }
  out[SPB_ZERO] = out[SPB_MEASURE] = (uint32_t)((nw * 64 * G + 255) / 256);
  out[SPB_ENERGY] = (uint32_t)en_blocks(d);
  out[SPB_PT] = (uint32_t)(nw * d.NR);
  out[SPB_PERMUTE] = (uint32_t)((nw * d.V * d.NR + kPermRows - 1) / kPermRows);
  if (cluster && d.nclust > 0) {
    const int ng = d.NR >= 4 ? 2 : 1;
    for (int g = 0; g < ng; ++g) {
      out[SPB_OVL0 + g] = out[SPB_FL0 + g] = (uint32_t)((nw * d.nclust * d.V + 255) / 256);
      out[SPB_CL0 + g] = (uint32_t)(nw * d.nclust * 8);
    }
  }
}

// Largest dynamic SMEM of a kernel: the 227 KB of a block less its static SMEM.
template <class K>
static cudaError_t max_dynamic_smem(K kernel) {
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, kernel);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - (int)fa.sharedSizeBytes);
}

cudaError_t sp_batch_setup() {
  cudaError_t e = max_dynamic_smem(kb_sp_pass);
  if (e == cudaSuccess) e = max_dynamic_smem(kb_sp_cluster);
  if (e == cudaSuccess) e = max_dynamic_smem(kb_sp_permute);
  if (e == cudaSuccess) e = sp_batch_ctr_setup();
  if (e == cudaSuccess) e = max_dynamic_smem(kb_sp_energy);
  if (e == cudaSuccess) e = max_dynamic_smem(kb_sp_pt);
  return e;
}

// Sweep `sweep` of the counters drawn last (sp_batch_ctr_chain), colour by colour.
cudaError_t sp_batch_sweep(const SpBatchDev &b, int ncol_max, int sweep, cudaStream_t st) {
  for (int c = 0; c < ncol_max; ++c)
    if (b.total[SPB_PASS0 + c]) kb_sp_pass<<<b.total[SPB_PASS0 + c], 512, b.pass_smem, st>>>(b, sweep, c);
  return cudaGetLastError();
}

static void spb_energy(const SpBatchDev &b, cudaStream_t st) {
  kb_sp_zero<<<b.total[SPB_ZERO], 256, 0, st>>>(b);
  kb_sp_energy<<<b.total[SPB_ENERGY], b.energy_threads, b.energy_smem, st>>>(b);
}

cudaError_t sp_batch_tempering(const SpBatchDev &b, cudaStream_t st) {
  spb_energy(b, st);
  kb_sp_pt<<<b.total[SPB_PT], kPtThreads, b.pt_smem, st>>>(b);
  kb_sp_permute<<<b.total[SPB_PERMUTE], kPermRows, b.perm_smem, st>>>(b);
  return cudaGetLastError();
}

cudaError_t sp_batch_houdayer(const SpBatchDev &b, cudaStream_t st) {
  kb_sp_pairs<<<(b.njobs + 127) / 128, 128, 0, st>>>(b);
  for (int g = 0; g < 2; ++g) {
    if (!b.total[SPB_CL0 + g]) continue;
    kb_sp_overlap<<<b.total[SPB_OVL0 + g], 256, 0, st>>>(b, g);
    kb_sp_cluster<<<b.total[SPB_CL0 + g], b.cluster_threads, b.cluster_smem, st>>>(b, g);
    kb_sp_flip<<<b.total[SPB_FL0 + g], 256, 0, st>>>(b, g);
  }
  return cudaGetLastError();
}

cudaError_t sp_batch_measure(const SpBatchDev &b, bool from_e, cudaStream_t st) {
  if (!from_e) spb_energy(b, st);
  kb_sp_measure<<<b.total[SPB_MEASURE], 256, 0, st>>>(b, from_e ? 1 : 0);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Persistent bin kernel: one cooperative launch runs whole bins of a set of
// jobs (one job, or a batch), every phase of the cadence -- colour passes
// with their counters, energies, tempering, permutes, Houdayer moves,
// measurements -- as a loop over the same packed (job, block) work list the
// batched kernels use, with a grid barrier between phases.  The bodies are
// the one-job kernels', in the same order, so the words are the same as with
// one launch per phase; what goes away is the launch and graph-node gap of
// every phase, which bounds jobs too small to fill the GPU.
// ---------------------------------------------------------------------------
constexpr int kPersistThreads = 512;
constexpr unsigned long long kBarrierWaitNs = 4000000000ull;  // 4 s

__device__ __forceinline__ unsigned long long sp_globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Grid barrier of a cooperative launch (every block resident): arrivals are
// counted in *bar (zero at launch); the k-th barrier of the launch waits for
// k x gridDim.x arrivals.  A wait gives up after kBarrierWaitNs, or as soon
// as another block has given up, counts that in *err and returns false; the
// kernel then returns, so no block waits for ever and the host reports the
// failure.
__device__ bool sp_grid_sync(const SpPersistDev &p, unsigned &epoch) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    ++epoch;
    const unsigned long long target = (unsigned long long)epoch * gridDim.x;
    __threadfence();
    atomicAdd(p.bar, 1ull);
    int ok = 1;
    const unsigned long long t0 = sp_globaltimer();
    for (;;) {
      unsigned long long v;
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p.bar) : "memory");
      if (v >= target) break;
      if (*(volatile int *)p.err) { ok = 0; break; }
      if (sp_globaltimer() - t0 > kBarrierWaitNs) { atomicAdd(p.err, 1); ok = 0; break; }
      __nanosleep(64);
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// The blocks of one work-list kind whose bodies need a whole thread block.
#define SPP_BLOCKS(KIND, BODY)                                                        \
  for (uint32_t vb = blockIdx.x; vb < b.total[KIND]; vb += gridDim.x) {              \
    __syncthreads();                                                                  \
    if (threadIdx.x == 0) {                                                           \
      const int jb_ = spb_job(b.pre[KIND], b.njobs, vb);                              \
      s_job[0] = b.jobs[jb_];                                                         \
      s_blk[0] = (int)(vb - __ldg(b.pre[KIND] + jb_));                                \
    }                                                                                 \
    __syncthreads();                                                                  \
    const SpDev &d = s_job[0];                                                        \
    const int blk = s_blk[0];                                                         \
    BODY;                                                                             \
  }

// Kinds whose one-job blocks have SUB threads and no barrier: each thread
// block takes kPersistThreads / SUB of them at a time.  They use no dynamic
// SMEM, so their job descriptors lie there.
#define SPP_SUB(KIND, SUB, BODY)                                                      \
  for (uint32_t vb0 = blockIdx.x * (kPersistThreads / SUB); vb0 < b.total[KIND];      \
       vb0 += gridDim.x * (kPersistThreads / SUB)) {                                 \
    const int sub = threadIdx.x / SUB, ltid = threadIdx.x % SUB;                      \
    SpDev *const sjob = reinterpret_cast<SpDev *>(smem);                              \
    const uint32_t vb = vb0 + sub;                                                    \
    __syncthreads();                                                                  \
    if (ltid == 0 && vb < b.total[KIND]) {                                            \
      const int jb_ = spb_job(b.pre[KIND], b.njobs, vb);                              \
      sjob[sub] = b.jobs[jb_];                                                        \
      s_blk[sub] = (int)(vb - __ldg(b.pre[KIND] + jb_));                              \
    }                                                                                 \
    __syncthreads();                                                                  \
    if (vb < b.total[KIND]) {                                                         \
      const SpDev &d = sjob[sub];                                                     \
      const int blk = s_blk[sub];                                                     \
      BODY;                                                                           \
    }                                                                                 \
  }

#define SPP_SYNC() \
  if (!sp_grid_sync(p, epoch)) return

__global__ void __launch_bounds__(kPersistThreads, 1) k_sp_persist(const __grid_constant__ SpPersistDev p) {
  extern __shared__ __align__(16) unsigned char smem[];
  // at most 512 bytes of static SMEM beside the widest tiles (sp_kt)
  __shared__ SpDev s_job[1];
  __shared__ int s_blk[kPersistThreads / 256];
  const SpBatchDev &b = p.b;
  unsigned epoch = 0;
  auto energy = [&]() -> bool {
    SPP_SUB(SPB_ZERO, 256, {
      const long long i = (long long)blk * 256 + ltid;
      if (i < (long long)d.nw * 64 * d.NR * d.NB) d.U2[i] = 0;
    })
    if (!sp_grid_sync(p, epoch)) return false;
    SPP_BLOCKS(SPB_ENERGY, sp_energy_body(d, blk, smem))
    return sp_grid_sync(p, epoch);
  };
  for (int it = 0; it < p.itmax; ++it) {
    for (int im = 0; im < p.mesfr; ++im) {
      for (int ih = 0; ih < p.houfr; ++ih) {
        for (int sw = 0; sw < p.ptfr; ++sw) {
          for (int c = 0; c < p.ncol_max; ++c) {
            for (int j = blockIdx.x; j < b.njobs; j += gridDim.x) {
              __syncthreads();
              if (threadIdx.x == 0) s_job[0] = b.jobs[j];
              __syncthreads();
              if (c < s_job[0].ncol) sp_fill_body(s_job[0]);
            }
            SPP_SYNC();
            SPP_BLOCKS(SPB_PASS0 + c, sp_pass_any(d, d.ctr, c, blk, smem))
            SPP_SYNC();
          }
        }
        if (!energy()) return;
        SPP_BLOCKS(SPB_PT, sp_pt_body(d, blk, smem))
        SPP_SYNC();
        SPP_BLOCKS(SPB_PERMUTE, sp_permute_body(d, blk, reinterpret_cast<u64 *>(smem)))
        SPP_SYNC();
      }
      if (p.cluster) {
        for (int j = blockIdx.x * kPersistThreads + threadIdx.x; j < b.njobs; j += gridDim.x * kPersistThreads)
          if (b.jobs[j].nclust > 0) sp_pairs_body(b.jobs[j]);
        SPP_SYNC();
        for (int g = 0; g < 2; ++g) {
          if (!b.total[SPB_CL0 + g]) continue;
          SPP_SUB(SPB_OVL0 + g, 256, sp_overlap_body(d, g, (long long)blk * 256 + ltid))
          SPP_SYNC();
          SPP_BLOCKS(SPB_CL0 + g, sp_cluster_any(d, g, blk, smem))
          SPP_SYNC();
          SPP_SUB(SPB_FL0 + g, 256, sp_flip_body(d, g, (long long)blk * 256 + ltid))
          SPP_SYNC();
        }
      }
    }
    if (p.cluster && !energy()) return;
    SPP_SUB(SPB_MEASURE, 256, sp_measure_u2_body(d, (long long)blk * 256 + ltid, !p.cluster))
    SPP_SYNC();
  }
}

#undef SPP_SYNC
#undef SPP_SUB
#undef SPP_BLOCKS

// Blocks of a cooperative launch of k_sp_persist with `smem` bytes of dynamic
// SMEM: every block resident at once (one per SM, the kernel's registers and
// SMEM allowing), and no more than the largest phase has work for.
int sp_persist_grid(const SpBatchDev &b, size_t smem) {
  int dev = 0, nsm = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 0;
  if (cudaFuncSetAttribute(k_sp_persist, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sp_persist, kPersistThreads, smem) != cudaSuccess ||
      per_sm < 1)
    return 0;
  uint32_t work = (uint32_t)b.njobs;
  for (int k = 0; k < SPB_COUNT; ++k) {
    const uint32_t sub = (k >= SPB_PASS0 && k <= SPB_PASS3) || k == SPB_ENERGY || k == SPB_PT || k == SPB_PERMUTE ||
                                 k == SPB_CL0 || k == SPB_CL1
                             ? 1 : kPersistThreads / 256;
    work = std::max(work, (b.total[k] + sub - 1) / sub);
  }
  return (int)std::min<uint32_t>(work, (uint32_t)(per_sm * nsm));
}

cudaError_t sp_launch_persist(const SpPersistDev &p, int grid, size_t smem, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(p.bar, 0, sizeof(unsigned long long), st);
  if (e != cudaSuccess) return e;
  void *args[] = {const_cast<SpPersistDev *>(&p)};
  return cudaLaunchCooperativeKernel((const void *)k_sp_persist, dim3(grid), dim3(kPersistThreads), args, smem, st);
}

// ---------------------------------------------------------------------------
// One-job kernels: the bodies above, one block per item
// ---------------------------------------------------------------------------
// Pseudo-random overlap words (a 64-bit mix of the index) for timing the
// labelling on clusters of a random overlap; only the autotuner uses it.
__global__ void k_sp_noise(unsigned long long *Q, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned long long x = (unsigned long long)i * 0x9E3779B97F4A7C15ull + 0x632BE59BD9B4E019ull;
  x ^= x >> 31; x *= 0xBF58476D1CE4E5B9ull; x ^= x >> 29; x *= 0x94D049BB133111EBull; x ^= x >> 32;
  Q[i] = x;
}
__global__ void __launch_bounds__(512, 2) k_sp_pass(const __grid_constant__ SpDev d, int pass, int off, int n) {
  extern __shared__ __align__(16) unsigned char smem[];
  sp_pass_body(d, d.ctrs + (size_t)pass * d.NR, off, n, blockIdx.x, smem);
}

__global__ void __launch_bounds__(kItemsThreads, 1) k_sp_pass_items(const __grid_constant__ SpDev d, int pass, int off,
                                                                     int n) {
  extern __shared__ __align__(16) unsigned char smem[];
  sp_pass_items_body(d, d.ctrs + (size_t)pass * d.NR, off, n, (long long)blockIdx.x * blockDim.x + threadIdx.x,
                     (long long)n * d.NR * d.NB, (long long)gridDim.x * blockDim.x, smem);
}
__global__ void __launch_bounds__(kEnMaxThreads, 4) k_sp_energy(const __grid_constant__ SpDev d) {
  extern __shared__ __align__(16) unsigned char smem[];
  sp_energy_body(d, blockIdx.x, smem);
}
__global__ void __launch_bounds__(kPtThreads) k_sp_pt(const __grid_constant__ SpDev d) {
  extern __shared__ __align__(16) unsigned char smem[];
  sp_pt_body(d, blockIdx.x, smem);
}
__global__ void __launch_bounds__(kPermRows) k_sp_permute(const __grid_constant__ SpDev d) {
  extern __shared__ u64 rows[];
  sp_permute_body(d, blockIdx.x, rows);
}
__global__ void k_sp_pairs(const __grid_constant__ SpDev d) {
  if (threadIdx.x == 0) sp_pairs_body(d);
}
__global__ void k_sp_overlap(const __grid_constant__ SpDev d, int g) {
  sp_overlap_body(d, g, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}
__global__ void __launch_bounds__(1024, 1) k_sp_cluster(const __grid_constant__ SpDev d, int g) {
  extern __shared__ __align__(16) uint32_t sm[];
  sp_cluster_any(d, g, blockIdx.x, reinterpret_cast<unsigned char *>(sm));
}
template <int NS>
__global__ void __launch_bounds__(1024, 1) k_sp_slab(const __grid_constant__ SpDev d) {
  extern __shared__ __align__(16) unsigned char sm8[];
  sp_slab_body<NS>(d, blockIdx.y, blockIdx.x, sm8);
}
__global__ void k_sp_slab_merge(const __grid_constant__ SpDev d) {
  sp_slab_merge_body(d, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}
__global__ void k_sp_slab_coins(const __grid_constant__ SpDev d, int g) {
  sp_slab_coins_body(d, g, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}
__global__ void k_sp_slab_flip(const __grid_constant__ SpDev d) {
  sp_slab_flip_body(d, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}
__global__ void k_sp_flip(const __grid_constant__ SpDev d, int g) {
  sp_flip_body(d, g, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}
__global__ void k_sp_measure_u2(const __grid_constant__ SpDev d, int from_e) {
  sp_measure_u2_body(d, (long long)blockIdx.x * blockDim.x + threadIdx.x, from_e);
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
size_t sp_cluster_smem(int L, int Lz);

size_t sp_sweep_smem(int NB, int NR, int kt) {
  return (size_t)NB * kPre11Stride + (size_t)NB * kt * NR * (16 + 8) + (size_t)kt * 7 * 4;
}
size_t sp_items_smem(int NB, int threads) { return (size_t)NB * kPre11Stride + threads / 32 * sizeof(ItemsWarp); }

// Grid of the per-item pass: every CTA resident at once (the kernel's
// registers and the threshold tables' SMEM allowing); 0 if none fits.
int sp_items_grid(int NB) {
  int dev = 0, nsm = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sp_pass_items, kItemsThreads, sp_items_smem(NB, kItemsThreads)) != cudaSuccess)
    return 0;
  return per_sm * nsm;
}

// Tile width: the smallest power of two whose random triples (NB x kt x NR)
// fill half of the CTA's 512 threads -- narrower tiles leave the CTA staging
// every threshold table for a few words -- then doubled while two tiles per
// SM remain and SMEM fits (large jobs amortise the staging over more sites).
int sp_kt(int NB, int NR, int nsites_colour) {
  int kt = 1;
  while (kt < 64 && NB * kt * NR < 256) kt <<= 1;
  const size_t lim = 227 * 1024 - 512;  // room for the kernels' static SMEM
  while (kt > 1 && sp_sweep_smem(NB, NR, kt) > lim) kt >>= 1;
  if (sp_sweep_smem(NB, NR, kt) > lim) return 0;
  auto two = [&](int k) { return 2 * (sp_sweep_smem(NB, NR, k) + 1536) <= 228 * 1024; };  // CTAs an SM
  while (kt < 32 && sp_sweep_smem(NB, NR, 2 * kt) <= lim && (two(2 * kt) || !two(kt)) &&
         (nsites_colour + 2 * kt - 1) / (2 * kt) >= 2 * 152)
    kt <<= 1;
  // In between, where whole rounds of the GPU make a colour shorter: 12^2 x 48
  // with 24 temperatures and 4 replicas takes 370 us a sweep of 4096 samples
  // with 8 sites a tile (1.4 rounds), 313 with 12 (0.95), of 256 samples 94 and
  // 82.  Never so wide that one CTA an SM is left: 24^2 x 96, 32 temperatures,
  // 128 samples takes 444 us with 16 sites, 571 with 24.
  auto rounds = [&](int k) {
    const int slots = two(k) ? 2 * 152 : 152, tiles = (nsites_colour + k - 1) / k;
    return (tiles + slots - 1) / slots;
  };
  int best = kt;
  for (int k = kt + 1; k < 2 * kt && k < 64 && sp_sweep_smem(NB, NR, k) <= lim && two(k) == two(kt); ++k)
    if (rounds(k) * k < rounds(best) * best) best = k;
  return best;
}

cudaError_t sp_setup() {
  cudaError_t e = cudaFuncSetAttribute(k_sp_pass, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - 512);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sp_pass_items, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  const int cl = (int)std::max(kRunSmem, (size_t)kSpClusterMaxV * 7);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sp_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, cl);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_sp_permute, cudaFuncAttributeMaxDynamicSharedMemorySize, kPermRows * 65 * 8);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sp_energy, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kEnSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sp_pt, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pt_smem(64));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sp_slab<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRunSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sp_slab<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRunSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sp_slab<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRunSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sp_slab<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRunSmem);
  return e;
}

// Colour pass `pass` of the counters drawn last (sp_launch_ctr_chain).
cudaError_t sp_launch_pass(const SpDev &d, int pass, int off, int n, cudaStream_t st) {
  if (n > 0 && d.pgrid > 0) {
    const long long blocks = ((long long)n * d.NR * d.NB + kItemsThreads - 1) / kItemsThreads;
    k_sp_pass_items<<<(unsigned)std::min<long long>(blocks, d.pgrid), kItemsThreads, sp_items_smem(d.NB, kItemsThreads), st>>>(
        d, pass, off, n);
  } else if (n > 0) {
    const int grid = (n + d.kt - 1) / d.kt;
    k_sp_pass<<<grid, 512, sp_sweep_smem(d.NB, d.NR, d.kt), st>>>(d, pass, off, n);
  }
  return cudaGetLastError();
}

cudaError_t sp_launch_energy(const SpDev &d, cudaStream_t st) {
  const int G = d.NR * d.NB;
  cudaError_t e = cudaMemsetAsync(d.U2, 0, sizeof(int32_t) * (size_t)d.nw * 64 * G, st);
  if (e != cudaSuccess) return e;
  const int nth = d.en.threads;
  k_sp_energy<<<(unsigned)en_blocks(d), nth, en_smem(d, nth), st>>>(d);
  return cudaGetLastError();
}

cudaError_t sp_launch_pt(const SpDev &d, cudaStream_t st) {
  k_sp_pt<<<d.nw * d.NR, kPtThreads, pt_smem(d.NB), st>>>(d);
  return cudaGetLastError();
}

cudaError_t sp_launch_permute(const SpDev &d, cudaStream_t st) {
  const long long n = (long long)d.nw * d.V * d.NR;
  k_sp_permute<<<(unsigned)((n + kPermRows - 1) / kPermRows), kPermRows, perm_smem(d.NB), st>>>(d);
  return cudaGetLastError();
}


size_t sp_cluster_smem(int L, int Lz) {
  const int ns = run_samples(L, Lz), V = L * L * Lz;
  return ns ? run_smem(run_shape(L, Lz), ns) : V <= kSpClusterMaxV ? (size_t)V * 7 : 0;
}

// Block size of the cluster labelling for a launch of `blocks` CTAs: its
// (column chunk, sample) items spread evenly over some passes, so that an SM's
// CTAs -- as many as SMEM, registers (56 a thread) and the launch leave it --
// take the most items side by side; of equal ones the smallest blocks, whose
// barriers hide behind other CTAs.  12 x 12 x 48: 768 threads (one CTA an SM, the
// passes that 1024 threads take) 4.91 ms a move, 512 6.51.  11 x 11 x 3, 24
// temperatures, 15 words: 224 threads 99 us a move, 992 (the fewest passes) 134;
// 15 x 15 x 3, 40 words: 384 272, 928 352; 10 x 10 x 10, 8 words: 288 85, 800 103.
// One word's launches of fewer CTAs than SMs keep the fewest passes.
int sp_cluster_threads(int L, int Lz, size_t blocks) {
  const int ns = run_samples(L, Lz);
  if (!ns) return 1024;
  const int items = run_shape(L, Lz).nseg * ns, few = (items + 1023) / 1024;
  const double smem = (double)sp_cluster_smem(L, Lz), most = std::max(1.0, blocks / 152.0);
  int best = 0;
  double rate = 0;  // items of an SM side by side, over all of a CTA's
  for (int p = few; p <= 3 * few + 4; ++p) {
    const int t = std::min(1024, ((items + p - 1) / p + 31) / 32 * 32);
    const double ctas = std::floor(std::min({227 * 1024 / (smem + 1024), 65536.0 / (56 * t), 2048.0 / t}));
    const double r = std::min(std::max(ctas, 1.0), most) / p;
    if (r >= 0.999 * rate) {
      best = t;
      rate = std::max(rate, r);
    }
    if (t <= 96) break;
  }
  return best;
}

// Planes per slab of the slab labelling of lattices above kSpClusterMaxV
// sites, and the samples labelled at a time: 8 when slabs of at least 6
// planes then fit SMEM (fewer planes leave more bonds to the union across
// slabs than the wider label slots save), else the fewest that give 6, else
// the thickest slab of any; 0 (the one-CTA labelling in global scratch) when
// a plane alone is too large or the labels of every (word, slot, group) would
// pass 4 GB.
int sp_slab_planes(int L, int Lz, int nw, int nclust, int *samples) {
  const long long L2 = (long long)L * L, V = L2 * Lz;
  if (V <= kSpClusterMaxV || L2 > 32768) return 0;
  if ((long long)nw * nclust * 8 * V * 33 > (4ll << 30)) return 0;
  int best = 0;
  for (int ns = 8; ns >= 1 && best < 6; ns >>= 1) {
    int D = 0;
    // at least two slabs: the z wrap is left to the union across slabs
    while (D < Lz - 1 && L2 * (D + 1) <= 65535 && run_smem(run_shape(L, D + 1), ns) <= kRunSmem) ++D;
    if (D > best) {
      best = D;
      if (samples) *samples = ns;
    }
  }
  return best;
}

cudaError_t sp_launch_houdayer(const SpDev &d, cudaStream_t st) {
  k_sp_pairs<<<1, 32, 0, st>>>(d);
  const int ng = d.NR >= 4 ? 2 : 1;
  for (int g = 0; g < ng; ++g) {
    const long long n = (long long)d.nw * d.nclust * d.V;
    k_sp_overlap<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(d, g);
    if (d.slabD > 0) {
      const int L2 = d.L * d.L, nslab = (d.Lz + d.slabD - 1) / d.slabD, nunits = d.nw * d.nclust * 8;
      const long long nu = (long long)nunits * d.V;
      const dim3 grid((unsigned)nslab, (unsigned)nunits);
      const size_t sm = run_smem(run_shape(d.L, d.slabD), d.slabNS);
      switch (d.slabNS) {
        case 8: k_sp_slab<8><<<grid, 1024, sm, st>>>(d); break;
        case 4: k_sp_slab<4><<<grid, 1024, sm, st>>>(d); break;
        case 2: k_sp_slab<2><<<grid, 1024, sm, st>>>(d); break;
        default: k_sp_slab<1><<<grid, 1024, sm, st>>>(d);
      }
      const long long nm = (long long)nunits * sp_face_planes(d.Lz, d.slabD) * L2;
      k_sp_slab_merge<<<(unsigned)((nm + 255) / 256), 256, 0, st>>>(d);
      k_sp_slab_coins<<<(unsigned)((nu + 255) / 256), 256, 0, st>>>(d, g);
      k_sp_slab_flip<<<(unsigned)((nu + 255) / 256), 256, 0, st>>>(d);
    } else {
      const size_t blocks = (size_t)d.nw * d.nclust * 8;
      const int threads = d.cthreads ? d.cthreads : sp_cluster_threads(d.L, d.Lz, blocks);
      k_sp_cluster<<<(unsigned)blocks, threads, sp_cluster_smem(d.L, d.Lz), st>>>(d, g);
    }
    k_sp_flip<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(d, g);
  }
  return cudaGetLastError();
}

cudaError_t sp_launch_measure_u2(const SpDev &d, bool from_e, cudaStream_t st) {
  const long long n = (long long)d.nw * 64 * d.NR * d.NB;
  k_sp_measure_u2<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(d, from_e ? 1 : 0);
  return cudaGetLastError();
}

cudaError_t sp_launch_dos(const SpDev &d, cudaStream_t st) {
  const int nlow = std::min(kDosLow, d.V - 1);
  const int npre = d.V - 1 - nlow;
  const unsigned long long nthreads = 1ull << npre;
  const dim3 grid((unsigned)((nthreads + 255) / 256), (unsigned)(d.nw * 64));
  k_sp_dos<<<grid, 256, 0, st>>>(d, npre);
  return cudaGetLastError();
}

cudaError_t sp_launch_exact(const SpDev &d, const double *betas, int nbeta, double *meanE, cudaStream_t st) {
  const int n = d.nw * 64 * nbeta;
  k_sp_exact<<<(n + 127) / 128, 128, 0, st>>>(d, betas, nbeta, meanE);
  return cudaGetLastError();
}

}  // namespace eagb

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
using namespace eagb;

namespace {
int spfail(int code, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  set_last_error(buf);
  if (code == EA_ERR_CUDA || code == EA_ERR_NOMEM) (void)cudaGetLastError();  // reported here, not by the next launch
  return code;
}
#define SCU(call)                                                                             \
  do {                                                                                        \
    cudaError_t e_ = (call);                                                                  \
    if (e_ != cudaSuccess) return spfail(EA_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
  } while (0)
}  // namespace

struct ea_sp {
  ea_sp_geom geom{};
  SpGraph g;
  int device = 0;
  cudaStream_t st = nullptr;
  SpDev d{};
  std::vector<void *> owned;
  std::vector<int32_t> expoff;
  bool exp_falls = false;             // no pair's table rises
  double *exptab = nullptr;
  bool have_temps = false;
  // one iteration of the bin cadence, replayed as a CUDA graph
  cudaGraphExec_t it_graph = nullptr;
  ea_cadence it_cad{};
  int q_cap = 0;  // slots the overlap buffer holds
  SpDev it_dev{};  // the descriptor the graph was captured with
  int last_itmax = 0;  // iterations of the last bin (alone or batched)
  // persistent bin kernel of the job alone (EA_BIN_*)
  int bin_mode = EA_BIN_AUTO;
  SpDev *p_jobs = nullptr;            // [1] descriptor of the work list
  uint32_t *p_pre = nullptr;          // [SPB_COUNT][2] block prefix sums
  unsigned long long *p_bar = nullptr;
  int *p_err = nullptr;
  SpDev p_up{};                       // descriptor last uploaded
  bool p_valid = false;
  // resident bin kernel (EA_BIN_RESIDENT): plan for the descriptor r_dev,
  // Philox counters and random words of one launch's passes
  SpResPlan r_plan{};
  SpDev r_dev{};
  int r_state = 0;                    // 0: not planned, 1: eligible, 2: not eligible
  uint4 *r_ctrs = nullptr;
  unsigned long long *r_R = nullptr;
  int32_t *r_X = nullptr;
  size_t r_cap_pass = 0, r_cap_sweep = 0, r_cap_pt = 0;
  bool pair_energy = false;           // see sp_pair_energy
};

namespace {
template <class T>
int sp_own(ea_sp *c, T *&p, size_t n) {
  cudaError_t e = cudaMalloc((void **)&p, sizeof(T) * (n ? n : 1));
  if (e != cudaSuccess) return spfail(EA_ERR_NOMEM, "cudaMalloc(%zu bytes): %s", sizeof(T) * n, cudaGetErrorString(e));
  c->owned.push_back((void *)p);
  cudaMemsetAsync(p, 0, sizeof(T) * (n ? n : 1), c->st);
  return EA_OK;
}

bool geom_ok(const ea_sp_geom *g) {
  return g && g->nbetas >= 2 && g->nbetas <= 64 && g->nrep >= 1 && g->nrep <= 64 && g->nwords >= 1 &&
         g->nwords <= (1 << 20);
}
}  // namespace

extern "C" {

int ea_sp_graph(int32_t L, int32_t Lz, int32_t bc, int32_t *nb, int32_t *mate, uint8_t *colour, int32_t *ncol) {
  SpGraph g;
  if (!sp_graph(L, Lz, bc, g)) return spfail(EA_ERR_ARG, "tube %d x %d x %d (bc %d) not supported", L, L, Lz, bc);
  if (nb) std::memcpy(nb, g.nb.data(), g.nb.size() * 4);
  if (mate) std::memcpy(mate, g.mate.data(), g.mate.size() * 4);
  if (colour) std::memcpy(colour, g.colour.data(), g.colour.size());
  if (ncol) *ncol = g.ncol;
  return EA_OK;
}

int ea_sp_host_init(const ea_sp_geom *gp, uint64_t seed_J, uint64_t seed_u, uint64_t *J, uint64_t *S) {
  SpGraph g;
  if (!geom_ok(gp) || !sp_graph(gp->L, gp->Lz, gp->bc, g)) return spfail(EA_ERR_ARG, "bad sample-packed geometry");
  if (J) sp_couplings(g, gp->nwords, seed_J, J);
  if (S) sp_spins(g, gp->nwords, gp->nrep, gp->nbetas, seed_u, S);
  return EA_OK;
}

int ea_sp_presearch11(const uint64_t *cum, uint8_t *pre) {
  if (!cum || !pre) return spfail(EA_ERR_ARG, "null argument");
  if (cum[255] != ~0ULL) return spfail(EA_ERR_ARG, "threshold 255 is not 2^64-1");
  presearch(cum, 11, pre);
  return EA_OK;
}

int ea_sp_create(const ea_sp_geom *gp, int32_t device, ea_sp **out) {
  if (!gp || !out) return spfail(EA_ERR_ARG, "null argument");
  if (!geom_ok(gp)) return spfail(EA_ERR_ARG, "2 <= nbetas <= 64, 1 <= nrep <= 64, nwords >= 1");
  ea_sp *c = new ea_sp();
  c->geom = *gp;
  if (!sp_graph(gp->L, gp->Lz, gp->bc, c->g)) {
    delete c;
    return spfail(EA_ERR_ARG, "tube %d x %d x %d (bc %d) not supported", gp->L, gp->L, gp->Lz, gp->bc);
  }
  const SpGraph &g = c->g;
  SpDev &d = c->d;
  d.L = g.L; d.Lz = g.Lz; d.V = g.V; d.bc = g.bc; d.NB = gp->nbetas; d.NR = gp->nrep; d.nw = gp->nwords;
  d.ncol = g.ncol;
  int maxc = 0;
  for (int k = 0; k < g.ncol; ++k) maxc = std::max(maxc, g.col_off[k + 1] - g.col_off[k]);
  d.kt = sp_kt(d.NB, d.NR, maxc);
  d.fd_NB.set((uint32_t)d.NB);
  d.esites = d.V;
  d.epair = 0;
  sp_energy_shape(d, sp_energy_chunk(d));
  for (int k = 0; k <= g.ncol && k < 9; ++k) d.col_off[k] = g.col_off[k];
  if (!d.kt) { delete c; return spfail(EA_ERR_ARG, "NB=%d x NR=%d does not fit in shared memory", d.NB, d.NR); }
  c->device = device;
  cudaError_t e = cudaSetDevice(device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&c->st, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = sp_setup();
  if (e == cudaSuccess) e = sp_res_setup();
  if (e != cudaSuccess) { delete c; return spfail(EA_ERR_CUDA, "set-up: %s", cudaGetErrorString(e)); }
  const size_t G = (size_t)d.NR * d.NB, V = g.V, nw = d.nw;
  int rc;
#define SOWN(p, n) if ((rc = sp_own(c, p, n)) != EA_OK) { ea_sp_destroy(c); return rc; }
  { int32_t *p; SOWN(p, V * 6); d.nb = p; }
  { int32_t *p; SOWN(p, V); d.col_sites = p; }
  SOWN(d.S, nw * V * G);
  { unsigned long long *p; SOWN(p, nw * V * 6); d.J = p; }
  { unsigned long long *p; SOWN(p, (size_t)d.NB * 256); d.cum = p; }
  { uint8_t *p; SOWN(p, (size_t)d.NB * kPre11Stride); d.pre11 = p; }
  SOWN(d.ctr, (size_t)d.NR);
  SOWN(d.ctrs, (size_t)kCtrPasses * d.NR);
  { uint32_t *p; SOWN(p, (size_t)d.NR); d.keys = p; }
  SOWN(d.prc, (size_t)d.NR);
  SOWN(d.xo, (size_t)d.NR);
  SOWN(d.iter, 1);
  SOWN(d.U2, nw * 64 * G);
  SOWN(d.E, nw * 64 * G);
  SOWN(d.perm, nw * 64 * G);
  SOWN(d.acc, nw * 64 * d.NR * (d.NB - 1));
  SOWN(d.M, nw * d.NR * (d.NB - 1));
  { double *p; SOWN(p, (size_t)d.NB); d.betas = p; }
  { int32_t *p; SOWN(p, (size_t)d.NB); d.expoff = p; }
  SOWN(d.ptstep, 1);
  SOWN(d.avgE, nw * 64 * G);
  SOWN(d.rc, 1);
  SOWN(d.pairs, 4);
  SOWN(d.move, 1);
#undef SOWN
  SCU(cudaMemcpyAsync((void *)d.nb, g.nb.data(), V * 6 * 4, cudaMemcpyHostToDevice, c->st));
  SCU(cudaMemcpyAsync((void *)d.col_sites, g.col_sites.data(), V * 4, cudaMemcpyHostToDevice, c->st));
  // identity slot -> configuration map
  std::vector<uint8_t> perm(nw * 64 * G);
  for (size_t i = 0; i < perm.size(); ++i) perm[i] = (uint8_t)(i % d.NB);
  SCU(cudaMemcpyAsync(d.perm, perm.data(), perm.size(), cudaMemcpyHostToDevice, c->st));
  SCU(cudaStreamSynchronize(c->st));
  // one-word jobs take the per-item pass: measured faster than every tile
  // width on one word (L=6 to 24, 12 to 32 temperatures); many words share
  // each tile's random words and keep the tiles
  if (nw == 1) d.pgrid = sp_items_grid(d.NB);
  *out = c;
  return EA_OK;
}

int ea_sp_destroy(ea_sp *c) {
  if (!c) return EA_OK;
  cudaSetDevice(c->device);
  if (c->st) cudaStreamSynchronize(c->st);
  for (void *p : c->owned) cudaFree(p);
  if (c->exptab) cudaFree(c->exptab);
  if (c->d.dos) cudaFree(c->d.dos);
  if (c->d.Q) cudaFree(c->d.Q);
  if (c->d.cscratch) cudaFree(c->d.cscratch);
  if (c->d.slab_lab) cudaFree(c->d.slab_lab);
  if (c->d.slab_coin) cudaFree(c->d.slab_coin);
  if (c->it_graph) cudaGraphExecDestroy(c->it_graph);
  if (c->p_jobs) cudaFree(c->p_jobs);
  if (c->p_pre) cudaFree(c->p_pre);
  if (c->p_bar) cudaFree(c->p_bar);
  if (c->p_err) cudaFree(c->p_err);
  if (c->r_ctrs) cudaFree(c->r_ctrs);
  if (c->r_R) cudaFree(c->r_R);
  if (c->r_X) cudaFree(c->r_X);
  if (c->st) cudaStreamDestroy(c->st);
  delete c;
  return EA_OK;
}

// The job's device view and stream, for the analysis entry points of
// sp_analysis.cu (current device set to the job's).
int ea_sp_device_view(ea_sp *c, SpDev *d, cudaStream_t *st) {
  if (!c || !d || !st) return spfail(EA_ERR_ARG, "null argument");
  SCU(cudaSetDevice(c->device));
  *d = c->d;
  *st = c->st;
  return EA_OK;
}

int ea_sp_info(const ea_sp *c, int32_t *ncol, int32_t *tile) {
  if (!c) return spfail(EA_ERR_ARG, "null job");
  if (ncol) *ncol = c->d.ncol;
  if (tile) *tile = c->d.pgrid ? 0 : c->d.kt;
  return EA_OK;
}

int ea_sp_stream(ea_sp *c, void **stream) {
  if (!c || !stream) return spfail(EA_ERR_ARG, "null argument");
  *stream = (void *)c->st;
  return EA_OK;
}

// After a synchronisation: did a persistent bin kernel give up on a barrier?
static int sp_check_persist(int *d_err, cudaStream_t st) {
  if (!d_err) return EA_OK;
  int err = 0;
  SCU(cudaMemcpyAsync(&err, d_err, sizeof(int), cudaMemcpyDeviceToHost, st));
  SCU(cudaStreamSynchronize(st));
  if (err) {
    SCU(cudaMemsetAsync(d_err, 0, sizeof(int), st));
    return spfail(EA_ERR_CUDA, "persistent bin kernel: a grid barrier wait gave up (%d blocks); the bin is incomplete", err);
  }
  return EA_OK;
}

int ea_sp_sync(ea_sp *c) {
  if (!c) return spfail(EA_ERR_ARG, "null job");
  SCU(cudaSetDevice(c->device));
  SCU(cudaStreamSynchronize(c->st));
  return sp_check_persist(c->p_err, c->st);
}

int ea_sp_set_tile(ea_sp *c, int32_t tile) {
  if (!c) return spfail(EA_ERR_ARG, "null job");
  SCU(cudaSetDevice(c->device));
  SpDev &d = c->d;
  if (tile == 0) {
    const int pg = sp_items_grid(d.NB);
    if (!pg) return spfail(EA_ERR_ARG, "the per-item pass does not fit NB=%d", d.NB);
    d.pgrid = pg;
    return EA_OK;
  }
  if (tile < 1 || tile > 64 || sp_sweep_smem(d.NB, d.NR, tile) > 227 * 1024 - 512)
    return spfail(EA_ERR_ARG, "tile %d: 1..64 sites whose tables fit in shared memory", tile);
  d.kt = tile;
  d.pgrid = 0;
  return EA_OK;
}

int ea_sp_set_bin_kernel(ea_sp *c, int32_t mode) {
  if (!c || mode < EA_BIN_AUTO || mode > EA_BIN_RESIDENT) return spfail(EA_ERR_ARG, "bad bin-kernel mode");
  c->bin_mode = mode;
  return EA_OK;
}

int ea_sp_set_temperatures(ea_sp *c, const double *betas, const uint64_t *cum) {
  if (!c || !betas || !cum) return spfail(EA_ERR_ARG, "null argument");
  const int NB = c->d.NB;
  for (int i = 0; i + 1 < NB; ++i)
    if (betas[i] < betas[i + 1]) return spfail(EA_ERR_ARG, "betas must be sorted from largest to smallest");
  std::vector<uint8_t> pre11((size_t)NB * kPre11Stride);
  for (int b = 0; b < NB; ++b) {
    if (cum[(size_t)b * 256 + 255] != ~0ULL) return spfail(EA_ERR_ARG, "threshold 255 of beta %d is not 2^64-1", b);
    presearch(cum + (size_t)b * 256, 11, pre11.data() + (size_t)b * kPre11Stride);
  }
  std::vector<double> tab;
  pt_exp_table(betas, NB, tab, c->expoff);
  SCU(cudaSetDevice(c->device));
  SCU(cudaStreamSynchronize(c->st));
  c->have_temps = false;  // until the new tables are in place
  if (c->exptab) cudaFree(c->exptab);
  c->exptab = nullptr;
  SCU(cudaMalloc((void **)&c->exptab, sizeof(double) * std::max<size_t>(1, tab.size())));
  SCU(cudaMemcpyAsync(c->exptab, tab.data(), sizeof(double) * tab.size(), cudaMemcpyHostToDevice, c->st));
  SCU(cudaMemcpyAsync((void *)c->d.cum, cum, sizeof(uint64_t) * 256 * NB, cudaMemcpyHostToDevice, c->st));
  SCU(cudaMemcpyAsync((void *)c->d.pre11, pre11.data(), pre11.size(), cudaMemcpyHostToDevice, c->st));
  SCU(cudaMemcpyAsync((void *)c->d.betas, betas, sizeof(double) * NB, cudaMemcpyHostToDevice, c->st));
  SCU(cudaMemcpyAsync((void *)c->d.expoff, c->expoff.data(), sizeof(int32_t) * NB, cudaMemcpyHostToDevice, c->st));
  SCU(cudaStreamSynchronize(c->st));
  c->d.exptab = c->exptab;
  c->have_temps = true;
  // the resident kernel's draws take the table's values to fall along each
  // pair's energies, as exp does
  c->exp_falls = true;
  for (int i = 0; i + 1 < NB; ++i)
    for (int k = c->expoff[i] + 1; k < c->expoff[i + 1]; ++k) c->exp_falls = c->exp_falls && tab[k] <= tab[k - 1];
  c->r_state = 0;
  return EA_OK;
}

int ea_sp_set_generators(ea_sp *c, const ea_generators *gen, uint64_t pt_seed) {
  if (!c || !gen) return spfail(EA_ERR_ARG, "null argument");
  const int NR = c->d.NR;
  SCU(cudaSetDevice(c->device));
  SCU(cudaMemcpyAsync(c->d.prc, gen->prc, sizeof(ea_hq) * NR, cudaMemcpyHostToDevice, c->st));
  SCU(cudaMemcpyAsync(c->d.xo, gen->xo, sizeof(ea_xoshiro) * NR, cudaMemcpyHostToDevice, c->st));
  SCU(cudaMemcpyAsync((void *)c->d.keys, gen->keys, sizeof(uint32_t) * NR, cudaMemcpyHostToDevice, c->st));
  SCU(cudaMemcpyAsync(c->d.rc, &gen->rc, sizeof(ea_hq), cudaMemcpyHostToDevice, c->st));
  SCU(cudaStreamSynchronize(c->st));
  c->d.pt_seed = pt_seed;
  return EA_OK;
}

int ea_sp_get_generators(ea_sp *c, ea_generators *gen) {
  if (!c || !gen) return spfail(EA_ERR_ARG, "null argument");
  const int NR = c->d.NR;
  std::memset(gen, 0, sizeof(*gen));
  SCU(cudaSetDevice(c->device));
  SCU(cudaMemcpyAsync(gen->prc, c->d.prc, sizeof(ea_hq) * NR, cudaMemcpyDeviceToHost, c->st));
  SCU(cudaMemcpyAsync(gen->xo, c->d.xo, sizeof(ea_xoshiro) * NR, cudaMemcpyDeviceToHost, c->st));
  SCU(cudaMemcpyAsync(gen->keys, c->d.keys, sizeof(uint32_t) * NR, cudaMemcpyDeviceToHost, c->st));
  SCU(cudaMemcpyAsync(&gen->rc, c->d.rc, sizeof(ea_hq), cudaMemcpyDeviceToHost, c->st));
  SCU(cudaStreamSynchronize(c->st));
  return EA_OK;
}

int ea_sp_init(ea_sp *c, const uint64_t seeds[4], uint32_t jobid) {
  if (!c || !seeds) return spfail(EA_ERR_ARG, "null argument");
  const SpDev &d = c->d;
  const size_t G = (size_t)d.NR * d.NB;
  std::vector<uint64_t> J((size_t)d.nw * d.V * 6), S((size_t)d.nw * d.V * G);
  sp_couplings(c->g, d.nw, seeds[0], J.data());
  sp_spins(c->g, d.nw, d.NR, d.NB, seeds[1], S.data());
  // Metropolis generators per replica as Init_Random seeds them
  // (random_generator.cu:94-158, 203-241), from seed_MC
  std::vector<uint64_t> sMC(d.NR);
  seeds_from_one(seeds[2], sMC.data(), d.NR);
  std::vector<ea_generators> gen(1);
  std::memset(gen.data(), 0, sizeof(ea_generators));
  for (int r = 0; r < d.NR; ++r) init_generators(sMC[r], gen[0].prc[r], gen[0].xo[r], gen[0].keys[r]);
  // replica-pair generator of the cluster moves, a Parisi-Rapuano stream
  // seeded from seed_PT as Init_Rand_HQ_64bits seeds one
  hq_seed(gen[0].rc, seeds[3]);
  int rc = ea_sp_set_couplings(c, J.data());
  if (!rc) rc = ea_sp_set_spins(c, S.data());
  if (!rc) rc = ea_sp_set_generators(c, gen.data(), seeds[3]);
  if (!rc) rc = ea_sp_set_counter(c, 0, 0, jobid);
  return rc;
}

int ea_sp_set_spins(ea_sp *c, const uint64_t *S) {
  if (!c || !S) return spfail(EA_ERR_ARG, "null argument");
  SCU(cudaSetDevice(c->device));
  SCU(cudaMemcpyAsync(c->d.S, S, (size_t)c->d.nw * c->d.V * c->d.NR * c->d.NB * 8, cudaMemcpyHostToDevice, c->st));
  SCU(cudaStreamSynchronize(c->st));
  return EA_OK;
}

int ea_sp_get_spins(ea_sp *c, uint64_t *S) {
  if (!c || !S) return spfail(EA_ERR_ARG, "null argument");
  SCU(cudaSetDevice(c->device));
  prefault(S, (size_t)c->d.nw * c->d.V * c->d.NR * c->d.NB * 8);
  SCU(cudaMemcpyAsync(S, c->d.S, (size_t)c->d.nw * c->d.V * c->d.NR * c->d.NB * 8, cudaMemcpyDeviceToHost, c->st));
  SCU(cudaStreamSynchronize(c->st));
  return EA_OK;
}

// Whether U2 equals twice the unsatisfied half-edges of the colour-1 sites:
// two colours, every half-edge's mate at the other end of its bond (on the
// other colour), and both ends holding the same coupling word.
static bool sp_pair_energy(const SpGraph &g, int nw, const uint64_t *J) {
  if (g.ncol != 2) return false;
  for (int h = 0; h < g.V * 6; ++h) {
    const int i = h / 6, m = g.mate[h], j = m / 6;
    if (m < 0 || m >= g.V * 6 || g.nb[h] != j || g.nb[m] != i || g.mate[m] != h || g.colour[i] == g.colour[j])
      return false;
    for (int w = 0; w < nw; ++w)
      if (J[(size_t)w * g.V * 6 + h] != J[(size_t)w * g.V * 6 + m]) return false;
  }
  return true;
}

int ea_sp_set_couplings(ea_sp *c, const uint64_t *J) {
  if (!c || !J) return spfail(EA_ERR_ARG, "null argument");
  SCU(cudaSetDevice(c->device));
  SCU(cudaMemcpyAsync((void *)c->d.J, J, (size_t)c->d.nw * c->d.V * 6 * 8, cudaMemcpyHostToDevice, c->st));
  SCU(cudaStreamSynchronize(c->st));
  c->pair_energy = sp_pair_energy(c->g, c->d.nw, J);
  c->d.epair = c->pair_energy ? 1 : 0;
  c->d.esites = c->pair_energy ? c->g.col_off[2] - c->g.col_off[1] : c->d.V;
  sp_energy_shape(c->d, sp_energy_chunk(c->d));
  return EA_OK;
}

int ea_sp_set_counter(ea_sp *c, int64_t iter, uint64_t ptstep, uint32_t jobid) {
  if (!c || jobid >= (1u << 14)) return spfail(EA_ERR_ARG, "job id < 2^14");
  SCU(cudaSetDevice(c->device));
  c->d.jobid = jobid;
  SCU(cudaMemcpyAsync(c->d.iter, &iter, 8, cudaMemcpyHostToDevice, c->st));
  SCU(cudaMemcpyAsync(c->d.ptstep, &ptstep, 8, cudaMemcpyHostToDevice, c->st));
  SCU(cudaStreamSynchronize(c->st));
  return EA_OK;
}

int ea_sp_get_counter(ea_sp *c, int64_t *iter, uint64_t *ptstep) {
  if (!c) return spfail(EA_ERR_ARG, "null job");
  SCU(cudaSetDevice(c->device));
  int64_t it = 0;
  uint64_t ps = 0;
  SCU(cudaMemcpyAsync(&it, c->d.iter, 8, cudaMemcpyDeviceToHost, c->st));
  SCU(cudaMemcpyAsync(&ps, c->d.ptstep, 8, cudaMemcpyDeviceToHost, c->st));
  SCU(cudaStreamSynchronize(c->st));
  if (iter) *iter = it;
  if (ptstep) *ptstep = ps;
  return EA_OK;
}

// Autotuner: times the launch shapes that leave the results unchanged -- the
// colour pass's tile width, the energy count's sites per thread and the
// labelling's block size -- on the job itself and keeps the fastest.  What
// the timing runs change (spin words, pass counter, Philox counters, the two
// generators feeding them, the energy counts) is copied aside on the device
// first and put back after; the labelling runs on pseudo-random overlap words
// in the job's overlap buffer, which every move rewrites.
static int sp_sweeps(ea_sp *c, int n);
static int sp_cluster_prepare(ea_sp *c, int &nclust);

int ea_sp_autotune(ea_sp *c, int32_t *tile, int32_t *echunk, int32_t *cthreads) {
  if (!c) return spfail(EA_ERR_ARG, "null job");
  if (!c->have_temps) return spfail(EA_ERR_STATE, "temperatures not set");
  SCU(cudaSetDevice(c->device));
  SpDev &d = c->d;
  const size_t G = (size_t)d.NR * d.NB;
  // whatever may be refused comes before the first timing run
  const bool cluster = d.V <= kSpClusterMaxV;  // lattices labelled in SMEM
  int nclust = 0;
  if (cluster) {
    const int rc = sp_cluster_prepare(c, nclust);
    if (rc) return rc;
  }
  struct Part { void *p; size_t n; };
  const Part parts[] = {{d.S, (size_t)d.nw * d.V * G * 8}, {d.iter, 8}, {d.ctr, sizeof(uint4) * d.NR},
                        {d.prc, sizeof(ea_hq) * d.NR}, {d.xo, sizeof(ea_xoshiro) * d.NR},
                        {d.U2, (size_t)d.nw * 64 * G * 4}};
  size_t total = 0;
  for (const Part &q : parts) total += (q.n + 255) & ~(size_t)255;
  char *save = nullptr;
  SCU(cudaMalloc((void **)&save, total));
  size_t off = 0;
  for (const Part &q : parts) {
    SCU(cudaMemcpyAsync(save + off, q.p, q.n, cudaMemcpyDeviceToDevice, c->st));
    off += (q.n + 255) & ~(size_t)255;
  }
  cudaEvent_t e0, e1;
  SCU(cudaEventCreate(&e0));
  SCU(cudaEventCreate(&e1));
  auto timed = [&](auto &&body) -> float {
    float best = 1e30f;
    for (int rep = 0; rep < 3; ++rep) {  // the first run warms up
      cudaEventRecord(e0, c->st);
      body();
      cudaEventRecord(e1, c->st);
      cudaEventSynchronize(e1);
      float ms = 0.f;
      cudaEventElapsedTime(&ms, e0, e1);
      if (rep) best = std::min(best, ms);
    }
    return cudaGetLastError() == cudaSuccess ? best : 1e30f;
  };
  int maxc = 0;
  for (int k = 0; k < d.ncol; ++k) maxc = std::max(maxc, d.col_off[k + 1] - d.col_off[k]);
  // colour pass: the heuristic's tile width and its neighbours that fit in
  // SMEM, and the per-item pass
  const int kt0 = d.kt, pg0 = d.pgrid;
  int best_kt = kt0, best_pg = pg0;
  float best = 1e30f;
  d.pgrid = 0;
  for (int kt : {kt0 / 2, kt0, kt0 * 2, kt0 * 4}) {
    if (kt < 1 || kt > 64 || sp_sweep_smem(d.NB, d.NR, kt) > 227 * 1024 - 512) continue;
    if ((maxc + kt - 1) / kt < 1) continue;
    d.kt = kt;
    const float ms = timed([&] { sp_sweeps(c, 2); });
    if (ms < best) { best = ms; best_kt = kt; best_pg = 0; }
  }
  d.kt = best_kt;
  if (const int pg = sp_items_grid(d.NB)) {
    d.pgrid = pg;
    const float ms = timed([&] { sp_sweeps(c, 2); });
    if (ms < best) { best = ms; best_pg = pg; }
  }
  d.pgrid = best_pg;
  // sites per thread of the energy count
  const int ec0 = d.echunk;
  int best_ec = ec0;
  best = 1e30f;
  for (int ec : {ec0 / 4, ec0 / 2, ec0, ec0 * 2, kEnSites}) {
    if (ec < 1 || ec > kEnSites) continue;
    sp_energy_shape(d, ec);
    const float ms = timed([&] { sp_launch_energy(d, c->st); });
    if (ms < best) { best = ms; best_ec = ec; }
  }
  sp_energy_shape(d, best_ec);
  // block size of the labelling
  int best_ct = d.cthreads;
  if (cluster) {
    const long long nq = (long long)d.nw * d.nclust * d.V;
    best = 1e30f;
    for (int ct : {256, 512, 1024}) {
      const float ms = timed([&] {
        k_sp_noise<<<(unsigned)((nq + 255) / 256), 256, 0, c->st>>>(d.Q, nq);
        k_sp_cluster<<<(unsigned)(d.nw * d.nclust * 8), ct, sp_cluster_smem(d.L, d.Lz), c->st>>>(d, 0);
      });
      if (ms < best) { best = ms; best_ct = ct; }
    }
  }
  d.cthreads = best_ct;
  off = 0;
  for (const Part &q : parts) {
    cudaMemcpyAsync(q.p, save + off, q.n, cudaMemcpyDeviceToDevice, c->st);
    off += (q.n + 255) & ~(size_t)255;
  }
  const cudaError_t e = cudaStreamSynchronize(c->st);
  cudaFree(save);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  SCU(e);
  if (tile) *tile = d.pgrid ? 0 : d.kt;
  if (echunk) *echunk = d.echunk;
  if (cthreads) *cthreads = d.cthreads ? d.cthreads : 1024;
  return EA_OK;
}

// The passes of n sweeps from pass `pass` of the counters drawn last.
static int sp_passes(ea_sp *c, int n, int pass) {
  const SpGraph &g = c->g;
  for (int s = 0; s < n; ++s)
    for (int k = 0; k < g.ncol; ++k)
      SCU(sp_launch_pass(c->d, pass++, g.col_off[k], g.col_off[k + 1] - g.col_off[k], c->st));
  return EA_OK;
}

static int sp_sweeps(ea_sp *c, int n) {
  while (n > 0) {
    const int m = std::min(n, kCtrPasses / c->g.ncol);
    SCU(sp_launch_ctr_chain(c->d, m * c->g.ncol, c->d.ctrs, c->st));
    const int rc = sp_passes(c, m, 0);
    if (rc) return rc;
    n -= m;
  }
  return EA_OK;
}

int ea_sp_sweeps(ea_sp *c, int32_t n) {
  if (!c || n < 0) return spfail(EA_ERR_ARG, "bad arguments");
  if (!c->have_temps) return spfail(EA_ERR_STATE, "temperatures not set");
  SCU(cudaSetDevice(c->device));
  return sp_sweeps(c, n);
}

int ea_sp_energy(ea_sp *c, int32_t *U2) {
  if (!c) return spfail(EA_ERR_ARG, "null job");
  SCU(cudaSetDevice(c->device));
  SCU(sp_launch_energy(c->d, c->st));
  if (U2) {
    prefault(U2, sizeof(int32_t) * (size_t)c->d.nw * 64 * c->d.NR * c->d.NB);
    SCU(cudaMemcpyAsync(U2, c->d.U2, sizeof(int32_t) * (size_t)c->d.nw * 64 * c->d.NR * c->d.NB,
                        cudaMemcpyDeviceToHost, c->st));
    SCU(cudaStreamSynchronize(c->st));
  }
  return EA_OK;
}

static int sp_pt(ea_sp *c) {
  SCU(sp_launch_energy(c->d, c->st));
  SCU(sp_launch_pt(c->d, c->st));
  SCU(sp_launch_permute(c->d, c->st));
  return EA_OK;
}

int ea_sp_parallel_tempering(ea_sp *c) {
  if (!c) return spfail(EA_ERR_ARG, "null job");
  if (!c->have_temps) return spfail(EA_ERR_STATE, "temperatures not set");
  SCU(cudaSetDevice(c->device));
  return sp_pt(c);
}

int ea_sp_get_tempering(ea_sp *c, int32_t *E, uint8_t *perm, uint32_t *acc, uint64_t *masks) {
  if (!c) return spfail(EA_ERR_ARG, "null job");
  const SpDev &d = c->d;
  const size_t n = (size_t)d.nw * 64 * d.NR * d.NB;
  SCU(cudaSetDevice(c->device));
  prefault(E, n * 4);
  prefault(perm, n);
  prefault(acc, (size_t)d.nw * 64 * d.NR * (d.NB - 1) * 4);
  prefault(masks, (size_t)d.nw * d.NR * (d.NB - 1) * 8);
  if (E) SCU(cudaMemcpyAsync(E, d.E, n * 4, cudaMemcpyDeviceToHost, c->st));
  if (perm) SCU(cudaMemcpyAsync(perm, d.perm, n, cudaMemcpyDeviceToHost, c->st));
  if (acc) SCU(cudaMemcpyAsync(acc, d.acc, (size_t)d.nw * 64 * d.NR * (d.NB - 1) * 4, cudaMemcpyDeviceToHost, c->st));
  if (masks) SCU(cudaMemcpyAsync(masks, d.M, (size_t)d.nw * d.NR * (d.NB - 1) * 8, cudaMemcpyDeviceToHost, c->st));
  SCU(cudaStreamSynchronize(c->st));
  return EA_OK;
}

// Overlap buffer for moves on nclust slots (allocated before any capture).
static int sp_cluster_prepare(ea_sp *c, int &nclust) {
  SpDev &d = c->d;
  if (d.NR < 2) return spfail(EA_ERR_ARG, "the Houdayer move needs 2 replicas");
  if (nclust <= 0) nclust = (int)std::lround(0.5 * d.NB);
  if (nclust > d.NB) nclust = d.NB;
  if (nclust > c->q_cap) {
    SCU(cudaStreamSynchronize(c->st));
    if (d.Q) cudaFree(d.Q);
    if (d.cscratch) cudaFree(d.cscratch);
    if (d.slab_lab) cudaFree(d.slab_lab);
    if (d.slab_coin) cudaFree(d.slab_coin);
    d.Q = nullptr;
    d.cscratch = nullptr;
    d.slab_lab = nullptr;
    d.slab_coin = nullptr;
    d.slabD = 0;
    c->q_cap = 0;  // until all of them are there
    SCU(cudaMalloc((void **)&d.Q, sizeof(unsigned long long) * (size_t)d.nw * nclust * d.V));
    if (d.V > kSpClusterMaxV) {
      SCU(cudaMalloc((void **)&d.cscratch, sizeof(uint32_t) * sp_cluster_words(d.V) * (size_t)d.nw * nclust * 8));
      int ns = 0;
      const int D = sp_slab_planes(d.L, d.Lz, d.nw, nclust, &ns);
      if (D > 0) {
        // without memory for the slabs' labels: in the scratch, one CTA a unit
        const size_t units = (size_t)d.nw * nclust * 8;
        if (cudaMalloc((void **)&d.slab_lab, sizeof(uint32_t) * units * 8 * d.V) == cudaSuccess &&
            cudaMalloc((void **)&d.slab_coin, units * d.V) == cudaSuccess) {
          d.slabD = D;
          d.slabNS = ns;
        } else {
          (void)cudaGetLastError();
          if (d.slab_lab) cudaFree(d.slab_lab);
          d.slab_lab = nullptr;
          d.slab_coin = nullptr;
        }
      }
    }
    c->q_cap = nclust;
  }
  d.nclust = nclust;
  return EA_OK;
}

static int sp_houdayer(ea_sp *c, int nclust) {
  const int rc = sp_cluster_prepare(c, nclust);
  if (rc) return rc;
  SCU(sp_launch_houdayer(c->d, c->st));
  return EA_OK;
}

int ea_sp_houdayer(ea_sp *c, int32_t nclust) {
  if (!c) return spfail(EA_ERR_ARG, "null job");
  SCU(cudaSetDevice(c->device));
  return sp_houdayer(c, nclust);
}

// EA_BIN_AUTO takes the graph.  Measured on GB300: a job alone, each phase of
// a small job is a latency-bound chain that a barrier does not shorten, and
// the graph's per-phase kernels run at twice the persistent kernel's
// occupancy (84 vs 106 us per sweep at L=6, Lz=24, NT=12); 64 small jobs of
// the serving mix, the phases in lock-step wait for each phase's slowest
// job, while the jobs' graphs on their own streams interleave (0.20 vs 0.42
// spin-updates/ps).
static bool sp_use_persist(int mode, const SpDev &) { return mode == EA_BIN_PERSISTENT; }

// The work list of the job alone (its blocks of every kind, as a batch of
// one), uploaded when the descriptor changed; then one cooperative launch.
static int sp_run_persist(ea_sp *c, const ea_cadence *cad) {
  const SpDev &d = c->d;
  if (d.ncol > kSpBatchMaxColours) return spfail(EA_ERR_ARG, "the persistent bin kernel takes up to %d colours", kSpBatchMaxColours);
  if (!c->p_jobs) SCU(cudaMalloc((void **)&c->p_jobs, sizeof(SpDev)));
  if (!c->p_pre) SCU(cudaMalloc((void **)&c->p_pre, sizeof(uint32_t) * SPB_COUNT * 2));
  if (!c->p_bar) SCU(cudaMalloc((void **)&c->p_bar, sizeof(unsigned long long)));
  if (!c->p_err) {
    SCU(cudaMalloc((void **)&c->p_err, sizeof(int)));
    SCU(cudaMemsetAsync(c->p_err, 0, sizeof(int), c->st));
  }
  uint32_t cnt[SPB_COUNT];
  sp_batch_blocks(d, cad->cluster != 0, cnt);
  if (!c->p_valid || std::memcmp(&c->p_up, &d, sizeof(SpDev))) {
    std::vector<uint32_t> pre((size_t)SPB_COUNT * 2);
    for (int k = 0; k < SPB_COUNT; ++k) { pre[2 * k] = 0; pre[2 * k + 1] = cnt[k]; }
    SCU(cudaMemcpyAsync(c->p_jobs, &d, sizeof(SpDev), cudaMemcpyHostToDevice, c->st));
    SCU(cudaMemcpyAsync(c->p_pre, pre.data(), sizeof(uint32_t) * pre.size(), cudaMemcpyHostToDevice, c->st));
    SCU(cudaStreamSynchronize(c->st));
    c->p_up = d;
    c->p_valid = true;
  }
  SpPersistDev p{};
  p.b.jobs = c->p_jobs;
  p.b.njobs = 1;
  for (int k = 0; k < SPB_COUNT; ++k) { p.b.pre[k] = c->p_pre + 2 * k; p.b.total[k] = cnt[k]; }
  p.itmax = cad->itmax; p.houfr = cad->houfr; p.mesfr = cad->mesfr; p.ptfr = cad->ptfr;
  p.cluster = cad->cluster != 0 && d.nclust > 0;
  p.ncol_max = d.ncol;
  p.bar = c->p_bar;
  p.err = c->p_err;
  size_t smem = std::max(d.pgrid ? sp_items_smem(d.NB, kPersistThreads) : sp_sweep_smem(d.NB, d.NR, d.kt), perm_smem(d.NB));
  smem = std::max(smem, std::max(en_smem(d, kPersistThreads), pt_smem(d.NB)));
  if (p.cluster) smem = std::max(smem, sp_cluster_smem(d.L, d.Lz));
  const int grid = sp_persist_grid(p.b, smem);
  if (grid < 1) return spfail(EA_ERR_CUDA, "persistent bin kernel: no co-resident grid for %zu bytes of shared memory", smem);
  SCU(sp_launch_persist(p, grid, smem, c->st));
  return EA_OK;
}

static bool sp_res_ok(ea_sp *c) {
  if (c->r_state == 0 || std::memcmp(&c->r_dev, &c->d, sizeof(SpDev))) {
    c->r_state = c->exp_falls && sp_res_plan(c->d, c->g.col_sites.data(), c->r_plan) ? 1 : 2;
    c->r_dev = c->d;
  }
  return c->r_state == 1;
}

// The resident path takes bins without cluster moves of jobs that fit one
// cluster: explicitly (EA_BIN_RESIDENT) or by default.
static bool sp_use_resident(ea_sp *c, const ea_cadence *cad) {
  if (c->bin_mode != EA_BIN_RESIDENT && c->bin_mode != EA_BIN_AUTO) return false;
  return sp_res_launch_sweeps(c->d.V, (size_t)c->d.NR * c->d.NB, cad) > 0 && sp_res_ok(c);
}

// The resident path's buffers for such bins: counters, random words, draws.
static int sp_res_buffers(ea_sp *c, const ea_cadence *cad) {
  const SpDev &d = c->d;
  const size_t words_sweep = (size_t)2 * d.V * d.NR * d.NB;
  const size_t nsweep = sp_res_launch_sweeps(d.V, (size_t)d.NR * d.NB, cad), npass = nsweep * d.ncol;
  const size_t npt = nsweep / cad->ptfr;                    // tempering steps per launch
  if (npass > c->r_cap_pass || nsweep > c->r_cap_sweep || npt > c->r_cap_pt) {
    SCU(cudaStreamSynchronize(c->st));
    if (c->r_ctrs) cudaFree(c->r_ctrs);
    if (c->r_R) cudaFree(c->r_R);
    if (c->r_X) cudaFree(c->r_X);
    c->r_ctrs = nullptr;
    c->r_R = nullptr;
    c->r_X = nullptr;
    c->r_cap_pass = c->r_cap_sweep = c->r_cap_pt = 0;
    SCU(cudaMalloc((void **)&c->r_ctrs, sizeof(uint4) * npass * d.NR));
    SCU(cudaMalloc((void **)&c->r_R, 8 * words_sweep * nsweep));
    SCU(cudaMalloc((void **)&c->r_X, 4 * npt * d.nw * d.NR * (d.NB - 1) * 64));
    c->r_cap_pass = npass;
    c->r_cap_sweep = nsweep;
    c->r_cap_pt = npt;
  }
  return EA_OK;
}

static int sp_run_resident(ea_sp *c, const ea_cadence *cad) {
  const SpDev &d = c->d;
  const SpResPlan &pl = c->r_plan;
  const int spi = cad->mesfr * cad->houfr * cad->ptfr;  // sweeps per iteration
  const size_t nsweep = sp_res_launch_sweeps(d.V, (size_t)d.NR * d.NB, cad);
  const int ipl = cad->cluster ? 1 : (int)(nsweep / spi);  // iterations per launch
  SpResDev p{};
  p.d = d;
  p.R = c->r_R;
  p.X = c->r_X;
  p.pair_energy = c->pair_energy ? 1 : 0;
  p.houfr = cad->houfr;
  p.mesfr = cad->mesfr;
  p.ptfr = cad->ptfr;
  p.ncta = pl.ncta;
  p.nslm = pl.nslm;
  p.parts = pl.parts;
  std::memcpy(p.kr, pl.kr, sizeof(p.kr));
  if (cad->cluster) {
    // per houfr block: one resident launch (sweeps and tempering steps, no
    // measurement), then the move's kernels on the words it wrote back; the
    // energies counted again and measured after each iteration, as the
    // graph path does
    p.nit = 1;
    p.mesfr = 1;
    p.nsweep = (int)nsweep;
    p.measure = 0;
    for (int it = 0; it < cad->itmax; ++it) {
      for (int im = 0; im < cad->mesfr; ++im) {
        SCU(sp_res_chunk(p, pl, p.nsweep * d.ncol, c->r_ctrs, c->st));
        SCU(sp_launch_houdayer(c->d, c->st));
      }
      SCU(sp_launch_energy(c->d, c->st));
      SCU(sp_launch_measure_u2(c->d, false, c->st));
    }
    return EA_OK;
  }
  p.measure = 1;
  for (int done = 0; done < cad->itmax;) {
    p.nit = std::min(ipl, cad->itmax - done);
    p.nsweep = p.nit * spi;
    SCU(sp_res_chunk(p, pl, p.nsweep * d.ncol, c->r_ctrs, c->st));
    done += p.nit;
  }
  return EA_OK;
}

int ea_sp_bin_kernel_for(ea_sp *c, const ea_cadence *cad, int32_t *mode) {
  if (!c || !cad || !mode || cad->itmax < 1 || cad->houfr < 1 || cad->mesfr < 1 || cad->ptfr < 1)
    return spfail(EA_ERR_ARG, "bad arguments");
  SCU(cudaSetDevice(c->device));
  if (sp_use_resident(c, cad)) *mode = EA_BIN_RESIDENT;
  else if (c->bin_mode == EA_BIN_RESIDENT) return spfail(EA_ERR_ARG, "the resident bin kernel does not take this bin");
  else *mode = c->bin_mode == EA_BIN_PERSISTENT ? EA_BIN_PERSISTENT : EA_BIN_GRAPH;
  return EA_OK;
}

int ea_sp_run(ea_sp *c, const ea_cadence *cad, double *avgE) {
  if (!c || !cad || cad->itmax < 1 || cad->houfr < 1 || cad->mesfr < 1 || cad->ptfr < 1)
    return spfail(EA_ERR_ARG, "bad cadence");
  if (!c->have_temps) return spfail(EA_ERR_STATE, "temperatures not set");
  SCU(cudaSetDevice(c->device));
  const SpDev &d = c->d;
  const size_t n = (size_t)d.nw * 64 * d.NR * d.NB;
  SCU(cudaMemsetAsync(d.avgE, 0, n * 8, c->st));
  int rc = EA_OK, nclust = cad->nclust;
  if (cad->cluster && (rc = sp_cluster_prepare(c, nclust))) return rc;
  if (c->bin_mode == EA_BIN_RESIDENT && !sp_use_resident(c, cad))
    return spfail(EA_ERR_ARG, "the resident bin kernel takes jobs whose words fit one thread-block cluster, bins "
                              "without cluster moves or with at least %d sweeps between moves", kResMinBlock);
  // without memory for the resident path's buffers the graph takes the bin,
  // unless the caller asked for the resident kernel
  const bool resident = sp_use_resident(c, cad);
  if (resident && (rc = sp_res_buffers(c, cad)) && c->bin_mode == EA_BIN_RESIDENT) return rc;
  if (resident && !rc) {
    if ((rc = sp_run_resident(c, cad))) return rc;
    c->last_itmax = cad->itmax;
    if (avgE) return ea_sp_bin_results(c, avgE);
    return EA_OK;
  }
  if (sp_use_persist(c->bin_mode, d)) {
    if ((rc = sp_run_persist(c, cad))) return rc;
    c->last_itmax = cad->itmax;
    if (avgE) return ea_sp_bin_results(c, avgE);
    return EA_OK;
  }
  // one iteration: every launch reads its counters (pass, tempering step,
  // move) from the device, so the captured graph replays each iteration
  auto iteration = [&]() -> int {
    // the counters of every sweep up to the move at once, when they fit
    const long long per = (long long)cad->ptfr * c->g.ncol;
    const bool ahead = per * cad->houfr <= kCtrPasses;
    for (int im = 0; im < cad->mesfr; ++im) {
      if (ahead) SCU(sp_launch_ctr_chain(c->d, (int)per * cad->houfr, c->d.ctrs, c->st));
      for (int ih = 0; ih < cad->houfr; ++ih) {
        int r = ahead ? sp_passes(c, cad->ptfr, (int)per * ih) : sp_sweeps(c, cad->ptfr);
        if (!r) r = sp_pt(c);
        if (r) return r;
      }
      if (cad->cluster) SCU(sp_launch_houdayer(c->d, c->st));
    }
    // without cluster moves the last tempering step's energies are current
    if (cad->cluster) SCU(sp_launch_energy(c->d, c->st));
    SCU(sp_launch_measure_u2(c->d, !cad->cluster, c->st));
    return EA_OK;
  };
  if (cad->itmax == 1) {
    if ((rc = iteration())) return rc;
  } else {
    if (!c->it_graph || std::memcmp(&c->it_cad, cad, sizeof(ea_cadence)) ||
        std::memcmp(&c->it_dev, &c->d, sizeof(SpDev))) {
      if (c->it_graph) { cudaGraphExecDestroy(c->it_graph); c->it_graph = nullptr; }
      cudaGraph_t graph = nullptr;
      SCU(cudaStreamBeginCapture(c->st, cudaStreamCaptureModeThreadLocal));
      rc = iteration();
      const cudaError_t e = cudaStreamEndCapture(c->st, &graph);
      if (rc) { if (graph) cudaGraphDestroy(graph); return rc; }
      SCU(e);
      const cudaError_t ei = cudaGraphInstantiate(&c->it_graph, graph, 0);
      cudaGraphDestroy(graph);
      SCU(ei);
      c->it_cad = *cad;
      c->it_dev = c->d;
    }
    for (int it = 0; it < cad->itmax; ++it) SCU(cudaGraphLaunch(c->it_graph, c->st));
  }
  c->last_itmax = cad->itmax;
  if (avgE) return ea_sp_bin_results(c, avgE);
  return EA_OK;
}

int ea_sp_bin_results(ea_sp *c, double *avgE) {
  if (!c || !avgE) return spfail(EA_ERR_ARG, "null argument");
  if (c->last_itmax < 1) return spfail(EA_ERR_STATE, "no bin has run");
  SCU(cudaSetDevice(c->device));
  const SpDev &d = c->d;
  const size_t n = (size_t)d.nw * 64 * d.NR * d.NB;
  std::vector<double> h(n);
  SCU(cudaMemcpyAsync(h.data(), d.avgE, n * 8, cudaMemcpyDeviceToHost, c->st));
  SCU(cudaStreamSynchronize(c->st));
  const int rc = sp_check_persist(c->p_err, c->st);
  if (rc) return rc;
  for (size_t i = 0; i < n; ++i) avgE[i] = h[i] / c->last_itmax;
  return EA_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Batches of sample-packed jobs
// ---------------------------------------------------------------------------
// A batch is split into classes -- one per job for batches of up to
// kSpBatchBranches jobs, else jobs with the same number of temperatures and
// lattices of similar size -- so that every launch is sized for its class
// (SMEM of the thresholds and of the cluster labelling, labelling block
// size); each class's bin iteration is a branch of one CUDA graph, so the
// classes run side by side and one graph launch advances the whole batch.
// (Measured on 72 jobs of mixed geometry: one class per job 0.83x / 0.97x of
// the jobs on their own streams for 72 / 1024 sample words, (NB, size)
// classes 0.78x / 0.90x, a single class 0.62x / 0.70x: fusing different
// geometries into one launch costs more than the launches it saves.)
struct SpClass {
  std::vector<ea_sp *> jobs;
  int ncol_max = 0;
  SpDev *d_jobs = nullptr;
  uint32_t *d_pre = nullptr;
  std::vector<SpDev> up_jobs;
  std::vector<uint32_t> up_pre;
  SpBatchDev bd{};
  cudaStream_t fs = nullptr;   // branch stream of the capture
  cudaEvent_t join = nullptr;
};

struct ea_sp_batch {
  std::vector<SpClass> classes;
  std::vector<ea_sp *> jobs;
  int device = 0;
  cudaStream_t bs = nullptr;
  cudaEvent_t done = nullptr, fork = nullptr;
  cudaGraphExec_t it_graph = nullptr;
  ea_cadence it_cad{};
  std::vector<SpBatchDev> it_bd;
  // persistent bin kernel: every job in one work list
  int bin_mode = EA_BIN_AUTO;
  SpClass all;
  unsigned long long *p_bar = nullptr;
  int *p_err = nullptr;
};

constexpr int kSpBatchBranches = 256;

static int sp_size_bucket(int V) { return V <= 2048 ? 0 : V <= 8192 ? 1 : V <= kSpClusterMaxV ? 2 : 3; }

static int spb_upload(SpClass &k, bool cluster, cudaStream_t bs) {
  const int n = (int)k.jobs.size();
  std::vector<SpDev> hj(n);
  std::vector<uint32_t> hp((size_t)SPB_COUNT * (n + 1), 0);
  int pass_smem = 0, prm_smem = 0, cl_smem = 0, e_smem = 0, t_smem = 0, e_threads = 32, nrep = 1, cl_threads = 32;
  for (int i = 0; i < n; ++i) {
    hj[i] = k.jobs[i]->d;
    uint32_t cnt[SPB_COUNT];
    sp_batch_blocks(hj[i], cluster, cnt);
    for (int q = 0; q < SPB_COUNT; ++q) hp[(size_t)q * (n + 1) + i + 1] = hp[(size_t)q * (n + 1) + i] + cnt[q];
    pass_smem = std::max(pass_smem, (int)(hj[i].pgrid ? sp_items_smem(hj[i].NB, kPersistThreads)  // the batched launch has as many threads
                                                       : sp_sweep_smem(hj[i].NB, hj[i].NR, hj[i].kt)));
    prm_smem = std::max(prm_smem, (int)perm_smem(hj[i].NB));
    nrep = std::max(nrep, hj[i].NR);
    e_threads = std::max(e_threads, hj[i].en.threads);
    e_smem = std::max(e_smem, (int)en_smem(hj[i], kPersistThreads));  // a persistent launch's blocks are the larger
    t_smem = std::max(t_smem, (int)pt_smem(hj[i].NB));
    if (cluster) {
      cl_smem = std::max(cl_smem, (int)sp_cluster_smem(hj[i].L, hj[i].Lz));
      cl_threads = std::max(cl_threads, sp_cluster_threads(hj[i].L, hj[i].Lz, cnt[SPB_CL0]));
    }
  }
  if (k.up_jobs.size() != hj.size() || std::memcmp(k.up_jobs.data(), hj.data(), sizeof(SpDev) * n) ||
      k.up_pre != hp) {
    SCU(cudaMemcpyAsync(k.d_jobs, hj.data(), sizeof(SpDev) * n, cudaMemcpyHostToDevice, bs));
    SCU(cudaMemcpyAsync(k.d_pre, hp.data(), sizeof(uint32_t) * hp.size(), cudaMemcpyHostToDevice, bs));
    SCU(cudaStreamSynchronize(bs));
    k.up_jobs = hj;
    k.up_pre = hp;
  }
  SpBatchDev &bd = k.bd;
  bd = SpBatchDev{};
  bd.jobs = k.d_jobs;
  bd.njobs = n;
  for (int q = 0; q < SPB_COUNT; ++q) {
    bd.pre[q] = k.d_pre + (size_t)q * (n + 1);
    bd.total[q] = hp[(size_t)q * (n + 1) + n];
  }
  bd.pass_smem = pass_smem;
  bd.perm_smem = prm_smem;
  bd.energy_smem = e_smem;
  bd.energy_threads = e_threads;
  bd.nrep = nrep;
  bd.pt_smem = t_smem;
  bd.cluster_smem = cl_smem;
  bd.cluster_threads = cl_threads;
  return EA_OK;
}

static cudaError_t spb_iteration(const SpClass &k, const ea_cadence *cad, cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  const int fit = kCtrPasses / k.ncol_max;  // sweeps whose counters are drawn at once
  for (int im = 0; im < cad->mesfr && e == cudaSuccess; ++im) {
    long long left = (long long)cad->houfr * cad->ptfr;  // sweeps up to the move
    int drawn = 0, next = 0;
    for (int ih = 0; ih < cad->houfr && e == cudaSuccess; ++ih) {
      for (int sw = 0; sw < cad->ptfr && e == cudaSuccess; ++sw) {
        if (next == drawn) {
          drawn = (int)std::min<long long>(left, fit);
          next = 0;
          e = sp_batch_ctr_chain(k.bd, drawn, st);
          if (e != cudaSuccess) break;
        }
        e = sp_batch_sweep(k.bd, k.ncol_max, next++, st);
        --left;
      }
      if (e == cudaSuccess) e = sp_batch_tempering(k.bd, st);
    }
    if (e == cudaSuccess && cad->cluster) e = sp_batch_houdayer(k.bd, st);
  }
  if (e == cudaSuccess) e = sp_batch_measure(k.bd, !cad->cluster, st);
  return e;
}

extern "C" {

int ea_sp_batch_create(ea_sp *const *jobs, int32_t njobs, ea_sp_batch **out) {
  if (!jobs || !out || njobs < 1) return spfail(EA_ERR_ARG, "at least one job");
  ea_sp_batch *b = new ea_sp_batch();
  std::vector<std::pair<int, int>> keys;
  for (int i = 0; i < njobs; ++i) {
    ea_sp *c = jobs[i];
    if (!c || std::find(b->jobs.begin(), b->jobs.end(), c) != b->jobs.end()) {
      delete b;
      return spfail(EA_ERR_ARG, "job %d is null or appears twice", i);
    }
    if (i && c->device != b->device) { delete b; return spfail(EA_ERR_ARG, "the jobs of a batch share the device"); }
    if (c->d.ncol > kSpBatchMaxColours) {
      delete b;
      return spfail(EA_ERR_ARG, "job %d needs %d colours (a batch takes %d)", i, c->d.ncol, kSpBatchMaxColours);
    }
    b->device = c->device;
    b->jobs.push_back(c);
    // one class per job up to kSpBatchBranches jobs (measured fastest: every
    // launch sized for its job, the jobs' branches side by side), else
    // classes of equal NB and lattice-size bucket
    const std::pair<int, int> key(njobs <= kSpBatchBranches ? i : c->d.NB, sp_size_bucket(c->d.V));
    size_t q = std::find(keys.begin(), keys.end(), key) - keys.begin();
    if (q == keys.size()) {
      keys.push_back(key);
      b->classes.emplace_back();
    }
    SpClass &k = b->classes[q];
    k.jobs.push_back(c);
    k.ncol_max = std::max(k.ncol_max, c->d.ncol);
  }
  cudaError_t e = cudaSetDevice(b->device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&b->bs, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->done, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->fork, cudaEventDisableTiming);
  b->all.jobs = b->jobs;
  for (ea_sp *c : b->jobs) b->all.ncol_max = std::max(b->all.ncol_max, c->d.ncol);
  if (e == cudaSuccess) e = cudaMalloc((void **)&b->all.d_jobs, sizeof(SpDev) * b->jobs.size());
  if (e == cudaSuccess) e = cudaMalloc((void **)&b->all.d_pre, sizeof(uint32_t) * SPB_COUNT * (b->jobs.size() + 1));
  if (e == cudaSuccess) e = cudaMalloc((void **)&b->p_bar, sizeof(unsigned long long));
  if (e == cudaSuccess) e = cudaMalloc((void **)&b->p_err, sizeof(int));
  if (e == cudaSuccess) e = cudaMemsetAsync(b->p_err, 0, sizeof(int), b->bs);
  for (SpClass &k : b->classes) {
    const size_t n = k.jobs.size();
    if (e == cudaSuccess) e = cudaMalloc((void **)&k.d_jobs, sizeof(SpDev) * n);
    if (e == cudaSuccess) e = cudaMalloc((void **)&k.d_pre, sizeof(uint32_t) * SPB_COUNT * (n + 1));
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&k.fs, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&k.join, cudaEventDisableTiming);
  }
  if (e == cudaSuccess) e = sp_batch_setup();
  if (e != cudaSuccess) {
    ea_sp_batch_destroy(b);
    return spfail(EA_ERR_CUDA, "batch set-up: %s", cudaGetErrorString(e));
  }
  *out = b;
  return EA_OK;
}

int ea_sp_batch_destroy(ea_sp_batch *b) {
  if (!b) return EA_OK;
  cudaSetDevice(b->device);
  if (b->bs) cudaStreamSynchronize(b->bs);
  if (b->it_graph) cudaGraphExecDestroy(b->it_graph);
  for (SpClass &k : b->classes) {
    if (k.d_jobs) cudaFree(k.d_jobs);
    if (k.d_pre) cudaFree(k.d_pre);
    if (k.join) cudaEventDestroy(k.join);
    if (k.fs) cudaStreamDestroy(k.fs);
  }
  if (b->all.d_jobs) cudaFree(b->all.d_jobs);
  if (b->all.d_pre) cudaFree(b->all.d_pre);
  if (b->p_bar) cudaFree(b->p_bar);
  if (b->p_err) cudaFree(b->p_err);
  if (b->done) cudaEventDestroy(b->done);
  if (b->fork) cudaEventDestroy(b->fork);
  if (b->bs) cudaStreamDestroy(b->bs);
  delete b;
  return EA_OK;
}

int ea_sp_batch_stream(ea_sp_batch *b, void **stream) {
  if (!b || !stream) return spfail(EA_ERR_ARG, "null argument");
  *stream = (void *)b->bs;
  return EA_OK;
}

int ea_sp_batch_sync(ea_sp_batch *b) {
  if (!b) return spfail(EA_ERR_ARG, "null batch");
  SCU(cudaSetDevice(b->device));
  SCU(cudaStreamSynchronize(b->bs));
  return sp_check_persist(b->p_err, b->bs);
}

int ea_sp_batch_set_bin_kernel(ea_sp_batch *b, int32_t mode) {
  if (!b || mode < EA_BIN_AUTO || mode > EA_BIN_PERSISTENT) return spfail(EA_ERR_ARG, "bad bin-kernel mode");
  b->bin_mode = mode;
  return EA_OK;
}

int ea_sp_batch_run(ea_sp_batch *b, const ea_cadence *cad) {
  if (!b || !cad || cad->itmax < 1 || cad->houfr < 1 || cad->mesfr < 1 || cad->ptfr < 1)
    return spfail(EA_ERR_ARG, "bad cadence");
  SCU(cudaSetDevice(b->device));
  int rc;
  for (ea_sp *c : b->jobs) {
    if (!c->have_temps) return spfail(EA_ERR_STATE, "temperatures not set");
    int nclust = cad->nclust;
    if (cad->cluster && (rc = sp_cluster_prepare(c, nclust))) return rc;
    // every job's earlier work comes first
    SCU(cudaEventRecord(b->done, c->st));
    SCU(cudaStreamWaitEvent(b->bs, b->done, 0));
  }
  const bool persist = b->bin_mode == EA_BIN_PERSISTENT;
  if (persist) {
    // one work list of every job, one cooperative launch per bin
    if ((rc = spb_upload(b->all, cad->cluster != 0, b->bs))) return rc;
    for (ea_sp *c : b->jobs)
      SCU(cudaMemsetAsync(c->d.avgE, 0, sizeof(double) * (size_t)c->d.nw * 64 * c->d.NR * c->d.NB, b->bs));
    SpPersistDev p{};
    p.b = b->all.bd;
    p.itmax = cad->itmax; p.houfr = cad->houfr; p.mesfr = cad->mesfr; p.ptfr = cad->ptfr;
    p.cluster = cad->cluster != 0;
    p.ncol_max = b->all.ncol_max;
    p.bar = b->p_bar;
    p.err = b->p_err;
    const size_t smem = (size_t)std::max({p.b.pass_smem, p.b.perm_smem, p.b.cluster_smem, p.b.energy_smem, p.b.pt_smem});
    const int grid = sp_persist_grid(p.b, smem);
    if (grid < 1) return spfail(EA_ERR_CUDA, "persistent bin kernel: no co-resident grid for %zu bytes of shared memory", smem);
    SCU(sp_launch_persist(p, grid, smem, b->bs));
  } else {
  std::vector<SpBatchDev> bds;
  for (SpClass &k : b->classes) {
    if ((rc = spb_upload(k, cad->cluster != 0, b->bs))) return rc;
    bds.push_back(k.bd);
  }
  for (ea_sp *c : b->jobs)
    SCU(cudaMemsetAsync(c->d.avgE, 0, sizeof(double) * (size_t)c->d.nw * 64 * c->d.NR * c->d.NB, b->bs));
  if (!b->it_graph || std::memcmp(&b->it_cad, cad, sizeof(ea_cadence)) || b->it_bd.size() != bds.size() ||
      std::memcmp(b->it_bd.data(), bds.data(), sizeof(SpBatchDev) * bds.size())) {
    if (b->it_graph) { cudaGraphExecDestroy(b->it_graph); b->it_graph = nullptr; }
    cudaGraph_t graph = nullptr;
    SCU(cudaStreamBeginCapture(b->bs, cudaStreamCaptureModeThreadLocal));
    cudaError_t e = cudaEventRecord(b->fork, b->bs);
    for (SpClass &k : b->classes) {
      if (e == cudaSuccess) e = cudaStreamWaitEvent(k.fs, b->fork, 0);
      if (e == cudaSuccess) e = spb_iteration(k, cad, k.fs);
      if (e == cudaSuccess) e = cudaEventRecord(k.join, k.fs);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(b->bs, k.join, 0);
    }
    const cudaError_t ec = cudaStreamEndCapture(b->bs, &graph);
    if (e != cudaSuccess || ec != cudaSuccess) {
      if (graph) cudaGraphDestroy(graph);
      return spfail(EA_ERR_CUDA, "batch capture: %s", cudaGetErrorString(e != cudaSuccess ? e : ec));
    }
    const cudaError_t ei = cudaGraphInstantiate(&b->it_graph, graph, 0);
    cudaGraphDestroy(graph);
    SCU(ei);
    b->it_cad = *cad;
    b->it_bd = bds;
  }
  for (int it = 0; it < cad->itmax; ++it) SCU(cudaGraphLaunch(b->it_graph, b->bs));
  }
  // later work of each job comes after the batch
  SCU(cudaEventRecord(b->done, b->bs));
  for (ea_sp *c : b->jobs) {
    SCU(cudaStreamWaitEvent(c->st, b->done, 0));
    c->last_itmax = cad->itmax;
  }
  return EA_OK;
}

int ea_sp_job_bytes(const ea_sp_geom *gp, const ea_cadence *cad, const double *betas, uint64_t *bytes) {
  SpGraph g;
  if (!bytes || !geom_ok(gp) || !sp_graph(gp->L, gp->Lz, gp->bc, g)) return spfail(EA_ERR_ARG, "bad sample-packed geometry");
  uint64_t tot = 0;
  auto add = [&](uint64_t n) {
    n = std::max<uint64_t>(n, 1);
    tot += n >= (1ull << 20) ? (n + (2ull << 20) - 1) & ~((2ull << 20) - 1) : (n + 511) & ~(uint64_t)511;
  };
  const uint64_t V = g.V, NB = gp->nbetas, NR = gp->nrep, nw = gp->nwords, G = NR * NB;
  add(V * 24); add(V * 4);                                   // neighbour table, colour lists
  add(nw * V * G * 8); add(nw * V * 48);                     // spins, couplings
  add(NB * 256 * 8); add(NB * kPre11Stride);  // thresholds, pre-search
  add(NR * 16); add(NR * 16 * kCtrPasses); add(NR * 4); add(NR * sizeof(ea_hq)); add(NR * sizeof(ea_xoshiro)); add(8);
  add(nw * 64 * G * 4); add(nw * 64 * G * 4); add(nw * 64 * G);   // U2, E, slot permutations
  add(nw * 64 * NR * (NB - 1) * 4); add(nw * NR * (NB - 1) * 8); // accepted swaps, lane masks
  add(NB * 8); add(NB * 4); add(8); add(nw * 64 * G * 8);   // betas, exp offsets, step, averages
  add(sizeof(ea_hq)); add(16); add(8);                      // random_c, pairs, move counter
  uint64_t nexp = (NB - 1) * 25001;
  if (betas) {
    std::vector<double> tab;
    std::vector<int32_t> off;
    pt_exp_table(betas, (int)NB, tab, off);
    nexp = tab.size();
  }
  add(nexp * 8);
  if (cad && cad->cluster) {
    const uint64_t nc = (uint64_t)(cad->nclust > 0 ? std::min<int>(cad->nclust, (int)NB) : std::lround(0.5 * NB));
    add(nw * nc * V * 8);
    if (V > (uint64_t)kSpClusterMaxV) add(nw * nc * 8 * sp_cluster_words((int)V) * 4);
    if (sp_slab_planes(gp->L, gp->Lz, (int)nw, (int)nc, nullptr) > 0) {   // slab labels and coins
      add(nw * nc * 8 * 8 * V * 4);
      add(nw * nc * 8 * V);
    }
  }
  if (cad && sp_res_fits(gp->L, gp->Lz, (int)nw, (int)NR, (int)NB)) {
    // the resident kernel's counters, random words and tempering draws
    const uint64_t ns = sp_res_launch_sweeps(V, G, cad);
    add(ns * g.ncol * NR * 16);
    add(ns * 16 * V * G);
    if (cad->ptfr > 0) add(ns / cad->ptfr * nw * NR * (NB - 1) * 64 * 4);
  }
  *bytes = tot + (2ull << 20);                               // stream, graph, small-allocation pages
  return EA_OK;
}

int ea_sp_exact(ea_sp *c, const double *betas, int32_t nbeta, uint64_t *dos, double *meanE) {
  if (!c) return spfail(EA_ERR_ARG, "null job");
  const SpDev &d0 = c->d;
  if (d0.V > 32) return spfail(EA_ERR_ARG, "exact enumeration needs V <= 32 sites (V = %d)", d0.V);
  if (meanE && (!betas || nbeta < 1)) return spfail(EA_ERR_ARG, "betas");
  SCU(cudaSetDevice(c->device));
  const size_t nbins = 6 * (size_t)d0.V + 1, ns = (size_t)d0.nw * 64;
  if (!c->d.dos) SCU(cudaMalloc((void **)&c->d.dos, ns * nbins * 8));
  const SpDev &d = c->d;
  SCU(cudaMemsetAsync(d.dos, 0, ns * nbins * 8, c->st));
  SCU(sp_launch_dos(d, c->st));
  if (dos) SCU(cudaMemcpyAsync(dos, d.dos, ns * nbins * 8, cudaMemcpyDeviceToHost, c->st));
  if (meanE) {
    double *db = nullptr, *dm = nullptr;
    SCU(cudaMalloc((void **)&db, sizeof(double) * nbeta));
    SCU(cudaMalloc((void **)&dm, sizeof(double) * ns * nbeta));
    SCU(cudaMemcpyAsync(db, betas, sizeof(double) * nbeta, cudaMemcpyHostToDevice, c->st));
    SCU(sp_launch_exact(d, db, nbeta, dm, c->st));
    SCU(cudaMemcpyAsync(meanE, dm, sizeof(double) * ns * nbeta, cudaMemcpyDeviceToHost, c->st));
    SCU(cudaStreamSynchronize(c->st));
    cudaFree(db);
    cudaFree(dm);
  }
  SCU(cudaStreamSynchronize(c->st));
  return EA_OK;
}

}  // extern "C"
