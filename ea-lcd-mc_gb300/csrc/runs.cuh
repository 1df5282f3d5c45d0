// runs.cuh -- cluster labelling of equal-overlap clusters by runs along z, for
// both layouts.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace eagb {

typedef unsigned long long u64;

// The 8 x 8 bit matrix with byte i, bit j at bit 8 i + j, transposed.
__device__ __forceinline__ u64 transpose8(u64 x) {
  u64 t = (x ^ (x >> 7)) & 0x00AA00AA00AA00AAull;
  x ^= t ^ (t << 7);
  t = (x ^ (x >> 14)) & 0x0000CCCC0000CCCCull;
  x ^= t ^ (t << 14);
  t = (x ^ (x >> 28)) & 0x00000000F0F0F0F0ull;
  return x ^ t ^ (t << 28);
}

// The labelling by runs.  A "run" is a maximal stretch of equal overlap along z
// of one (x, y) column of one sample; its sites share a cluster, so only its
// lowest site -- its smallest index -- carries a label, and the bonds along x
// and y are needed once per pair of touching runs (a "contact").  A thread
// holds the q bits of one (sample, column, chunk of at most 31 planes) in a
// word: run starts and contacts are a few bit operations, and walking them
// touches 2 to 3 times fewer labels than sites.
//   hook:  every pending contact whose two labels differ hangs the larger
//          label below the smaller by a plain store (SMEM has no 16-bit
//          atomicMin): of several stores to one root one stays, and the other
//          contacts are still pending in the next round.  A contact whose
//          labels are equal is done for good: they lie in one tree, or are
//          joined by the pending contact of the thread that stored one of
//          them in these rounds of the loop.
//   jump:  every run walks to its root; roots do not change meanwhile, so one
//          pass leaves every label a root.
// until a hook pass finds no difference: 3 passes on overlaps of production
// tubes.  Labels only decrease and stay inside the cluster, so every run ends
// labelled by its cluster's smallest site, the root the reference takes.
// NS samples at a time (lanes: NS samples of 32 / NS neighbouring columns, so
// one 2 NS-byte label slot serves the NS lanes of a column).
//
// Bound by instruction issue (61 % of the slots busy with 37 % of the warps, 44 %
// of the SMEM path, 19 of 32 lanes active; 83 % and 78 % of the warps in slabs).  The forms it replaces labelled every
// site, 8 samples in lock step with vector label slots, at 72 % of the SMEM
// path.  A launch on 6144 x 8 lattices of 12 x 12 x 48: 5.08 -> 2.27 ms; one
// word of it (96 blocks): 155 -> 62 us; 24 x 24 x 192 in slabs: 1.83 -> 0.83
// ms a group; a move of 16 x 16 x 64 (once one sample at a time): 4.84 -> 0.77
// ms.
struct RunShape {
  int S, nz, H, nch, nseg;  // sites of a plane, planes, planes of a chunk, chunks, column chunks
};
__host__ __device__ inline RunShape run_shape(int L, int nz) {
  RunShape r;
  r.S = L * L;
  r.nz = nz;
  const int n = (nz + 30) / 31;
  r.H = (nz + n - 1) / n;
  r.nch = (nz + r.H - 1) / r.H;
  r.nseg = r.S * r.nch;
  return r;
}
// SMEM: run words and contacts [3][nseg][NS] u32, labels [nz S][NS] u16, the
// column at x + 1 [S] u16, the 8 samples' q bytes [nz S] and (NS < 8) their
// flip bytes.
__host__ __device__ inline size_t run_smem(const RunShape &r, int NS) {
  return (size_t)12 * r.nseg * NS + (size_t)r.nz * r.S * (2 * NS + (NS < 8 ? 2 : 1)) + (size_t)2 * r.S;
}
// The part before the q bytes, one sample at a time (the multispin layout).
__host__ __device__ inline size_t run_label_smem(const RunShape &r) {
  return ((size_t)12 * r.nseg + (size_t)2 * r.nz * r.S + (size_t)2 * r.S + 15) & ~(size_t)15;
}
constexpr size_t kRunSmem = 224 * 1024;  // leaves 3 KB for the static SMEM of the batched and persistent kernels
__device__ __forceinline__ uint32_t run_mask(const RunShape &r, int ch) {
  return (1u << min(r.H, r.nz - ch * r.H)) - 1u;
}
__device__ __forceinline__ uint32_t run_starts(uint32_t m, uint32_t mask) { return ((m ^ (m << 1)) | 1u) & mask; }

template <int NS>
struct RunLab {
  RunShape r;
  int L;
  uint32_t *qm, *cx, *cy;  // [nseg][NS]: q bits, pending contacts with the column at x + 1 / y + 1 (bit 31 of cy: towards z + H)
  uint16_t *lab;           // [nz S][NS], valid at run starts
  uint16_t *nx;            // [S]
  uint8_t *qb, *fb;        // [nz S]

  __device__ __forceinline__ RunLab(unsigned char *sm, int L_, int nz) : r(run_shape(L_, nz)), L(L_) {
    qm = reinterpret_cast<uint32_t *>(sm);
    cx = qm + (size_t)r.nseg * NS;
    cy = cx + (size_t)r.nseg * NS;
    lab = reinterpret_cast<uint16_t *>(cy + (size_t)r.nseg * NS);
    nx = lab + (size_t)r.nz * r.S * NS;
    qb = reinterpret_cast<uint8_t *>(nx + r.S);
    fb = qb + (NS < 8 ? (size_t)r.nz * r.S : 0);
  }
  __device__ __forceinline__ void columns() const {
    for (int i = threadIdx.x; i < r.S; i += blockDim.x) nx[i] = (uint16_t)(i % L == L - 1 ? i - (L - 1) : i + 1);
  }
  // the 8 samples' q bytes of the sites from Qb on, one byte of 8 a site
  __device__ __forceinline__ void load(const uint8_t *Qb) const {
    for (int i = threadIdx.x; i < r.nz * r.S; i += blockDim.x) qb[i] = Qb[(size_t)i * 8];
    columns();
    __syncthreads();
  }
  // the thread's (column chunk, sample) items: body(item, chunk, column)
  template <class F>
  __device__ __forceinline__ void items(F &&body) const {
    const int step = blockDim.x / NS;
    int sg = threadIdx.x / NS, ch = sg / r.S, col = sg - ch * r.S;
    for (; sg < r.nseg; sg += step) {
      body(sg * NS + (int)(threadIdx.x % NS), ch, col);
      for (col += step; col >= r.S; col -= r.S) ++ch;
    }
  }
  // body(byte of the chunk's plane words, column chunk, chunk, column, planes of that byte)
  template <class F>
  __device__ __forceinline__ void bytes(F &&body) const {
    for (int u = threadIdx.x; u < 4 * r.nseg; u += blockDim.x) {
      const int j = u / r.nseg, sg = u - j * r.nseg, ch = sg / r.S, col = sg - ch * r.S;
      body(j, sg, ch, col, min(8, min(r.H, r.nz - ch * r.H) - 8 * j));
    }
  }
  __device__ __forceinline__ uint16_t *slot(int ch, int col) const {
    return lab + ((size_t)ch * r.H * r.S + col) * NS + threadIdx.x % NS;
  }
  __device__ __forceinline__ int next_y(int col) const { return col + L >= r.S ? col + L - r.S : col + L; }
  // M: the bits of a slot that are its label
  template <int M = 0xFFFF>
  __device__ __forceinline__ int root(int x) const {
    const uint16_t *lane = lab + threadIdx.x % NS;
    for (int y; (y = lane[x * NS] & M) != x;) x = y;
    return x;
  }

  // The pending contacts of two columns: those whose labels still differ.
  // WALK: the labels may have been hung below others since they were roots.
  template <bool WALK>
  __device__ __forceinline__ uint32_t hook(uint32_t c, uint32_t sa, uint32_t sb, const uint16_t *la,
                                           const uint16_t *lb) const {
    const int zs = r.S * NS;
    uint16_t *lane = lab + threadIdx.x % NS;
    uint32_t keep = 0;
    while (c) {
      const uint32_t bit = c & (0u - c), low = bit + (bit - 1u);  // bits up to and with the contact
      c ^= bit;
      int a = la[(31 - __clz(sa & low)) * zs], b = lb[(31 - __clz(sb & low)) * zs];
      if (WALK) {
        a = root(a);
        b = root(b);
      }
      if (a != b) {
        keep |= bit;
        lane[max(a, b) * NS] = (uint16_t)min(a, b);
      }
    }
    return keep;
  }
  // One hook pass; whether this thread found labels that differ.
  template <bool WALK>
  __device__ __forceinline__ int hooks() const {
    const int zs = r.S * NS;
    int hooked = 0;
    items([&](int it, int ch, int col) {
      uint32_t c = cx[it];
      const uint32_t d = cy[it];
      if (!(c | d)) return;
      const uint32_t mask = run_mask(r, ch), st = run_starts(qm[it], mask);
      const int row = it - col * NS;  // item of column 0 of the chunk
      const uint16_t *la = slot(ch, col);
      if (c) {
        const int nc = nx[col];
        c = hook<WALK>(c, st, run_starts(qm[row + nc * NS], mask), la, slot(ch, nc));
        cx[it] = c;
        hooked |= c != 0;
      }
      if (d) {
        const int nc = next_y(col);
        uint32_t e = 0;
        if (d & 0x7FFFFFFFu)
          e = hook<WALK>(d & 0x7FFFFFFFu, st, run_starts(qm[row + nc * NS], mask), la, slot(ch, nc));
        if (d >> 31) {
          int a = la[(31 - __clz(st)) * zs], b = *slot(ch == r.nch - 1 ? 0 : ch + 1, col);
          if (WALK) {
            a = root(a);
            b = root(b);
          }
          if (a != b) {
            e |= 0x80000000u;
            lab[max(a, b) * NS + threadIdx.x % NS] = (uint16_t)min(a, b);
          }
        }
        cy[it] = e;
        hooked |= e != 0;
      }
    });
    return __syncthreads_or(hooked);
  }
  // Every run's label a root; found(slot of the column, its first index, the
  // item's roots) may set bits outside M in the roots' slots.
  template <int M = 0xFFFF, class F>
  __device__ __forceinline__ void jump(F &&found) const {
    const int zs = r.S * NS;
    items([&](int it, int ch, int col) {
      uint16_t *l = slot(ch, col);
      const int id = ch * r.H * r.S + col;
      uint32_t roots = 0;
      for (uint32_t st = run_starts(qm[it], run_mask(r, ch)); st; st &= st - 1u) {
        const uint32_t bit = st & (0u - st);
        const int z = 31 - __clz(bit), x = l[z * zs] & M;
        if (x == id + z * r.S) {
          roots |= bit;
          continue;
        }
        const int y = root<M>(x);
        if (y != x) l[z * zs] = (uint16_t)y;
      }
      found(l, id, roots);
    });
  }

  // The q words of samples [h NS, (h + 1) NS) from the q bytes.
  __device__ __forceinline__ void words(int h) const {
    bytes([&](int j, int sg, int ch, int col, int n) {
      const uint8_t *p = qb + (ch * r.H + 8 * j) * r.S + col;
      u64 x = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k < n) x |= (u64)p[k * r.S] << (8 * k);
      x = transpose8(x) >> (8 * NS * h);
      uint8_t *o = reinterpret_cast<uint8_t *>(qm + (size_t)sg * NS) + j;
#pragma unroll
      for (int l = 0; l < NS; ++l) o[4 * l] = (uint8_t)(x >> (8 * l));
    });
  }

  // Labels from the q words; the runs' labels are left one walk from their
  // roots (jump).  wrap: the last plane is bonded to the first; corner: only its
  // last column is.  bonds(chunk, column, mask of planes bonded along x) may
  // change the mask.
  template <class Bonds>
  __device__ __forceinline__ void label(bool wrap, bool corner, Bonds &&bonds) const {
    const int zs = r.S * NS;
    __syncthreads();
    items([&](int it, int ch, int col) {
      const uint32_t mask = run_mask(r, ch), m = qm[it], st = run_starts(m, mask);
      const int row = it - col * NS, id = ch * r.H * r.S + col;
      uint16_t *l0 = slot(ch, col);
      for (uint32_t s = st; s; s &= s - 1u) {
        const int z = 31 - __clz(s & (0u - s));
        l0[z * zs] = (uint16_t)(id + z * r.S);
      }
      uint32_t n = qm[row + nx[col] * NS], eq = bonds(ch, col, ~(m ^ n) & mask);
      cx[it] = eq & (st | run_starts(n, mask) | ~(eq << 1));
      n = qm[row + next_y(col) * NS];
      eq = ~(m ^ n) & mask;
      uint32_t c = eq & (st | run_starts(n, mask) | ~(eq << 1));
      const bool last = ch == r.nch - 1;
      if (!last || wrap || (corner && col == r.S - 1)) {
        n = qm[last ? it - ch * r.S * NS : it + r.S * NS];  // the chunk above: its first plane
        const uint32_t top = (m >> (31 - __clz(mask))) & 1u;
        if (top == (n & 1u)) c |= 0x80000000u;
      }
      cy[it] = c;
    });
    __syncthreads();
    // two rounds on root labels join nearly everything; the few contacts left
    // walk, which saves a jump pass a round
    if (!hooks<false>()) return;
    jump([](uint16_t *, int, uint32_t) {});
    __syncthreads();
    if (!hooks<false>()) return;
    while (hooks<true>()) {
    }
  }
};

}  // namespace eagb
