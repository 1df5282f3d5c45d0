// xorwow.cuh -- the cluster coins of the multispin layout: the bits
// [U < 0.5] of the uniforms the reference draws with cuRAND's default
// generator (HoudayerXEA.cu:174-195), without the uniforms.
//
// That generator is Marsaglia's xorwow (Xorshift RNGs, J. Stat. Softw. 8(14),
// 2003): 4096 streams, number i of the sequence being number i / 4096 of
// stream i mod 4096 (the documented default ordering), a double taking two
// draws of its stream.  A double lies below 1/2 exactly when the second
// draw's top bit is 0 -- the only thing a cluster move asks of it -- so one
// bit per site stands for eight bytes, and no FP64 is left.
//
// A "row" is one double of each of the 4096 streams.  The job's sequence runs
// on from move to move; position p of it is stream p mod 4096 of row p / 4096
// (an offset o into the sequence starts it at position o mod 4096).
#pragma once
#include <cstdint>
#include <vector>
#include <cuda_runtime.h>
#include "kernels.cuh"

namespace eagb {

constexpr int kXwStreams = 4096;
constexpr int kXwMat = 160 * 8;     // words of a jump matrix: the image of each of the 160 state bits, padded to 8 words
constexpr uint32_t kXwWeyl = 362437u;

// Segments of a move of n2 coins: each of the 4096 streams is cut into that
// many runs of W rows, one thread each, so that a large move fills the GPU
// (64 x 4096 threads) and a small one keeps runs of about 128 rows (the jump
// to the next move costs as much as about 60 rows).
int xw_segments(unsigned long long n2);
int xw_rows(unsigned long long n2, int seg);
inline size_t xw_words(unsigned long long n2) { return (size_t)((n2 + 62) / 32); }
// The matrix that advances a state by `rows` rows.
void xw_jump(uint64_t rows, uint32_t m[kXwMat]);

// States of every segment's first row for the sequence of (seed, offset);
// mat: [0] the jump by W rows (unused for one segment).
cudaError_t launch_xw_init(const JobDev &j, unsigned long long seed, unsigned long long offset, const uint32_t *jump_w,
                           cudaStream_t st);
// The start of a move: its replica pairs and its coins (from position
// xw_pos[1], which then becomes xw_pos[0]).
cudaError_t launch_move_start(const JobDev &j, cudaStream_t st);

#ifdef __CUDACC__
__device__ __forceinline__ void xw_step(uint32_t v[5]) {
  const uint32_t t = v[0] ^ (v[0] >> 2);
  v[0] = v[1]; v[1] = v[2]; v[2] = v[3]; v[3] = v[4];
  v[4] = (v[4] ^ (v[4] << 4)) ^ (t ^ (t << 1));
}

__device__ __forceinline__ void xw_apply(const uint32_t *m, uint32_t v[5]) {
  uint32_t a[5] = {0, 0, 0, 0, 0};
#pragma unroll
  for (int w = 0; w < 5; ++w) {
#pragma unroll 8
    for (int b = 0; b < 32; ++b) {
      const uint32_t on = 0u - ((v[w] >> b) & 1u);
      const uint32_t *r = m + (w * 32 + b) * 8;
      const uint4 q = *reinterpret_cast<const uint4 *>(r);
      a[0] ^= q.x & on; a[1] ^= q.y & on; a[2] ^= q.z & on; a[3] ^= q.w & on;
      a[4] ^= r[4] & on;
    }
  }
#pragma unroll
  for (int k = 0; k < 5; ++k) v[k] = a[k];
}

// Block blk of a move's coins: 16 blocks of 256 threads per segment, a thread
// per (segment, stream).  A warp's 32 streams are 32 consecutive positions, so
// a row of them is one ballot and one word.  Bound by instruction issue: ~17
// instructions a row and thread, ~1300 for the jump; no traffic but one word a
// warp and row.  219 M coins of a move (L=24, Lz=192, 32 temperatures, 31
// samples): 163 us on the whole GPU, against 2 x 2.36 ms for cuRAND's doubles
// on 32 SMs (FP64-bound), the move's read of them included 1.75 GB less.  s_m: kXwMat words of SMEM for the
// jump matrix (read from global memory by every thread, its 160 rows were a
// chain of L2 latencies: 28 us of a small move).
__device__ __forceinline__ void xw_body(const JobDev &j, int blk, uint32_t *s_m) {
  const int t = (blk & 15) * 256 + threadIdx.x, k = blk >> 4;
  const unsigned long long B = j.xw_pos[1];
  uint32_t *st = j.xw_state + (size_t)k * 6 * kXwStreams + t;
  uint32_t d = st[0], v[5];
#pragma unroll
  for (int q = 0; q < 5; ++q) v[q] = st[(q + 1) * kXwStreams];
  if (j.xw_seg > 1)
    for (int i = threadIdx.x; i < kXwMat; i += 256) s_m[i] = __ldg(j.xw_jump + i);
  __syncthreads();
  const int row0 = (int)(B & (kXwStreams - 1));                     // positions into the first row
  const int nrows = (int)((row0 + j.xw_n - 1) / kXwStreams) + 1;    // rows this move touches
  const int adv = (int)((row0 + j.xw_n) / kXwStreams);              // rows to the next move's first row
  const bool lane0 = (threadIdx.x & 31) == 0;
  auto draw = [&]() {
    xw_step(v);
    xw_step(v);
    d += 2 * kXwWeyl;
    return __ballot_sync(0xffffffffu, (int)(v[4] + d) >= 0);
  };
  // words of the first row below the move's first position belong to the last
  // move (row0 / 32 of them, not kept), those past its last to the next
  const int nwords = (int)(((B & 31) + j.xw_n + 31) >> 5), w0 = (t >> 5) - (row0 >> 5);
  auto edge_row = [&](int r) {
    const unsigned sel = draw();
    const int w = r * (kXwStreams / 32) + w0;
    if (lane0 && w >= 0 && w < nwords) j.xw_bits[w] = sel;
  };
  if (j.xw_seg == 1) {
    for (int r = 0; r < adv; ++r) edge_row(r);
  } else {
    int r = k * j.xw_w;
    const int rend = r + j.xw_w, rin = min(rend, nrows - 1);
    if (r == 0) edge_row(r++);
    uint32_t *p = j.xw_bits + (size_t)r * (kXwStreams / 32) + w0;
    for (; r + 5 <= rin; r += 5) {
#pragma unroll
      for (int u = 0; u < 5; ++u) {
        const unsigned sel = draw();
        if (lane0) p[u * (kXwStreams / 32)] = sel;
      }
      p += 5 * (kXwStreams / 32);
    }
    for (; r < min(rend, nrows); ++r) edge_row(r);
    for (; r < rend; ++r) { xw_step(v); xw_step(v); d += 2 * kXwWeyl; }
    // on to this segment's rows of the next move: a whole number of rows
    // fixed per job, and one more row in some moves
    xw_apply(s_m, v);
    const int base = (int)(j.xw_n / kXwStreams);
    d += 2 * kXwWeyl * (uint32_t)(base - j.xw_w);
    if (adv > base) { xw_step(v); xw_step(v); d += 2 * kXwWeyl; }
  }
  st[0] = d;
#pragma unroll
  for (int q = 0; q < 5; ++q) st[(q + 1) * kXwStreams] = v[q];
  if (j.xw_seg == 1 && nrows > adv) edge_row(adv);
}

// A block of a move's start is done: the last one moves the positions on.
__device__ __forceinline__ void xw_done(const JobDev &j) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(j.xw_pos + 2, 1ull) + 1 == (unsigned long long)j.xw_seg * (kXwStreams / 256) + 1) {
      const unsigned long long p = j.xw_pos[1];
      j.xw_pos[0] = p;
      j.xw_pos[1] = p + j.xw_n;
      j.xw_pos[2] = 0;
    }
  }
}

// [U < 0.5] of (group g, index i of its call): bit base + i of j.xw_bits.
__device__ __forceinline__ unsigned long long xw_base(const JobDev &j, int g) {
  return (j.xw_pos[0] & 31) + (unsigned long long)g * (j.xw_n >> 1);
}
__device__ __forceinline__ bool xw_coin(const uint32_t *bits, uint32_t i) {
  return (__ldg(bits + (i >> 5)) >> (i & 31)) & 1u;
}
#endif

}  // namespace eagb
