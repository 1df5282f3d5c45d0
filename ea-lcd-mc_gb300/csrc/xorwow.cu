// xorwow.cu -- set-up and launch of the cluster coins (xorwow.cuh).
#include <curand_kernel.h>

#include <algorithm>
#include <mutex>

#include "kernels_dev.cuh"
#include "xorwow.cuh"

namespace eagb {

int xw_segments(unsigned long long n2) {
  const unsigned long long rows = n2 / kXwStreams;
  return (int)std::min<unsigned long long>(64, std::max<unsigned long long>(1, rows / 128));
}

// Rows a segment covers: the move touches at most n2 / 4096 + 2 rows.
int xw_rows(unsigned long long n2, int seg) { return (int)((n2 / kXwStreams + 2 + seg - 1) / seg); }

namespace {
struct Mat {
  uint32_t r[160][5];
};

void apply(const Mat &m, const uint32_t v[5], uint32_t out[5]) {
  uint32_t a[5] = {0, 0, 0, 0, 0};
  for (int i = 0; i < 160; ++i)
    if ((v[i >> 5] >> (i & 31)) & 1u)
      for (int k = 0; k < 5; ++k) a[k] ^= m.r[i][k];
  for (int k = 0; k < 5; ++k) out[k] = a[k];
}

void then(const Mat &a, const Mat &b, Mat &out) {  // first a, then b
  Mat o;
  for (int i = 0; i < 160; ++i) apply(b, a.r[i], o.r[i]);
  out = o;
}

// Advances by 2^k rows, k = 0..39 (constants of the recurrence, built once).
const std::vector<Mat> &powers() {
  static std::once_flag once;
  static std::vector<Mat> p;
  std::call_once(once, [] {
    p.resize(40);
    for (int i = 0; i < 160; ++i) {
      uint32_t v[5] = {0, 0, 0, 0, 0};
      v[i >> 5] = 1u << (i & 31);
      for (int s = 0; s < 2; ++s) {  // a row is two steps
        const uint32_t t = v[0] ^ (v[0] >> 2);
        v[0] = v[1]; v[1] = v[2]; v[2] = v[3]; v[3] = v[4];
        v[4] = (v[4] ^ (v[4] << 4)) ^ (t ^ (t << 1));
      }
      for (int k = 0; k < 5; ++k) p[0].r[i][k] = v[k];
    }
    for (size_t k = 1; k < p.size(); ++k) then(p[k - 1], p[k - 1], p[k]);
  });
  return p;
}
}  // namespace

void xw_jump(uint64_t rows, uint32_t m[kXwMat]) {
  Mat o;
  for (int i = 0; i < 160; ++i)
    for (int k = 0; k < 5; ++k) o.r[i][k] = (i >> 5) == k ? 1u << (i & 31) : 0u;
  const std::vector<Mat> &p = powers();
  for (size_t k = 0; k < p.size() && (rows >> k); ++k)
    if ((rows >> k) & 1) then(o, p[k], o);
  for (int i = 0; i < 160; ++i)
    for (int k = 0; k < 8; ++k) m[i * 8 + k] = k < 5 ? o.r[i][k] : 0u;
}

// Streams below offset mod 4096 have given one draw more when the sequence
// starts, and their first double belongs to row 1: their row-0 state lies one
// draw before the start of the others (the step run backwards at offset 0).
__global__ void __launch_bounds__(64) k_xw_init(const __grid_constant__ JobDev j, unsigned long long seed,
                                                unsigned long long offset, const uint32_t *jump_w) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= kXwStreams) return;
  const unsigned long long q = offset / kXwStreams;
  const bool early = (unsigned long long)t < offset % kXwStreams;
  curandStateXORWOW_t s;
  curand_init(seed, (unsigned long long)t, early && q ? q - 1 : q, &s);
  uint32_t d = s.d, v[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) v[k] = s.v[k];
  if (early && !q) {
    uint32_t m = v[4] ^ v[3] ^ (v[3] << 4);   // t ^ (t << 1)
    m ^= m << 1; m ^= m << 2; m ^= m << 4; m ^= m << 8; m ^= m << 16;
    m ^= m >> 2; m ^= m >> 4; m ^= m >> 8; m ^= m >> 16;  // x from x ^ (x >> 2)
    v[4] = v[3]; v[3] = v[2]; v[2] = v[1]; v[1] = v[0]; v[0] = m;
    d -= kXwWeyl;
  }
  for (int k = 0; k < j.xw_seg; ++k) {
    if (k) {
      xw_apply(jump_w, v);
      d += 2 * kXwWeyl * (uint32_t)j.xw_w;
    }
    uint32_t *st = j.xw_state + (size_t)k * 6 * kXwStreams + t;
    st[0] = d;
#pragma unroll
    for (int i = 0; i < 5; ++i) st[(i + 1) * kXwStreams] = v[i];
  }
  if (t == 0) {
    j.xw_pos[0] = j.xw_pos[1] = offset % kXwStreams;
    j.xw_pos[2] = 0;
  }
}

// The replica pairs ride in block 0 (one thread, a chain of a few generator
// steps): one launch less in a small job's chain.
__global__ void __launch_bounds__(256) k_move_start(const __grid_constant__ JobDev j) {
  __shared__ __align__(16) uint32_t s_m[kXwMat];
  if (blockIdx.x > 0) xw_body(j, blockIdx.x - 1, s_m);
  else if (threadIdx.x == 0) pairs_body(j);
  xw_done(j);
}

cudaError_t launch_xw_init(const JobDev &j, unsigned long long seed, unsigned long long offset, const uint32_t *jump_w,
                           cudaStream_t st) {
  k_xw_init<<<kXwStreams / 64, 64, 0, st>>>(j, seed, offset, jump_w);
  return cudaGetLastError();
}

cudaError_t launch_move_start(const JobDev &j, cudaStream_t st) {
  k_move_start<<<1 + j.xw_seg * (kXwStreams / 256), 256, 0, st>>>(j);
  return cudaGetLastError();
}

}  // namespace eagb
