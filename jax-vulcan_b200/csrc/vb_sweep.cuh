// The serial chain of the block solves' sweeps: one n x n block product per
// layer with stored inverses that stream through shared memory (one CTA per
// atmosphere).
//
// A layer's latency is what counts when a few atmospheres are solved. A warp
// takes eight rows, four lanes each, in one unrolled pass; the lane that forms a
// row's result keeps that row's vector element and its operands, loaded two
// layers ahead; a warp of its own issues the copies and waits for them, so the
// chain meets one block barrier a layer and no other wait. Two passes over the
// rows, run-time bounds, the vectors through shared memory and three barriers
// took 2.0 us a layer at n = 69 (B200, one atmosphere, the blocks in L2), this
// 0.65 (the block's shared-memory reads, 324 cycles, and the barrier bound it).
// Batches beyond an SM each are bound by HBM (the blocks, 38 KB a layer).
#pragma once
#include <cuda_runtime.h>

#include "vb_common.cuh"

namespace vb {

constexpr int SWEEP_MAX_STAGES = 8;   // mbarriers of a ring

// Row of a thread of the row warps. The eight rows of a warp are dealt so that
// a half-warp holds the even or the odd ones: with a row stride of 2 mod 4
// doubles (odd ni / 2) their four-column reads then fall into different banks
// (in order: two-way conflicts).
__device__ __forceinline__ int sweep_row() {
  const int q = (threadIdx.x >> 2) & 7;
  return (threadIdx.x >> 5) * 8 + ((2 * q) & 7) + (q >> 2);
}

// Row `row` of A v, by the four lanes that share it (8 (N8 - 1) < n <= 8 N8):
// two interleaved partial sums each (columns sub + 8 t and sub + 4 + 8 t), then
// two shuffle levels. Every lane of the warp calls it (rows past the block
// return a repeat of the last row's value).
template <int N8, typename T>
__device__ __forceinline__ double row_dot(const T* __restrict__ A, int n, int lda, int row, const double* v) {
  const int sub = threadIdx.x & 3;
  const T* a = A + min(row, n - 1) * lda + sub;
  v += sub;
  double s0 = 0.0, s1 = 0.0;
#pragma unroll
  for (int t = 0; t < N8 - 1; ++t) {
    s0 = fma((double)a[8 * t], v[8 * t], s0);
    s1 = fma((double)a[8 * t + 4], v[8 * t + 4], s1);
  }
  constexpr int e = 8 * (N8 - 1);
  if (e + sub < n) s0 = fma((double)a[e], v[e], s0);
  if (e + sub + 4 < n) s1 = fma((double)a[e + 4], v[e + 4], s1);
  double s = s0 + s1;
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  return s;
}

// `count` equally sized blocks, block s at src(s), taken in order through a
// ring of `stages` shared-memory buffers. One thread issues and waits (copy());
// the others follow with block() / next().
template <typename Src>
struct BlockStream {
  Src src;
  char* ring;
  uint64_t* bars;
  uint32_t bytes;
  size_t stride;
  int stages, count;
  int issued = 0, into = 0;   // copying thread: copies issued, the next one's stage
  int stage = 0;              // stage and barrier phase of the current block
  uint32_t phase = 0;

  __device__ const char* block() const { return ring + stage * stride; }
  __device__ void next() {
    if (++stage == stages) {
      stage = 0;
      phase ^= 1u;
    }
  }
  __device__ void issue() {
    mbar_expect_tx(&bars[into], bytes);
    bulk_g2s(ring + into * stride, src(issued), bytes, &bars[into]);
    ++issued;
    if (++into == stages) into = 0;
  }
  __device__ bool wait(long long limit) const { return mbar_wait(&bars[stage], phase, limit); }

  // The copying warp's side of a sweep: fills the ring, and arrives at the
  // sweep's barrier before the first block and after each block (as the other
  // warps do) once the next block is there. A ring of one stage takes a barrier
  // more per block, since the copy into it starts when the block has been used
  // (used()). false: a wait gave up (every thread sees it at that barrier); the
  // copies in flight have been waited for.
  __device__ void used() const {
    if (stages == 1) __syncthreads_or(0);
  }
  __device__ bool copy(long long limit) {
    const bool me = (threadIdx.x & 31) == 0;
    if (me) {
      for (int st = 0; st < stages; ++st) mbar_init(&bars[st], 1);
      fence_proxy_async();
      while (issued < stages && issued < count) issue();
    }
    for (int s = 0; s <= count; ++s) {
      if (s > 0) used();
      bool ok = true;
      if (me) {
        // block s - 2 (one stage: s - 1) has been used: its stage takes the next copy
        if (s >= (stages == 1 ? 1 : 2) && issued < count) {
          fence_proxy_async();
          issue();
        }
        if (s < count) ok = wait(limit);
      }
      if (__syncthreads_or(!ok)) {
        if (me)
          for (int q = s; q < issued; ++q) {
            wait(WAIT_LIMIT);
            next();
          }
        return false;
      }
      next();
    }
    return true;
  }
};

}  // namespace vb
