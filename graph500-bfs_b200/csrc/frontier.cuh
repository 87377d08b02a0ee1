// Device code shared by the kernels that run a whole search (persistent.cu,
// noalloc.cu): the barrier between their blocks and the top-down frontier
// list with its edge-balanced expansion.
#pragma once

#include "common.cuh"

namespace b200bfs {

// polls of the grid barrier before it gives up (well over ten seconds)
constexpr unsigned kSpinLimit = 1u << 25;

__device__ __forceinline__ unsigned load_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Barrier of a cooperative launch's blocks on the arrival count *bar, which
// is zero before the launch; *target counts the arrivals that end the barrier.
// False when a block gave up waiting (*error; *fail is in shared memory,
// zero at first): every block then leaves the kernel.  The fences around
// the arrival make each block's writes visible to every block behind the
// barrier; state that the kernel writes is read with ordinary loads.
__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned* error, unsigned* target,
                                             int* fail) {
  *target += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(bar, 1u);
    unsigned n = 0;
    while ((int)(load_acquire(bar) - *target) < 0) {
      if (++n == kSpinLimit || ((n & 1023u) == 0 && load_acquire(error) != 0)) {
        atomicExch(error, 1u);
        *fail = 1;
        break;
      }
    }
    __threadfence();
  }
  __syncthreads();
  return *(volatile int*)fail == 0;
}

// Largest i in [0, hi] with pre[i] <= t (pre[0] = 0), for the whole warp, 32
// probes per round.
__device__ __forceinline__ int64_t segment_search(const uint32_t* pre, int64_t hi, uint32_t t) {
  const int lane = lane_id();
  int64_t lo = 0;
  while (hi - lo > 31) {
    const int64_t step = (hi - lo + 31) / 32;
    const int64_t probe = lo + step * lane;
    const unsigned le = __ballot_sync(kFull, probe <= hi && pre[probe] <= t);
    const int last = 31 - __clz(le);
    const int64_t next = lo + step * (last + 1);  // first probe known to be > t
    lo += step * last;
    if (last < 31 && next <= hi) hi = next - 1;
  }
  const int64_t probe = lo + lane;
  const unsigned le = __ballot_sync(kFull, probe <= hi && pre[probe] <= t);
  return lo + (31 - __clz(le));
}

// Appends a warp's rows to a frontier list whose *q is rows << kShift | their
// adjacency entries: lane's n rows with d entries together (d < 2^31).  One
// atomic gives the slots and the entry offset of the first of them, so that
// the list carries its degree prefix without a scan.  Returns the lane's slot
// and offset, and in lane 31 *q after the warp's rows.
template <int kShift>
__device__ __forceinline__ void reserve(unsigned long long* q, uint32_t n, uint32_t d,
                                        int64_t* slot, uint32_t* offset,
                                        unsigned long long* after) {
  const int lane = lane_id();
  unsigned long long x = (unsigned long long)n << kShift | d, incl = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += t;
  }
  unsigned long long at = 0;
  if (lane == 31) at = atomicAdd(q, incl);
  *after = at + incl;
  at = __shfl_sync(kFull, at, 31) + incl - x;
  *slot = (int64_t)(at >> kShift);
  *offset = (uint32_t)at;
}

// Edge-balanced expansion of a frontier list of nrows rows with `total`
// entries: tiles of a multiple of 32 entries (as small as one warp per tile
// allows) of the concatenated rows, 32 * kPer entries per step.  A step
// inside one row needs no lookup; else the rows of each 32 entries are found
// among the next 32 list entries (a row has at least one entry, so no more
// can start there).  total + 32 * kPer is below 2^32, so that a step's end does
// not wrap.  claim(u, p) gets a lane's kPer neighbours (-1: none) and
// parent(row) of their rows.
template <int kPer, typename Parent, typename Claim>
__device__ __forceinline__ void expand_frontier(const int64_t* __restrict__ row_ptr,
                                                const int32_t* __restrict__ col,
                                                const int32_t* rows, const uint32_t* pre,
                                                int64_t nrows, uint32_t total, int64_t gw,
                                                int64_t nwarps, Parent parent, Claim claim) {
  const int lane = lane_id();
  const uint32_t tile =
      32u * (uint32_t)min((int64_t)8, max((int64_t)1, (total + 32 * nwarps - 1) / (32 * nwarps)));
  const int64_t ntiles = ((int64_t)total + tile - 1) / tile;
  for (int64_t t = gw; t < ntiles; t += nwarps) {
    const uint32_t t0 = (uint32_t)(t * tile), t1 = (uint32_t)min((int64_t)total, (t + 1) * tile);
    int64_t i = segment_search(pre, nrows - 1, t0);
    for (uint32_t e0 = t0; e0 < t1; e0 += 32 * kPer) {
      int32_t u[kPer], p[kPer];
      const uint32_t seg_hi = i + 1 < nrows ? pre[i + 1] : total;
      if (seg_hi >= t1 || seg_hi - e0 >= 32 * kPer) {
        const int32_t src = rows[i];
        const int64_t rb = __ldg(row_ptr + src) - pre[i] + e0;
        const int32_t par = parent(src);
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
          const uint32_t x = q * 32 + lane;
          u[q] = e0 + x < t1 ? __ldg(col + rb + x) : -1;
          p[q] = par;
        }
        if (seg_hi == e0 + 32 * kPer) ++i;
      } else {
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
          u[q] = -1;
          p[q] = 0;
          const uint32_t b = e0 + q * 32;
          if (b >= t1) continue;  // warp-uniform
          const uint32_t st = i + lane < nrows ? pre[i + lane] : total;
          const uint32_t x = b + lane;
          // last row that starts at or before entry x
          int k = 0;
#pragma unroll
          for (int o = 16; o; o >>= 1) {
            const uint32_t v = __shfl_sync(kFull, st, (k + o) & 31);
            if (v <= x) k += o;
          }
          const uint32_t first = __shfl_sync(kFull, st, k);
          if (x < t1) {
            const int32_t src = rows[i + k];
            u[q] = __ldg(col + __ldg(row_ptr + src) + (x - first));
            p[q] = parent(src);
          }
          // the row of entry b + 32
          i += __shfl_sync(kFull, k, 31);
          if (i + 1 < nrows && pre[i + 1] <= b + 32) ++i;
        }
      }
      claim(u, p);
    }
  }
}

}  // namespace b200bfs
