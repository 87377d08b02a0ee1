// BFS entry point that allocates no device memory.
//
// Some callers cannot call cudaMalloc: applications whose caching allocator
// owns the device memory (a framework's memory pool that must not be
// bypassed, or that has already reserved nearly all of the GPU), and hosts
// that give a library a fixed device-memory budget at start-up and forbid
// allocations after it.  b200bfs_bfs_noalloc serves them: the caller passes a
// CSR and the output array already on the device, and the search keeps its
// two visited bitmaps and its counter in one file-scope device array of fixed
// size (B200BFS_NOALLOC_MAX_ROWS vertices, 4 MiB of bitmaps), which every GPU
// that loads the library holds until the process exits.
//
// The whole search is one cooperative kernel: its blocks, all resident, go
// through the levels together with a grid barrier after each.  Small
// frontiers are kept as a list of rows with their degree prefix and expanded
// top-down, edge-balanced; large ones (more than a 14th of the adjacency
// entries, or more rows than the list has room for) are searched bottom-up:
// a warp owns 32 vertices, each unvisited one looks for a neighbour visited
// before the level, and the next bitmap word is built with __ballot_sync.
// Bottom-up alone is a correct BFS on a symmetric CSR too, with a kernel and a
// readback per level, but its first levels read nearly the whole CSR and wait
// for the warps that sweep the hubs' rows alone: a SCALE 20 Kronecker graph in
// its own vertex order takes 1,400-1,870 us so and 102-118 in this form (levels
// extracted by the caller included).  What bounds it is the dependent loads
// and the barrier of each level.
// The host reads the result after the kernel, so the call synchronises its
// stream; a stream that is being captured into a CUDA graph is refused before
// anything is enqueued on it.
#include <algorithm>
#include <mutex>
#include "common.cuh"
#include "engine.h"
#include "frontier.cuh"

namespace b200bfs {
namespace {

constexpr int64_t kMaxRows = B200BFS_NOALLOC_MAX_ROWS;
constexpr int64_t kMaxWords = kMaxRows / 32;
constexpr int kThreads = 1024;
constexpr int64_t kListRows = 1 << 16;  // rows of a frontier list
// A list's prefix is in 32 bits: rows count as at most this many entries, and
// a list of that many is not expanded top-down.
constexpr long long kLongRow = 1ll << 29;

struct NoallocCounters {        // of one level
  unsigned long long q;         // next frontier's list: rows << 40 | their adjacency entries
  unsigned long long nq;        // vertices found
};
struct NoallocCtl {             // zero between searches
  unsigned bar, blocks_done, error, pad;
  NoallocCounters c[3];         // of level L: c[L % 3]
};
struct NoallocResult {
  int status;                   // 1 finished, 3 too many levels, 4 gave up
  int level;
};
struct Scratch {
  uint32_t vis[2][kMaxWords];
  int32_t rows[2][kListRows];
  uint32_t pre[2][kListRows];
  NoallocCtl ctl;
  NoallocResult result;
};
static __device__ __align__(256) Scratch g_noalloc_scratch;

// A device's array and the mutex that a search holds from its launch until it
// is complete: overlapping searches would share the barrier's count and read
// each other's frontier lists, whose rows may be beyond their own graph.
struct DeviceScratch {
  std::mutex mu;
  Scratch* ptr = nullptr;
};
DeviceScratch g_scratch[256];

struct Shared {
  long long level, nq, q_rows, in_edges;
  int forward, cur, qcur, done, fail, stop;
  unsigned long long b_nq;
};

// Entries of row v; none where the row pointers decrease.
__device__ __forceinline__ long long row_entries(const int64_t* __restrict__ row_ptr, int64_t v) {
  return max((long long)(row_ptr[v + 1] - row_ptr[v]), 0ll);
}

// Bottom-up level: bitmap words w of 32 vertices per warp.  A lane tries up to
// 16 neighbours, four loads at a time, then the warp sweeps the rest of its
// row, 128 at a time.  Ids outside [0, n) are ignored rather than read out of
// the bitmap.
__device__ __forceinline__ uint32_t bottom_up(const int64_t* __restrict__ row_ptr,
                                              const int32_t* __restrict__ col, int64_t n,
                                              const uint32_t* cur, uint32_t* nxt, int64_t gw,
                                              int64_t nwarps, int64_t* __restrict__ pred,
                                              int64_t level) {
  const int lane = lane_id();
  const int64_t W = (n + 31) >> 5;
  uint32_t total = 0;  // lane 0
  for (int64_t w = gw; w < W; w += nwarps) {
    const uint32_t c = cur[w];
    if (c == kFull) {
      if (lane == 0) nxt[w] = c;
      continue;
    }
    const int64_t v = w * 32 + lane;
    int64_t b = 0, e = 0;
    int32_t parent = -1;
    if (!((c >> lane) & 1u)) {
      b = row_ptr[v];
      e = row_ptr[v + 1];
    }
#pragma unroll 1
    for (int round = 0; round < 4; ++round) {
      const bool need = parent < 0 && b < e;
      if (!__any_sync(kFull, need)) break;
      if (!need) continue;
      int32_t u[4];
      uint32_t m[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) u[q] = b + q < e ? __ldg(col + b + q) : -1;
#pragma unroll
      for (int q = 0; q < 4; ++q) m[q] = (uint32_t)u[q] < (uint64_t)n ? cur[u[q] >> 5] : 0u;
#pragma unroll
      for (int q = 3; q >= 0; --q)
        if ((m[q] >> (u[q] & 31)) & 1u) parent = u[q];
      b += 4;
    }
    unsigned rem = __ballot_sync(kFull, parent < 0 && b < e);
    while (rem) {
      const int l = __ffs(rem) - 1;
      rem &= rem - 1;
      const int64_t jb = __shfl_sync(kFull, b, l), je = __shfl_sync(kFull, e, l);
      int32_t p = -1;
      for (int64_t j = jb; j < je && p < 0; j += 128) {
        int32_t u[4];
        uint32_t m[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          u[q] = j + q * 32 + lane < je ? __ldg(col + j + q * 32 + lane) : -1;
#pragma unroll
        for (int q = 0; q < 4; ++q) m[q] = (uint32_t)u[q] < (uint64_t)n ? cur[u[q] >> 5] : 0u;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const unsigned hm = __ballot_sync(kFull, (m[q] >> (u[q] & 31)) & 1u);
          if (hm && p < 0) p = __shfl_sync(kFull, u[q], __ffs(hm) - 1);
        }
      }
      if (lane == l) parent = p;
    }
    const unsigned fm = __ballot_sync(kFull, parent >= 0);
    if (lane == 0) {
      nxt[w] = c | fm;
      total += __popc(fm);
    }
    if (parent >= 0) pred[v] = pred_entry(parent, level);
  }
  return total;
}

// The frontier list of a top-down level that follows a bottom-up one: the
// vertices new in `now` against `before` that have entries.
__device__ __forceinline__ void list_new(const int64_t* __restrict__ row_ptr, int64_t n,
                                         const uint32_t* now, const uint32_t* before, int64_t gw,
                                         int64_t nwarps, int32_t* rows, uint32_t* pre,
                                         unsigned long long* q) {
  const int64_t W = (n + 31) >> 5;
  const int lane = lane_id();
  // a lane per vertex, so that a warp's entries are few
  for (int64_t w = gw; w < W; w += nwarps) {
    const uint32_t f = now[w] & ~before[w];
    if (!f) continue;
    const int64_t v = w * 32 + lane;
    const long long len =
        ((f >> lane) & 1u) ? min(row_entries(row_ptr, v), kLongRow) : 0;
    int64_t slot;
    uint32_t offset;
    unsigned long long after;
    reserve<40>(q, len > 0, (uint32_t)len, &slot, &offset, &after);
    if (len > 0 && slot < kListRows) {
      rows[slot] = (int32_t)v;
      pre[slot] = offset;
    }
  }
}

__global__ void __launch_bounds__(kThreads, 1)
    noalloc_search_kernel(const int64_t* __restrict__ row_ptr, const int32_t* __restrict__ col,
                          int64_t n, int64_t root, int64_t* __restrict__ pred,
                          Scratch* __restrict__ sc) {
  __shared__ Shared s;
  const int lane = lane_id();
  const int64_t t0 = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * kThreads;
  const int64_t gw = t0 >> 5, nwarps = nthreads >> 5;
  const int64_t W = (n + 31) >> 5;
  NoallocCtl* ctl = &sc->ctl;
  unsigned target = 0;
  for (int64_t i = t0; i < n; i += nthreads) pred[i] = i == root ? root : -1;
  for (int64_t w = t0; w < W; w += nthreads) {
    // bits at or beyond n are padding and start "visited"
    const int64_t first = w * 32;
    uint32_t v = first + 32 > n ? kFull << (n - first) : 0u;
    if (w == (root >> 5)) v |= 1u << (root & 31);
    sc->vis[0][w] = v;
  }
  // switch thresholds: adjacency entries of a frontier that go bottom-up, and
  // vertices of one that come back to top-down
  const long long entries = row_ptr[n];
  const long long most = min(entries / 14, kLongRow - 1), few = n / (14 * 32);
  const long long rdeg = row_entries(row_ptr, root);
  if (t0 == 0) {
    sc->rows[0][0] = (int32_t)root;
    sc->pre[0][0] = 0;
  }
  if (threadIdx.x == 0) {
    s.level = 0;
    s.nq = 1;
    s.q_rows = rdeg > 0 ? 1 : 0;
    s.in_edges = rdeg;
    // the root alone is a list of one row, whatever its length, up to 2^31
    s.forward = rdeg <= 0x7FFFFFFFll;
    s.cur = s.qcur = s.done = s.fail = s.stop = 0;
    s.b_nq = 0;
  }
  bool alive = grid_barrier(&ctl->bar, &ctl->error, &target, &s.fail);
  while (alive) {
    const long long level = s.level + 1;
    const int forward = s.forward, cur = s.cur, qcur = s.qcur;
    NoallocCounters* c = &ctl->c[level % 3];
    if (t0 == 0) memset(&ctl->c[(level + 1) % 3], 0, sizeof(NoallocCounters));
    uint32_t found = 0;
    if (forward) {
      uint32_t* vis = sc->vis[cur];
      int32_t* rows = sc->rows[qcur ^ 1];
      uint32_t* pre = sc->pre[qcur ^ 1];
      expand_frontier<4>(
          row_ptr, col, sc->rows[qcur], sc->pre[qcur], s.q_rows, (uint32_t)s.in_edges, gw, nwarps,
          [](int32_t row) { return row; },
          [&](const int32_t(&u)[4], const int32_t(&p)[4]) {
            uint32_t word[4], len[4], m = 0, d = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q)
              word[q] = (uint32_t)u[q] < (uint64_t)n ? vis[u[q] >> 5] : kFull;
            // a stale word only costs an OR that wins nothing
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint32_t bit = 1u << (u[q] & 31);
              word[q] = word[q] & bit ? kFull : atomicOr(vis + (u[q] >> 5), bit);
            }
            const int stopped =
                __shfl_sync(kFull, lane == 0 ? *(volatile int*)&s.stop : 0, 0);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              len[q] = 0;
              if ((word[q] >> (u[q] & 31)) & 1u) continue;
              pred[u[q]] = pred_entry(p[q], level);
              ++found;
              if (stopped) continue;
              // a row too long for the prefix ends the list: its length alone
              // sends the next level bottom-up
              len[q] = (uint32_t)min(row_entries(row_ptr, u[q]), kLongRow);
              m += len[q] > 0;
              d += len[q];
            }
            if (stopped || !__any_sync(kFull, m != 0)) return;
            int64_t slot;
            uint32_t offset;
            unsigned long long after;
            reserve<40>(&c->q, m, d, &slot, &offset, &after);
            if (lane == 31 && ((long long)(after >> 40) > kListRows ||
                               (long long)(after & ((1ull << 40) - 1)) > most))
              *(volatile int*)&s.stop = 1;  // the next level is bottom-up
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              if (len[q] == 0 || slot >= kListRows) continue;
              rows[slot] = u[q];
              pre[slot] = offset;
              ++slot;
              offset += len[q];
            }
          });
    } else {
      found = bottom_up(row_ptr, col, n, sc->vis[cur], sc->vis[cur ^ 1], gw, nwarps, pred, level);
    }
    found = __reduce_add_sync(kFull, found);
    if (lane == 0 && found) atomicAdd(&s.b_nq, (unsigned long long)found);
    __syncthreads();
    if (threadIdx.x == 0 && s.b_nq) atomicAdd(&c->nq, s.b_nq);
    alive = grid_barrier(&ctl->bar, &ctl->error, &target, &s.fail);
    if (!alive) break;
    if (threadIdx.x == 0) {
      const unsigned long long q = __ldcg(&c->q);
      const long long nq = (long long)__ldcg(&c->nq);
      s.level = level;
      s.b_nq = 0;
      s.stop = 0;
      s.nq = nq;
      s.q_rows = (long long)(q >> 40);
      s.in_edges = (long long)(q & ((1ull << 40) - 1));
      s.qcur = qcur ^ 1;
      if (forward) {
        s.forward = s.q_rows <= kListRows && s.in_edges <= most;
      } else {
        s.cur = cur ^ 1;
        s.forward = nq < few;
      }
      if (nq == 0) s.done = 1;
      else if (level >= kMaxLevel) s.done = 3;
    }
    __syncthreads();
    if (s.done) break;
    if (!forward && s.forward) {
      list_new(row_ptr, n, sc->vis[s.cur], sc->vis[s.cur ^ 1], gw, nwarps, sc->rows[s.qcur],
               sc->pre[s.qcur], &c->q);
      alive = grid_barrier(&ctl->bar, &ctl->error, &target, &s.fail);
      if (threadIdx.x == 0) {
        const unsigned long long q = __ldcg(&c->q);
        s.q_rows = (long long)(q >> 40);
        s.in_edges = (long long)(q & ((1ull << 40) - 1));
        s.forward = s.q_rows <= kListRows && s.in_edges <= most;
      }
      __syncthreads();
    }
  }
  if (t0 == 0) {
    sc->result.status = alive ? s.done : 4;
    sc->result.level = (int)s.level;
  }
  // the last block leaves the counters zero for the next search
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&ctl->blocks_done, 1u) == gridDim.x - 1) memset((void*)ctl, 0, sizeof(*ctl));
  }
}

}  // namespace
}  // namespace b200bfs

extern "C" int b200bfs_bfs_noalloc(const int64_t* row_ptr, const int32_t* col, int64_t nrows,
                                   int64_t root, int64_t* pred, void* stream,
                                   int32_t* num_levels) {
  using namespace b200bfs;
  if (!row_ptr || !col || !pred) return B200BFS_ERR_INVALID;
  if (nrows < 1 || nrows > kMaxRows) return B200BFS_ERR_INVALID;  // beyond the fixed scratch
  if (root < 0 || root >= nrows) return B200BFS_ERR_INVALID;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  {
    // The read-back of the result and the synchronisation are not allowed
    // during stream capture: refuse before enqueuing anything, so that the
    // caller's capture stays intact.
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cs) != cudaSuccess) {
      cudaGetLastError();
      return B200BFS_ERR_INVALID;
    }
    if (cs != cudaStreamCaptureStatusNone) return B200BFS_ERR_INVALID;
  }
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 256) {
    cudaGetLastError();
    return B200BFS_ERR_CUDA;
  }
  DeviceScratch& ds = g_scratch[dev];
  std::lock_guard<std::mutex> lk(ds.mu);
  if (!ds.ptr) {
    // Once per device, with that device current: the host-side name of the
    // array is not a device address, so fetch the address the kernels use.
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) {
      cudaGetLastError();
      return B200BFS_ERR_CUDA;
    }
    ds.ptr = static_cast<Scratch*>(p);
  }
  Scratch* scratch = ds.ptr;
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  void* params[] = {&row_ptr, &col, &nrows, &root, &pred, &scratch};
  // a block per SM; fewer when a part of the device is all there is (MPS)
  cudaError_t e = cudaErrorCooperativeLaunchTooLarge;
  for (int grid = sms; grid > 0 && e == cudaErrorCooperativeLaunchTooLarge; grid /= 2)
    e = cudaLaunchCooperativeKernel((const void*)noalloc_search_kernel, dim3(grid),
                                    dim3(kThreads), params, 0, s);
  NoallocResult r = {0, 0};
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(&r, &scratch->result, sizeof(r), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  cudaGetLastError();
  if (e != cudaSuccess) return B200BFS_ERR_CUDA;
  if (r.status == 3) return B200BFS_ERR_OVERFLOW;
  if (r.status != 1) return B200BFS_ERR_TIMEOUT;
  if (num_levels) *num_levels = r.level;
  return B200BFS_OK;
}
