// Counting and compacting the entries of CSR rows that a predicate keeps, for
// the construction passes (duplicates dropped, pruned neighbours dropped).
//
// A warp per row leaves the pass to the warps that hold the hubs: a SCALE 22
// hub has 400,000 entries, 12,000 dependent steps of one warp, and the four
// passes of a SCALE 22 CoreBFS build took 6.7, 5.4, 4.3 and 3.1 ms with the
// rest of the GPU idle; in this form 0.8, 0.5, 0.9 and 0.6 ms.
// Rows of more than kLongRow entries are therefore cut into pieces of
// kRowPiece, each a block's: the count pass stores every piece's count, and the
// fill pass finds a piece's place from those before it in its row.
#pragma once

#include "common.cuh"
#include "engine.h"

namespace b200bfs {

constexpr int kLongRow = 2048;
constexpr int kRowPiece = 4096;
constexpr int kRowThreads = 256;

// (row, piece) of every piece of the long rows of ptr[0..R]; a row's pieces
// are consecutive.
struct RowPieces {
  int2* list = nullptr;
  int32_t* count = nullptr;  // entries kept in each piece
  int64_t n = 0;
};

static __global__ void row_pieces_count_kernel(const int64_t* __restrict__ ptr, int64_t R,
                                        unsigned long long* __restrict__ n) {
  unsigned long long c = 0;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < R;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t len = ptr[r + 1] - ptr[r];
    if (len > kLongRow) c += (unsigned long long)((len + kRowPiece - 1) / kRowPiece);
  }
  if (c) atomicAdd(n, c);
}

static __global__ void row_pieces_list_kernel(const int64_t* __restrict__ ptr, int64_t R,
                                       unsigned long long* __restrict__ n,
                                       int2* __restrict__ list) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < R;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t len = ptr[r + 1] - ptr[r];
    if (len <= kLongRow) continue;
    const int64_t k = (len + kRowPiece - 1) / kRowPiece;
    const int64_t at = (int64_t)atomicAdd(n, (unsigned long long)k);
    for (int64_t i = 0; i < k; ++i) list[at + i] = make_int2((int32_t)r, (int32_t)i);
  }
}

// Kept entries of every row.  keep(r, j, b) tells whether entry j of row r,
// which begins at b, is kept; put(r, count) takes a row's count (from one
// thread; for a long row once per piece, to be added up).
template <typename Keep, typename Put>
__global__ void __launch_bounds__(kRowThreads)
    row_count_kernel(const int64_t* __restrict__ ptr, int64_t R, Keep keep, Put put) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int lane = lane_id();
  for (int64_t r = warp; r < R; r += nwarps) {
    const int64_t b = ptr[r], e = ptr[r + 1];
    if (e - b > kLongRow) continue;
    int64_t cnt = 0;
    for (int64_t j = b + lane; j - lane < e; j += 32)
      cnt += __popc(__ballot_sync(kFull, j < e && keep(r, j, b)));
    if (lane == 0) put(r, cnt);
  }
}

template <typename Keep, typename Put>
__global__ void __launch_bounds__(kRowThreads)
    piece_count_kernel(const int64_t* __restrict__ ptr, const int2* __restrict__ list, int64_t n,
                       int32_t* __restrict__ count, Keep keep, Put put) {
  for (int64_t i = blockIdx.x; i < n; i += gridDim.x) {
    const int2 x = list[i];
    const int64_t b = ptr[x.x], jb = b + (int64_t)x.y * kRowPiece;
    const int64_t je = min(ptr[x.x + 1], jb + kRowPiece);
    int c = 0;
    for (int64_t j = jb; j < je; j += kRowThreads)
      c += __syncthreads_count(j + threadIdx.x < je && keep(x.x, j + threadIdx.x, b));
    if (threadIdx.x == 0) {
      count[i] = c;
      put(x.x, (int64_t)c);
    }
  }
}

// Kept entries in order from out(r): set(position, r, j).
template <typename Keep, typename Out, typename Set>
__global__ void __launch_bounds__(kRowThreads)
    row_fill_kernel(const int64_t* __restrict__ ptr, int64_t R, Keep keep, Out out, Set set) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int lane = lane_id();
  for (int64_t r = warp; r < R; r += nwarps) {
    const int64_t b = ptr[r], e = ptr[r + 1];
    if (e - b > kLongRow) continue;
    int64_t at = out(r);
    if (at < 0) continue;
    for (int64_t j = b + lane; j - lane < e; j += 32) {
      const bool k = j < e && keep(r, j, b);
      const unsigned m = __ballot_sync(kFull, k);
      if (k) set(at + __popc(m & ((1u << lane) - 1)), r, j);
      at += __popc(m);
    }
  }
}

template <typename Keep, typename Out, typename Set>
__global__ void __launch_bounds__(kRowThreads)
    piece_fill_kernel(const int64_t* __restrict__ ptr, const int2* __restrict__ list, int64_t n,
                      const int32_t* __restrict__ count, Keep keep, Out out, Set set) {
  __shared__ int64_t s_at;
  __shared__ int s_warp[kRowThreads / 32];
  const int lane = lane_id(), wid = threadIdx.x >> 5;
  for (int64_t i = blockIdx.x; i < n; i += gridDim.x) {
    const int2 x = list[i];
    const int64_t b = ptr[x.x], jb = b + (int64_t)x.y * kRowPiece;
    const int64_t je = min(ptr[x.x + 1], jb + kRowPiece);
    const int64_t base = out(x.x);
    if (base < 0) continue;  // the same for the whole block
    if (wid == 0) {
      // the pieces of this row before this one
      int64_t before = 0;
      for (int64_t k = i - x.y + lane; k < i; k += 32) before += count[k];
#pragma unroll
      for (int o = 16; o; o >>= 1) before += __shfl_xor_sync(kFull, before, o);
      if (lane == 0) s_at = base + before;
    }
    __syncthreads();
    int64_t at = s_at;
    for (int64_t j0 = jb; j0 < je; j0 += kRowThreads) {
      const int64_t j = j0 + threadIdx.x;
      const bool k = j < je && keep(x.x, j, b);
      const unsigned m = __ballot_sync(kFull, k);
      if (lane == 0) s_warp[wid] = __popc(m);
      __syncthreads();
      int before = 0, total = 0;
#pragma unroll
      for (int w = 0; w < kRowThreads / 32; ++w) {
        before += w < wid ? s_warp[w] : 0;
        total += s_warp[w];
      }
      if (k) set(at + before + __popc(m & ((1u << lane) - 1)), x.x, j);
      at += total;
      __syncthreads();
    }
  }
}

// The pieces of the rows of ptr; synchronises the stream.
inline RowPieces row_pieces(DeviceArena& arena, cudaStream_t s, int sms, const int64_t* ptr,
                            int64_t R) {
  RowPieces p;
  unsigned long long* n = arena_alloc<unsigned long long>(arena, 1, "row pieces");
  check_cuda(cudaMemsetAsync(n, 0, 8, s), "memset");
  row_pieces_count_kernel<<<grid_for(R, 256, sms, 16), 256, 0, s>>>(ptr, R, n);
  unsigned long long h = 0;
  check_cuda(cudaMemcpyAsync(&h, n, 8, cudaMemcpyDeviceToHost, s), "copy");
  check_cuda(cudaMemsetAsync(n, 0, 8, s), "memset");
  check_cuda(cudaStreamSynchronize(s), "row pieces");
  p.n = (int64_t)h;
  if (p.n > 0) {
    p.list = arena_alloc<int2>(arena, p.n, "row pieces");
    p.count = arena_alloc<int32_t>(arena, p.n, "row piece counts");
    row_pieces_list_kernel<<<grid_for(R, 256, sms, 16), 256, 0, s>>>(ptr, R, n, p.list);
  }
  arena.free(n);
  return p;
}

inline void free_row_pieces(DeviceArena& arena, RowPieces& p) {
  arena.free(p.list);
  arena.free(p.count);
  p = RowPieces();
}

// put is called once per short row and per piece of a long row.
template <typename Keep, typename Put>
void count_rows(cudaStream_t s, int sms, const int64_t* ptr, int64_t R, const RowPieces& p,
                Keep keep, Put put) {
  row_count_kernel<<<grid_for(R * 32, kRowThreads, sms, 16), kRowThreads, 0, s>>>(ptr, R, keep,
                                                                                 put);
  if (p.n > 0)
    piece_count_kernel<<<(unsigned)std::min<int64_t>(p.n, (int64_t)sms * 8), kRowThreads, 0, s>>>(
        ptr, p.list, p.n, p.count, keep, put);
}

// After count_rows with the same keep; out(r) < 0 leaves a row out.
template <typename Keep, typename Out, typename Set>
void fill_rows(cudaStream_t s, int sms, const int64_t* ptr, int64_t R, const RowPieces& p,
               Keep keep, Out out, Set set) {
  row_fill_kernel<<<grid_for(R * 32, kRowThreads, sms, 16), kRowThreads, 0, s>>>(ptr, R, keep, out,
                                                                                set);
  if (p.n > 0)
    piece_fill_kernel<<<(unsigned)std::min<int64_t>(p.n, (int64_t)sms * 8), kRowThreads, 0, s>>>(
        ptr, p.list, p.n, p.count, keep, out, set);
}

}  // namespace b200bfs
