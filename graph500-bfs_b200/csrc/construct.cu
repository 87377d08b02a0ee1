// Edge list -> degree-ordered, de-duplicated CSR on the device.
//
// Replaces make_symmetry_edge_list (mpi/benchmark_helper.hpp:383-497) and
// GraphConstructor2DCSR::construct (mpi/graph_constructor.hpp:1009-1033) for
// one rank:
//   1. estimate SCALE from the OR of all endpoints of non-loop edges
//      (benchmark_helper.hpp:488-494);
//   2. count the pre-dedup symmetric degree of every vertex
//      (DegreeCalculation::calc_degree, graph_constructor.hpp:572-592);
//   3. order vertices by descending degree, dropping degree-0 vertices
//      (VERTEX_REORDERING=2, :632-637; with group reordering the order is
//      taken within groups of 2^16 original ids, SMALL_REORDER_BIT :594-732);
//   4. place every directed entry into its row (two-pass counting placement),
//      sort each row and drop duplicates (sortEdgesInner, :1986-2056) to get
//      num_global_edges_ (:2100) and num_global_verts_ (:2103-2128).  Rows
//      are sorted by the neighbours' global degree rank (highest degree
//      first) even with group reordering, where the reference sorts by the
//      group-ordered id: adjacency order changes neither levels nor the
//      validity of parents, and hub-first lists let the bottom-up searches
//      stop early.
// Self-loops are dropped as in make_symmetry_edge_list (:409, 429, 447).
// Most passes are bandwidth-bound integer streams; the placement is bound by its
// random atomics.  CUB supplies the radix sorts and scans.
#include <algorithm>
#include <cub/cub.cuh>
#include "common.cuh"
#include "engine.h"
#include "row_filter.cuh"

namespace b200bfs {
namespace {

__global__ void or_ids_kernel(const uint2* __restrict__ e, int64_t m, unsigned long long* out) {
  uint32_t acc = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += (int64_t)gridDim.x * blockDim.x) {
    uint2 x = e[i];
    if (x.x != x.y) acc |= x.x | x.y;
  }
  for (int o = 16; o; o >>= 1) acc |= __shfl_xor_sync(kFull, acc, o);
  if (lane_id() == 0 && acc) atomicOr(out, (unsigned long long)acc);
}

__global__ void count_degree_kernel(const uint2* __restrict__ e, int64_t m, bool mirror,
                                    uint32_t* __restrict__ deg) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += (int64_t)gridDim.x * blockDim.x) {
    uint2 x = e[i];
    if (x.x == x.y) continue;
    atomicAdd(deg + x.x, 1u);
    if (mirror) atomicAdd(deg + x.y, 1u);
  }
}

// key = (degree==0) << 63 | group << 32 | (2^32-1 - degree): ascending order
// puts degree-0 vertices last and the rest in descending degree per group.
__global__ void make_keys_kernel(const uint32_t* __restrict__ deg, int64_t n, int group_bits,
                                 uint64_t* __restrict__ keys, int32_t* __restrict__ ids) {
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n;
       v += (int64_t)gridDim.x * blockDim.x) {
    uint32_t d = deg[v];
    uint64_t g = group_bits > 0 ? (uint64_t)(v >> group_bits) : 0;
    keys[v] = ((uint64_t)(d == 0) << 63) | (g << 32) | (uint64_t)(0xFFFFFFFFu - d);
    ids[v] = (int32_t)v;
  }
}

__global__ void fill_i32_kernel(int32_t* p, int64_t n, int32_t v) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    p[i] = v;
}

__global__ void rank_kernel(const int32_t* __restrict__ inv, const uint32_t* __restrict__ deg,
                            int64_t R, int32_t* __restrict__ rank, int32_t* __restrict__ mdeg,
                            int64_t* __restrict__ len64) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < R;
       r += (int64_t)gridDim.x * blockDim.x) {
    int32_t v = inv[r];
    rank[v] = (int32_t)r;
    uint32_t d = deg[v];
    mdeg[r] = (int32_t)d;
    len64[r] = d;
  }
}

// Places every edge in its source row; the stored value is the neighbour's
// sort key nkey[v] (its row id, or its global degree rank when rows follow
// the group order).  *bad is set if a neighbour has no row: a list said to be
// symmetric in which it is no edge's source.
__global__ void scatter_kernel(const uint2* __restrict__ e, int64_t m, bool mirror,
                               const int32_t* __restrict__ rank, const int32_t* __restrict__ nkey,
                               const int64_t* __restrict__ raw_ptr,
                               uint32_t* __restrict__ cursor, int32_t* __restrict__ raw,
                               unsigned long long* __restrict__ bad) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += (int64_t)gridDim.x * blockDim.x) {
    uint2 x = e[i];
    if (x.x == x.y) continue;
    int32_t ra = rank[x.x], rb = rank[x.y];
    if (rb < 0) {
      *bad = 1;
      continue;
    }
    raw[raw_ptr[ra] + atomicAdd(cursor + ra, 1u)] = nkey[x.y];
    if (mirror) raw[raw_ptr[rb] + atomicAdd(cursor + rb, 1u)] = nkey[x.x];
  }
}

// Group order: nkey[v] = position of v in the global degree order,
// row_of_key[k] = row of the vertex at global position k.
__global__ void global_rank_kernel(const int32_t* __restrict__ gorder, int64_t R,
                                   const int32_t* __restrict__ rank, int32_t* __restrict__ nkey,
                                   int32_t* __restrict__ row_of_key) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < R;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int32_t v = gorder[k];
    nkey[v] = (int32_t)k;
    row_of_key[k] = rank[v];
  }
}

__global__ void rel_offsets_kernel(const int64_t* __restrict__ raw_ptr, int64_t r0, int64_t nr,
                                   int32_t* __restrict__ rel) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= nr;
       i += (int64_t)gridDim.x * blockDim.x)
    rel[i] = (int32_t)(raw_ptr[r0 + i] - raw_ptr[r0]);
}

// Largest row index r1 in (r0, R] with raw_ptr[r1] - raw_ptr[r0] <= limit.
__global__ void chunk_end_kernel(const int64_t* __restrict__ raw_ptr, int64_t R, int64_t r0,
                                 int64_t limit, int64_t* out) {
  int64_t lo = r0 + 1, hi = R, base = raw_ptr[r0];
  // invariant: answer in [lo, hi]; at least one row even if it exceeds limit
  while (lo < hi) {
    int64_t mid = lo + (hi - lo + 1) / 2;
    if (raw_ptr[mid] - base <= limit) lo = mid;
    else hi = mid - 1;
  }
  *out = lo;
}

// First index of the sorted keys with the degree-0 bit (one thread).
__global__ void boundary_kernel(const uint64_t* __restrict__ keys, int64_t n, int64_t* out) {
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    const int64_t mid = (lo + hi) / 2;
    if (keys[mid] >> 63) hi = mid;
    else lo = mid + 1;
  }
  *out = lo;
}

// Rows are sorted by their length.  Up to 256 entries: a warp per row, in
// registers.  Up to 16384: a block per row in shared memory, over the bits
// that a key has.  From long_row (R / 512 entries, above 16384): by bitmap,
// setting the row's keys' bits (keys are below R) and reading them back in
// order, which drops the duplicates as well; all rows of a batch together and
// every pass spread over the grid.  Between the two, on graphs of more than 8 M
// rows: CUB's segmented sort, which gives a row of more than some hundred
// entries to a block that goes through global memory over all 32 bits.  The
// rows of a SCALE 22 build: 10.3 ms by the segmented sort alone, 3.4 ms so.
constexpr int kWarpRow = 256, kBlockRow = 16384;
constexpr int kSortClasses = 6;  // 0..3 block sorts, 4 bitmap, 5 segmented sort
__host__ __device__ __forceinline__ bool in_segmented_sort(int64_t len, int64_t long_row) {
  return len > kBlockRow && len < long_row;
}
__device__ __forceinline__ int sort_class(int64_t len, int64_t long_row) {
  if (len <= kWarpRow) return -1;
  if (len >= long_row) return 4;
  return len <= 512 ? 0 : len <= 2048 ? 1 : len <= 8192 ? 2 : len <= kBlockRow ? 3 : 5;
}

struct Less {
  __device__ bool operator()(int32_t a, int32_t b) const { return a < b; }
};

template <int kItems>
__device__ __forceinline__ void warp_sort(int32_t* __restrict__ row, int len, void* smem) {
  using Sort = cub::WarpMergeSort<int32_t, kItems, 32>;
  const int lane = lane_id();
  int32_t key[kItems];
#pragma unroll
  for (int q = 0; q < kItems; ++q) {
    const int x = lane * kItems + q;
    key[q] = x < len ? row[x] : 0x7FFFFFFF;
  }
  Sort(*static_cast<typename Sort::TempStorage*>(smem)).Sort(key, Less());
#pragma unroll
  for (int q = 0; q < kItems; ++q) {
    const int x = lane * kItems + q;
    if (x < len) row[x] = key[q];
  }
  __syncwarp();
}

__global__ void __launch_bounds__(256) warp_sort_kernel(const int64_t* __restrict__ ptr, int64_t R,
                                                        int32_t* __restrict__ raw) {
  __shared__ __align__(16) int32_t smem[8][kWarpRow + 32];
  static_assert(sizeof(cub::WarpMergeSort<int32_t, 8, 32>::TempStorage) <= sizeof(smem[0]),
                "shared memory of a warp");
  void* tmp = smem[threadIdx.x >> 5];
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = warp; r < R; r += nwarps) {
    const int64_t b = ptr[r], n = ptr[r + 1] - b;
    if (n <= 1 || n > kWarpRow) continue;
    if (n <= 32) warp_sort<1>(raw + b, (int)n, tmp);
    else if (n <= 64) warp_sort<2>(raw + b, (int)n, tmp);
    else if (n <= 128) warp_sort<4>(raw + b, (int)n, tmp);
    else warp_sort<8>(raw + b, (int)n, tmp);
  }
}
// of a batch's bitmaps, and no more than all entries take: a second buffer of
// that size is what sorting them elsewhere needs, so a budget that has room for
// the one has room for the other (one row's bitmap, R / 8 bytes, is smaller)
constexpr int64_t kBitmapBytes = int64_t(256) << 20;
constexpr int kBitTile = 8192;                        // words per block: 32 per thread

// Rows of each class: counted (list null), then listed from start[class].
__global__ void sort_classes_kernel(const int64_t* __restrict__ ptr, int64_t R, int64_t long_row,
                                    unsigned long long* __restrict__ start,
                                    int32_t* __restrict__ list) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < R;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int k = sort_class(ptr[r + 1] - ptr[r], long_row);
    if (k < 0) continue;
    const unsigned long long at = atomicAdd(start + k, 1ull);
    if (list) list[at] = (int32_t)r;
  }
}

// A block per row of at most kThreads * kItems entries.
template <int kThreads, int kItems>
__global__ void __launch_bounds__(kThreads)
    block_sort_kernel(const int64_t* __restrict__ ptr, const int32_t* __restrict__ list, int64_t n,
                      int pad, int bits, int32_t* __restrict__ raw) {
  using Sort = cub::BlockRadixSort<int32_t, kThreads, kItems>;
  extern __shared__ __align__(16) unsigned char smem[];
  typename Sort::TempStorage& tmp = *reinterpret_cast<typename Sort::TempStorage*>(smem);
  for (int64_t i = blockIdx.x; i < n; i += gridDim.x) {
    const int64_t b = ptr[list[i]];
    const int len = (int)(ptr[list[i] + 1] - b);
    int32_t key[kItems];
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
      const int x = q * kThreads + threadIdx.x;
      key[q] = x < len ? raw[b + x] : pad;  // pad: above every key
    }
    Sort(tmp).SortBlockedToStriped(key, 0, bits);
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
      const int x = q * kThreads + threadIdx.x;
      if (x < len) raw[b + x] = key[q];
    }
    __syncthreads();
  }
}

template <int kThreads, int kItems>
void block_sort(cudaStream_t s, int sms, const int64_t* ptr, const int32_t* list, int64_t n,
                int64_t R, int32_t* raw) {
  if (n <= 0) return;
  const int bytes =
      (int)sizeof(typename cub::BlockRadixSort<int32_t, kThreads, kItems>::TempStorage);
  auto kernel = block_sort_kernel<kThreads, kItems>;
  if (bytes > 48 * 1024)
    check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes),
               "block sort");
  int bits = 1;
  while ((int64_t(1) << bits) <= R) ++bits;
  kernel<<<(unsigned)std::min<int64_t>(n, (int64_t)sms * 32), kThreads, bytes, s>>>(
      ptr, list, n, (int)R, bits, raw);
}

// blockIdx.y: row of the batch, in the next four kernels.
__global__ void bits_set_kernel(const int64_t* __restrict__ ptr, const int32_t* __restrict__ list,
                                const int32_t* __restrict__ raw, int64_t words,
                                uint32_t* __restrict__ bits) {
  const int32_t r = list[blockIdx.y];
  uint32_t* bm = bits + blockIdx.y * words;
  for (int64_t j = ptr[r] + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < ptr[r + 1];
       j += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t k = (uint32_t)raw[j];
    red_or(bm + (k >> 5), 1u << (k & 31));
  }
}

__global__ void __launch_bounds__(256)
    bits_count_kernel(const uint32_t* __restrict__ bits, int64_t words, int64_t tiles,
                      int32_t* __restrict__ count) {
  __shared__ int s_sum;
  const uint32_t* bm = bits + blockIdx.y * words;
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    if (threadIdx.x == 0) s_sum = 0;
    __syncthreads();
    int c = 0;
    for (int i = threadIdx.x; i < kBitTile; i += 256)
      if (t * kBitTile + i < words) c += __popc(bm[t * kBitTile + i]);
    c = __reduce_add_sync(kFull, c);
    if (lane_id() == 0) atomicAdd(&s_sum, c);
    __syncthreads();
    if (threadIdx.x == 0) count[blockIdx.y * tiles + t] = s_sum;
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256)
    bits_write_kernel(const int64_t* __restrict__ ptr, const int32_t* __restrict__ list,
                      const uint32_t* __restrict__ bits, int64_t words, int64_t tiles,
                      const int32_t* __restrict__ count, int32_t* __restrict__ raw) {
  __shared__ int64_t s_at;
  __shared__ int s_warp[8];
  const uint32_t* bm = bits + blockIdx.y * words;
  const int lane = lane_id(), wid = threadIdx.x >> 5;
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    if (wid == 0) {
      int64_t before = 0;
      for (int64_t k = lane; k < t; k += 32) before += count[blockIdx.y * tiles + k];
#pragma unroll
      for (int o = 16; o; o >>= 1) before += __shfl_xor_sync(kFull, before, o);
      if (lane == 0) s_at = ptr[list[blockIdx.y]] + before;
    }
    const int64_t w0 = t * kBitTile + threadIdx.x * 32;
    int c = 0;
    for (int i = 0; i < 32; ++i) c += w0 + i < words ? __popc(bm[w0 + i]) : 0;
    int incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += x;
    }
    if (lane == 31) s_warp[wid] = incl;
    __syncthreads();
    int64_t at = s_at + incl - c;
    for (int w = 0; w < wid; ++w) at += s_warp[w];
    for (int i = 0; i < 32 && w0 + i < words; ++i)
      for (uint32_t x = bm[w0 + i]; x; x &= x - 1)
        raw[at++] = (int32_t)((w0 + i) * 32 + __ffs(x) - 1);
    __syncthreads();
  }
}

// The places of a row's dropped duplicates repeat its last key.
__global__ void bits_tail_kernel(const int64_t* __restrict__ ptr, const int32_t* __restrict__ list,
                                 int64_t tiles, const int32_t* __restrict__ count,
                                 int32_t* __restrict__ raw) {
  const int32_t r = list[blockIdx.y];
  int64_t n = 0;
  for (int64_t k = 0; k < tiles; ++k) n += count[blockIdx.y * tiles + k];
  const int64_t b = ptr[r];
  const int32_t last = raw[b + n - 1];
  for (int64_t j = b + n + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < ptr[r + 1];
       j += (int64_t)gridDim.x * blockDim.x)
    raw[j] = last;
}

// Segment ends of the segmented sort: the rows sorted elsewhere are empty.
__global__ void segment_ends_kernel(const int32_t* __restrict__ rel, int64_t nr, int64_t long_row,
                                    int32_t* __restrict__ end) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nr;
       i += (int64_t)gridDim.x * blockDim.x)
    end[i] = in_segmented_sort(rel[i + 1] - rel[i], long_row) ? rel[i + 1] : rel[i];
}

// The rows that the segmented sort left in its other buffer (warp per row).
__global__ void segments_back_kernel(const int32_t* __restrict__ rel,
                                     const int32_t* __restrict__ end, int64_t nr,
                                     const int32_t* __restrict__ alt, int32_t* __restrict__ raw) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t i = warp; i < nr; i += nwarps)
    for (int64_t j = rel[i] + lane_id(); j < end[i]; j += 32) raw[j] = alt[j];
}

// Of a sorted row, the first entry of each run of equal values.
struct Distinct {
  const int32_t* raw;
  __device__ bool operator()(int64_t, int64_t j, int64_t b) const {
    return j == b || raw[j] != raw[j - 1];
  }
};
struct AddLength {  // a row's length, from one piece or several
  unsigned long long* len;
  __device__ void operator()(int64_t r, int64_t c) const {
    atomicAdd(len + r, (unsigned long long)c);
  }
};
struct RowStart {
  const int64_t* row_ptr;
  __device__ int64_t operator()(int64_t r) const { return row_ptr[r]; }
};
struct PutNeighbour {  // the neighbour's row id
  const int32_t *raw, *row_of_key;
  int32_t* col;
  __device__ void operator()(int64_t at, int64_t, int64_t j) const {
    col[at] = row_of_key ? row_of_key[raw[j]] : raw[j];
  }
};

__global__ void first_kernel(const int64_t* __restrict__ row_ptr, const int32_t* __restrict__ col,
                             const int32_t* __restrict__ inv, int64_t R,
                             int32_t* __restrict__ first, int2* __restrict__ first_pair) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < R;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int32_t f = row_ptr[r + 1] > row_ptr[r] ? col[row_ptr[r]] : -1;
    first[r] = f;
    if (first_pair) first_pair[r] = make_int2(f, f >= 0 ? inv[f] : -1);
  }
}

__global__ void max_degree_kernel(const int64_t* __restrict__ row_ptr, int64_t R,
                                  unsigned long long* out) {
  unsigned long long acc = 0;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < R;
       r += (int64_t)gridDim.x * blockDim.x)
    acc = max(acc, (unsigned long long)(row_ptr[r + 1] - row_ptr[r]));
  for (int o = 16; o; o >>= 1) acc = max(acc, __shfl_xor_sync(kFull, acc, o));
  if (lane_id() == 0) atomicMax(out, acc);
}

int msb_index(uint64_t v) { return v ? 63 - __builtin_clzll(v) : -1; }

}  // namespace

void build_csr(DeviceArena& arena, cudaStream_t s, const uint2* edges, int64_t m, bool mirror,
               bool group_reorder, int scale_hint, Graph& g, int sms) {
  const int B = 256;
  auto grid = [&](int64_t n) { return grid_for(n, B, sms, 16); };

  // 1. SCALE estimate.
  unsigned long long* d_u64 = arena_alloc<unsigned long long>(arena, 2, "scalars");
  check_cuda(cudaMemsetAsync(d_u64, 0, 16, s), "memset");
  or_ids_kernel<<<grid(m), B, 0, s>>>(edges, m, d_u64);
  unsigned long long orv = 0;
  check_cuda(cudaMemcpyAsync(&orv, d_u64, 8, cudaMemcpyDeviceToHost, s), "copy");
  check_cuda(cudaStreamSynchronize(s), "scale estimate");
  int est = msb_index(orv) + 1;
  if (est <= 0) est = 1;
  if (scale_hint > 0 && est > scale_hint)
    throw Error{B200BFS_ERR_INVALID, "edge endpoints exceed 2^scale"};
  if (est > 30) throw Error{B200BFS_ERR_INVALID, "SCALE above 30 is not supported"};
  g.scale = est;
  g.nverts = int64_t(1) << est;
  g.pred_size = std::max<int64_t>(g.nverts, int64_t(1) << 16);
  g.group_reorder = group_reorder;
  // Group width of the group order: min(16, 48 - local id bits)
  // (graph_constructor.hpp:704-712), which is 16 for every SCALE <= 30 here.
  // Below SCALE 16 one group holds every id, as with a narrower group.
  const int group_bits = group_reorder ? 16 : 0;
  g.reorder_bits = group_bits;
  const int64_t n = g.nverts;

  // 2. pre-dedup degree
  uint32_t* deg = arena_alloc<uint32_t>(arena, n, "degree");
  check_cuda(cudaMemsetAsync(deg, 0, n * 4, s), "memset");
  count_degree_kernel<<<grid(m), B, 0, s>>>(edges, m, mirror, deg);

  // 3. degree order
  uint64_t* keys = arena_alloc<uint64_t>(arena, n, "sort keys");
  uint64_t* keys2 = arena_alloc<uint64_t>(arena, n, "sort keys");
  int32_t* ids = arena_alloc<int32_t>(arena, n, "sort values");
  int32_t* ids2 = arena_alloc<int32_t>(arena, n, "sort values");
  make_keys_kernel<<<grid(n), B, 0, s>>>(deg, n, group_bits, keys, ids);
  {
    size_t tmp = 0;
    check_cuda(cub::DeviceRadixSort::SortPairs(nullptr, tmp, keys, keys2, ids, ids2, (int)n, 0,
                                               64, s),
               "sort size");
    void* t = arena.alloc(tmp, "sort temp");
    check_cuda(cub::DeviceRadixSort::SortPairs(t, tmp, keys, keys2, ids, ids2, (int)n, 0, 64, s),
               "sort");
    arena.free(t);
  }
  arena.free(keys);
  // R = number of keys without the degree-0 bit, which sorts them last.
  int64_t R = 0;
  boundary_kernel<<<1, 1, 0, s>>>(keys2, n, reinterpret_cast<int64_t*>(d_u64));
  check_cuda(cudaMemcpyAsync(&R, d_u64, 8, cudaMemcpyDeviceToHost, s), "row count");
  check_cuda(cudaStreamSynchronize(s), "row count");
  arena.free(keys2);
  arena.free(ids);
  if (R == 0) throw Error{B200BFS_ERR_INVALID, "graph has no edges"};
  Csr& c = g.csr;
  c.nrows = R;
  c.inv = arena_alloc<int32_t>(arena, R, "inv map");
  check_cuda(cudaMemcpyAsync(c.inv, ids2, R * 4, cudaMemcpyDeviceToDevice, s), "copy inv");
  arena.free(ids2);
  c.rank = arena_alloc<int32_t>(arena, n, "rank map");
  fill_i32_kernel<<<grid(n), B, 0, s>>>(c.rank, n, -1);
  c.mdeg = arena_alloc<int32_t>(arena, R, "mdeg");
  int64_t* raw_ptr = arena_alloc<int64_t>(arena, R + 1, "raw row ptr");
  int64_t* len64 = arena_alloc<int64_t>(arena, R, "row len");
  rank_kernel<<<grid(R), B, 0, s>>>(c.inv, deg, R, c.rank, c.mdeg, len64);
  // Neighbour lists are sorted by the neighbours' global degree rank, highest
  // degree first, whatever the row numbering: the bottom-up searches stop at
  // the first neighbour found, and the hubs are found first.  With one global
  // degree order the rank is the row id; with the group order it comes from a
  // second sort by degree alone.
  int32_t* nkey = c.rank;
  int32_t* row_of_key = nullptr;
  if (group_bits > 0) {
    uint64_t* k1 = arena_alloc<uint64_t>(arena, n, "sort keys");
    uint64_t* k2 = arena_alloc<uint64_t>(arena, n, "sort keys");
    int32_t* i1 = arena_alloc<int32_t>(arena, n, "sort values");
    int32_t* i2 = arena_alloc<int32_t>(arena, n, "sort values");
    make_keys_kernel<<<grid(n), B, 0, s>>>(deg, n, 0, k1, i1);
    size_t tmp = 0;
    check_cuda(cub::DeviceRadixSort::SortPairs(nullptr, tmp, k1, k2, i1, i2, (int)n, 0, 64, s),
               "sort size");
    void* t = arena.alloc(tmp, "sort temp");
    check_cuda(cub::DeviceRadixSort::SortPairs(t, tmp, k1, k2, i1, i2, (int)n, 0, 64, s),
               "sort");
    arena.free(t);
    arena.free(k1);
    arena.free(k2);
    arena.free(i1);
    nkey = arena_alloc<int32_t>(arena, n, "neighbour keys");
    row_of_key = arena_alloc<int32_t>(arena, R, "key to row");
    global_rank_kernel<<<grid(R), B, 0, s>>>(i2, R, c.rank, nkey, row_of_key);
    arena.free(i2);
  }
  arena.free(deg);
  check_cuda(cudaMemsetAsync(raw_ptr, 0, 8, s), "memset");
  {
    size_t tmp = 0;
    check_cuda(cub::DeviceScan::InclusiveSum(nullptr, tmp, len64, raw_ptr + 1, (int)R, s),
               "scan size");
    void* t = arena.alloc(tmp, "scan temp");
    check_cuda(cub::DeviceScan::InclusiveSum(t, tmp, len64, raw_ptr + 1, (int)R, s), "scan");
    arena.free(t);
  }
  int64_t total = 0;
  check_cuda(cudaMemcpyAsync(&total, raw_ptr + R, 8, cudaMemcpyDeviceToHost, s), "copy");
  check_cuda(cudaStreamSynchronize(s), "total");

  // 4. placement
  int32_t* raw = arena_alloc<int32_t>(arena, total, "raw adjacency");
  uint32_t* cursor = arena_alloc<uint32_t>(arena, R, "cursor");
  check_cuda(cudaMemsetAsync(cursor, 0, R * 4, s), "memset");
  scatter_kernel<<<grid(m), B, 0, s>>>(edges, m, mirror, c.rank, nkey, raw_ptr, cursor, raw,
                                       d_u64 + 1);
  if (!mirror) {
    unsigned long long bad = 0;
    check_cuda(cudaMemcpyAsync(&bad, d_u64 + 1, 8, cudaMemcpyDeviceToHost, s), "copy");
    check_cuda(cudaStreamSynchronize(s), "placement");
    if (bad) throw Error{B200BFS_ERR_INVALID, "edge list is not symmetric"};
  }
  if (nkey != c.rank) arena.free(nkey);
  arena.free(cursor);

  // 5. per-row sort (see sort_class); the segmented sort in chunks of at most
  // 2^30 entries
  const int64_t long_row = std::max<int64_t>(kBlockRow + 1, R / 512);
  int32_t* sort_list = nullptr;
  unsigned long long first[kSortClasses + 1] = {0};  // of each class in sort_list
  {
    unsigned long long* d_class = arena_alloc<unsigned long long>(arena, 8, "sort classes");
    check_cuda(cudaMemsetAsync(d_class, 0, 64, s), "memset");
    sort_classes_kernel<<<grid(R), B, 0, s>>>(raw_ptr, R, long_row, d_class, nullptr);
    check_cuda(cudaMemcpyAsync(first + 1, d_class, kSortClasses * 8, cudaMemcpyDeviceToHost, s), "copy");
    check_cuda(cudaStreamSynchronize(s), "sort classes");
    for (int k = 1; k <= kSortClasses; ++k) first[k] += first[k - 1];
    warp_sort_kernel<<<grid(R * 32), 256, 0, s>>>(raw_ptr, R, raw);
    if (first[kSortClasses] > 0) {
      sort_list = arena_alloc<int32_t>(arena, (int64_t)first[kSortClasses], "sort list");
      check_cuda(cudaMemcpyAsync(d_class, first, kSortClasses * 8, cudaMemcpyHostToDevice, s), "copy");
      sort_classes_kernel<<<grid(R), B, 0, s>>>(raw_ptr, R, long_row, d_class, sort_list);
      auto n = [&](int k) { return (int64_t)(first[k + 1] - first[k]); };
      block_sort<128, 4>(s, sms, raw_ptr, sort_list + first[0], n(0), R, raw);
      block_sort<256, 8>(s, sms, raw_ptr, sort_list + first[1], n(1), R, raw);
      block_sort<512, 16>(s, sms, raw_ptr, sort_list + first[2], n(2), R, raw);
      block_sort<1024, 16>(s, sms, raw_ptr, sort_list + first[3], n(3), R, raw);
    }
    arena.free(d_class);
  }
  const int64_t nlong = (int64_t)(first[5] - first[4]);
  const int32_t* long_list = sort_list + first[4];
  if (nlong > 0) {
    const int64_t words = (R + 31) / 32, tiles = (words + kBitTile - 1) / kBitTile;
    const int64_t bytes = std::min(kBitmapBytes, total * 4);
    const int64_t batch =
        std::min({nlong, std::max<int64_t>(1, bytes / (words * 4)), (int64_t)32768});
    uint32_t* bits = arena_alloc<uint32_t>(arena, batch * words, "long row bitmaps");
    int32_t* count = arena_alloc<int32_t>(arena, batch * tiles, "long row counts");
    for (int64_t i = 0; i < nlong; i += batch) {
      const unsigned k = (unsigned)std::min(batch, nlong - i);
      const int64_t per = (2 * (int64_t)sms * 8 + k - 1) / k;  // blocks per row
      const dim3 by_entry((unsigned)per, k);
      const dim3 by_tile((unsigned)std::min(tiles, per), k);
      check_cuda(cudaMemsetAsync(bits, 0, k * words * 4, s), "memset");
      bits_set_kernel<<<by_entry, B, 0, s>>>(raw_ptr, long_list + i, raw, words, bits);
      bits_count_kernel<<<by_tile, 256, 0, s>>>(bits, words, tiles, count);
      bits_write_kernel<<<by_tile, 256, 0, s>>>(raw_ptr, long_list + i, bits, words, tiles, count,
                                                raw);
      bits_tail_kernel<<<by_entry, B, 0, s>>>(raw_ptr, long_list + i, tiles, count, raw);
    }
    arena.free(bits);
    arena.free(count);
  }
  if (total > int64_t(1) << 30 || first[6] > first[5]) {
    const int64_t kChunk = int64_t(1) << 30;
    int64_t* d_end = reinterpret_cast<int64_t*>(d_u64);
    int32_t* alt = nullptr;
    if (first[6] > first[5])
      alt = arena_alloc<int32_t>(arena, std::min(total, kChunk) + 1, "sort alt");
    int32_t *rel = nullptr, *seg_end = nullptr;
    int64_t rel_cap = 0;
    void* tmp = nullptr;
    size_t tmp_cap = 0;
    for (int64_t r0 = 0; r0 < R;) {
      chunk_end_kernel<<<1, 1, 0, s>>>(raw_ptr, R, r0, kChunk, d_end);
      int64_t r1, lo, hi;
      check_cuda(cudaMemcpyAsync(&r1, d_end, 8, cudaMemcpyDeviceToHost, s), "copy");
      check_cuda(cudaMemcpyAsync(&lo, raw_ptr + r0, 8, cudaMemcpyDeviceToHost, s), "copy");
      check_cuda(cudaStreamSynchronize(s), "chunk");
      check_cuda(cudaMemcpyAsync(&hi, raw_ptr + r1, 8, cudaMemcpyDeviceToHost, s), "copy");
      check_cuda(cudaStreamSynchronize(s), "chunk");
      const int64_t nr = r1 - r0, ni = hi - lo;
      if (ni > kChunk) throw Error{B200BFS_ERR_INVALID, "row longer than 2^30 entries"};
      if (nr + 1 > rel_cap) {
        arena.free(rel);
        arena.free(seg_end);
        rel_cap = nr + 1;
        rel = arena_alloc<int32_t>(arena, rel_cap, "segment offsets");
        seg_end = arena_alloc<int32_t>(arena, rel_cap, "segment ends");
      }
      rel_offsets_kernel<<<grid(nr + 1), B, 0, s>>>(raw_ptr, r0, nr, rel);
      segment_ends_kernel<<<grid(nr), B, 0, s>>>(rel, nr, long_row, seg_end);
      if (ni > 1 && first[6] > first[5]) {
        cub::DoubleBuffer<int32_t> db(raw + lo, alt);
        size_t need = 0;
        check_cuda(cub::DeviceSegmentedSort::SortKeys(nullptr, need, db, (int)ni, (int)nr, rel,
                                                       seg_end, s),
                   "segsort size");
        if (need > tmp_cap) {
          if (tmp) arena.free(tmp);
          tmp_cap = need;
          tmp = arena.alloc(tmp_cap, "segsort temp");
        }
        check_cuda(cub::DeviceSegmentedSort::SortKeys(tmp, need, db, (int)ni, (int)nr, rel,
                                                       seg_end, s),
                   "segsort");
        if (db.Current() != raw + lo)
          segments_back_kernel<<<grid(nr * 32), B, 0, s>>>(rel, seg_end, nr, db.Current(),
                                                          raw + lo);
      }
      r0 = r1;
    }
    check_cuda(cudaStreamSynchronize(s), "segsort");
    if (tmp) arena.free(tmp);
    arena.free(rel);
    arena.free(seg_end);
    arena.free(alt);
  }
  arena.free(sort_list);

  // 6. de-duplicate and compact
  int64_t* dlen = len64;
  RowPieces pieces = row_pieces(arena, s, sms, raw_ptr, R);
  check_cuda(cudaMemsetAsync(dlen, 0, R * 8, s), "memset");
  count_rows(s, sms, raw_ptr, R, pieces, Distinct{raw},
             AddLength{reinterpret_cast<unsigned long long*>(dlen)});
  c.row_ptr = arena_alloc<int64_t>(arena, R + 1, "row ptr");
  check_cuda(cudaMemsetAsync(c.row_ptr, 0, 8, s), "memset");
  {
    size_t tmp = 0;
    check_cuda(cub::DeviceScan::InclusiveSum(nullptr, tmp, dlen, c.row_ptr + 1, (int)R, s),
               "scan size");
    void* t = arena.alloc(tmp, "scan temp");
    check_cuda(cub::DeviceScan::InclusiveSum(t, tmp, dlen, c.row_ptr + 1, (int)R, s), "scan");
    arena.free(t);
  }
  check_cuda(cudaMemcpyAsync(&c.nedges, c.row_ptr + R, 8, cudaMemcpyDeviceToHost, s), "copy");
  check_cuda(cudaStreamSynchronize(s), "dedup count");
  c.col = arena_alloc<int32_t>(arena, c.nedges, "adjacency");
  fill_rows(s, sms, raw_ptr, R, pieces, Distinct{raw}, RowStart{c.row_ptr},
            PutNeighbour{raw, row_of_key, c.col});
  check_cuda(cudaMemsetAsync(d_u64, 0, 8, s), "memset");
  max_degree_kernel<<<grid(R), B, 0, s>>>(c.row_ptr, R, d_u64);
  unsigned long long maxd = 0;
  check_cuda(cudaMemcpyAsync(&maxd, d_u64, 8, cudaMemcpyDeviceToHost, s), "copy");
  check_cuda(cudaStreamSynchronize(s), "compact");
  c.max_degree = (int64_t)maxd;
  free_row_pieces(arena, pieces);
  arena.free(raw);
  arena.free(raw_ptr);
  arena.free(len64);
  arena.free(d_u64);
  if (row_of_key) arena.free(row_of_key);
  build_first(arena, s, c, sms);
  check_cuda(cudaGetLastError(), "build_csr");
}

void build_first(DeviceArena& arena, cudaStream_t s, Csr& c, int sms, bool parent_ids) {
  arena.free(c.first);
  arena.free(c.first_pair);
  c.first_pair = nullptr;
  c.first = arena_alloc<int32_t>(arena, c.nrows, "first neighbours");
  if (parent_ids) {
    // rounded up to whole 32-row bitmap words: the bottom-up sweep's early
    // loads read the entries of all 32 rows of a word, the last word's
    // padding rows included (their entries are discarded); the padding
    // holds (-1, -1)
    const int64_t padded = (c.nrows + 31) / 32 * 32;
    c.first_pair = arena_alloc<int2>(arena, padded, "first neighbour pairs");
    check_cuda(cudaMemsetAsync(c.first_pair, 0xFF, padded * sizeof(int2), s), "memset");
  }
  first_kernel<<<grid_for(c.nrows, 256, sms, 16), 256, 0, s>>>(c.row_ptr, c.col, c.inv, c.nrows,
                                                               c.first, c.first_pair);
  check_cuda(cudaGetLastError(), "first neighbours");
}

}  // namespace b200bfs
