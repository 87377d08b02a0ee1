// Graph500 result validation on the device.
//
// Restates BfsValidation::validate (mpi/validate.hpp:607-976) for one GPU,
// stopping at the first group of checks that finds errors, as the reference
// does: value ranges (:994-1016), root is its own parent, no other self-parent,
// the depth map (check_bfs_depth_map_using_predecessors :1145-1254, or
// build_bfs_depth_map :1040-1141 with CoreBFS, which leaves tree levels
// unknown), then one pass over the input edges: endpoint depths must differ
// by at most one or both be unreached, tree edges must match depths
// (check_pred_depth :1018-1034), each reached vertex must have an input edge
// to its parent, and the edges with both endpoints reached are counted
// (edge_visit_count, the TEPS numerator).
#include <algorithm>
#include "common.cuh"
#include "validate.h"
#include "corebfs.h"

namespace b200bfs {
namespace {

__device__ __forceinline__ int64_t parent_of(int64_t x) { return (int64_t)((uint64_t)x << 16) >> 16; }
__device__ __forceinline__ int depth_of(int64_t x) { return (int)(((uint64_t)x >> 48) & 0xFFFF); }
__device__ __forceinline__ int64_t with_depth(int64_t x, int d) {
  return (int64_t)(((uint64_t)x & 0xFFFFFFFFFFFFull) | ((uint64_t)(d & 0xFFFF) << 48));
}

// What the checks before the edge pass need, gathered in one pass over pred.
struct Checks {
  unsigned long long below;      // parents below -1
  unsigned long long self;       // self-parents other than the root
  unsigned long long depth;      // wrong depths (without CoreBFS)
  unsigned long long edge;       // errors of the edge pass
  unsigned long long visited;    // input edges with both ends reached
  unsigned long long deep;       // chains the depth map left to depth_build_kernel
  unsigned long long max_parent; // + 1
  unsigned long long max_used;   // highest vertex with an edge, + 1
  long long root_entry;
};

__device__ __forceinline__ void add_up(unsigned long long* to, unsigned long long x) {
#pragma unroll
  for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
  if (lane_id() == 0 && x) atomicAdd(to, x);
}
__device__ __forceinline__ void max_up(unsigned long long* to, unsigned long long x) {
#pragma unroll
  for (int o = 16; o; o >>= 1) x = max(x, __shfl_xor_sync(kFull, x, o));
  if (lane_id() == 0 && x) atomicMax(to, x);
}

// Value ranges, self-parents, depths and the highest used vertex
// (find_max_used_vertex, benchmark_helper.hpp:564-582: rank or tree parent as
// in has_edge) of every id, whichever of them the verdict turns out to need:
// one pass of 75 us at SCALE 23, whose counters are read with those of the
// edge pass, where six with a readback after each take 130 us of kernels and
// as much waiting.  An entry is looked at only if its index is in range.
// kMap: with CoreBFS, the depth map (build_bfs_depth_map) is written to map
// in the same pass instead of a check of the depths: entries of unknown depth
// take that of the first ancestor with a known one, plus the steps.  map may
// be pred itself: an ancestor that has its depth already only ends the climb
// sooner, with the same depth, and parents are not changed.
template <bool kMap>
__global__ void pred_checks_kernel(const int64_t* pred, int64_t n, int64_t root,
                                   const int32_t* __restrict__ rank,
                                   const int32_t* __restrict__ tp, int64_t nverts,
                                   int64_t* map, Checks* __restrict__ out) {
  unsigned long long below = 0, self = 0, bad = 0, deep = 0, top = 0, used = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t x = pred[i];
    const int64_t p = parent_of(x);
    const int d = depth_of(x);
    if (i < nverts && (rank[i] >= 0 || (tp && tp[i] >= 0))) used = (unsigned long long)i + 1;
    if (p < -1) ++below;
    if (p >= 0) top = max(top, (unsigned long long)p + 1);
    if (i == root) out->root_entry = x;
    else if (p == i) ++self;
    if (kMap) {
      int64_t y = i == root ? with_depth(x, 0) : x;
      if (i != root && p >= 0 && d == 0xFFFF) {
        int64_t q = p;
        for (int up = 1;; ++up) {
          if (q < 0 || q >= n) break;  // no known ancestor
          if (up > 64) {
            ++deep;
            break;
          }
          const int64_t z = pred[q];
          const int dq = q == root ? 0 : depth_of(z);
          if (dq != 0xFFFF) {
            if (dq + up < 0xFFFF) y = with_depth(x, dq + up);
            else ++deep;
            break;
          }
          q = parent_of(z);
        }
      }
      map[i] = y;
    } else {
      if (p == -1 && d != 0xFFFF) ++bad;
      else if (p != -1 && d == 0xFFFF) ++bad;
      if (i == root) {
        if (d != 0) ++bad;
      } else if (p != -1) {
        const int dp = p >= 0 && p < n ? depth_of(__ldg(pred + p)) : 0xFFFF;
        if (dp == 0xFFFF) ++bad;
        if (d != dp + 1) ++bad;
      }
    }
  }
  add_up(&out->below, below);
  add_up(&out->self, self);
  add_up(&out->depth, bad);
  add_up(&out->deep, deep);
  max_up(&out->max_parent, top);
  max_up(&out->max_used, used);
}

__global__ void range_kernel(const int64_t* __restrict__ pred, int64_t n, int64_t nglobal,
                             unsigned long long* err) {
  unsigned long long e = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = parent_of(pred[i]);
    if (p < -1 || p >= nglobal) ++e;
  }
  if (e) atomicAdd(err, e);
}

__global__ void depth_build_kernel(int64_t* __restrict__ pred, int64_t n, int64_t root,
                                   int* changed) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    if (i == root) continue;
    const int64_t x = pred[i];
    const int64_t p = parent_of(x);
    if (p < 0 || depth_of(x) != 0xFFFF) continue;
    const int dp = depth_of(pred[p]);
    if (dp != 0xFFFF) {
      pred[i] = with_depth(x, dp + 1);
      *changed = 1;
    }
  }
}

__global__ void edge_check_kernel(const uint2* __restrict__ edges, int64_t m, int64_t n,
                                  const int64_t* __restrict__ pred, uint8_t* __restrict__ valid,
                                  unsigned long long* err, unsigned long long* count) {
  unsigned long long e = 0, c = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += (int64_t)gridDim.x * blockDim.x) {
    const uint2 ed = edges[i];
    const int64_t s = ed.x, t = ed.y;
    if (s >= n || t >= n) {  // endpoint outside pred[]
      ++e;
      continue;
    }
    const int64_t ps = pred[s], pt = pred[t];
    const int sd = depth_of(ps), td = depth_of(pt);
    if (sd != 0xFFFF && td == 0xFFFF) ++e;
    else if (sd == 0xFFFF && td != 0xFFFF) ++e;
    else if (sd - td < -1 || sd - td > 1) ++e;
    else if (sd != 0xFFFF) ++c;
    if (parent_of(ps) == t) {
      if (s != t && td + 1 != sd) ++e;
      valid[s] = 1;
    }
    if (parent_of(pt) == s) {
      if (s != t && sd + 1 != td) ++e;
      valid[t] = 1;
    }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    e += __shfl_xor_sync(kFull, e, o);
    c += __shfl_xor_sync(kFull, c, o);
  }
  if (lane_id() == 0) {
    if (e) atomicAdd(err, e);
    if (c) atomicAdd(count, c);
  }
}

__global__ void parent_edge_kernel(const int64_t* __restrict__ pred, int64_t n, int64_t root,
                                   const uint8_t* __restrict__ valid, unsigned long long* err) {
  unsigned long long e = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    if (i == root || parent_of(pred[i]) == -1) continue;
    if (!valid[i]) ++e;
  }
  if (e) atomicAdd(err, e);
}

}  // namespace

void validate_device(DeviceArena& arena, cudaStream_t s, int sms, const Graph& g,
                     const int64_t* pred, bool on_device, bool corebfs, int64_t root,
                     int64_t* errors, int64_t* edge_visit_count) {
  const int B = 256;
  const int64_t n = g.pred_size;
  auto grid = [&](int64_t items) { return grid_for(items, B, sms, 16); };
  if (root < 0 || root >= g.nverts) throw Error{B200BFS_ERR_INVALID, "root out of range"};
  if (!g.input_edges) throw Error{B200BFS_ERR_STATE, "input edges are not resident"};
  // The caller's pred on the device; with CoreBFS the depth map, in the copy's
  // place or beside the engine's pred.
  int64_t* copy = nullptr;
  if (!on_device) {
    copy = arena_alloc<int64_t>(arena, n, "pred copy");
    check_cuda(cudaMemcpyAsync(copy, pred, n * 8, cudaMemcpyDefault, s), "copy");
    pred = copy;
  }
  int64_t* beside = corebfs && !copy ? arena_alloc<int64_t>(arena, n, "depth map") : nullptr;
  int64_t* map = copy ? copy : beside;
  uint8_t* valid = arena_alloc<uint8_t>(arena, n, "pred valid");
  Checks* out = arena_alloc<Checks>(arena, 1, "validation counters");
  const int64_t* p = corebfs ? map : pred;
  const int32_t* tp = g.core.enabled ? g.core.tree_parent : nullptr;
  auto edge_pass = [&] {
    check_cuda(cudaMemsetAsync(valid, 0, n, s), "memset");
    edge_check_kernel<<<grid(g.num_input_edges), B, 0, s>>>(
        g.input_edges, g.num_input_edges, n, p, valid, &out->edge, &out->visited);
    parent_edge_kernel<<<grid(n), B, 0, s>>>(p, n, root, valid, &out->edge);
  };
  Checks h;
  auto read = [&](const char* what) {
    check_cuda(cudaMemcpyAsync(&h, out, sizeof(h), cudaMemcpyDeviceToHost, s), "copy");
    check_cuda(cudaStreamSynchronize(s), what);
  };
  check_cuda(cudaMemsetAsync(out, 0, sizeof(Checks), s), "memset");
  if (corebfs)
    pred_checks_kernel<true><<<grid(n), B, 0, s>>>(pred, n, root, g.csr.rank, tp, g.nverts, map,
                                                   out);
  else
    pred_checks_kernel<false><<<grid(n), B, 0, s>>>(pred, n, root, g.csr.rank, tp, g.nverts,
                                                    nullptr, out);
  edge_pass();
  read("validation");
  // The checks count in the reference's order and stop at the first that
  // fails (validate.hpp:612-664): value ranges, the root's own parent, other
  // self-parents, the depth map, then the pass over the input edges.
  *edge_visit_count = 0;
  const int64_t nglobal = std::max<int64_t>((int64_t)h.max_used, 1);
  int64_t err = (int64_t)h.below;
  if ((int64_t)h.max_parent > nglobal) {
    // parents beyond the used vertices: how many
    check_cuda(cudaMemsetAsync(&out->below, 0, 8, s), "memset");
    range_kernel<<<grid(n), B, 0, s>>>(pred, n, nglobal, &out->below);
    unsigned long long e = 0;
    check_cuda(cudaMemcpyAsync(&e, &out->below, 8, cudaMemcpyDeviceToHost, s), "copy");
    check_cuda(cudaStreamSynchronize(s), "validate ranges");
    err = (int64_t)e;
  }
  // a root beyond the used vertex range counts as one more range error
  if (root >= nglobal) ++err;
  if (err == 0 && ((int64_t)((uint64_t)h.root_entry << 16) >> 16) != root) err = 1;
  if (err == 0) err = (int64_t)h.self;
  if (err == 0) err = (int64_t)h.depth;
  if (err == 0) {
    if (h.deep) {
      // unknown depths further than 64 steps from a known one (or on a cycle):
      // parent's depth + 1, pass by pass, then the edge pass again
      int* changed = arena_alloc<int>(arena, 1, "flag");
      for (int pass = 0; pass < 0x10000; ++pass) {
        check_cuda(cudaMemsetAsync(changed, 0, 4, s), "memset");
        depth_build_kernel<<<grid(n), B, 0, s>>>(map, n, root, changed);
        int hc = 0;
        check_cuda(cudaMemcpyAsync(&hc, changed, 4, cudaMemcpyDeviceToHost, s), "copy");
        check_cuda(cudaStreamSynchronize(s), "depth map");
        if (!hc) break;
      }
      arena.free(changed);
      check_cuda(cudaMemsetAsync(&out->edge, 0, 16, s), "memset");
      edge_pass();
      read("validate edges");
    }
    err = (int64_t)h.edge;
    *edge_visit_count = (int64_t)h.visited;
  }
  *errors = err;
  arena.free(out);
  arena.free(valid);
  arena.free(beside);
  arena.free(copy);
}

}  // namespace b200bfs
