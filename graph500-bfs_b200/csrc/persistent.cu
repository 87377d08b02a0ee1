// Single-source search as one kernel.
//
// On graphs whose levels take microseconds the level loop of bfs.cu is bound
// by its launches: a search of a SCALE 20 graph is 23 kernels and eight host
// round trips, 273 us of which the GPU works 160.  Here the whole search is
// one kernel: its blocks, all resident, go through the levels together with
// a barrier after each (a cooperative grid, or one cluster on small graphs).
// Every block evaluates the direction rule (bfs.hpp:3413-3457) from the level's
// counters by itself, and the pred assembly follows in the same launch.  The
// host launches once and waits once.
//
// Top-down levels claim a vertex with an OR that returns the old word, so
// that exactly one entry wins it; the winner counts it and appends it to the
// next frontier, with its degree prefix from the same atomic that gives the
// slot, so that a level needs no pass over the bitmaps and no scan.  Bottom-up
// levels are those of the level kernels (search_device.cuh).
//
// us per search (16 roots, default alpha and beta), level loop -> one kernel:
// SCALE 12 152 -> 60, 16 207 -> 70, 20 273 -> 94, 22 333 -> 151, 24 494 -> 315,
// 26 973 -> 856; with CoreBFS and group reordering SCALE 24 355 -> 261, 26
// 731 -> 656.  What bounds it: on the small graphs a chain of about ten
// dependent loads, three atomics and the barrier (2 us) per level; from
// SCALE 24 the bottom-up sweep and the assembly, as in the level loop.
#include <algorithm>
#include <atomic>
#include <cstring>
#include "common.cuh"
#include "bfs_internal.h"
#include "search_device.cuh"
#include "frontier.cuh"
#include "level_rule.h"

namespace b200bfs {
namespace {

// The barrier between the kernel's blocks: those of one cluster (kCluster,
// the grid is one cluster; the hardware schedules it as one) or of a
// cooperative grid.
template <bool kCluster>
__device__ __forceinline__ bool blocks_barrier(PersistCtl* ctl, unsigned* target, int* fail) {
  if (kCluster) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    return true;
  }
  return grid_barrier(&ctl->bar, &ctl->error, target, fail);
}

struct Shared : LevelState {
  int fail, stop, nrec;
  unsigned long long b_nq, b_ne, b_sc;  // the block's share of the level's counters
  PersistRec rec[kPersistRecs];   // kept by block 0
};

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Frontier output of a top-down level.
struct Emit {
  int32_t* rows;
  uint32_t* pre;
  PersistCounters* c;
  // per lane, of the vertices that were not appended: their number and their
  // pre-dedup degree sum
  uint32_t nq;
  unsigned long long ne;
};

// Claims kPer neighbours per lane (u < 0: none) for the parents par: the
// vertices won are counted and appended to the next frontier.  Once the
// level's totals decide that the next level is bottom-up, the frontier is not
// needed and the appending stops (s.stop): stop_nq and stop_ne are those
// thresholds, stop_ne < 0 if the rule does not apply.
template <int kPer>
__device__ __forceinline__ void claim(const PersistArgs& a, Emit& e, Shared& s, uint32_t* vis,
                                      const int32_t (&u)[kPer], const int32_t (&par)[kPer],
                                      int64_t level, long long stop_nq, long long stop_ne) {
  uint32_t word[kPer];
#pragma unroll
  for (int q = 0; q < kPer; ++q) word[q] = u[q] >= 0 ? vis[u[q] >> 5] : kFull;
  // a stale word only costs an OR that wins nothing
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const uint32_t bit = 1u << (u[q] & 31);
    if (u[q] >= 0 && !(word[q] & bit)) word[q] = atomicOr(vis + (u[q] >> 5), bit);
    else word[q] = kFull;
  }
  const int stopped = __shfl_sync(kFull, lane_id() == 0 ? *(volatile int*)&s.stop : 0, 0);
  uint32_t n = 0, d = 0, len[kPer];
  unsigned long long m = 0;
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    len[q] = 0;
    if ((word[q] >> (u[q] & 31)) & 1u) continue;
    a.rp[u[q]] = pred_entry(par[q], level);
    m += (unsigned)__ldg(a.mdeg + u[q]);
    ++n;
    if (!stopped) {
      len[q] = (uint32_t)(__ldg(a.row_ptr + u[q] + 1) - __ldg(a.row_ptr + u[q]));
      d += len[q];
    }
  }
  if (stopped) {
    e.nq += n;
    e.ne += m;
    return;
  }
  if (!__any_sync(kFull, n != 0)) return;
#pragma unroll
  for (int o = 16; o; o >>= 1) m += __shfl_xor_sync(kFull, m, o);
  unsigned long long ne = 0, after;
  if (lane_id() == 31) ne = atomicAdd(&e.c->nq_edges, m) + m;
  int64_t slot;
  uint32_t offset;
  reserve<32>(&e.c->q, n, d, &slot, &offset, &after);
  if (lane_id() == 31 && stop_ne >= 0 && (long long)ne > stop_ne &&
      (long long)(after >> 32) > stop_nq)
    *(volatile int*)&s.stop = 1;
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    if (len[q] == 0) continue;  // every row has an entry
    e.rows[slot] = u[q];
    e.pre[slot] = offset;
    ++slot;
    offset += len[q];
  }
}

// The frontier of a top-down level that follows a bottom-up one: the rows
// new in `now` against `before`.
__device__ __forceinline__ void frontier_from_bits(const PersistArgs& a, const uint32_t* now,
                                                   const uint32_t* before, int64_t gw,
                                                   int64_t nwarps, int32_t* rows, uint32_t* pre,
                                                   PersistCounters* c) {
  const int lane = lane_id();
  for (int64_t w0 = gw * 32; w0 < a.W; w0 += nwarps * 32) {
    const int64_t w = w0 + lane;
    const uint32_t f = w < a.W ? now[w] & ~before[w] : 0u;
    if (!__any_sync(kFull, f != 0)) continue;
    uint32_t d = 0;
    for (uint32_t g = f; g; g &= g - 1) {
      const int64_t v = w * 32 + __ffs(g) - 1;
      d += (uint32_t)(__ldg(a.row_ptr + v + 1) - __ldg(a.row_ptr + v));
    }
    int64_t slot;
    uint32_t offset;
    unsigned long long after;
    reserve<32>(&c->q, __popc(f), d, &slot, &offset, &after);
    for (uint32_t g = f; g; g &= g - 1) {
      const int64_t v = w * 32 + __ffs(g) - 1;
      rows[slot] = (int32_t)v;
      pre[slot] = offset;
      ++slot;
      offset += (uint32_t)(__ldg(a.row_ptr + v + 1) - __ldg(a.row_ptr + v));
    }
  }
}

// Adds the block's share to the level's counters (thread 0, before it
// arrives at the barrier).
__device__ __forceinline__ void add_counters(PersistCounters* c, Shared& s) {
  if (s.b_nq) atomicAdd(&c->nq, s.b_nq);
  if (s.b_ne) atomicAdd(&c->nq_edges, s.b_ne);
  if (s.b_sc) atomicAdd(&c->scanned, s.b_sc);
  s.b_nq = s.b_ne = s.b_sc = 0;
}

__device__ __forceinline__ unsigned long long warp_add(unsigned long long x) {
#pragma unroll
  for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
  return x;
}

template <int kWords, int kPer, int kThreads, int kMinBlocks, bool kCluster>
__global__ void __launch_bounds__(kThreads, kMinBlocks)
    persistent_search_kernel(const __grid_constant__ PersistArgs a) {
  static_assert(kPersistEntries + 32 * kPer < int64_t(1) << 32, "steps of expand_frontier");
  __shared__ Shared s;
  const int lane = lane_id();
  const int64_t t0 = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * kThreads;
  const int64_t gw = t0 >> 5, nwarps = nthreads >> 5;
  const bool lead = t0 == 0;
  PersistCtl* ctl = a.ctl;
  unsigned target = 0;
  unsigned long long stamp = 0;
  if (lead) stamp = globaltimer_ns();

  // initialize_memory and first_expand (bfs.hpp:315-349, 562-631)
  const int32_t r = __ldg(a.rank + a.root);
  const int64_t rdeg = r >= 0 ? __ldg(a.row_ptr + r + 1) - __ldg(a.row_ptr + r) : 0;
  for (int64_t w = t0; w < a.W; w += nthreads) {
    // bits at or beyond R are padding and start "visited"
    const int64_t first = w * 32;
    uint32_t v = first + 32 > a.R ? kFull << (a.R - first) : 0u;
    if (r >= 0 && w == (r >> 5)) v |= 1u << (r & 31);
    a.vis[0][w] = v;
  }
  if (lead) {
    if (r >= 0) a.rp[r] = a.root;
    a.rows[0][0] = r;
    a.pre[0][0] = 0;
  }
  if (threadIdx.x == 0) {
    s.level = a.root_level;
    s.visited = 1;
    s.nq = 0;
    s.in_edges = rdeg;
    s.q_rows = r >= 0 ? 1 : 0;
    s.next_forward = s.growing = 1;
    s.cur = s.qcur = 0;
    s.done = s.fail = s.stop = 0;
    s.b_nq = s.b_ne = s.b_sc = 0;
    s.at_set = 0;
  }
  int nrec = 0;
  bool alive = blocks_barrier<kCluster>(ctl, &target, &s.fail);

  while (alive) {
    if (threadIdx.x == 0) {
      ++s.level;
      s.prev_nq = s.nq;
      s.forward = s.next_forward;
      s.stop = a.force_direction == 2;
    }
    __syncthreads();
    const long long level = s.level;
    const int forward = s.forward, cur = s.cur, qcur = s.qcur;
    PersistCounters* c = &ctl->c[level % 3];
    if (lead) memset(&ctl->c[(level + 1) % 3], 0, sizeof(PersistCounters));
    const long long unvisited = a.R - s.visited;
    if (forward) {
      Emit e;
      e.rows = a.rows[qcur ^ 1];
      e.pre = a.pre[qcur ^ 1];
      e.c = c;
      e.nq = 0;
      e.ne = 0;
      const bool rule = s.growing && a.force_direction == 0;
      const long long stop_nq = s.prev_nq;
      const long long stop_ne = rule ? a.t2b : -1;
      expand_frontier<kPer>(
          a.row_ptr, a.col, a.rows[qcur], a.pre[qcur], s.q_rows, (uint32_t)s.in_edges, gw, nwarps,
          [&](int32_t row) { return __ldg(a.inv + row); },
          [&](const int32_t(&u)[kPer], const int32_t(&p)[kPer]) {
            claim<kPer>(a, e, s, a.vis[cur], u, p, level, stop_nq, stop_ne);
          });
      if (__any_sync(kFull, e.nq != 0)) {
        const unsigned long long n = warp_add(e.nq), d = warp_add(e.ne);
        if (lane == 0) {
          atomicAdd(&s.b_nq, n);
          atomicAdd(&s.b_ne, d);
        }
      }
    } else {
      uint32_t found = 0, scanned = 0;
      uint32_t* now = a.vis[cur];
      uint32_t* nxt = a.vis[cur ^ 1];
      // the same rules as in the level loop (run_bfs_core)
      if (4 * unvisited < a.W)
        bu_wide_words<kWords, true, true, false, true>(now, nxt, a.W, a.row_ptr, a.col, a.fpair,
                                                       a.inv, nullptr, a.rp, level, found,
                                                       scanned);
      else if (2 * unvisited > a.R)
        bu_wide_words<kWords, true, false, true, true>(now, nxt, a.W, a.row_ptr, a.col, a.fpair,
                                                       a.inv, nullptr, a.rp, level, found,
                                                       scanned);
      else
        bu_wide_words<kWords, true, false, false, true>(now, nxt, a.W, a.row_ptr, a.col, a.fpair,
                                                        a.inv, nullptr, a.rp, level, found,
                                                        scanned);
      if (__any_sync(kFull, (found | scanned) != 0)) {
        const unsigned long long n = warp_add(found), x = warp_add(scanned);
        if (lane == 0) {
          if (n) atomicAdd(&s.b_nq, n);
          atomicAdd(&s.b_sc, x);
        }
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) add_counters(c, s);
    alive = blocks_barrier<kCluster>(ctl, &target, &s.fail);
    if (!alive) break;
    if (threadIdx.x == 0) {
      PersistCounters end;
      end.q = __ldcg(&c->q);
      end.nq = __ldcg(&c->nq);
      end.nq_edges = __ldcg(&c->nq_edges);
      end.scanned = __ldcg(&c->scanned);
      const long long in_edges = s.in_edges;
      level_end(s, a, end);
      if (lead) {
        const unsigned long long now = globaltimer_ns();
        PersistRec rec;
        rec.bottom_up = forward ? 0 : 1;
        rec.discovered = (uint32_t)s.nq;
        rec.scanned = (uint32_t)(forward ? in_edges : (long long)end.scanned);
        rec.ns = (uint32_t)min(now - stamp, 0xFFFFFFFFull);
        stamp = now;
        (nrec < kPersistRecs ? s.rec[nrec] : a.more[nrec - kPersistRecs]) = rec;
        ++nrec;
      }
    }
    __syncthreads();
    if (s.done) break;
    if (!forward && s.next_forward) {
      frontier_from_bits(a, a.vis[s.cur], a.vis[s.cur ^ 1], gw, nwarps, a.rows[s.qcur],
                         a.pre[s.qcur], c);
      alive = blocks_barrier<kCluster>(ctl, &target, &s.fail);
      if (threadIdx.x == 0) {
        const unsigned long long q = __ldcg(&c->q);
        s.q_rows = (long long)(q >> 32);
        s.in_edges = (long long)(q & 0xFFFFFFFFull);
      }
      __syncthreads();
    }
  }
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0) {
      ctl->stamp = globaltimer_ns();
      a.out->level = s.level;
      a.out->visited = s.visited;
      a.out->nrec = nrec;
      ctl->done = alive ? s.done : 4;
      a.out->at_set = s.at_set | 1u << 8;
      s.at[8] = s.level;  // AUTO_LEVEL
      for (int i = 0; i < 9; ++i) a.out->at[i] = s.at[i];
      s.nrec = nrec;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < min(s.nrec, kPersistRecs); i += kThreads) a.out->rec[i] = s.rec[i];
    __threadfence_system();
  }
  if (alive && s.done == 1)
    assemble_body<true>(a.pmap, a.pred_size, a.vis[s.cur], a.rp, a.root, a.prev_root, a.sparse,
                        a.pred);
  // the last block publishes the result and leaves the counters zero for the
  // next search
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&ctl->blocks_done, 1u) == gridDim.x - 1) {
      __threadfence_system();
      a.out->done = published_status(*(volatile unsigned*)&ctl->done,
                                     *(volatile unsigned*)&ctl->error);
      a.out->pred_ns = (long long)(globaltimer_ns() - *(volatile unsigned long long*)&ctl->stamp);
      memset((void*)ctl, 0, sizeof(*ctl));
      __threadfence_system();
      *(volatile unsigned long long*)&a.out->seq = a.seq;
    }
  }
}

}  // namespace

bool run_bfs_core_persistent(const Graph& g, BfsState& st, cudaStream_t s, int sms, int64_t root,
                             int64_t root_level, int edgefactor, double alpha, double beta,
                             int64_t* at, const RunOptions& opt, b200bfs_run_stats* stats) {
  if (!st.pmap) throw Error{B200BFS_ERR_STATE, "pred assembly map not built"};
  const Csr& c = g.csr;
  const bool sparse = st.assembled && st.pred_clean;
  PersistArgs a;
  memset(&a, 0, sizeof(a));
  a.row_ptr = c.row_ptr;
  a.col = c.col;
  a.inv = c.inv;
  a.mdeg = c.mdeg;
  a.rank = c.rank;
  a.fpair = c.first_pair;
  a.R = st.R;
  a.W = st.W;
  a.nedges = c.nedges;
  a.vis[0] = st.vis[0];
  a.vis[1] = st.vis[1];
  // two frontier lists: rows and the degree prefix in 32 bits
  a.rows[0] = st.queue;
  a.rows[1] = st.queue2;
  a.pre[0] = reinterpret_cast<uint32_t*>(st.qdeg);
  a.pre[1] = a.pre[0] + st.R + 2;
  a.rp = st.rp;
  a.pmap = st.pmap;
  a.pred = st.pred;
  a.pred_size = st.pred_size;
  a.ctl = st.pctl;
  a.out = st.dout;
  a.more = st.prec;
  a.root = root;
  a.prev_root = sparse ? st.prev_root : -1;
  a.sparse = sparse ? 1 : 0;
  a.root_level = root_level;
  a.t2b = t2b_limit(c.nedges, alpha);
  a.b2t = b2t_limit(st.R, edgefactor, beta);
  a.force_direction = opt.force_direction;
  a.seq = ++st.out_seq;
  // Up to 80 K rows: one cluster of 16 blocks, whose barrier is the hardware's;
  // beyond, 16 SMs no longer do.  us per search by rows, cooperative grid /
  // cluster: 3 K 62.3 / 60.1, 47 K 77.2 / 76.5, 57 K 82.0 / 78.2, 64 K 92.4 /
  // 86.0, 73 K (a 2-core) 77.2 / 79.5, 78 K 85.3 / 83.3, 90 K 88.0 / 85.4, 101 K
  // 83.5 / 80.9, 123 K 92.9 / 96.3, 149 K 84.6 / 97.8, 174 K 92.3 / 101.9.
  // Else a cooperative grid.  Threads per SM: 1024 with the registers the level
  // code asks for (no spills) while a level is a few rounds of loads per warp;
  // from 6 M rows 2048 threads at 32 registers, whose loads in flight are worth
  // more than their spills.  us per search, 16 roots, 1024 / 2048 threads:
  // SCALE 20 (R 0.6 M) 94 / 115, SCALE 22 (2.4 M) 151 / 168, SCALE 24 (8.9 M)
  // 321 / 315, its 2-core (6.7 M) 269 / 261, SCALE 26 (33 M) 983 / 856.
  constexpr int kThreads = 1024, kCluster = 16;
  const bool small = opt.persistent == 4 || (opt.persistent == 1 && st.R <= 80 * 1024);
  const bool wide =
      opt.persistent == 3 || (opt.persistent == 1 && st.R >= (int64_t(6) << 20));
  bool launched = false;
  if (small) {
    auto kernel = persistent_search_kernel<2, 4, kThreads, 1, true>;
    cudaLaunchAttribute dim;
    dim.id = cudaLaunchAttributeClusterDimension;
    dim.val.clusterDim.x = kCluster;
    dim.val.clusterDim.y = dim.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kCluster);
    cfg.blockDim = dim3(kThreads);
    cfg.stream = s;
    cfg.attrs = &dim;
    cfg.numAttrs = 1;
    if (st.clusters < 0) {
      // 16 blocks are beyond the portable cluster size: the device has to have
      // a group of SMs of that many
      int n = 0;
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
              cudaSuccess ||
          cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
      }
      st.clusters = n;
    }
    if (st.clusters > 0) {
      check_cuda(cudaLaunchKernelEx(&cfg, kernel, a), "search kernel");
      launched = true;
    }
  }
  if (!launched) {
    auto kernel = wide ? persistent_search_kernel<2, 2, kThreads, 2, false>
                       : persistent_search_kernel<2, 4, kThreads, 1, false>;
    void* params[] = {&a};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void*)kernel,
                                                      dim3(sms * blocks_per_sm(kernel, kThreads)),
                                                      dim3(kThreads), params, 0, s);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
      // a part of the device only (MPS): not every block can be resident
      cudaGetLastError();
      return false;
    }
    check_cuda(e, "search kernel");
  }
  volatile unsigned long long* flag = &st.hout->seq;
  for (unsigned long long n = 1; *flag != a.seq; ++n) {
    if ((n & 4095) == 0) {
      const cudaError_t e = cudaStreamQuery(s);
      if (e == cudaSuccess) {
        if (*flag != a.seq) throw Error{B200BFS_ERR_CUDA, "search result not published"};
        break;
      }
      if (e != cudaErrorNotReady) check_cuda(e, "search");
    }
  }
  std::atomic_thread_fence(std::memory_order_acquire);
  const PersistOut& o = *st.hout;
  if (o.done != 1) {
    // pred may hold a part of this search: the next one writes all of it
    st.assembled = false;
    st.pred_clean = false;
  }
  if (o.done == 3) throw Error{B200BFS_ERR_OVERFLOW, "more than 0xFFFE BFS levels"};
  if (o.done != 1) throw Error{B200BFS_ERR_TIMEOUT, "search kernel gave up waiting for its blocks"};
  st.asm_ev = -1;
  st.asm_sparse = sparse;
  st.pred_clean = true;
  st.prev_root = root;
  st.assembled = true;
  if (at)
    for (int i = 0; i < 9; ++i)
      if ((o.at_set >> i) & 1u) at[i] = o.at[i];
  // the records beyond the published ones (searches of more levels)
  std::vector<PersistRec> more;
  if (o.nrec > kPersistRecs) {
    more.resize((size_t)(o.nrec - kPersistRecs));
    check_cuda(cudaMemcpyAsync(more.data(), st.prec, more.size() * sizeof(PersistRec),
                               cudaMemcpyDeviceToHost, s),
               "level records");
    check_cuda(cudaStreamSynchronize(s), "level records");
  }
  b200bfs_run_stats rs;
  memset(&rs, 0, sizeof(rs));
  int64_t bytes = 4 * st.W;
  st.levels.clear();
  int64_t visited = 1, frontier = 1;
  for (int i = 0; i < o.nrec; ++i) {
    const PersistRec& x = i < kPersistRecs ? o.rec[i] : more[(size_t)(i - kPersistRecs)];
    const double ms = std::max<uint32_t>(x.ns, 1) * 1e-6;
    const int32_t level = (int32_t)(root_level + 1 + i);
    const int64_t found = x.discovered, scanned = x.scanned;
    const int64_t input = x.bottom_up ? st.R - visited : frontier;
    int64_t b = 16 * input + 8 * scanned + 12 * found;
    if (x.bottom_up) {
      b += 3 * (st.W * 4);
      ++rs.num_bu_levels;
      if (level < 64) rs.bu_level_mask |= 1ull << level;
      rs.edges_scanned_bu += scanned;
      rs.bu_bytes += b;
      rs.bu_ms += ms;
    } else {
      ++rs.num_td_levels;
      rs.edges_scanned_td += scanned;
      rs.td_bytes += b;
      rs.td_ms += ms;
    }
    bytes += b;
    visited += found;
    frontier = found;
    st.levels.push_back({level, (int32_t)x.bottom_up, input, found, scanned, b, ms});
  }
  rs.pred_bytes = assembly_bytes(st, o.visited, sparse);
  rs.pred_ms = std::max<long long>(o.pred_ns, 1) * 1e-6;
  rs.kernel_launches = 1;
  rs.levels = (int32_t)o.level;
  rs.visited = o.visited;
  rs.algorithmic_bytes = bytes + rs.pred_bytes;
  if (stats) *stats = rs;
  return true;
}

}  // namespace b200bfs
