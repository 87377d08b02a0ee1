// Device code shared by the level kernels (bfs.cu) and the one-kernel search
// (persistent.cu): the pred assembly pass and the bottom-up row search.
#pragma once

#include "common.cuh"

namespace b200bfs {

// kLive: the word or entry may have been written earlier in the running
// kernel, so it is read with an ordinary load instead of a read-only one.
template <bool kLive, typename T>
__device__ __forceinline__ T load_state(const T* p) {
  return kLive ? *p : __ldg(p);
}

template <bool kLive>
__device__ __forceinline__ bool bit_test_state(const uint32_t* bm, int64_t v) {
  return (load_state<kLive>(bm + (v >> 5)) >> (v & 31)) & 1u;
}

// Assembly of pred from the row-order buffer rp (engine option
// pred_assemble).  pmap[u] for original id u: its row (>= 0), -1 (no parent:
// no edge, or beyond the graph), or -(p + 2) for a CoreBFS pruned vertex with
// tree parent p.  A reached row gives its rp entry, an unreached row -1, a
// pruned vertex its tree entry (level 0xFFFF, as write_tree_kernel writes),
// the root itself.  The pass runs over u in order, so pred is written in full
// lines; with group reordering the rows of a group of 2^16 ids are
// contiguous, so the rp reads of the ids a wave of warps covers fall in a few
// windows that stay in L2.  Scattering the entries by original id during the
// levels instead costs a random 32-byte sector per entry.
// A row's visited word and rp entry are loaded together (both only for
// rows), so the entry costs one round trip after the map; nearly every row
// is reached in a search of the giant component, so the rp reads of the
// unreached rows are few.
template <bool kLive>
__device__ __forceinline__ int64_t assembled_entry(int32_t m, int64_t u, const uint32_t* vis,
                                                   const int64_t* rp, int64_t root) {
  int64_t e = -1;
  if (m >= 0) {
    const uint32_t vw = load_state<kLive>(vis + (m >> 5));
    const int64_t r = load_state<kLive>(rp + m);
    if ((vw >> (m & 31)) & 1u) e = r;
  } else if (m < -1) {
    e = pred_entry(-(int64_t)m - 2, 0xFFFF);
  }
  return u == root ? root : e;
}

// Four ids per thread: one 16-byte map load, two 16-byte pred stores
// (pred and pmap are 256-byte aligned; n4 = n / 4, the tail done by thread 0).
// sparse: pred already holds the entries of every vertex outside the
// searched rows (-1, or its tree parent at level 0xFFFF), except at
// prev_root (and the previous CoreBFS climb, which the caller restores), so
// a group of four such vertices is not written: a third of the ids are rows
// at SCALE 28, and one group in five has none.
template <bool kLive>
__device__ __forceinline__ void assemble_body(const int32_t* __restrict__ pmap, int64_t n,
                                              const uint32_t* vis, const int64_t* rp,
                                              int64_t root, int64_t prev_root, int sparse,
                                              int64_t* __restrict__ pred) {
  const int64_t n4 = n >> 2;
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int4* m4 = reinterpret_cast<const int4*>(pmap);
  longlong2* p2 = reinterpret_cast<longlong2*>(pred);
  for (int64_t i = t0; i < n4; i += stride) {
    const int4 m = __ldg(m4 + i);
    const int64_t u = 4 * i;
    if (sparse && (m.x & m.y & m.z & m.w) < 0 && (uint64_t)(root - u) >= 4 &&
        (uint64_t)(prev_root - u) >= 4)
      continue;
    p2[2 * i] = make_longlong2(assembled_entry<kLive>(m.x, u, vis, rp, root),
                               assembled_entry<kLive>(m.y, u + 1, vis, rp, root));
    p2[2 * i + 1] = make_longlong2(assembled_entry<kLive>(m.z, u + 2, vis, rp, root),
                                   assembled_entry<kLive>(m.w, u + 3, vis, rp, root));
  }
  if (t0 == 0)
    for (int64_t u = 4 * n4; u < n; ++u) pred[u] = assembled_entry<kLive>(pmap[u], u, vis, rp, root);
}

// Bottom-up step, second form: a warp step covers kWords bitmap words, so
// every lane owns kWords vertices and issues their row-offset loads, then
// their neighbour-id loads (two neighbours per round), then the visited
// probes, back to back: kWords * 2 independent loads are in flight per lane
// instead of one dependent chain.  Rows unresolved after 8 probes are swept
// by the whole warp as in bu_kernel.
// kFirst: each open row first probes its first neighbour, read from the
// dense fpair[] array together with that neighbour's original id (one
// coalesced 8-byte read per row), and loads its row offsets only when that
// probe misses; the offset rounds then start at the second neighbour.  A
// parent found by the first probe has its pred entry's id at hand: no
// second load, no gather into inv[].
// kSpec (with kFirst): the fpair[] loads are issued for every row of the
// words, beside the loads of the words themselves, and the visited rows'
// entries are dropped afterwards: one round trip fewer per step, for the
// levels where most rows are still unvisited.
// The row search of the bottom-up forms for kWords bitmap words w[k] (w[k]
// < 0: no word) whose current visited words are c[k]: lane l handles row
// w[k] * 32 + l of each word, and the word's next value c[k] | found is
// written to nxt.
template <int kWords, bool kFirst, bool kSpec = false, bool kLive = false>
__device__ __forceinline__ void bu_rows(
    const int64_t (&w)[kWords], const uint32_t (&c)[kWords], const uint32_t* cur,
    uint32_t* nxt, const int64_t* __restrict__ row_ptr,
    const int32_t* __restrict__ col, const int2* __restrict__ fpair,
    const int32_t* __restrict__ inv, const int32_t* __restrict__ pidx,
    int64_t* __restrict__ pred, int64_t level, uint32_t& found_total, uint32_t& scanned) {
  const int lane = lane_id();
  // open row w[k] * 32 + lane: its next neighbour is col[b[k]] and
  // rem[k] of them are left (a row has fewer than 2^31 neighbours)
  int64_t b[kWords];
  int32_t rem[kWords];
  // par[k]: the parent's row id, or with pf[k] (found by the first probe)
  // already its original id
  int32_t par[kWords];
  bool pf[kWords];
  if (kFirst) {
    int2 f[kWords];
#pragma unroll
    for (int k = 0; k < kWords; ++k) {
      par[k] = -1;
      pf[k] = false;
      b[k] = 0;
      rem[k] = 0;
      f[k] = make_int2(-1, -1);
      if (kSpec ? w[k] >= 0 : (((~c[k]) >> lane) & 1u) != 0)
        f[k] = __ldg(fpair + w[k] * 32 + lane);
    }
    if (kSpec) {
#pragma unroll
      for (int k = 0; k < kWords; ++k)
        if (((c[k] >> lane) & 1u) != 0) f[k].x = -1;
    }
    uint32_t mf[kWords];
#pragma unroll
    for (int k = 0; k < kWords; ++k) mf[k] = f[k].x >= 0 ? load_state<kLive>(cur + (f[k].x >> 5)) : 0u;
#pragma unroll
    for (int k = 0; k < kWords; ++k) {
      if (f[k].x < 0) continue;
      scanned += 1;
      if ((mf[k] >> (f[k].x & 31)) & 1u) {
        par[k] = f[k].y;
        pf[k] = true;
      } else {
        const int64_t v = w[k] * 32 + lane;
        const int64_t rb = row_ptr[v];
        b[k] = rb + 1;
        rem[k] = (int32_t)(row_ptr[v + 1] - rb - 1);
      }
    }
  } else {
#pragma unroll
    for (int k = 0; k < kWords; ++k) {
      par[k] = -1;
      pf[k] = false;
      b[k] = 0;
      rem[k] = 0;
      if (((~c[k]) >> lane) & 1u) {
        const int64_t v = w[k] * 32 + lane;
        b[k] = row_ptr[v];
        rem[k] = (int32_t)(row_ptr[v + 1] - b[k]);
      }
    }
  }
  // four rounds of two probes per vertex
#pragma unroll
  for (int round = 0; round < 4; ++round) {
    int32_t u0[kWords], u1[kWords];
    bool need = false;
#pragma unroll
    for (int k = 0; k < kWords; ++k) {
      u0[k] = u1[k] = -1;
      if (par[k] < 0 && rem[k] > 0) {
        u0[k] = __ldg(col + b[k]);
        if (rem[k] > 1) u1[k] = __ldg(col + b[k] + 1);
        need = true;
      }
    }
    if (!__any_sync(kFull, need)) break;
    uint32_t m0[kWords], m1[kWords];
#pragma unroll
    for (int k = 0; k < kWords; ++k) {
      m0[k] = u0[k] >= 0 ? load_state<kLive>(cur + (u0[k] >> 5)) : 0u;
      m1[k] = u1[k] >= 0 ? load_state<kLive>(cur + (u1[k] >> 5)) : 0u;
    }
#pragma unroll
    for (int k = 0; k < kWords; ++k) {
      if (u0[k] < 0) continue;
      if ((m0[k] >> (u0[k] & 31)) & 1u) {
        par[k] = u0[k];
        scanned += 1;
      } else if (u1[k] >= 0 && ((m1[k] >> (u1[k] & 31)) & 1u)) {
        par[k] = u1[k];
        scanned += 2;
      } else {
        const int32_t t = (u1[k] >= 0) ? 2 : 1;
        scanned += t;
        b[k] += t;
        rem[k] -= t;
      }
    }
  }
  // cooperative sweep of the rows still unresolved
#pragma unroll
  for (int k = 0; k < kWords; ++k) {
    unsigned left = __ballot_sync(kFull, par[k] < 0 && rem[k] > 0);
    while (left) {
      const int l = __ffs(left) - 1;
      left &= left - 1;
      const int64_t jb = __shfl_sync(kFull, b[k], l);
      const int64_t je = jb + __shfl_sync(kFull, rem[k], l);
      int32_t p = -1;
      for (int64_t j = jb; j < je; j += 32) {
        const int64_t jj = j + lane;
        int32_t u = 0;
        bool hit = false;
        if (jj < je) {
          u = __ldg(col + jj);
          hit = bit_test_state<kLive>(cur, u);
        }
        const unsigned hm = __ballot_sync(kFull, hit);
        if (hm) {
          const int fl = __ffs(hm) - 1;
          p = __shfl_sync(kFull, u, fl);
          if (lane == l) scanned += (uint32_t)(j - jb + fl + 1);
          break;
        }
      }
      if (p < 0 && lane == l) scanned += (uint32_t)(je - jb);
      if (lane == l) par[k] = p;
    }
  }
#pragma unroll
  for (int k = 0; k < kWords; ++k) {
    const unsigned fm = __ballot_sync(kFull, par[k] >= 0);
    if (lane == 0 && w[k] >= 0) {
      nxt[w[k]] = c[k] | fm;
      found_total += __popc(fm);
    }
    if (par[k] >= 0) {
      const int64_t v = w[k] * 32 + lane;
      const int32_t po = pf[k] ? par[k] : __ldg(inv + par[k]);
      pred[pred_slot(pidx, v)] = pred_entry(po, level);
    }
  }
}

// A warp's share of a bottom-up level.  found_total (lane 0) and scanned (per
// lane; a lane scans far fewer than 2^32 entries) are added to.
template <int kWords, bool kFirst, bool kSparse, bool kSpec = false, bool kLive = false>
__device__ __forceinline__ void bu_wide_words(
    const uint32_t* cur, uint32_t* nxt, int64_t W,
    const int64_t* __restrict__ row_ptr, const int32_t* __restrict__ col,
    const int2* __restrict__ fpair, const int32_t* __restrict__ inv,
    const int32_t* __restrict__ pidx, int64_t* __restrict__ pred, int64_t level,
    uint32_t& found_total, uint32_t& scanned) {
  const int lane = lane_id();
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  if (kSparse) {
    // Few unvisited rows left (the last levels): a warp takes blocks of 32
    // bitmap words, one per lane; full words are copied to nxt at once and
    // only the words with unvisited rows go through the row search, kWords
    // at a time.  A block costs one load per lane instead of 32 / kWords
    // dependent word steps.
    const int64_t nblk = (W + 31) >> 5;
    for (int64_t blk = gw; blk < nblk; blk += nwarps) {
      const int64_t wl = (blk << 5) + lane;
      const uint32_t cl = wl < W ? cur[wl] : kFull;
      if (cl == kFull && wl < W) nxt[wl] = kFull;
      unsigned om = __ballot_sync(kFull, cl != kFull);
      while (om) {
        int64_t w[kWords];
        uint32_t c[kWords];
#pragma unroll
        for (int k = 0; k < kWords; ++k) {
          w[k] = -1;
          c[k] = kFull;
          if (om) {
            const int l = __ffs(om) - 1;
            om &= om - 1;
            w[k] = (blk << 5) + l;
            c[k] = __shfl_sync(kFull, cl, l);
          }
        }
        bu_rows<kWords, kFirst, false, kLive>(w, c, cur, nxt, row_ptr, col, fpair, inv, pidx, pred,
                                level, found_total, scanned);
      }
    }
  } else {
    // kWords consecutive words per warp step, strided over the warps
    for (int64_t w0 = gw * kWords; w0 < W; w0 += nwarps * kWords) {
      int64_t w[kWords];
      uint32_t c[kWords];
      bool all_full = true;
#pragma unroll
      for (int k = 0; k < kWords; ++k) {
        w[k] = w0 + k < W ? w0 + k : -1;
        c[k] = w[k] >= 0 ? cur[w0 + k] : kFull;
        all_full &= (c[k] == kFull);
      }
      // (kSpec issues the row loads before the words arrive: no early exit)
      if (!kSpec && all_full) {
        if (lane < kWords && w0 + lane < W) nxt[w0 + lane] = kFull;
        continue;
      }
      bu_rows<kWords, kFirst, kSpec, kLive>(w, c, cur, nxt, row_ptr, col, fpair, inv, pidx, pred, level,
                              found_total, scanned);
    }
  }
}

}  // namespace b200bfs
