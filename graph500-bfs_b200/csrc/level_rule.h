// End of a level in the one-kernel search (persistent.cu): the host loop's
// bookkeeping and direction switch, evaluated by every block for itself.
#pragma once

#include "bfs_internal.h"
#include "common.cuh"

namespace b200bfs {

// A block's copy of what the level loop of bfs.cu keeps in local variables.
struct LevelState {
  long long level, visited, prev_nq, nq, in_edges;
  long long q_rows;               // rows of the level's frontier list
  int forward, next_forward, growing, cur, qcur, done;
  long long at[9];                // auto_tuning_data, and the slots written
  unsigned at_set;
};

// All blocks have to come to the same state, so nothing that is used here may
// change between the barrier that ends the level and the next one.  q does
// after a bottom-up level: a block that is through with the rule appends the
// next frontier to it (frontier_from_bits) while a later one may still be
// here, so after a bottom-up level it says nothing about the level's vertices.
__host__ __device__ __forceinline__ void level_end(LevelState& s, const PersistArgs& a,
                                                   const PersistCounters& c) {
  const bool forward = s.forward != 0;
  const long long ne = (long long)c.nq_edges;
  const long long nq = (long long)(c.nq + (forward ? c.q >> 32 : 0));
  s.nq = nq;
  s.visited += nq;
  if (!forward) s.cur ^= 1;
  bool next_forward = s.next_forward != 0;
  if (nq == 0) {
    s.done = 1;
  } else if (s.growing && nq > s.prev_nq) {
    if (forward) {
      if (ne > a.t2b) {
        next_forward = false;
        s.at[0] = ne;          // AUTO_GLOBAL_NQ_EDGES
        s.at[1] = a.nedges;    // AUTO_NUM_GLOBAL_EDGES
        s.at[2] = s.level;     // AUTO_T2B_LEVEL
        s.at_set |= 7u;
      } else {
        s.at[6] = ne;  // AUTO_PRE_GLOBAL_NQ_EDGES
        s.at_set |= 1u << 6;
      }
    }
  } else if (!forward) {
    if (nq < a.b2t) {
      next_forward = true;
      s.growing = 0;
      s.at[3] = nq;       // AUTO_GLOBAL_NQ_SIZE
      s.at[4] = a.R;      // AUTO_NUM_GLOBAL_VERTS
      s.at[5] = s.level;  // AUTO_B2T_LEVEL
      s.at_set |= 7u << 3;
    } else {
      s.at[7] = nq;  // AUTO_PRE_GLOBAL_NQ_SIZE
      s.at_set |= 1u << 7;
    }
  }
  if (s.done == 0 && s.level >= kMaxLevel) s.done = 3;
  if (a.force_direction == 1) next_forward = true;
  if (a.force_direction == 2) next_forward = false;
  s.next_forward = next_forward;
  if (forward) {  // else the list is made, and its size read, before the next barrier
    s.q_rows = (long long)(c.q >> 32);
    s.in_edges = (long long)(c.q & 0xFFFFFFFFull);
  }
  s.qcur ^= 1;
}

// What the last block to finish publishes.  A block that gave up waiting left
// without its share of the level or of the assembly, even if the blocks it
// waited for arrived right after and went on to the end.
__host__ __device__ __forceinline__ int published_status(unsigned done, unsigned error) {
  return error ? 4 : (int)done;
}

}  // namespace b200bfs
