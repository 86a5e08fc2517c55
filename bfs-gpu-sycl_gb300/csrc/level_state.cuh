// level_state.cuh -- the start of a BFS on a filled workspace, shared by the
// init kernel and the narrow-level kernel.
#pragma once
#include <cuda_runtime.h>

#include "bfs_internal.h"

namespace bfsgb {

// One thread: seeds the root and the first frontier of a filled state.
__device__ __forceinline__ void init_state(BfsDevState *st, unsigned long long cond, int use_cond) {
  const uint32_t r = st->root;                     // original id
  const uint32_t ri = st->pinv ? st->pinv[r] : r;  // internal id
  st->root_id = ri;
  st->vis[ri >> 5] |= 1u << (ri & 31u);
  st->prev[ri >> 5] |= 1u << (ri & 31u);
  st->lv8[ri] = 0;
  if (st->parent) st->parent[r] = (int32_t)r;
  const bool expanded = ri < st->n_rows;  // run_bfs_cpu.hpp:31
  uint32_t b = 0, e = 0;
  if (expanded) {
    b = st->indptr[ri];
    e = st->indptr[ri + 1];
  }
  if (expanded && e > b) {
    const uint32_t nch = edge_chunks(b, e - b, st->inds_off);
    st->qb[0][0] = b;
    st->qd[0][0] = e - b;
    st->qc[0][0] = 0;
    st->qc[0][1] = nch;
    st->qv[0][0] = r;
    st->F = 1;
    st->EF = e - b;
    st->EC = nch;
  } else {
    st->qc[0][0] = 0;
    st->F = 0;
    st->EF = 0;
    st->EC = 0;
  }
  st->edges_count = expanded ? (unsigned long long)(e - b) : 0ull;
  st->cur = 0;
  st->lvl = 0;
  st->reached = 1;
  st->reached_prev = 1;
  st->max_level = 0;
  st->next_packed = 0;
  st->next_edges = 0;
  st->next_walk = 0;
  st->skip_full = 0;
  st->explore_done = 0;
  st->done_blocks = 0;
  st->lg_cursor = 0;
  st->error = 0;
  st->launches = 2;  // fill and the level output after the loop
  st->arm = st->fixed_arm >= 0 ? st->fixed_arm : 0;
  if (st->rec_cap > 0) {
    st->rec_frontier[0] = st->F;
    st->rec_edges[0] = st->EF;
    st->rec_arm[0] = -1;
  }
  if (use_cond) cudaGraphSetConditional((cudaGraphConditionalHandle)cond, st->F > 0);
}

}  // namespace bfsgb
