// kernels.h -- host-visible entry points of kernels.cu.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "bfs_internal.h"

namespace bfsgb {

constexpr int kLevelgenBlock = 256;
// Block size of the explore kernel that runs any arm (learned schedule and
// every GLB launch); one block per SM.
constexpr int kAnyBlock = 1024;
// Explore kernels keep U warp rounds (U edges per lane) in flight; U is the
// "items per thread" tunable (4 or 8).  A GLB warp chunk is at least
// kGlbGroups groups of U rounds (more when the level is large: about eight
// chunks per warp of the grid).
constexpr int kGlbGroups = 4;
inline uint32_t glb_chunk_edges(int ipt) { return 32u * (uint32_t)ipt * kGlbGroups; }

// ---- narrow levels (narrow.cu) ----
constexpr uint32_t kNarrowBlock = 512;
// Degree from which an entry goes to the list.  A warp takes a queue entry's
// chunks 32 at a time, a chain of round trips each; R-MAT scale 12, whole BFS:
// 57 us with 32 to 96, 63 with 128, 76 with 512, 105 with 1024.
constexpr uint32_t kNarrowHeavy = 64;
constexpr uint32_t kNarrowHeavyBound = 512;  // the same where only a bound on degrees is known
// Largest level.  It costs the cluster by its new vertices, whose entries and
// levels it writes one by one, more than by its edges.  Whole BFS of a graph
// with one such level (GLB/256), cluster against two-kernel loop: level of 70 K
// edges 82 us against 95, 131 K 87 against 98 (103 against 107 with 79 K new
// vertices), 160 K 90 against 98 (110 against 112 with 96 K new), 200 K 90 to
// 102 against 97 (138 against 111 with 120 K new), 260 K 166 against 109 with
// 156 K new.  Above 2^17 a level of few new vertices would still gain a tenth,
// and nothing tells the two apart beforehand.
constexpr uint32_t kNarrowEdges = 1u << 17;
constexpr uint32_t kNarrowList = 8192;         // entries walked by the whole cluster
constexpr uint32_t kNarrowEntries = 48u << 10;  // they fit the cluster's queues
// Whether the narrow-level kernel takes a level of F entries and EF edges;
// with `heavy`, `list` of them may hold many edges (or wait in global memory)
// and are walked by the whole cluster.
BFS_HD bool narrow_level(uint32_t F, uint32_t EF, bool heavy, uint32_t list) {
  return F > 0u && EF <= kNarrowEdges && (heavy ? list : 0u) <= kNarrowList;
}
BFS_HD bool narrow_level(uint32_t F, uint32_t EF, bool heavy) {
  return narrow_level(F, EF, heavy, F) && F <= kNarrowEntries;
}
// The same after init or level generation, in loops that run the kernel
// (no entry has more than EF - F + 1 edges: each has at least one).
BFS_HD bool narrow_next(const BfsDevState *st, uint32_t F, uint32_t EF) {
  return st->narrow != 0u && narrow_level(F, EF, EF - F + 1u > kNarrowHeavyBound);
}
// Arguments (BfsDevState*, conditional_handle, use_conditional, int first);
// first: seeds the root before it looks at the level (no init kernel then).
// One cluster
// of kNarrowBlock-thread blocks, grid = cluster size,
// narrow_smem_bytes(parents) of dynamic shared memory.
const void *narrow_kernel_fn(int cluster, bool parents);
size_t narrow_smem_bytes(bool parents);
// The largest cluster (16 or 8 blocks) the current device runs the kernel
// on; raises the kernel's attributes for it.  0 and an error if none.
cudaError_t narrow_cluster_size(int *cluster);

// Kernel function pointers (for CUDA-graph kernel nodes and direct launches).
// Every kernel takes (BfsDevState*) first; levelgen and init also take
// (unsigned long long conditional_handle, int use_conditional), fill the
// state's contents (BfsDevState).
// parents: the variant that also records BFS-tree parents.
const void *explore_kernel_fn(int arm, int ipt, bool parents);
// The explore kernel that runs any arm: arguments (BfsDevState*, int arm),
// arm < 0 = the arm stored in st->arm; kAnyBlock threads, one block per SM,
// dynamic shared memory of st->hub_words words for GLB levels behind the hub
// filter (the function's maximum dynamic shared memory must be raised first).
const void *explore_any_kernel_fn(int ipt, bool parents);
// Level generation: kLevelgenBlock threads, levelgen_smem(parents) bytes of
// dynamic shared memory (above the default limit: the function's maximum
// dynamic shared memory must be raised first).
const void *levelgen_kernel_fn(bool parents);
size_t levelgen_smem(bool parents);
const void *init_kernel_fn();
// fill writes the state, clears the visited bitmaps (vis, prev: st->words words each), marks
// every working level unvisited and sets parents (when recorded) to -1.
const void *fill_kernel_fn();
// Writes the output levels (st->level, every entry) from the working levels;
// runs once after the level loop; copies the state to its `result`, if any.
// Arguments (BfsDevState*).
const void *level_out_kernel_fn();

cudaError_t launch_validate(const uint32_t *indptr, const uint32_t *inds, uint32_t n_rows,
                            uint32_t n_cols, uint32_t root, const int32_t *level,
                            const int32_t *parent, uint8_t *witness, uint8_t *parent_ok,
                            unsigned long long *bad, cudaStream_t s);
// Counts the CSC's errors in *bad; where there are any and rows is given,
// sets *rows to 0 (init then queues no root).
cudaError_t launch_check_csc(const uint32_t *indptr, const uint32_t *inds, uint32_t n_cols,
                             uint64_t nnz, unsigned long long *bad, cudaStream_t s,
                             uint32_t *rows = nullptr);

}  // namespace bfsgb
