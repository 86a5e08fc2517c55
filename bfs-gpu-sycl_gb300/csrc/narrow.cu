// narrow.cu -- runs of levels with few edges, in one launch.
//
// A level of the two-kernel loop costs 12 to 19 us however small it is: two
// launches of the loop's body, a grid-wide scan of the visited bitmap, a
// ticket and, for learned plans, the scheduler's inference.  A grid spends
// all of its time there (thousands of levels of a few thousand vertices),
// and a power-law graph its first and last levels.  This kernel runs such
// levels back to back on one thread-block cluster: an edge's claim is an
// atomicOr whose winner (exactly one per vertex) stores the working level,
// reads the vertex's offsets and appends it to the next frontier, so no
// bitmap is scanned and nothing is launched between levels; the cluster
// barrier is the level barrier.  It runs in front of the level loop and
// after every level generation in it, returns at once when the next level is
// not narrow (narrow_level in kernels.h), and leaves the state and the queue
// as level generation would.
//
// The frontier stays on the chip: entries are pushed into the shared memory
// of the cluster's blocks, each warp to one block (another one every level, so
// that the load evens out), through that block's counter.  Entries with many
// edges, and those that find a block's queue full, go to a list in global
// memory that the whole cluster walks together, balanced by chunk: every block
// scans the list's chunk counts into shared memory, kNarrowTile entries at a
// time, and each lane finds its chunk's owner by binary search.
//
// Bound: the latency of a level's chain -- counters, edge chunk, claim and
// offsets side by side, queue slot, entry, barrier -- each link one round trip
// to L2 or across the cluster.  Work is dealt in 16-byte chunks of the edge
// array, one per lane (up to four edges, whose claims are in flight together).
// Measured per level, learned plan: 2.5 us on a 300 x 300 grid (200 entries a
// level) against 18.3 in the two-kernel loop, 4.6 against 21.8 on 4096 x 4096
// (3600 entries, where the scattered loads and claims of 16 SMs bound it);
// R-MAT scale 12, whole BFS: 57 us against 117.  Blocks of 512 threads: 1024
// spill and wait longer at the barrier (2.8 -> 4.3 us on 1023 x 1537), 256
// have too few lanes (4.6 -> 7.3 on 4096 x 4096).  Clusters of 8 instead of
// 16: 5.6 -> 7.4 there in an earlier form.  With the queue in global memory
// and one counter for the cluster a level took 4.0 us instead of 2.5 on
// 300 x 300.  No gain: queue entries kept in their own block (no remote
// counter), prefetching the next level's edges, testing claims with a load
// first on levels with fewer edges than lanes (2.84 -> 3.08).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "bfs_internal.h"
#include "device_util.cuh"
#include "kernels.h"
#include "bfs_sched_dev.cuh"
#include "level_state.cuh"

namespace bfsgb {
namespace {

namespace cg = cooperative_groups;

constexpr uint32_t kNarrowTile = 2048;  // list entries scanned at a time
// Entries of one block's queue (two queues per block: this level's, the next)
constexpr uint32_t kNarrowQueue = 6144;

// Counters of a block for the next level, one set per level modulo 3.
struct __align__(16) NarrowCounters {
  uint32_t count;    // entries pushed to this block's queue
  uint32_t edges;    // degrees of the entries this block pushed
  uint32_t reached;  // new vertices this block claimed (those without edges too)
  uint32_t list;     // entries of the list in global memory (rank 0's)
};

__device__ __forceinline__ uint32_t map_to_rank(const void *p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
               : "=r"(r)
               : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ uint32_t cluster_add(uint32_t addr, uint32_t v) {
  uint32_t r;
  asm volatile("atom.relaxed.cluster.shared::cluster.add.u32 %0, [%1], %2;"
               : "=r"(r)
               : "r"(addr), "r"(v)
               : "memory");
  return r;
}
__device__ __forceinline__ void cluster_store2(uint32_t addr, uint32_t x, uint32_t y) {
  asm volatile("st.shared::cluster.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void cluster_store(uint32_t addr, uint32_t x) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(x) : "memory");
}
__device__ __forceinline__ uint4 cluster_load4(uint32_t addr) {
  uint4 r;
  asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
               : "r"(addr)
               : "memory");
  return r;
}

__device__ __forceinline__ uint32_t chunks_of(uint32_t b, uint32_t d) {
  return edge_chunks(b, d, 0u);
}

// Dynamic shared memory: two queues of (position, degree), with parents two
// of vertex ids.
constexpr size_t narrow_smem(bool parents) {
  return (size_t)2 * kNarrowQueue * (parents ? 12 : 8);
}

template <int C, bool PAR>
__global__ void __cluster_dims__(C, 1, 1) __launch_bounds__(kNarrowBlock, 1)
    narrow_kernel(BfsDevState *__restrict__ st, unsigned long long cond, int use_cond, int first) {
  constexpr uint32_t NW = kNarrowBlock / 32;
  constexpr uint32_t kPer = kNarrowTile / kNarrowBlock;  // list entries per thread and tile
  static_assert(kPer * kNarrowBlock == kNarrowTile && NW <= 32, "block size");
  static_assert(kNarrowEntries <= 8u * kNarrowQueue, "the first level fits the queues");
  // positions are edge indexes counted from inds0, the 16-byte boundary at or
  // below inds
  extern __shared__ __align__(16) uint2 s_q[];  // [2][kNarrowQueue] (position, degree)
  uint32_t *const s_v = reinterpret_cast<uint32_t *>(s_q + 2 * kNarrowQueue);
  __shared__ uint32_t s_off[kNarrowTile];  // first chunk of a list entry, in the tile's chunks
  __shared__ uint32_t s_beg[kNarrowTile];
  __shared__ uint32_t s_deg[kNarrowTile];
  __shared__ uint32_t s_vid[PAR ? kNarrowTile : 1];
  __shared__ uint32_t s_wsum[32];
  __shared__ NarrowCounters s_ctr[3];
  __shared__ NarrowCounters s_all;  // the cluster's totals
  __shared__ float s_w[kSchedParams];  // rank 0: the scheduler's model
  __shared__ uint2 s_out;           // chunks of this block's part of the queue, at the end

  const uint32_t rank = cg::this_cluster().block_rank();
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t le_mask = (2u << lane) - 1u;
  if (first) {
    if (rank == 0 && tid == 0) init_state(st, cond, use_cond);
    cg::this_cluster().sync();
  }
  const float *const w = st->sched_w;
  // F entries in all, L of them in this block's queue and G in the list
  uint32_t F = st->F, EF = st->EF, lvl = st->lvl, cur = st->cur;
  // no entry has more edges than this (every entry has at least one)
  const bool heavy = EF - F + 1u > kNarrowHeavyBound;
  const bool run = narrow_level(F, EF, heavy);  // uniform over the cluster
  if (rank == 0 && w != nullptr && (run || first)) stage_weights(s_w, w);
  if (!run) {
    if (rank == 0 && tid == 0) st->launches += 1;
    if (first && F > 0u && w != nullptr && rank == 0) {
      __syncthreads();
      if (warp == 0) fused_sched_pick(st, level_counters(st), s_w);
    }
    return;
  }
  uint32_t *const __restrict__ vis = st->vis;
  uint32_t *const __restrict__ prev = st->prev;
  uint8_t *const __restrict__ lv8 = st->lv8;
  const uint32_t *const __restrict__ indptr = st->indptr;
  int32_t *const __restrict__ level = st->level;
  int32_t *const __restrict__ parent = st->parent;
  const uint32_t *const __restrict__ moved = st->moved;
  const uint32_t *const __restrict__ perm = st->perm;
  const uint32_t n_rows = st->n_rows, level_cap = st->level_cap;
  const uint32_t off = st->inds_off;
  const uint32_t *const __restrict__ inds0 = st->inds - off;
  const uint32_t lo4 = off ? 1u : 0u, hi4 = (st->nnz + off) >> 2;  // chunks wholly inside inds
  uint32_t reached = st->reached, max_level = st->max_level, error = 0;
  unsigned long long edges_count = st->edges_count;
  if (tid < 3) s_ctr[tid] = NarrowCounters{0u, 0u, 0u, 0u};
  uint32_t L = 0, G = F;
  if (F > kNarrowTile && !heavy) {  // many entries of few edges: into the queues
    const uint32_t *const qb = st->qb[cur], *const qd = st->qd[cur], *const qv = st->qv[cur];
    for (uint32_t i = tid * C + rank; i < F; i += kNarrowBlock * C) {
      s_q[cur * kNarrowQueue + i / C] = make_uint2(qb[i] + off, qd[i]);
      if (PAR) s_v[cur * kNarrowQueue + i / C] = qv[i];
    }
    L = (F - rank + C - 1u) / C;  // F > rank
    G = 0;
  }
  const uint32_t list_ctr = map_to_rank(s_ctr, 0) + 12u;  // NarrowCounters::list
  cg::this_cluster().sync();

  uint32_t set = 0;  // the level's counters
  while (true) {     // one level
    const uint32_t next_set = set == 2u ? 0u : set + 1u;
    // everyone read this set two barriers ago
    if (tid == 0) s_ctr[next_set] = NarrowCounters{0u, 0u, 0u, 0u};
    const uint32_t nxt = cur ^ 1u;
    const uint32_t lvl_next = lvl + 1u;
    const uint8_t rep = lvl_next < (uint32_t)kLv8Deep ? (uint8_t)lvl_next : kLv8Deep;
    // more edges than lanes: a claim is tested with a load first
    const bool pretest = EF > C * kNarrowBlock;
    uint32_t my_edges = 0, my_reached = 0;
    // the block this warp pushes to
    const uint32_t dest = (rank + warp + lvl) & (C - 1u);
    const uint32_t dest_ctr = map_to_rank(s_ctr + set, dest);  // NarrowCounters::count
    const uint32_t dest_q = map_to_rank(s_q + nxt * kNarrowQueue, dest);
    const uint32_t dest_v = PAR ? map_to_rank(s_v + nxt * kNarrowQueue, dest) : 0u;

    auto push_list = [&](uint32_t b, uint32_t d, uint32_t v) {
      const uint32_t i = cluster_add(list_ctr + set * (uint32_t)sizeof(NarrowCounters), 1u);
      st->qb[nxt][i] = b;
      st->qd[nxt][i] = d;
      if (PAR) st->qv[nxt][i] = v;
    };
    // Chunk a4 (counted from inds0) of the entry whose edges start at
    // position sb with degree sd; `on` lanes only.  Claims its targets and
    // pushes the new vertices: all lanes of the warp take part.
    auto visit_chunk = [&](bool on, uint32_t a4, uint32_t sb, uint32_t sd, uint32_t from) {
      uint32_t n4[4] = {0u, 0u, 0u, 0u}, m = 0u;
      if (on) {
        const uint32_t p0 = a4 << 2;
        const uint32_t lo = sb > p0 ? sb - p0 : 0u;
        const uint32_t left = sb + sd - p0;
        m = (0xFu >> (4u - (left < 4u ? left : 4u))) & (0xFu << lo);
        if (a4 >= lo4 && a4 < hi4) {
          const uint4 q = __ldg(reinterpret_cast<const uint4 *>(inds0) + a4);
          n4[0] = q.x;
          n4[1] = q.y;
          n4[2] = q.z;
          n4[3] = q.w;
        } else {
#pragma unroll
          for (int i = 0; i < 4; i++)
            if ((m >> i) & 1u) n4[i] = __ldg(inds0 + p0 + i);
        }
      }
      uint32_t word[4];
      if (pretest) {
#pragma unroll
        for (int i = 0; i < 4; i++) word[i] = ((m >> i) & 1u) ? __ldcg(vis + (n4[i] >> 5)) : kFull;
#pragma unroll
        for (int i = 0; i < 4; i++)
          if ((word[i] >> (n4[i] & 31u)) & 1u) m &= ~(1u << i);
      }
      // the claims, and beside them the targets' offsets, whoever wins: one
      // round trip instead of two
      uint32_t b[4], d[4], cnt = 0;
#pragma unroll
      for (int i = 0; i < 4; i++)
        word[i] = ((m >> i) & 1u) ? atomicOr(vis + (n4[i] >> 5), 1u << (n4[i] & 31u)) : kFull;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        b[i] = d[i] = 0u;
        if (((m >> i) & 1u) && n4[i] < n_rows) {
          b[i] = __ldg(indptr + n4[i]);
          d[i] = __ldg(indptr + n4[i] + 1u);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const uint32_t n = n4[i];
        d[i] -= b[i];
        if ((word[i] >> (n & 31u)) & 1u) {
          d[i] = 0u;  // another edge reached n
          continue;
        }
        red_or(prev + (n >> 5), 1u << (n & 31u));
        lv8[n] = rep;
        my_reached++;
        my_edges += d[i];
        if (PAR || rep == kLv8Deep) {
          if (moved && ((moved[n >> 5] >> (n & 31u)) & 1u)) n4[i] = perm[n];
          if (PAR) parent[n4[i]] = (int32_t)from;
          if (rep == kLv8Deep) level[n4[i]] = (int32_t)lvl_next;
        }
        if (d[i] > kNarrowHeavy) {
          push_list(b[i], d[i], n4[i]);
          d[i] = 0u;
        }
        cnt += d[i] ? 1u : 0u;
      }
      const uint32_t incl = warp_incl_scan(cnt, lane);
      const uint32_t total = __shfl_sync(kFull, incl, 31);
      if (total == 0u) return;  // uniform over the warp
      uint32_t base = 0;
      if (lane == 0) base = cluster_add(dest_ctr, total);
      uint32_t slot = __shfl_sync(kFull, base, 0) + incl - cnt;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        if (!d[i]) continue;
        if (slot < kNarrowQueue) {
          cluster_store2(dest_q + 8u * slot, b[i] + off, d[i]);
          if (PAR) cluster_store(dest_v + 4u * slot, n4[i]);
        } else {
          push_list(b[i], d[i], n4[i]);
        }
        slot++;
      }
    };

    // this block's queue: E entries per warp and step
    if (L) {
      const uint32_t E = min((L + NW - 1u) / NW, 32u);
      const uint2 *const q = s_q + cur * kNarrowQueue;
      for (uint32_t t = warp * E; t < L; t += NW * E) {
        uint32_t b = 0, d = 0, v = 0;
        if (lane < E && t + lane < L) {
          const uint2 x = q[t + lane];
          b = x.x;
          d = x.y;
          if (PAR) v = s_v[cur * kNarrowQueue + t + lane];
        }
        const uint32_t nch = chunks_of(b, d);
        const uint32_t incl = warp_incl_scan(nch, lane);
        const uint32_t total = __shfl_sync(kFull, incl, 31);
        const uint32_t excl = d ? incl - nch : kFull;
        uint32_t before = 0;  // entries that start before x0
        for (uint32_t x0 = 0; x0 < total; x0 += 32u) {
          const uint32_t x = x0 + lane;
          // starts are distinct; entries that start before x0 wrap past 32
          const uint32_t starts = __reduce_or_sync(kFull, bit_or_zero(excl - x0));
          const uint32_t o = before + __popc(starts & le_mask) - 1u;
          before += __popc(starts);
          const uint32_t sb = __shfl_sync(kFull, b, o), sd = __shfl_sync(kFull, d, o);
          const uint32_t so = __shfl_sync(kFull, excl, o);
          const uint32_t sv = PAR ? __shfl_sync(kFull, v, o) : 0u;
          visit_chunk(x < total, (sb >> 2) + (x - so), sb, sd, sv);
        }
      }
    }
    // the list, walked by the whole cluster
    for (uint32_t t0 = 0; t0 < G; t0 += kNarrowTile) {
      const uint32_t i0 = tid * kPer;
      uint32_t nch[kPer], own = 0;
#pragma unroll
      for (uint32_t k = 0; k < kPer; k++) {
        uint32_t b = 0, d = 0;
        if (t0 + i0 + k < G) {
          b = __ldcg(st->qb[cur] + t0 + i0 + k) + off;
          d = __ldcg(st->qd[cur] + t0 + i0 + k);
          if (PAR) s_vid[i0 + k] = __ldcg(st->qv[cur] + t0 + i0 + k);
        }
        s_beg[i0 + k] = b;
        s_deg[i0 + k] = d;
        nch[k] = own;
        own += chunks_of(b, d);
      }
      const uint32_t incl = warp_incl_scan(own, lane);
      if (lane == 31) s_wsum[warp] = incl;
      __syncthreads();
      const uint32_t winc = warp_incl_scan(lane < NW ? s_wsum[lane] : 0u, lane);
      const uint32_t total = __shfl_sync(kFull, winc, 31);
      const uint32_t wprev = __shfl_sync(kFull, winc, (warp + 31u) & 31u);
      const uint32_t e0 = (warp ? wprev : 0u) + incl - own;
#pragma unroll
      for (uint32_t k = 0; k < kPer; k++) s_off[i0 + k] = e0 + nch[k];
      __syncthreads();
      const uint32_t n_ent = min(G - t0, kNarrowTile);
      for (uint32_t x0 = (warp * C + rank) * 32u; x0 < total; x0 += C * kNarrowBlock) {
        const uint32_t x = x0 + lane;
        uint32_t lo = 0, hi = n_ent;  // s_off[lo] <= x
        while (hi - lo > 1u) {
          const uint32_t mid = (lo + hi) >> 1;
          if (s_off[mid] <= x) lo = mid; else hi = mid;
        }
        const uint32_t sb = s_beg[lo], sd = s_deg[lo];
        visit_chunk(x < total, (sb >> 2) + (x - s_off[lo]), sb, sd, PAR ? s_vid[lo] : 0u);
      }
      __syncthreads();  // the tile's arrays are free
    }
    my_edges = __reduce_add_sync(kFull, my_edges);
    my_reached = __reduce_add_sync(kFull, my_reached);
    if (lane == 0 && my_reached) {
      if (my_edges) atomicAdd(&s_ctr[set].edges, my_edges);
      atomicAdd(&s_ctr[set].reached, my_reached);
    }
    cg::this_cluster().sync();
    // the level's totals: one lane per block of the cluster, for all warps
    if (warp == 0) {
      uint4 c = make_uint4(0u, 0u, 0u, 0u);
      if (lane < (uint32_t)C) c = cluster_load4(map_to_rank(s_ctr + set, lane));
      const uint32_t f = __reduce_add_sync(kFull, min(c.x, kNarrowQueue));
      const uint32_t ef = __reduce_add_sync(kFull, c.y), rc = __reduce_add_sync(kFull, c.z);
      const uint32_t g = __shfl_sync(kFull, c.w, 0);
      if (lane == 0) s_all = NarrowCounters{f + g, ef, rc, g};
    }
    __syncthreads();
    const NarrowCounters all = s_all;
    F = all.count;
    EF = all.edges;
    G = all.list;
    L = min(s_ctr[set].count, kNarrowQueue);
    reached += all.reached;
    if (all.reached) max_level = lvl_next;
    edges_count += EF;
    lvl = lvl_next;
    cur = nxt;
    set = next_set;
    if (F > 0u && lvl >= level_cap) {
      error = BFS_DEVERR_LEVEL_LIMIT;
      F = 0u;
    }
    // the list is in global memory, the queues' entries have few edges
    if (!narrow_level(F, EF, true, G)) break;  // uniform over the cluster
  }

  // What level generation would have left: the queue with its chunk prefix
  // (the list, then the blocks' queues), the counters and the next level's arm.
  uint32_t EC = 0;
  if (F > 0u) {
    uint32_t *const qb = st->qb[cur], *const qd = st->qd[cur];
    uint32_t *const qc = st->qc[cur], *const qv = st->qv[cur];
    const uint2 *const q = s_q + cur * kNarrowQueue;
    // this block's part of the list, and its chunks
    const uint32_t per = (G + C - 1u) / C;
    const uint32_t g0 = min(G, rank * per), g1 = min(G, g0 + per);
    uint32_t sum_g = 0, sum_l = 0;
    for (uint32_t i = g0 + tid; i < g1; i += kNarrowBlock)
      sum_g += chunks_of(__ldcg(qb + i) + off, __ldcg(qd + i));
    for (uint32_t i = tid; i < L; i += kNarrowBlock) sum_l += chunks_of(q[i].x, q[i].y);
    if (tid == 0) s_out = make_uint2(0u, 0u);
    __syncthreads();
    sum_g = __reduce_add_sync(kFull, sum_g);
    sum_l = __reduce_add_sync(kFull, sum_l);
    if (lane == 0) {
      atomicAdd(&s_out.x, sum_g);
      atomicAdd(&s_out.y, sum_l);
    }
    cg::this_cluster().sync();
    // entries and chunks before this block's parts
    const uint32_t last = set == 0u ? 2u : set - 1u;  // the last level's counters
    uint32_t ent = 0, cg_ = 0, cl_ = 0;
    if (lane < (uint32_t)C) {
      ent = min(cluster_load4(map_to_rank(s_ctr + last, lane)).x, kNarrowQueue);
      const uint32_t a = map_to_rank(&s_out, lane);
      asm volatile("ld.shared::cluster.v2.u32 {%0, %1}, [%2];" : "=r"(cg_), "=r"(cl_) : "r"(a) : "memory");
    }
    const uint32_t all_g = __reduce_add_sync(kFull, cg_);
    EC = all_g + __reduce_add_sync(kFull, cl_);
    const uint32_t base_g = __reduce_add_sync(kFull, lane < rank ? cg_ : 0u);
    const uint32_t base_l = all_g + __reduce_add_sync(kFull, lane < rank ? cl_ : 0u);
    const uint32_t out0 = G + __reduce_add_sync(kFull, lane < rank ? ent : 0u);
    // part 0: the list's chunk prefix in place; part 1: the queue's entries
    for (uint32_t part = 0; part < 2u; part++) {
      const uint32_t n = part ? L : g1 - g0;
      uint32_t base = part ? base_l : base_g;
      for (uint32_t j0 = 0; j0 < n; j0 += kNarrowBlock) {  // uniform over the block
        const uint32_t j = j0 + tid;
        uint32_t b = 0, d = 0;
        if (j < n) {
          b = part ? q[j].x : __ldcg(qb + g0 + j) + off;
          d = part ? q[j].y : __ldcg(qd + g0 + j);
        }
        const uint32_t nch = chunks_of(b, d);
        const uint32_t incl = warp_incl_scan(nch, lane);
        __syncthreads();  // s_wsum's last readers are done
        if (lane == 31) s_wsum[warp] = incl;
        __syncthreads();
        const uint32_t winc = warp_incl_scan(lane < NW ? s_wsum[lane] : 0u, lane);
        const uint32_t wprev = __shfl_sync(kFull, winc, (warp + 31u) & 31u);
        if (j < n) {
          const uint32_t i = part ? out0 + j : g0 + j;
          qc[i] = base + (warp ? wprev : 0u) + incl - nch;
          if (part) {
            qb[i] = b - off;
            qd[i] = d;
            if (PAR) qv[i] = s_v[cur * kNarrowQueue + j];
          }
        }
        base += __shfl_sync(kFull, winc, 31);
      }
    }
    if (rank == 0 && tid == 0) qc[F] = EC;
  }
  if (rank == 0 && tid == 0) {
    st->F = F;
    st->EF = EF;
    st->EC = EC;
    st->lvl = lvl;
    st->cur = cur;
    st->reached = st->reached_prev = reached;
    st->max_level = max_level;
    st->edges_count = edges_count;
    st->error |= error;
    st->launches += 1;
    if (use_cond) cudaGraphSetConditional((cudaGraphConditionalHandle)cond, F > 0u);
  }
  __syncthreads();
  if (rank == 0 && F > 0u && w != nullptr && warp == 0)
    fused_sched_pick(st, LevelCounters{F, EF, reached, lvl}, s_w);
  cg::this_cluster().sync();  // no block leaves while another reads its shared memory
}

template <int C>
const void *fn_of(bool parents) {
  return parents ? (const void *)narrow_kernel<C, true> : (const void *)narrow_kernel<C, false>;
}

}  // namespace

const void *narrow_kernel_fn(int cluster, bool parents) {
  return cluster == 16 ? fn_of<16>(parents) : fn_of<8>(parents);
}

size_t narrow_smem_bytes(bool parents) { return narrow_smem(parents); }

namespace {
// Whether one cluster of c blocks fits the current device, both variants.
bool cluster_fits(int c) {
  for (int par = 0; par < 2; par++) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(kNarrowBlock);
    cfg.dynamicSmemBytes = narrow_smem(par != 0);
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = c;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, narrow_kernel_fn(c, par != 0), &cfg) != cudaSuccess ||
        n < 1) {
      cudaGetLastError();
      return false;
    }
  }
  return true;
}
constexpr int kMaxDevices = 64;
std::atomic<int> g_cluster[kMaxDevices];  // what fits each device (0: not asked yet, -1: none)
}  // namespace

cudaError_t narrow_cluster_size(int *cluster) {
  *cluster = 0;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorNotSupported;
  for (int c : {16, 8}) {
    const int known = g_cluster[dev].load(std::memory_order_relaxed);
    if (known != 0 && known != c) continue;
    for (int par = 0; par < 2; par++) {
      const void *fn = narrow_kernel_fn(c, par != 0);
      e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)narrow_smem(par != 0));
      if (e == cudaSuccess && c > 8)
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      if (e != cudaSuccess) break;
    }
    if (e != cudaSuccess) {
      cudaGetLastError();
      continue;
    }
    if (known == c || cluster_fits(c)) {
      g_cluster[dev].store(c, std::memory_order_relaxed);
      *cluster = c;
      return cudaSuccess;
    }
  }
  g_cluster[dev].store(-1, std::memory_order_relaxed);
  return cudaErrorNotSupported;
}

}  // namespace bfsgb
