// hub_layout.cu -- the degree-ordered hub layout of a graph handle.
//
// In a top-down BFS every edge costs one probe of the visited bitmap, a
// random 4-byte gather over an n/8-byte bitmap, and on power-law graphs most
// of the edges of the large levels point at a few high in-degree vertices
// ("hubs") that were reached levels earlier.  The hub layout gives the
// explore kernel a cheap test for exactly those probes: the graph is
// relabelled so that internal ids 0 .. K-1 are the K vertices of highest
// in-degree, in that order, and the explore kernel keeps bits 0 .. K-1 of
// the visited bitmap in shared memory.  A probe of a hub already visited is
// then answered by shared memory; every other probe goes to the bitmap in
// global memory as before, so levels stay exact.
//
// Relabelling (a permutation perm: internal -> original, pinv its inverse):
//   internal i < K              -> the i-th vertex by in-degree (ties by id)
//   internal v >= K, original position of a hub
//                               -> a non-hub whose original id was < K
//                                  (the displaced and vacated ids are paired
//                                  in increasing order)
//   every other v               -> itself
// so outside the hub prefix almost every vertex keeps its id (and the
// locality of the original numbering).  The relabelled CSC lists, for
// internal vertex i, the out-neighbours of perm[i] mapped through pinv,
// ordered by target class: class c holds the internal ids below limit[c] that
// no earlier class holds, and skip[c][i] counts i's targets below limit[c].
// Once every vertex of the first classes is visited -- on R-MAT scale 25 the
// 2 M vertices of highest degree, which take 89 % of the edge endpoints, are
// by the second of its two large levels -- an edge to them can reach nothing
// new, and level generation queues a vertex without those edges, by one load
// of skip.  About a sixteenth of the vertices are ordered by degree for this,
// more than the shared-memory prefix holds; ordering more would cost the
// output pass more gathers than the edges saved.  R-MAT scale 25, learned,
// mean of 12 roots: 2.72 -> 2.07 ms (levels of 696 M and 348 M edges:
// 1.55 -> 1.30 and 0.75 -> 0.26 ms); scale 23: 831 -> 662 us; scale 21: 379 ->
// 279 us.
// Level and parent arrays are still written in original ids (the level
// generation kernel writes level[perm[v]]), so callers see no difference.
//
// A graph whose K highest in-degree vertices take less than a quarter of all
// edge endpoints (grids, uniform random graphs) gets no layout at all: the
// prefix would catch few probes, and the copy would cost memory and the
// shared-memory copy time for nothing.
//
// Graphs with n_cols <= K need no relabelling: the whole bitmap fits in
// shared memory and the layout is the identity (no copy).  Graphs with
// n_rows < n_cols keep the identity too (a relabelling could move a vertex
// across the n_rows boundary, which decides whether it is expanded); their
// shared-memory prefix is then simply the first K original ids.
#include <cuda_runtime.h>
#include <cub/cub.cuh>

#include <algorithm>
#include <string>

#include "bfs_internal.h"
#include "dev_alloc.h"
#include "engine.h"
#include "hub_layout.h"

namespace bfsgb {
namespace {

constexpr uint32_t kNone = 0xFFFFFFFFu;

__global__ void indeg_kernel(const uint32_t *__restrict__ inds, uint64_t nnz, uint32_t *indeg) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += stride)
    atomicAdd(indeg + inds[e], 1u);
}

__global__ void init_perm_kernel(uint32_t n, uint32_t *iota, uint32_t *perm, uint32_t *pinv) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) {
    iota[v] = v;
    perm[v] = v;
    pinv[v] = kNone;
  }
}

// Sum of the K largest in-degrees (the edge endpoints the prefix covers).
__global__ void top_sum_kernel(const uint32_t *__restrict__ sorted_deg, uint32_t K,
                               unsigned long long *sum) {
  unsigned long long t = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < K; i += gridDim.x * blockDim.x)
    t += sorted_deg[i];
  for (int d = 16; d > 0; d >>= 1) t += __shfl_down_sync(0xFFFFFFFFu, t, d);
  if ((threadIdx.x & 31u) == 0 && t) atomicAdd(sum, t);
}

// internal i < K takes the i-th vertex by in-degree
__global__ void place_hubs_kernel(const uint32_t *__restrict__ by_degree, uint32_t K,
                                  uint32_t *perm, uint32_t *pinv) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < K; i += stride) {
    const uint32_t h = by_degree[i];
    perm[i] = h;
    pinv[h] = i;
  }
}

// displaced: non-hubs with original id < K; vacated: hub ids >= K
__global__ void flags_kernel(const uint32_t *__restrict__ pinv, uint32_t K, uint32_t n,
                             uint8_t *displaced, uint8_t *vacated) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) {
    const bool hub = pinv[v] != kNone;
    displaced[v] = (v < K && !hub) ? 1 : 0;
    vacated[v] = (v >= K && hub) ? 1 : 0;
  }
}

__global__ void pair_kernel(const uint32_t *__restrict__ displaced,
                            const uint32_t *__restrict__ vacated, const uint32_t *count,
                            uint32_t *perm, uint32_t *pinv) {
  const uint32_t m = *count;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < m; j += stride) {
    perm[vacated[j]] = displaced[j];
    pinv[displaced[j]] = vacated[j];
  }
}

__global__ void finish_pinv_kernel(uint32_t n, uint32_t *pinv, const uint32_t *__restrict__ indptr,
                                   const uint32_t *__restrict__ perm, uint32_t *deg) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += stride) {
    if (v < n && pinv[v] == kNone) pinv[v] = v;
    deg[v] = v < n ? indptr[perm[v] + 1] - indptr[perm[v]] : 0u;
  }
}

// Bit v of `moved` is set when perm[v] != v (one ballot per 32 vertices).
__global__ void moved_kernel(const uint32_t *__restrict__ perm, uint32_t n, uint32_t words,
                             uint32_t *moved) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < words * 32u; v += stride) {
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, v < n && perm[v] != v);
    if ((threadIdx.x & 31u) == 0) moved[v >> 5] = m;
  }
}

// ---- relabelled lists ------------------------------------------------------
// Internal vertex i's list is the list of perm[i], every destination mapped
// through pinv and the targets ordered by class (hub_layout.h), with skip[c][i]
// the number of targets below limit[c].
struct Classes {
  uint32_t n;      // classes
  uint32_t shift;  // limit[0] = 1 << shift; every limit is 4 times the one before
  uint32_t *skip;  // n arrays, stride apart
  size_t stride;
};

// limit[0] = 2^s and limit[c] = 4 limit[c - 1]: the class from the top bit of
// the id (n: no class).
__device__ __forceinline__ uint32_t class_of(uint32_t t, const Classes &cl) {
  const uint32_t x = t >> cl.shift;
  const uint32_t c = x ? ((31u - __clz(x)) >> 1) + 1u : 0u;
  return c < cl.n ? c : cl.n;
}

// Lists longer than kMidList edges take a block of 256 threads each, those
// longer than kLongList a block of 1024.  The ids in front are ordered by
// degree, so a warp of relabel_kernel gets 32 lists of like length: with up to
// 4096 edges per list left to it, it took 3.5 of the build's 5.0 ms on R-MAT
// scale 21, and 0.6 of 2.4 so.  (One warp per list whatever its length, as
// before lists were ordered by class, took 34 of 49 ms on scale 25, where the
// build takes 31 ms now.)
constexpr uint32_t kMidList = 256;
constexpr uint32_t kLongList = 8192;

// One warp per 32 internal vertices: their edges in rounds of 32, whatever the
// lists' lengths.  Two passes, counting and placing; an edge's place is its
// rank among the warp's edges of the same vertex and class (match_any), after
// the counts of the rounds before.
__global__ void __launch_bounds__(256) relabel_kernel(
    const uint32_t *__restrict__ indptr, const uint32_t *__restrict__ inds,
    const uint32_t *__restrict__ perm, const uint32_t *__restrict__ pinv,
    const uint32_t *__restrict__ indptr_h, uint32_t n, Classes cl, uint32_t *inds_h,
    uint32_t *mid_list, uint32_t *long_list, uint32_t *n_list) {
  constexpr uint32_t NW = 256 / 32, kC = kHubClasses + 1;
  __shared__ uint32_t s_cnt[NW][32][kC];
  __shared__ uint32_t s_in[NW][32], s_out[NW][32], s_first[NW][32];
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u, le = (2u << lane) - 1u;
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t i0 = (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32u; i0 < n;
       i0 += warps * 32u) {
    const uint32_t i = (uint32_t)i0 + lane;
    uint32_t b = 0, d = 0;
    if (i < n) {
      const uint32_t src = perm[i];
      b = indptr[src];
      d = indptr[src + 1] - b;
      if (d > kMidList) {
        const bool lng = d > kLongList;
        (lng ? long_list : mid_list)[atomicAdd(n_list + (lng ? 1 : 0), 1u)] = i;
        d = kNone;
      }
    }
    const bool is_long = d == kNone;
    if (is_long) d = 0;
    const uint32_t some = __ballot_sync(kNone, d > 0u);  // vertices with edges here
    uint32_t first = d;  // exclusive prefix of d
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const uint32_t y = __shfl_up_sync(kNone, first, s);
      if (lane >= (uint32_t)s) first += y;
    }
    const uint32_t total = __shfl_sync(kNone, first, 31);
    first -= d;
    const uint32_t slot = __popc(some & lt);  // of a vertex with edges
    const uint32_t m = __popc(some);
    __syncwarp();
    if (d) {
      s_in[w][slot] = b - first;  // mod 2^32
      s_out[w][slot] = indptr_h[i];
      s_first[w][slot] = first;
    }
    if (lane < m)
#pragma unroll
      for (uint32_t c = 0; c < kC; c++) s_cnt[w][lane][c] = 0u;
    __syncwarp();
    const uint32_t start = lane < m ? s_first[w][lane] : kNone;
    for (int pass = 0; pass < 2; pass++) {
      uint32_t before = 0;  // vertices whose edges start before x0
      for (uint32_t x0 = 0; x0 < total; x0 += 32u) {
        const uint32_t x = x0 + lane, p = start - x0;
        const uint32_t starts = __reduce_or_sync(kNone, p < 32u ? 1u << p : 0u);
        const uint32_t o = before + __popc(starts & le) - 1u;
        before += __popc(starts);
        uint32_t t = 0, key = kNone;
        if (x < total) {
          t = pinv[inds[s_in[w][o] + x]];
          key = o * 8u + class_of(t, cl);
        }
        const uint32_t same = __match_any_sync(kNone, key);
        if (x < total) {
          uint32_t *const cnt = &s_cnt[w][o][key & 7u];
          const uint32_t base = pass ? *cnt : 0u;
          if (pass) inds_h[s_out[w][o] + base + __popc(same & lt)] = t;
        }
        __syncwarp();
        if (x < total && (same & lt) == 0u) s_cnt[w][o][key & 7u] += __popc(same);
        __syncwarp();
      }
      if (pass == 0) {  // counts to first places
        if (lane < m) {
          uint32_t run = 0;
#pragma unroll
          for (uint32_t c = 0; c < kC; c++) {
            const uint32_t y = s_cnt[w][lane][c];
            s_cnt[w][lane][c] = run;
            run += y;
          }
        }
        __syncwarp();
        if (i < n && !is_long)  // targets below limit[c]: the place of class c + 1
          for (uint32_t c = 0; c < cl.n; c++)
            cl.skip[c * cl.stride + i] = d ? s_cnt[w][slot][c + 1u] : 0u;
        __syncwarp();
      }
    }
  }
}

// One block per list.
template <int B>
__global__ void __launch_bounds__(B) relabel_long_kernel(
    const uint32_t *__restrict__ indptr, const uint32_t *__restrict__ inds,
    const uint32_t *__restrict__ perm, const uint32_t *__restrict__ pinv,
    const uint32_t *__restrict__ indptr_h, uint32_t n, Classes cl, uint32_t *inds_h,
    const uint32_t *__restrict__ long_list, const uint32_t *__restrict__ n_long) {
  __shared__ uint32_t s_cnt[kHubClasses + 1];
  const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  const uint32_t total = *n_long;
  for (uint32_t k = blockIdx.x; k < total; k += gridDim.x) {
    const uint32_t i = long_list[k], src = perm[i];
    const uint32_t b = indptr[src], d = indptr[src + 1] - b, o = indptr_h[i];
    __syncthreads();
    if (threadIdx.x <= cl.n) s_cnt[threadIdx.x] = 0u;
    __syncthreads();
    for (int pass = 0; pass < 2; pass++) {
      uint32_t mine = 0;  // pass 0: lane c counts class c
      for (uint32_t j0 = threadIdx.x & ~31u; j0 < d; j0 += blockDim.x) {
        const uint32_t j = j0 + lane;
        const uint32_t t = j < d ? pinv[inds[b + j]] : 0u;
        const uint32_t c = j < d ? class_of(t, cl) : kNone;
        uint32_t same = 0, num = 0;
        for (uint32_t y = 0; y <= cl.n; y++) {
          const uint32_t bal = __ballot_sync(kNone, c == y);
          if (c == y) same = bal;
          if (lane == y) num = __popc(bal);
        }
        if (pass == 0) {
          mine += num;
        } else {
          const uint32_t base = lane <= cl.n && num ? atomicAdd(&s_cnt[lane], num) : 0u;
          const uint32_t at = __shfl_sync(kNone, base, j < d ? c : 0u);
          if (j < d) inds_h[o + at + __popc(same & lt)] = t;
        }
      }
      if (pass == 0) {
        if (lane <= cl.n && mine) atomicAdd(&s_cnt[lane], mine);
        __syncthreads();
        if (threadIdx.x == 0) {
          uint32_t run = 0;
          for (uint32_t c = 0; c <= cl.n; c++) {
            const uint32_t y = s_cnt[c];
            s_cnt[c] = run;
            run += y;
            if (c < cl.n) cl.skip[c * cl.stride + i] = run;
          }
        }
        __syncthreads();
      }
    }
  }
}

}  // namespace

void free_hub(bfs_graph *g) {
  HubLayout *h = g->hub;
  if (!h) return;
  if (h->relabelled) {
    cudaFree(h->mem);
    cudaFree(h->inds);
  }
  delete h;
  g->hub = nullptr;
}

uint32_t hub_max_vertices(const bfs_graph *g, size_t static_bytes) {
  // dynamic shared memory of the explore kernel: what the device allows a
  // block beside the kernel's static arrays, in whole 16-byte rows
  int optin = 0;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, g->device) !=
          cudaSuccess ||
      optin <= 0 || (size_t)optin <= static_bytes + 1024) {
    cudaGetLastError();
    return 0;
  }
  const size_t bytes = (size_t)optin - static_bytes - 1024;
  return (uint32_t)(bytes * 8 / 128 * 128);
}

bfs_status build_hub(bfs_graph *g, uint32_t K) {
  free_hub(g);
  if (K == 0) return BFS_OK;
  const uint32_t n = g->n_cols;
  HubLayout *h = new (std::nothrow) HubLayout();
  if (!h) return fail(BFS_ERR_OOM, "host allocation failed");
  h->indptr = g->indptr;
  h->inds = g->inds;
  // identity for small graphs, graphs whose rows are not all expanded and
  // graphs of 2^31 vertices or more (level generation marks moved ids in
  // bit 31 of its vertex lists)
  if (n <= K || g->n_rows != n || n > 0x80000000u) {
    // identity: the prefix is the first min(K, all) original ids
    const uint32_t bits = (uint32_t)std::min<uint64_t>((uint64_t)K, (uint64_t)g->words * 32u);
    h->vertices = bits / 128u * 128u;
    h->relabelled = false;
    g->hub = h;
    return BFS_OK;
  }
  // Ids ordered by degree: the prefix, and for the target classes about a
  // sixteenth of the vertices (rounded down to a power of two); the classes'
  // limits are quarters of each other, none below 128 ids.
  uint32_t top = 128;
  while (top < (1u << 30) && (top * 2u <= K || top * 2u <= n / 16u)) top *= 2u;
  const uint32_t ordered = std::min(n, std::max(K, top));
  Classes cl = {};
  for (uint32_t lim = top; lim >= 128u && cl.n < (uint32_t)kHubClasses && lim < n; lim >>= 2) {
    cl.n++;
    cl.shift = 31u - (uint32_t)__builtin_clz(lim);
  }
  for (uint32_t c = 0; c < cl.n; c++) h->limit[c] = 1u << (cl.shift + 2u * c);
  h->classes = cl.n;
  h->vertices = K;
  h->relabelled = true;  // from here on the arrays below are the layout's own
  h->indptr = h->inds = nullptr;
  cudaStream_t s = g->stream;
  uint32_t *indeg = nullptr, *iota = nullptr, *sorted_deg = nullptr, *by_degree = nullptr;
  uint32_t *list_d = nullptr, *list_v = nullptr, *count = nullptr, *deg = nullptr;
  uint32_t *mid_list = nullptr, *long_list = nullptr;
  char *build = nullptr;
  unsigned long long *cover = nullptr, h_cover = 0;
  bool flat = false;
  uint8_t *flags = nullptr;
  void *tmp = nullptr;
  size_t tmp_bytes = 0, t_sort = 0, t_sel = 0, t_scan = 0;
  cudaError_t e = cudaSuccess;
  const int grid = g->num_sms * 8;
#define HUB_CK(x)                    \
  do {                               \
    e = (x);                         \
    if (e != cudaSuccess) goto done; \
  } while (0)
  // two allocations for the layout's own arrays and one for the build's (each
  // cudaMalloc and cudaFree of its own cost the first run more than a kernel)
  {
    auto al = [](size_t bytes) { return (bytes + 255) / 256 * 256; };
    const size_t v4 = al(sizeof(uint32_t) * ((size_t)n + 1)), o4 = al(sizeof(uint32_t) * (size_t)ordered);
    const size_t mw = al(sizeof(uint32_t) * (size_t)g->words);
    // lists of more than kMidList, kLongList edges: at most so many
    const size_t ml = al(sizeof(uint32_t) * (size_t)(g->nnz / kMidList + 1));
    const size_t ll = al(sizeof(uint32_t) * (size_t)(g->nnz / kLongList + 1));
    char *p = nullptr;
    HUB_CK(dev_malloc(&p, (3 + cl.n) * v4 + mw));
    h->mem = p;
    h->perm = (uint32_t *)p; p += v4;
    h->pinv = (uint32_t *)p; p += v4;
    h->indptr = (uint32_t *)p; p += v4;
    h->moved = (uint32_t *)p; p += mw;
    cl.skip = (uint32_t *)p;
    cl.stride = v4 / sizeof(uint32_t);
    for (uint32_t c = 0; c < cl.n; c++) h->skip[c] = cl.skip + c * cl.stride;
    HUB_CK(dev_malloc(&h->inds, sizeof(uint32_t) * (g->nnz ? g->nnz : 1)));
    HUB_CK(cub::DeviceRadixSort::SortPairsDescending(nullptr, t_sort, indeg, sorted_deg, iota,
                                                     by_degree, (int64_t)n, 0, 32, s));
    HUB_CK(cub::DeviceSelect::Flagged(nullptr, t_sel, iota, flags, list_d, count, (int64_t)n, s));
    HUB_CK(cub::DeviceScan::ExclusiveSum(nullptr, t_scan, deg, h->indptr, (int64_t)n + 1, s));
    tmp_bytes = std::max(t_sort, std::max(t_sel, t_scan));
    HUB_CK(dev_malloc(&build, 5 * v4 + 2 * o4 + ml + ll + al(2 * (size_t)n) + 512 + tmp_bytes));
    p = build;
    indeg = (uint32_t *)p; p += v4;
    iota = (uint32_t *)p; p += v4;
    sorted_deg = (uint32_t *)p; p += v4;
    by_degree = (uint32_t *)p; p += v4;
    deg = (uint32_t *)p; p += v4;
    list_d = (uint32_t *)p; p += o4;
    list_v = (uint32_t *)p; p += o4;
    mid_list = (uint32_t *)p; p += ml;
    long_list = (uint32_t *)p; p += ll;
    flags = (uint8_t *)p; p += al(2 * (size_t)n);
    count = (uint32_t *)p; p += 256;
    cover = (unsigned long long *)p; p += 256;
    tmp = p;
  }

  HUB_CK(cudaMemsetAsync(indeg, 0, sizeof(uint32_t) * (size_t)n, s));
  indeg_kernel<<<grid, 256, 0, s>>>(g->inds, g->nnz, indeg);
  init_perm_kernel<<<grid, 256, 0, s>>>(n, iota, h->perm, h->pinv);
  HUB_CK(cudaGetLastError());
  // stable radix sort: equal in-degrees keep increasing ids
  {
    size_t t = tmp_bytes;
    HUB_CK(cub::DeviceRadixSort::SortPairsDescending(tmp, t, indeg, sorted_deg, iota, by_degree,
                                                     (int64_t)n, 0, 32, s));
  }
  HUB_CK(cudaMemsetAsync(cover, 0, sizeof(unsigned long long), s));
  top_sum_kernel<<<grid, 256, 0, s>>>(sorted_deg, K, cover);
  HUB_CK(cudaMemcpyAsync(&h_cover, cover, sizeof(h_cover), cudaMemcpyDeviceToHost, s));
  HUB_CK(cudaStreamSynchronize(s));
  if (h_cover * 4ull < g->nnz) {
    flat = true;  // no hubs to speak of: no layout
    goto done;
  }
  place_hubs_kernel<<<grid, 256, 0, s>>>(by_degree, ordered, h->perm, h->pinv);
  flags_kernel<<<grid, 256, 0, s>>>(h->pinv, ordered, n, flags, flags + n);
  HUB_CK(cudaGetLastError());
  {
    size_t t = tmp_bytes;
    HUB_CK(cub::DeviceSelect::Flagged(tmp, t, iota, flags, list_d, count, (int64_t)n, s));
    t = tmp_bytes;
    HUB_CK(cub::DeviceSelect::Flagged(tmp, t, iota, flags + n, list_v, count + 1, (int64_t)n, s));
  }
  pair_kernel<<<grid, 256, 0, s>>>(list_d, list_v, count, h->perm, h->pinv);
  finish_pinv_kernel<<<grid, 256, 0, s>>>(n, h->pinv, g->indptr, h->perm, deg);
  moved_kernel<<<grid, 256, 0, s>>>(h->perm, n, g->words, h->moved);
  HUB_CK(cudaGetLastError());
  {
    size_t t = tmp_bytes;
    HUB_CK(cub::DeviceScan::ExclusiveSum(tmp, t, deg, h->indptr, (int64_t)n + 1, s));
  }
  HUB_CK(cudaMemsetAsync(count + 2, 0, 2 * sizeof(uint32_t), s));
  relabel_kernel<<<grid, 256, 0, s>>>(g->indptr, g->inds, h->perm, h->pinv, h->indptr, n, cl,
                                      h->inds, mid_list, long_list, count + 2);
  relabel_long_kernel<1024><<<g->num_sms, 1024, 0, s>>>(g->indptr, g->inds, h->perm, h->pinv,
                                                        h->indptr, n, cl, h->inds, long_list,
                                                        count + 3);
  relabel_long_kernel<256><<<g->num_sms * 8, 256, 0, s>>>(g->indptr, g->inds, h->perm, h->pinv,
                                                          h->indptr, n, cl, h->inds, mid_list,
                                                          count + 2);
  HUB_CK(cudaGetLastError());
  {
    uint32_t hc[2] = {0, 0};
    HUB_CK(cudaMemcpyAsync(hc, count, sizeof(hc), cudaMemcpyDeviceToHost, s));
    HUB_CK(cudaStreamSynchronize(s));
    if (hc[0] != hc[1]) {
      e = cudaErrorUnknown;  // the two lists must pair up exactly
      goto done;
    }
  }
done:
#undef HUB_CK
  cudaStreamSynchronize(s);
  cudaFree(build);
  if (e != cudaSuccess || flat) {
    cudaGetLastError();
    g->hub = h;  // frees the layout's own arrays, never the graph's
    free_hub(g);
    if (flat) return BFS_OK;
    if (e == cudaErrorMemoryAllocation) return BFS_OK;  // no layout: plain kernels
    return fail(BFS_ERR_CUDA, std::string("hub layout: ") + cudaGetErrorString(e));
  }
  g->hub = h;
  return BFS_OK;
}

}  // namespace bfsgb
