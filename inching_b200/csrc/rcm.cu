// Level-synchronous Cuthill-McKee that reproduces the sequential BFS of the
// reference (InchingLiteInteger/Fuel/Coordinate/T1.py:254-323) bit for bit.
//
// Sequential rule: frontier atoms are processed in order; each appends its
// still-unvisited neighbours (descending index) and then stably sorts that run by
// degree.  Hence, within one level,
//   * child j belongs to the EARLIEST frontier position q adjacent to it
//     (atomicMin over positions),
//   * the children of q are ordered by (degree ascending, index descending),
//   * runs are concatenated in parent order (prefix sum of run lengths),
// and a component starts at its first atom in the caller's argsort(degree) order.
//
// What bounds it is the chain of levels, not the edges (500,000 atoms in 60
// components: 655 levels of about 760 atoms).  As five launches, a scan and two
// copies to the host a level took 65 us, 43 ms in all.  So
//   * all levels run in one cooperative kernel, one contiguous piece of the frontier
//     a block, three grid barriers a level, its bounds kept on the device;
//   * every component advances at once: components come from a union-find over the
//     edges whose root is the component's earliest seed, the first frontier holds
//     the roots in seed order, and a stable sort by component at the end puts the
//     runs where the sequential order has them (12 levels instead of 655).
// Whole call, before and now: assembly of 20 globules, 100,000 atoms, 75 and 0.52 ms;
// one globule of 20,000, 1.32 and 0.34 ms; 100,000 atoms at 15 A (18 levels of 800
// neighbours a row) 1.94 and 1.48 ms.  It loses where levels are few and wide: random
// lists of 16 neighbours a row, 8 or 9 levels, 150,000 atoms 0.59 and 0.54 ms, 300,000
// 0.67 and 0.78 ms, 1,000,000 1.16 and 2.3 ms (union-find over edges without locality, and
// 32 warps an SM instead of 56 for the gathers).  No structure has such lists.
// A directed adjacency (one that lists j under i and not i under j) may leave atoms
// that their component's first seed does not reach; the same kernel then runs again
// with one component at a time, each seeded when the frontier is empty.
#include <algorithm>

#include <cub/cub.cuh>

#include "common.cuh"

namespace inch {

extern thread_local int last_launches;

namespace {

constexpr int kWarps = 16;                  // warps of a BFS block
constexpr int kCap = INCH_MAX_DEGREE;
constexpr int kUnset = 0x7fffffff;
constexpr int kTimeout = 8;
constexpr unsigned kBarrierPolls = 1u << 24;   // bound of one grid barrier (seconds)

struct Ctl {
  unsigned arrive;      // grid barrier
  int bad;              // 1: seeds, 2: row length, 3: column (found before the BFS)
  int flag;             // 4: more children than atoms, kTimeout: a barrier ran out
  int levels;
  int64_t visited;
  int64_t seedptr;      // one component at a time: the next seed to look at
};

__global__ void k_check_seeds(const int64_t* __restrict__ seed_order, int64_t n, int* __restrict__ seen, Ctl* ctl) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    int64_t s = seed_order[i];
    if (s < 0 || s >= n || atomicAdd(&seen[s], 1) != 0) atomicExch(&ctl->bad, 1);
  }
}

// One warp per row (coalesced reads of the lists).
__global__ void k_check_rows(const int64_t* __restrict__ rowptr, const int* __restrict__ cols, int64_t n, Ctl* ctl) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps) {
    const int64_t e0 = rowptr[i], d = rowptr[i + 1] - e0;
    if (d < 0 || d > kCap) {
      if (lane == 0) atomicExch(&ctl->bad, 2);
      continue;
    }
    bool out = false;
    for (int64_t e = lane; e < d; e += 32) out |= cols[e0 + e] < 0 || cols[e0 + e] >= n;
    if (out) atomicExch(&ctl->bad, 3);
  }
}

__global__ void k_init(const int64_t* __restrict__ seed_order, int64_t n, int* __restrict__ order,
                       int* __restrict__ claim, int* __restrict__ par, int* __restrict__ rank, const Ctl* ctl) {
  if (ctl->bad) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    order[i] = -1;
    claim[i] = kUnset;
    par[i] = static_cast<int>(i);
    rank[seed_order[i]] = static_cast<int>(i);
  }
}

// ---------------------------------------------------------------------------
// Components: union-find (Tarjan & van Leeuwen's path halving), parents always of
// lower seed rank, so a root is its component's earliest seed whatever the order of
// the unions.  Nothing waits: a failed exchange means that another union went ahead.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int find_root(int* par, int x) {
  int p = __ldcg(par + x);
  while (p != x) {
    const int g = __ldcg(par + p);
    if (g == p) return p;
    par[x] = g;                     // an ancestor of x; x is no root and never becomes one again
    x = g;
    p = __ldcg(par + x);
  }
  return x;
}

// Joins the components of root a and atom j; the root of both afterwards.
__device__ __forceinline__ int join(int* par, const int* __restrict__ rank, int a, int j) {
  int b = find_root(par, j);
  while (a != b) {
    int hi = a, lo = b;
    if (rank[hi] < rank[lo]) {
      hi = b;
      lo = a;
    }
    const int old = atomicCAS(par + hi, hi, lo);
    if (old == hi) return lo;
    a = find_root(par, old);
    b = lo;
  }
  return a;
}

// A thread per row joins it to its first and middle neighbour: after it most rows
// hang in few trees, and the pass over all edges mostly compares two parents.
__global__ void k_join_few(const int64_t* __restrict__ rowptr, const int* __restrict__ cols, int64_t n,
                           const int* __restrict__ rank, int* par, const Ctl* ctl) {
  if (ctl->bad) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e0 = rowptr[i], d = rowptr[i + 1] - e0;
    if (d == 0) continue;
    int r = find_root(par, static_cast<int>(i));
    r = join(par, rank, r, cols[e0]);
    join(par, rank, r, cols[e0 + d / 2]);
  }
}

__global__ void k_join_all(const int64_t* __restrict__ rowptr, const int* __restrict__ cols, int64_t n,
                           const int* __restrict__ rank, int* par, const Ctl* ctl) {
  if (ctl->bad) return;
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps) {
    const int64_t e1 = rowptr[i + 1];
    int r = find_root(par, static_cast<int>(i));
#pragma unroll 4
    for (int64_t e = rowptr[i] + lane; e < e1; e += 32) {
      const int j = cols[e];
      if (__ldcg(par + j) != r) r = join(par, rank, find_root(par, r), j);
    }
  }
}

__global__ void k_flatten(int64_t n, int* par, const Ctl* ctl) {
  if (ctl->bad) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    // read-only walk: a halving store here could put an inner node over a finished root
    int x = static_cast<int>(i), p = __ldcg(par + x);
    while (p != x) {
      x = p;
      p = __ldcg(par + x);
    }
    par[i] = x;
  }
}

// root[r] = 1 where the r-th seed is a root (root[n] = 0): its prefix sum numbers
// the components in seed order.
__global__ void k_roots(const int64_t* __restrict__ seed_order, int64_t n, const int* __restrict__ par,
                        int* __restrict__ root, const Ctl* ctl) {
  const bool bad = ctl->bad != 0;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r <= n; r += (int64_t)gridDim.x * blockDim.x)
    root[r] = !bad && r < n && par[seed_order[r]] == static_cast<int>(seed_order[r]);
}

__global__ void k_seed(const int64_t* __restrict__ seed_order, int64_t n, const int* __restrict__ cidx,
                       int* __restrict__ order, int* __restrict__ claim, const Ctl* ctl) {
  if (ctl->bad) return;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x)
    if (cidx[r + 1] != cidx[r]) {
      const int s = static_cast<int>(seed_order[r]);
      order[cidx[r]] = s;
      claim[s] = -1;
    }
}

// Component of the atom at each BFS position, the key of the last sort.
__global__ void k_keys(const int* __restrict__ order, int64_t n, const int* __restrict__ par,
                       const int* __restrict__ rank, const int* __restrict__ cidx, int* __restrict__ key) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x)
    key[p] = cidx[rank[par[order[p]]]];
}

__global__ void k_finish(const int* __restrict__ order, int64_t n, int64_t* __restrict__ rcm,
                         int64_t* __restrict__ undo) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    int64_t a = order[n - 1 - i];
    rcm[i] = a;
    undo[a] = i;
  }
}

// ---------------------------------------------------------------------------
// The BFS
// ---------------------------------------------------------------------------
// Grid barrier of a cooperative launch (every block resident).  The wait is bounded:
// a block whose wait runs out records it and leaves, and so do the others.
__device__ bool grid_barrier(Ctl* ctl, unsigned& target, unsigned max_polls) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    target += gridDim.x;
    __threadfence();
    atomicAdd(&ctl->arrive, 1u);
    int ok = 1;
    const volatile unsigned* at = &ctl->arrive;
    for (unsigned polls = 0; static_cast<int>(*at - target) < 0; ++polls)
      if (polls > max_polls || ((polls & 1023) == 1023 && *(volatile int*)&ctl->flag == kTimeout)) {
        atomicExch(&ctl->flag, kTimeout);
        ok = 0;
        break;
      }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// Everything that another block writes during the kernel is read past L1 (__ldcg).
// `comp` (n_comp at comp_count): all components at once; else one at a time.
__global__ void __launch_bounds__(kWarps * 32, 2)
k_bfs(const int64_t* __restrict__ rowptr, const int* __restrict__ cols, const int* __restrict__ degree,
      const int64_t* __restrict__ seed_order, const int* __restrict__ par, const int* __restrict__ comp_count,
      int64_t n, int* order, int* claim, int* cnt, int* blocksum, Ctl* ctl, int all,
      unsigned max_polls) {
  extern __shared__ int s_buf[];            // kCap per warp
  __shared__ int64_t s_pre[kWarps], s_tot[kWarps];
  if (ctl->bad) return;                     // set by earlier kernels only: the same for every block
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int* s = s_buf + w * kCap;
  unsigned target = 0;
  int64_t ls = 0, le = all ? *comp_count : 0;
  int levels = 0;
  for (;;) {
    if (ls == le) {
      if (all || le >= n) break;
      // The first seed that no earlier component reached: the whole first block looks,
      // 512 seeds at a time, because the other blocks' wait is bounded (one warp would
      // pass 10^8 seeds in about their limit).
      if (blockIdx.x == 0) {
        int64_t p = ctl->seedptr;
        for (; p < n; p += kWarps * 32) {
          const int64_t q = p + threadIdx.x;
          const bool open = q < n && __ldcg(claim + seed_order[q]) == kUnset;
          const unsigned b = __ballot_sync(0xffffffffu, open);
          if (lane == 0) s_tot[w] = b != 0 ? q + __ffs(b) - 1 : n;
          if (__syncthreads_or(open)) break;
        }
        if (threadIdx.x == 0 && p < n) {
          for (int k = kWarps - 1; k >= 0; --k)
            if (s_tot[k] < n) p = s_tot[k];
          const int sd = static_cast<int>(seed_order[p]);
          order[le] = sd;
          claim[sd] = -1;
          ctl->seedptr = p + 1;
        }
      }
      if (!grid_barrier(ctl, target, max_polls)) break;
      le = ls + 1;
    }
    const int64_t L = le - ls;
    const int64_t per = (L + gridDim.x - 1) / gridDim.x;
    const int64_t q0 = min(ls + (int64_t)blockIdx.x * per, le), q1 = min(q0 + per, le);
    // claim: an atom visited before this level carries a smaller position than any q
    for (int64_t q = q0 + w; q < q1; q += kWarps) {
      const int i = __ldcg(order + q);
      if (i < 0) continue;                  // duplicated entries left a hole: refused below
      const int64_t e1 = rowptr[i + 1];
#pragma unroll 4
      for (int64_t e = rowptr[i] + lane; e < e1; e += 32) {
        const int j = cols[e];
        if (__ldcg(claim + j) > static_cast<int>(q)) atomicMin(claim + j, static_cast<int>(q));
      }
    }
    if (!grid_barrier(ctl, target, max_polls)) break;
    // count the children of each q, prefix sums within the block's piece
    for (int64_t q = q0 + w; q < q1; q += kWarps) {
      const int i = __ldcg(order + q);
      int c = 0;
      if (i >= 0) {
        const int64_t e1 = rowptr[i + 1];
#pragma unroll 4
        for (int64_t e = rowptr[i] + lane; e < e1; e += 32) c += __ldcg(claim + cols[e]) == static_cast<int>(q);
        c = warp_sum(c);
      } else if (lane == 0) {
        atomicExch(&ctl->flag, 4);          // a hole: some row lists an atom twice
      }
      if (lane == 0) {
        cnt[q] = c;
        if (q == ls) {
          ++levels;
        } else if (all && i >= 0) {
          const int h = __ldcg(order + q - 1);
          levels += h >= 0 && par[h] != par[i];   // a level of every component in the frontier
        }
      }
    }
    __syncthreads();
    if (w == 0) {
      int run = 0;
      for (int64_t q = q0; q < q1; q += 32) {
        const int v = q + lane < q1 ? cnt[q + lane] : 0;
        int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, x, o);
          if (lane >= o) x += y;
        }
        if (q + lane < q1) cnt[q + lane] = run + x - v;
        run += __shfl_sync(0xffffffffu, x, 31);
      }
      if (lane == 0) blocksum[blockIdx.x] = run;
    }
    if (!grid_barrier(ctl, target, max_polls)) break;
    int64_t pre = 0, tot = 0;
    for (int b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
      const int v = __ldcg(blocksum + b);
      tot += v;
      pre += b < blockIdx.x ? v : 0;
    }
    pre = warp_sum(pre);
    tot = warp_sum(tot);
    if (lane == 0) {
      s_pre[w] = pre;
      s_tot[w] = tot;
    }
    __syncthreads();
    pre = tot = 0;
#pragma unroll
    for (int k = 0; k < kWarps; ++k) {
      pre += s_pre[k];
      tot += s_tot[k];
    }
    // write the children of q, ordered by (degree asc, index desc), after the level
    for (int64_t q = q0 + w; q < q1; q += kWarps) {
      const int i = __ldcg(order + q);
      if (i < 0) continue;
      const int64_t e1 = rowptr[i + 1];
      int m = 0;
#pragma unroll 4
      for (int64_t e0 = rowptr[i]; e0 < e1; e0 += 32) {
        const int64_t e = e0 + lane;
        const int j = e < e1 ? cols[e] : 0;
        const bool ok = e < e1 && __ldcg(claim + j) == static_cast<int>(q);
        const unsigned b = __ballot_sync(0xffffffffu, ok);
        if (ok) s[m + __popc(b & ((1u << lane) - 1u))] = j;   // m + rank < row length <= kCap
        m += __popc(b);
      }
      __syncwarp();
      const bool both = 2 * m <= kCap;      // degrees beside the indices
      if (both)
        for (int t = lane; t < m; t += 32) s[m + t] = degree[s[t]];
      __syncwarp();
      const int64_t base = le + pre + cnt[q];
      for (int t = lane; t < m; t += 32) {
        const int jt = s[t];
        const int dt = both ? s[m + t] : degree[jt];
        int rank = 0;
        for (int u = 0; u < m; ++u) {
          const int ju = s[u];
          const int du = both ? s[m + u] : degree[ju];
          rank += (du < dt) || (du == dt && ju > jt);
        }
        if (base + rank < n) order[base + rank] = jt;
        else atomicExch(&ctl->flag, 4);
      }
      __syncwarp();
    }
    ls = le;
    le += tot;
    if (le > n) break;                      // the same in every block
    if (!grid_barrier(ctl, target, max_polls)) break;
  }
  levels = warp_sum(levels);                // lane 0 of each warp counted
  if (lane == 0 && levels != 0) atomicAdd(&ctl->levels, levels);
  if (blockIdx.x == 0 && threadIdx.x == 0) ctl->visited = le;
}

struct RcmWs {
  int *order, *claim, *par, *rank, *cidx, *cnt, *key, *order2, *blocksum;
  Ctl* ctl;
  void* cub_tmp;
  size_t cub_bytes;
};

constexpr int kMaxBlocks = 1024;            // blocks of the BFS kernel, at most

size_t cub_bytes_for(int64_t n) {
  size_t a = 0, b = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, a, (int*)nullptr, (int*)nullptr, (int)(n + 1));
  cub::DeviceRadixSort::SortPairs(nullptr, b, (const int*)nullptr, (int*)nullptr, (const int*)nullptr, (int*)nullptr,
                                  (int)n);
  return a > b ? a : b;
}

template <class C>
void carve_rcm(C& c, int64_t n, RcmWs* w) {
  const size_t cb = cub_bytes_for(n);
  if constexpr (std::is_same<C, Carver>::value) {
    w->order = c.template take<int>(n);
    w->claim = c.template take<int>(n);
    w->par = c.template take<int>(n);
    w->rank = c.template take<int>(n);
    w->cidx = c.template take<int>(n + 1);
    w->cnt = c.template take<int>(n + 1);
    w->key = c.template take<int>(n);
    w->order2 = c.template take<int>(n);
    w->blocksum = c.template take<int>(kMaxBlocks);
    w->ctl = c.template take<Ctl>(1);
    w->cub_tmp = c.template take<char>(cb);
    w->cub_bytes = cb;
  } else {
    for (int k = 0; k < 4; ++k) c.template take<int>(n);
    for (int k = 0; k < 2; ++k) c.template take<int>(n + 1);
    for (int k = 0; k < 2; ++k) c.template take<int>(n);
    c.template take<int>(kMaxBlocks);
    c.template take<Ctl>(1);
    c.template take<char>(cb);
  }
}

}  // namespace
}  // namespace inch

using namespace inch;

extern "C" size_t inch_rcm_workspace_size(int64_t n) {
  if (n < 1) return 0;
  Sizer s;
  RcmWs w;
  carve_rcm(s, n, &w);
  return s.bytes();
}

extern "C" inch_status inch_rcm(const int64_t* rowptr, const int32_t* cols, const int32_t* degree,
                                const int64_t* seed_order, int64_t n, int64_t* rcm_order, int64_t* undo,
                                int32_t* n_levels_host, void* ws, size_t ws_bytes, cudaStream_t stream) {
  return inch_rcm_bounded(rowptr, cols, degree, seed_order, n, rcm_order, undo, n_levels_host, kBarrierPolls, ws,
                          ws_bytes, stream);
}

extern "C" inch_status inch_rcm_bounded(const int64_t* rowptr, const int32_t* cols, const int32_t* degree,
                                        const int64_t* seed_order, int64_t n, int64_t* rcm_order, int64_t* undo,
                                        int32_t* n_levels_host, uint32_t max_polls, void* ws, size_t ws_bytes,
                                        cudaStream_t stream) {
  INCH_REQUIRE(rowptr && cols && degree && seed_order && rcm_order && undo, INCH_INVALID_ARG,
               "inch_rcm: NULL argument");
  INCH_REQUIRE(n >= 1 && n < (int64_t(1) << 31), INCH_INVALID_ARG, "inch_rcm: n_atoms out of range");
  Carver c(ws, ws_bytes);
  RcmWs w;
  carve_rcm(c, n, &w);
  INCH_REQUIRE(c.ok, INCH_OOM, "inch_rcm: workspace of %zu bytes, need %zu", ws_bytes, inch_rcm_workspace_size(n));
  constexpr int kSmem = kWarps * kCap * (int)sizeof(int);
  int dev = 0, sms = 0, per_sm = 0;
  INCH_CUDA(cudaGetDevice(&dev));
  INCH_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  INCH_CUDA(cudaFuncSetAttribute(k_bfs, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  INCH_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bfs, kWarps * 32, kSmem));
  INCH_REQUIRE(per_sm >= 1, INCH_CUDA_ERROR, "inch_rcm: the BFS kernel does not fit on an SM");
  // One block per SM for small inputs (fewer blocks to wait for at a barrier: 2,000-atom
  // path 17.3 ms, with two 17.6), two where a level's rows outnumber a block's warps:
  // globules of 20,000 / 100,000 / 400,000 atoms 358 / 677 / 1,976 us with one,
  // 338 / 543 / 1,350 with two; 100,000 atoms at 15 A (800 neighbours) 2,121 and 1,596.
  const int64_t want = n > 10000 ? 2 : 1;
  const int blocks = static_cast<int>(std::min<int64_t>(std::min<int64_t>(want, per_sm) * sms, kMaxBlocks));
  const int bl = grid_for(n, 256, 148 * 16), bw = grid_for(n, 8, 148 * 16);

  INCH_CUDA(cudaMemsetAsync(w.ctl, 0, sizeof(Ctl), stream));
  INCH_CUDA(cudaMemsetAsync(w.cnt, 0, sizeof(int) * n, stream));
  // Validate the inputs that index memory: seed_order must be a permutation, rows at
  // most kCap long with in-range columns.  The kernels that follow do nothing where
  // they are not.
  k_check_seeds<<<bl, 256, 0, stream>>>(seed_order, n, w.cnt, w.ctl);
  INCH_LAUNCH_CHECK();
  k_check_rows<<<bw, 256, 0, stream>>>(rowptr, cols, n, w.ctl);
  INCH_LAUNCH_CHECK();
  k_init<<<bl, 256, 0, stream>>>(seed_order, n, w.order, w.claim, w.par, w.rank, w.ctl);
  INCH_LAUNCH_CHECK();
  k_join_few<<<bl, 256, 0, stream>>>(rowptr, cols, n, w.rank, w.par, w.ctl);
  INCH_LAUNCH_CHECK();
  k_flatten<<<bl, 256, 0, stream>>>(n, w.par, w.ctl);
  INCH_LAUNCH_CHECK();
  k_join_all<<<bw, 256, 0, stream>>>(rowptr, cols, n, w.rank, w.par, w.ctl);
  INCH_LAUNCH_CHECK();
  k_flatten<<<bl, 256, 0, stream>>>(n, w.par, w.ctl);
  INCH_LAUNCH_CHECK();
  k_roots<<<grid_for(n + 1, 256, 148 * 16), 256, 0, stream>>>(seed_order, n, w.par, w.cnt, w.ctl);
  INCH_LAUNCH_CHECK();
  size_t cb = w.cub_bytes;
  INCH_CUDA(cub::DeviceScan::ExclusiveSum(w.cub_tmp, cb, w.cnt, w.cidx, (int)(n + 1), stream));
  k_seed<<<bl, 256, 0, stream>>>(seed_order, n, w.cidx, w.order, w.claim, w.ctl);
  INCH_LAUNCH_CHECK();

  int launched = 10;                        // so far; a CUB scan or sort counts as one
  Ctl h{};
  int comps = 0;
  const int* count = w.cidx + n;
  for (int all = 1; all >= 0; --all) {
    if (all == 0) {
      INCH_CUDA(cudaMemsetAsync(w.ctl, 0, sizeof(Ctl), stream));
      k_init<<<bl, 256, 0, stream>>>(seed_order, n, w.order, w.claim, w.par, w.rank, w.ctl);
      INCH_LAUNCH_CHECK();
      ++launched;
    }
    void* args[] = {&rowptr, &cols, &degree, &seed_order, &w.par, &count, &n, &w.order, &w.claim, &w.cnt,
                    &w.blocksum, &w.ctl, &all, &max_polls};
    INCH_CUDA(cudaLaunchCooperativeKernel((const void*)k_bfs, dim3(blocks), dim3(kWarps * 32), args, kSmem, stream));
    ++launched;
    INCH_CUDA(cudaMemcpyAsync(&h, w.ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, stream));
    if (all) INCH_CUDA(cudaMemcpyAsync(&comps, count, sizeof(int), cudaMemcpyDeviceToHost, stream));
    INCH_CUDA(cudaStreamSynchronize(stream));
    INCH_REQUIRE(h.bad != 1, INCH_INVALID_ARG, "inch_rcm: seed_order is not a permutation of 0..n-1");
    INCH_REQUIRE(h.bad != 2, INCH_LIMIT, "inch_rcm: a row has more than %d neighbours", kCap);
    INCH_REQUIRE(h.bad == 0, INCH_INVALID_ARG, "inch_rcm: column index out of range");
    INCH_REQUIRE(h.flag != kTimeout, INCH_TIMEOUT, "inch_rcm: the blocks of the search lost each other");
    INCH_REQUIRE(h.flag == 0 && h.visited <= n, INCH_INVALID_ARG, "inch_rcm: adjacency lists contain duplicates");
    if (h.visited == n) {
      if (!all) comps = 1;                  // already in sequential order
      break;
    }
  }
  INCH_REQUIRE(h.visited == n, INCH_INVALID_ARG, "inch_rcm: visited %lld of %lld atoms", (long long)h.visited,
               (long long)n);
  const int* order = w.order;
  if (comps > 1) {
    k_keys<<<bl, 256, 0, stream>>>(w.order, n, w.par, w.rank, w.cidx, w.key);
    INCH_LAUNCH_CHECK();
    int bits = 1;
    while (bits < 31 && (int64_t(1) << bits) < comps) ++bits;
    cb = w.cub_bytes;
    INCH_CUDA(cub::DeviceRadixSort::SortPairs(w.cub_tmp, cb, w.key, w.cnt, w.order, w.order2, (int)n, 0, bits, stream));
    order = w.order2;
    launched += 2;
  }
  k_finish<<<bl, 256, 0, stream>>>(order, n, rcm_order, undo);
  INCH_LAUNCH_CHECK();
  last_launches = launched + 1;
  if (n_levels_host) *n_levels_host = h.levels;
  return INCH_OK;
}
