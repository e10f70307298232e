// H0: minimum spanning forest (reference: boruvka.py:17-113) and the H0 rows
// (persistence.py:169-192).
//
// One kernel runs all Boruvka rounds on the device. Weights are the edge ranks
// (positions), which are distinct, so the forest is unique and equals the
// reference's. Edges are taken in passes of ascending rank: the forest of a
// prefix is a part of the whole forest, so an edge of a later pass that lies
// inside one component is done with after one look, and in a dense graph,
// whose forest lies in its first few n edges, that is nearly all of them. The
// first pass takes 4 n edges, the others as many as the threads hold in
// registers (MST_SLOTS each), the next pass's edges loaded ahead.
//
// A round, three barriers: every edge between two components offers (rank <<
// 32 | the other root) to both roots with a 64-bit atomicMin, so the winning
// word names the chosen edge and the component across it; every root with an
// offer marks the edge and points to the other root (of a mutual pair only the
// larger one hooks, so no cycle can form); the roots that hooked jump along
// their parents, all at the same time, so that the hook trees collapse in a
// logarithmic number of steps. Edges carry their roots from round to round, so only roots
// need be flat during a pass; all vertices are at its end. Offer words alternate
// between two arrays by round, the idle one being cleared during the hooks.
//
// Once a single component is left, the remaining edges are not looked at.
//
// Three forms, by the barrier: one block with parents and offers in shared
// memory (a lookup costs 30 cycles instead of an L2 round trip), a 16-block
// cluster and a cooperative grid, both with them in global memory. A batch of
// clouds takes a block a cloud.
// Every loop is bounded; overruns set PH_ERR_ITER_LIMIT in the device status
// word instead of spinning.
//
// Measured, every edge looked at in every round (cluster form up to 2^18 edges,
// else a grid of 592 blocks with unions by CAS) -> this form:
//   211 vertices, 2860 edges        68 -> 17 us (block)
//   4001, 105,525                  133 -> 81 (cluster)
//   1501, 157,995                  131 -> 85 (cluster)
//   20,000, 30,966                  96 -> 68 (cluster)
//   50,021, 308,535                420 -> 166 (grid)
//   200,000, 173,484               336 -> 138 (grid)
//   200,000, 326,323               440 -> 156 (grid)
// What is left are the barriers and the L2 round trips between them (6 to 13
// rounds of 8 to 15 us), not the edges' bytes.
#include <cooperative_groups.h>

#include <mutex>

#include <algorithm>
#include <climits>

#include "pipeline.cuh"

namespace cg = cooperative_groups;

namespace ph {
namespace {

constexpr int MST_NT = 1024;
constexpr int MST_SLOTS = 8;          // edges a thread holds
// A block passes 8192 edges in 4 us and its per-vertex steps take n / 1024 turns,
// a cluster 131,072 in 15 us, the grid's barriers cost twice the cluster's. us,
// block / cluster / grid, random clouds in 8 dimensions:
//   n 500, E 16,030: 47 / 52 / 67      n 1000, E 100,059: 114 / 82 / 104
//   n 2000, E 16,063: 62 / 63 / 90     n 4000, E 31,791: 95 / 92 / 105
//   n 8000, E 15,142: 82 / 62 / 74     n 8000, E 254,958: 400 / 133 / 127
//   n 16,000, E 30,636: - / 79 / 93    n 32,000, E 70,484: - / 113 / 97
constexpr i64 MST_BLOCK_N = 8192;  // vertices that fit one block's shared memory
bool takes_block(i64 n, i64 E) { return 8 * n + E <= 40 * 1024; }
bool takes_cluster(i64 n, i64 E) { return 16 * n + E <= 360 * 1024; }
constexpr u64 NO_OFFER = ~0ull;

struct MstCtl {
  int offered;  // the last tick (round of all passes) in which some edge was live
  int hooked;   // roots that became children so far
  i32 rest[8];  // clouds of a batch left to the grid
};

// A block passes a connected cloud's edges once its first few n are done with,
// but looks at all of them where several components stay, 1 us for 1000. A
// cloud of a batch with more than MST_MANY edges, and more than an eighth of
// all, is given up after MST_TRY of them and left to the grid (0.1 ms and more a
// cloud, one after another: two clouds of 0.4M edges lose by it, 1265 -> 1365 us
// a call).
constexpr i64 MST_TRY = i64(1) << 16, MST_MANY = i64(1) << 19;
__host__ __device__ inline i64 mst_many(i64 E) { return E / 8 > MST_MANY ? E / 8 : MST_MANY; }

// barriers; any(): whether some thread passed true (tick: the same for all, new each time)
struct BlockBar {
  MstCtl* ctl;
  __device__ void sync() { __syncthreads(); }
  __device__ bool any(bool b, int) { return __syncthreads_or(b) != 0; }
};
template <typename Group>
struct GroupBar {
  Group g;
  MstCtl* ctl;
  __device__ void sync() { g.sync(); }
  __device__ bool any(bool b, int tick) {
    if (__syncthreads_or(b) && threadIdx.x == 0) *(volatile int*)&ctl->offered = tick;
    g.sync();
    return *(volatile int*)&ctl->offered == tick;
  }
};

// pointer jumping of K vertices in lockstep (their loads overlap), each left
// pointing at its root; slots < 0 are padding. A thread writes only its own
// vertices' parents, so no slower walk can put an older ancestor back.
template <int K>
__device__ __forceinline__ void flatten(volatile i32* par, const i32 (&v)[K], bool* bad) {
  i32 p[K];
#pragma unroll
  for (int k = 0; k < K; ++k) p[k] = v[k] >= 0 ? par[v[k]] : -1;
  for (int it = 0; it < (1 << 20); ++it) {
    bool moved = false;
    i32 gp[K];
#pragma unroll
    for (int k = 0; k < K; ++k) gp[k] = p[k] >= 0 ? par[p[k]] : -1;
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (gp[k] != p[k]) {
        p[k] = gp[k];
        par[v[k]] = gp[k];
        moved = true;
      }
    if (!moved) return;
  }
  *bad = true;
}

struct MstArgs {
  const i32 *ei, *ej;  // endpoints less vbase are vertices 0 .. n-1
  i64 E, n;
  i32 vbase;
  i32* minv;
  uint8_t* mst;
  i32* comp;
  i64* ncomp;
  int* status;
  int max_rounds;
  i64 give_up;  // edges after which to leave off
};

// thread t of T; false where it left off
template <typename Bar>
__device__ bool forest(Bar bar, i64 t, i64 T, const MstArgs& a, volatile i32* par, u64* offer) {
  volatile u64* voff = offer;
  const i64 n = a.n, E = a.E;
  for (i64 v = t; v < n; v += T) {
    par[v] = (i32)v;
    offer[v] = NO_OFFER;
    offer[n + v] = NO_OFFER;
    a.minv[v] = INT_MAX;
  }
  {  // the mask: bytes up to a 16-byte boundary, 16-byte stores, bytes
    const i64 head = min(E, (i64)((16 - ((uintptr_t)a.mst & 15)) & 15)), quads = (E - head) / 16;
    uint4* body = reinterpret_cast<uint4*>(a.mst + head);
    for (i64 q = t; q < quads; q += T) body[q] = make_uint4(0, 0, 0, 0);
    for (i64 e = t; e < head; e += T) a.mst[e] = 0;
    for (i64 e = head + 16 * quads + t; e < E; e += T) a.mst[e] = 0;
  }
  if (t == 0) {
    bar.ctl->offered = -1;
    bar.ctl->hooked = 0;
  }
  bool bad = false;
  i32 nu[MST_SLOTS], nv[MST_SLOTS];  // the next pass's edges
  auto load = [&](i64 lo, i64 hi) {
#pragma unroll
    for (int k = 0; k < MST_SLOTS; ++k) {
      const i64 e = lo + t + k * T;
      nu[k] = e < hi ? __ldg(a.ei + e) - a.vbase : -1;
      nv[k] = e < hi ? __ldg(a.ej + e) - a.vbase : -1;
    }
  };
  const i64 full = T * MST_SLOTS;
  i64 lo = 0, hi = min(E, min(full, max(4 * n, T)));
  load(lo, hi);
  bar.sync();
  bool one = n == 1;  // a single component: no later edge can join two
  for (int tick = 0; lo < E && !one;) {
    if (lo >= a.give_up) return false;
    i32 u[MST_SLOTS], v[MST_SLOTS];
    u32 live = 0;
#pragma unroll
    for (int k = 0; k < MST_SLOTS; ++k) {
      u[k] = nu[k];
      v[k] = nv[k];
      live |= (u[k] >= 0 ? 1u : 0u) << k;
    }
    const i64 base = lo;
    lo = hi;
    hi = min(E, lo + full);
    load(lo, hi);
    for (int round = 0;; ++round, ++tick) {
      if (round >= a.max_rounds) {  // the same for all threads
        if (t == 0) set_status(a.status, PH_ERR_ITER_LIMIT);
        return true;
      }
      // offers: the lowest-ranked edge leaving each root; parents of the
      // vertices held are flat (all at a pass's start, roots after a round)
      u64* cur = offer + (size_t)(tick & 1) * n;
      volatile u64* vcur = voff + (size_t)(tick & 1) * n;
      if (base || round) {
#pragma unroll
        for (int k = 0; k < MST_SLOTS; ++k)
          if ((live >> k) & 1u) {
            u[k] = par[u[k]];
            v[k] = par[v[k]];
          }
      }
#pragma unroll
      for (int k = 0; k < MST_SLOTS; ++k)
        if (u[k] == v[k]) live &= ~(1u << k);  // inside one component for good
#pragma unroll
      for (int k0 = 0; k0 < MST_SLOTS; k0 += 4) {
        // a read first: most offers to a busy root lose to a smaller one
        u64 ou[4], ov[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if ((live >> (k0 + k)) & 1u) {
            ou[k] = vcur[u[k0 + k]];
            ov[k] = vcur[v[k0 + k]];
          }
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if ((live >> (k0 + k)) & 1u) {
            const u64 e = (u64)(base + t + (k0 + k) * T) << 32;
            const u64 wu = e | (u32)v[k0 + k], wv = e | (u32)u[k0 + k];
            if (wu < ou[k]) atomicMin((unsigned long long*)&cur[u[k0 + k]], (unsigned long long)wu);
            if (wv < ov[k]) atomicMin((unsigned long long*)&cur[v[k0 + k]], (unsigned long long)wv);
          }
      }
      if (!bar.any(live != 0, tick)) {
        if (round) {  // every vertex to its root: the next pass's edges are met with one load
          for (i64 x0 = t; x0 < n; x0 += 4 * T) {
            i32 x[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) x[k] = x0 + k * T < n ? (i32)(x0 + k * T) : -1;
            flatten(par, x, &bad);
          }
          bar.sync();
        }
        tick += 2;  // the array of this round is the clean one, and any() takes each tick once
        break;
      }
      // hooks; the other offer array (last read in the previous round) is cleared
      u64* idle = offer + (size_t)((tick + 1) & 1) * n;
      u64 hooked = 0;  // of the thread's first 64 vertices
      int hooks = 0;
      i64 j = 0;
      for (i64 x = t; x < n; x += T, ++j) {
        if (par[x] != (i32)x) continue;
        idle[x] = NO_OFFER;
        const u64 w = vcur[x];
        if (w == NO_OFFER) continue;
        const i32 e = (i32)(w >> 32), o = (i32)(w & 0xffffffffull);
        a.mst[e] = 1;
        if ((vcur[o] >> 32) == (u64)e && o > (i32)x) continue;  // mutual choice: the larger root hooks
        par[x] = o;
        ++hooks;
        hooked |= j < 64 ? 1ull << j : 0ull;
      }
      hooks = __reduce_add_sync(0xffffffffu, hooks);
      if ((threadIdx.x & 31) == 0 && hooks) atomicAdd(&bar.ctl->hooked, hooks);
      bar.sync();
      one = *(volatile int*)&bar.ctl->hooked == n - 1;  // the same for all: next added to after a barrier
      if (one) break;
      if (j <= 64) {
        while (hooked) {
          i32 x[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            x[k] = hooked ? (i32)(t + (i64)(__ffsll((long long)hooked) - 1) * T) : -1;
            hooked &= hooked - 1;
          }
          flatten(par, x, &bad);
        }
      } else {  // more vertices a thread than the mask holds: all of them
        for (i64 x0 = t; x0 < n; x0 += 4 * T) {
          i32 x[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) x[k] = x0 + k * T < n ? (i32)(x0 + k * T) : -1;
          flatten(par, x, &bad);
        }
      }
      bar.sync();
    }
  }
  if (one) {
    for (i64 x = t; x < n; x += T) a.comp[x] = a.vbase;
    if (t == 0) atomicAdd((unsigned long long*)a.ncomp, 1ull);
    if (bad) set_status(a.status, PH_ERR_ITER_LIMIT);
    return true;
  }
  // labels: the smallest vertex of each component, and the component count.
  // Vertices ascend over the lanes, so the first lane of those with one root
  // holds the least of them.
  long long roots = 0;
  for (i64 x0 = t - (threadIdx.x & 31); x0 < n; x0 += T) {
    const i64 x = x0 + (threadIdx.x & 31);
    const i32 r = x < n ? par[x] : -1;
    const u32 same = __match_any_sync(0xffffffffu, r);
    if (r >= 0 && (same & lanemask_lt()) == 0 && (i32)x < *(volatile i32*)(a.minv + r)) atomicMin(a.minv + r, (i32)x);
    roots += r == (i32)x && x < n;
  }
  for (int o = 16; o > 0; o >>= 1) roots += __shfl_xor_sync(0xffffffffu, roots, o);
  if ((threadIdx.x & 31) == 0 && roots) atomicAdd((unsigned long long*)a.ncomp, (unsigned long long)roots);
  bar.sync();
  for (i64 x = t; x < n; x += T) a.comp[x] = a.vbase + *(volatile i32*)(a.minv + par[x]);
  if (bad) set_status(a.status, PH_ERR_ITER_LIMIT);
  return true;
}

__global__ void __launch_bounds__(MST_NT, 1) k_mst_block(const MstArgs a) {
  ph::pdl_wait();
  ph::pdl_trigger();
  extern __shared__ u64 mst_smem[];
  __shared__ MstCtl ctl;
  if (threadIdx.x == 0) *a.ncomp = 0;
  forest(BlockBar{&ctl}, (i64)threadIdx.x, (i64)MST_NT, a, reinterpret_cast<i32*>(mst_smem + 2 * a.n), mst_smem);
}

// one cloud of a batch: edges [e_off[c], e_off[c + 1]), vertices from its segment
__device__ __forceinline__ MstArgs cloud_args(MstArgs a, const i64* __restrict__ e_off,
                                              const ph_cloud_seg* __restrict__ segs, int c) {
  const i64 e0 = e_off[c];
  const ph_cloud_seg g = segs[c];
  a.ei += e0;
  a.ej += e0;
  a.E = e_off[c + 1] - e0;
  a.n = g.n;
  a.vbase = (i32)g.vbase;
  a.minv += g.vbase;
  a.mst += e0;
  a.comp += g.vbase;
  return a;
}

// a block a cloud; ncomp and nrest start at zero
__global__ void __launch_bounds__(MST_NT, 1) k_mst_clouds(const MstArgs all, const i64* __restrict__ e_off,
                                                          const ph_cloud_seg* __restrict__ segs, MstCtl* rest,
                                                          int* nrest) {
  ph::pdl_wait();
  ph::pdl_trigger();
  extern __shared__ u64 mst_smem[];
  __shared__ MstCtl ctl;
  MstArgs a = cloud_args(all, e_off, segs, blockIdx.x);
  a.give_up = a.E > mst_many(all.E) ? MST_TRY : LLONG_MAX;
  const bool done = forest(BlockBar{&ctl}, (i64)threadIdx.x, (i64)MST_NT, a, reinterpret_cast<i32*>(mst_smem + 2 * a.n), mst_smem);
  if (!done && threadIdx.x == 0) rest->rest[atomicAdd(nrest, 1)] = blockIdx.x;  // fewer than eight
}

__global__ void __launch_bounds__(MST_NT, 1) k_mst_cluster(const MstArgs a, i32* par, u64* offer, MstCtl* ctl) {
  ph::pdl_wait();
  ph::pdl_trigger();
  cg::cluster_group cl = cg::this_cluster();
  if (cl.block_rank() == 0 && threadIdx.x == 0) *a.ncomp = 0;
  forest(GroupBar<cg::cluster_group>{cl, ctl}, (i64)cl.block_rank() * MST_NT + threadIdx.x,
         (i64)cl.num_blocks() * MST_NT, a, par, offer);
}

__global__ void __launch_bounds__(MST_NT, 1) k_mst_grid(const MstArgs a, i32* par, u64* offer, MstCtl* ctl) {
  ph::pdl_wait();
  ph::pdl_trigger();
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.ncomp = 0;
  forest(GroupBar<cg::grid_group>{cg::this_grid(), ctl}, (i64)blockIdx.x * MST_NT + threadIdx.x,
         (i64)gridDim.x * MST_NT, a, par, offer);
}

// the clouds that the blocks left off, one after another
__global__ void __launch_bounds__(MST_NT, 1) k_mst_rest(const MstArgs all, const i64* __restrict__ e_off,
                                                        const ph_cloud_seg* __restrict__ segs, i32* par, u64* offer,
                                                        MstCtl* ctl, const int* nrest) {
  ph::pdl_wait();
  ph::pdl_trigger();
  cg::grid_group g = cg::this_grid();
  for (int q = 0; q < *nrest; ++q) {
    forest(GroupBar<cg::grid_group>{g, ctl}, (i64)blockIdx.x * MST_NT + threadIdx.x, (i64)gridDim.x * MST_NT,
           cloud_args(all, e_off, segs, ctl->rest[q]), par, offer);
    g.sync();
  }
}

__global__ void k_h0_rows(const float* __restrict__ filt, const uint8_t* __restrict__ mst,
                          const i32* __restrict__ pos, i64 E, i64 n, float* __restrict__ rows) {
  ph::pdl_wait();
  ph::pdl_trigger();
  const i64 cnt = pos[E];
  for (i64 e = (i64)blockIdx.x * blockDim.x + threadIdx.x; e < E; e += (i64)gridDim.x * blockDim.x)
    if (mst[e]) {
      rows[2 * pos[e]] = 0.0f;
      rows[2 * pos[e] + 1] = filt[e];
    }
  for (i64 r = cnt + (i64)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (i64)gridDim.x * blockDim.x) {
    rows[2 * r] = 0.0f;
    rows[2 * r + 1] = __int_as_float(0x7f800000);
  }
}

}  // namespace
}  // namespace ph

using namespace ph;

namespace {

// Cluster size of the cluster form on the current device (16 where a 16-block
// cluster of this kernel can be resident, else 8, 0 when neither can). The
// function attribute belongs to a device, so it is set, and the answer
// cached, once per device.
int cluster_size() {
  static std::mutex mu;
  static int cached[64];
  static bool known[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    cudaGetLastError();
    return 0;
  }
  std::lock_guard<std::mutex> lock(mu);
  if (known[dev]) return cached[dev];
  known[dev] = true;
  cached[dev] = 0;
  cudaFuncSetAttribute((const void*)k_mst_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  for (int cs : {16, 8}) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(cs);
    cfg.blockDim = dim3(MST_NT);
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, (const void*)k_mst_cluster, &cfg) == cudaSuccess && clusters > 0) {
      cached[dev] = cs;
      break;
    }
  }
  cudaGetLastError();
  return cached[dev];
}

// a round at least halves the components that an edge still leaves
int rounds_bound(i64 n) {
  int r = 2;
  while ((i64(1) << (r - 2)) < n && r < 64) ++r;
  return r + 4;
}

size_t block_smem(i64 n) { return (size_t)n * (2 * sizeof(u64) + sizeof(i32)); }

}  // namespace

extern "C" size_t ph_boruvka_workspace_bytes(int64_t n, int64_t E) {
  (void)E;
  // parents, labels and two offer arrays
  return 2 * Carve::need((size_t)n * 4) + Carve::need(sizeof(MstCtl)) + Carve::need((size_t)n * 16);
}

extern "C" int ph_boruvka_mst(const int32_t* edge_i, const int32_t* edge_j, int64_t E, int64_t n,
                              uint8_t* mst_mask, int32_t* comp, int64_t* d_ncomp, int* d_status,
                              void* workspace, size_t workspace_bytes, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (n < 0 || E < 0 || n >= (int64_t(1) << 31) || E >= (int64_t(1) << 31)) return PH_ERR_OVERFLOW;
  if (n == 0) {
    ph::zero_async(d_ncomp, sizeof(int64_t), s);
    PH_CHECK_LAUNCH();
    return PH_OK;
  }
  Carve c(workspace, workspace_bytes);
  i32* parent = c.take<i32>(n);
  i32* minv = c.take<i32>(n);
  MstCtl* ctl = c.take<MstCtl>(1);
  u64* offer = c.take<u64>(2 * n);
  if (!parent || !minv || !ctl || !offer) return PH_ERR_ARG;
  const int max_rounds = rounds_bound(n);
  MstArgs a{edge_i, edge_j, E, n, 0, minv, mst_mask, comp, d_ncomp, d_status, max_rounds, LLONG_MAX};
  const i64 work = std::max<i64>(n, E);
  const int cs = takes_cluster(n, E) ? cluster_size() : 0;
  ph::count_launch();
  if (takes_block(n, E)) {
    if (ph::allow_dynamic_smem((const void*)k_mst_block) != cudaSuccess) {
      PH_CHECK_LAUNCH();
      return PH_ERR_CUDA;
    }
    ph::launch_pdl(k_mst_block, dim3(1), dim3(MST_NT), block_smem(n), s, a);
  } else if (cs > 0) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(cs);
    cfg.blockDim = dim3(MST_NT);
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, k_mst_cluster, a, parent, offer, ctl) != cudaSuccess) return PH_ERR_CUDA;
  } else {
    if (ph::occupancy((const void*)k_mst_grid, MST_NT, 0) < 1) return PH_ERR_CUDA;
    const i64 want = (work + 2 * MST_NT - 1) / (2 * MST_NT);
    const int blocks = (int)std::max<i64>(2, std::min<i64>(want, ph::device_sms()));
    void* args[] = {(void*)&a, (void*)&parent, (void*)&offer, (void*)&ctl};
    if (cudaLaunchCooperativeKernel((const void*)k_mst_grid, blocks, MST_NT, args, 0, s) != cudaSuccess)
      return PH_ERR_CUDA;
  }
  PH_CHECK_LAUNCH();
  return PH_OK;
}

int ph::pl::batch_forest(const i32* edge_i, const i32* edge_j, i64 E, i64 n, const i64* e_off,
                         const ph_cloud_seg* segs, int K, i64 max_n, uint8_t* mst_mask, i32* comp, i64* d_ncomp,
                         int* d_left, int* d_status, void* workspace, size_t workspace_bytes, cudaStream_t s) {
  // A block takes 1 us for 1000 edges, the grid 0.26 us for 1000 of the union's
  // (many passes, each with its rounds): blocks where the largest cloud, by its
  // share of the vertices, has less than a quarter of the edges, or where a
  // block would take it on its own. 192 clouds of 64 to 4096 points, 11.0M
  // edges: 2500 us by the grid -> 601 us. The share is a guess: a cloud that
  // turns out dense and in several components goes to the grid after all (40
  // sparse clouds and one of two times 4000 points, 16M edges: whole call 14.5 ms by the
  // grid, 16.2 by blocks alone, 6.6 this way).
  const i64 most = (i64)((double)E * max_n / n);
  if (max_n > MST_BLOCK_N || !(4 * max_n <= n || takes_block(max_n, most)))
    return ph_boruvka_mst(edge_i, edge_j, E, n, mst_mask, comp, d_ncomp, d_status, workspace, workspace_bytes, s);
  Carve c(workspace, workspace_bytes);
  i32* parent = c.take<i32>(n);
  i32* minv = c.take<i32>(n);
  MstCtl* ctl = c.take<MstCtl>(1);
  u64* offer = c.take<u64>(2 * n);
  if (!parent || !minv || !ctl || !offer) return PH_ERR_ARG;
  if (ph::allow_dynamic_smem((const void*)k_mst_clouds) != cudaSuccess) {
    PH_CHECK_LAUNCH();
    return PH_ERR_CUDA;
  }
  const MstArgs a{edge_i, edge_j, E, 0, 0, minv, mst_mask, comp, d_ncomp, d_status, rounds_bound(max_n), LLONG_MAX};
  ph::count_launch();
  ph::launch_pdl(k_mst_clouds, dim3((unsigned)K), dim3(MST_NT), block_smem(max_n), s, a, e_off, segs, ctl,
                 d_left);
  if (std::min<i64>(E, max_n * (max_n - 1) / 2) > mst_many(E)) {  // else no cloud can have been given up
    if (ph::occupancy((const void*)k_mst_rest, MST_NT, 0) < 1) return PH_ERR_CUDA;
    void* args[] = {(void*)&a, (void*)&e_off, (void*)&segs, (void*)&parent, (void*)&offer, (void*)&ctl, (void*)&d_left};
    ph::count_launch();
    if (cudaLaunchCooperativeKernel((const void*)k_mst_rest, ph::device_sms(), MST_NT, args, 0, s) != cudaSuccess)
      return PH_ERR_CUDA;
  }
  PH_CHECK_LAUNCH();
  return PH_OK;
}

extern "C" size_t ph_h0_rows_workspace_bytes(int64_t E) {
  return Carve::need((size_t)(E + 1) * 4) + scan_workspace_bytes(E);
}

extern "C" int ph_h0_rows(const float* edge_filt, const uint8_t* mst_mask, int64_t E, int64_t n,
                          float* out_rows, void* workspace, size_t workspace_bytes, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (E < 0 || n < 0) return PH_ERR_ARG;
  if (n == 0) return PH_OK;
  Carve c(workspace, workspace_bytes);
  i32* pos = c.take<i32>(E + 1);
  void* sws = c.take<char>((i64)scan_workspace_bytes(E));
  if (!pos || !sws) return PH_ERR_ARG;
  PH_TRY(scan_exclusive_u8_i32(mst_mask, pos, E, sws, scan_workspace_bytes(E), s));
  const i64 work = std::max<i64>(E, n);
  const int g = (int)std::max<i64>(1, std::min<i64>((work + 255) / 256, 148 * 8));
  ph::count_launch();
  ph::launch_pdl(k_h0_rows, dim3(g), dim3(256), 0, s, edge_filt, mst_mask, pos, E, n, out_rows);
  PH_CHECK_LAUNCH();
  return PH_OK;
}
