// Rips filtration on the GPU: pairwise edge enumeration, the filtration
// sort and the per-vertex adjacency.
//
// Edge enumeration (reference: kernels/edge_kernel.py:23-224) is the one
// FP32-ALU-bound stage of the pipeline: n(n-1)/2 pairs x d dimensions, two
// FP32 instructions (subtract, fused multiply-add) per pair and dimension.
// One CTA of 256 threads owns a 128 x 128 tile of the upper triangle of the
// pair matrix; both point tiles are staged in shared memory transposed
// (dimension-major, chunks of 16 dimensions) so that each thread reads its
// 8 x 8 register block with four 128-bit shared loads per dimension. The
// squared distance is accumulated in dimension order with one fused
// multiply-add per step, the arithmetic of the reference's compiled kernel.
// Hits are rare (density ~1e-4 at the benchmark sizes), so they are
// compacted with one warp-aggregated atomic on a global counter and sorted
// afterwards; the emission order does not need to be reproduced here.
#include <algorithm>
#include <cmath>

#include "edges.cuh"

namespace ph {
namespace {


__device__ __forceinline__ void tile_coords(i64 b, i64 nt, i64& I, i64& J) {
  // b-th tile of the row-major upper triangle (I <= J) of an nt x nt grid
  const double a = 2.0 * (double)nt + 1.0;
  i64 r = (i64)floor((a - sqrt(a * a - 8.0 * (double)b)) * 0.5);
  if (r < 0) r = 0;
  auto start = [nt](i64 x) { return x * nt - x * (x - 1) / 2; };
  while (r > 0 && start(r) > b) --r;
  while (start(r + 1) <= b) ++r;
  I = r;
  J = r + (b - start(r));
}

// Finds the cloud owning work item b: the last segment with tile_off <= b.
__device__ __forceinline__ int find_seg(const ph_cloud_seg* segs, int nsegs, i64 b) {
  int lo = 0, hi = nsegs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (segs[mid].tile_off <= b) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// One CTA per 128 x 128 tile of one cloud's upper triangle. Single clouds
// pass their segment by value (segs == nullptr); batches pass a device table
// of ph_cloud_seg records, ordered by tile_off. Vertex indices are written
// as global indices (vbase + local).
__global__ void __launch_bounds__(ENT, 2)
    k_edges(const float* __restrict__ pts_all, const ph_cloud_seg* __restrict__ segs, int nsegs,
            ph_cloud_seg seg0, i32* __restrict__ oi, i32* __restrict__ oj, float* __restrict__ od,
            i64 cap, unsigned long long* __restrict__ count) {
  ph::pdl_wait();
  ph::pdl_trigger();
  __shared__ EdgeTile sh;
  const ph_cloud_seg sg = segs ? segs[find_seg(segs, nsegs, (i64)blockIdx.x)] : seg0;
  const i64 n = sg.n, nt = (n + ET - 1) / ET;
  i64 I, J;
  tile_coords((i64)blockIdx.x - sg.tile_off, nt, I, J);
  edge_tile(sh, pts_all + sg.pt_off, n, sg.d, sg.thr_sq, I * ET, J * ET, cap, count,
            [&](unsigned long long at, i64 gi, i64 gj, float dsq) {
              oi[at] = (i32)(sg.vbase + gi);
              oj[at] = (i32)(sg.vbase + gj);
              od[at] = dsq;
            });
}

// ---- filtration sort -------------------------------------------------------
__global__ void k_edge_keys(const i32* __restrict__ ei, const i32* __restrict__ ej,
                            const float* __restrict__ dsq, i64 E, u64* __restrict__ keys,
                            u32* __restrict__ vals) {
  ph::pdl_wait();
  ph::pdl_trigger();
  for (i64 e = (i64)blockIdx.x * blockDim.x + threadIdx.x; e < E; e += (i64)gridDim.x * blockDim.x) {
    const u64 i = (u64)ei[e], j = (u64)ej[e];
    const u64 colex = j * (j - 1) / 2 + i;
    keys[e] = ((u64)float_bits(dsq[e]) << 32) | (colex & 0xffffffffull);
    vals[e] = (u32)e;
  }
}

// Position of pair (i, j), i < j, in the reference kernel's emission order:
// tiles of 32 points row-major over (I, J), row-major inside the tile.
__device__ __forceinline__ u64 emission_order(u64 i, u64 j, u64 nb32) {
  return (((i >> 5) * nb32 + (j >> 5)) << 10) | ((i & 31) << 5) | (j & 31);
}

// Runs of equal packed keys (possible only when the 32-bit colex part wraps,
// n > 92682) are put into emission order, which is what the reference's
// stable argsort of its emitted edge list produces.
__global__ void k_fix_ties(const u64* __restrict__ keys, u32* __restrict__ vals,
                           const i32* __restrict__ ei, const i32* __restrict__ ej, i64 E, u64 nb32) {
  ph::pdl_wait();
  ph::pdl_trigger();
  for (i64 p = (i64)blockIdx.x * blockDim.x + threadIdx.x; p < E; p += (i64)gridDim.x * blockDim.x) {
    const bool starts = (p == 0 || keys[p - 1] != keys[p]) && (p + 1 < E && keys[p + 1] == keys[p]);
    if (!starts) continue;
    i64 q = p + 1;
    while (q < E && keys[q] == keys[p]) ++q;
    for (i64 a = p + 1; a < q; ++a) {  // insertion sort of the run (runs are tiny)
      const u32 v = vals[a];
      const u64 ov = emission_order((u64)ei[v], (u64)ej[v], nb32);
      i64 b = a - 1;
      while (b >= p) {
        const u32 w = vals[b];
        if (emission_order((u64)ei[w], (u64)ej[w], nb32) <= ov) break;
        vals[b + 1] = w;
        --b;
      }
      vals[b + 1] = v;
    }
  }
}

__global__ void k_gather_edges(const u32* __restrict__ perm, const i32* __restrict__ ei,
                               const i32* __restrict__ ej, const float* __restrict__ dsq, i64 E,
                               i32* __restrict__ oi, i32* __restrict__ oj, float* __restrict__ od) {
  ph::pdl_wait();
  ph::pdl_trigger();
  for (i64 e = (i64)blockIdx.x * blockDim.x + threadIdx.x; e < E; e += (i64)gridDim.x * blockDim.x) {
    const u32 s = perm[e];
    oi[e] = ei[s];
    oj[e] = ej[s];
    od[e] = dsq[s];
  }
}

// ---- vertex CSR ---------------------------------------------------------------
// half-edge keys (vertex << sh) | neighbour, sh = the bits of a vertex index
__global__ void k_half_keys(const i32* __restrict__ ei, const i32* __restrict__ ej, i64 E, int sh,
                            u64* __restrict__ keys, u32* __restrict__ vals) {
  ph::pdl_wait();
  ph::pdl_trigger();
  for (i64 e = (i64)blockIdx.x * blockDim.x + threadIdx.x; e < E; e += (i64)gridDim.x * blockDim.x) {
    const u64 i = (u64)(u32)ei[e], j = (u64)(u32)ej[e];
    keys[2 * e] = (i << sh) | j;
    vals[2 * e] = (u32)e;
    keys[2 * e + 1] = (j << sh) | i;
    vals[2 * e + 1] = (u32)e;
  }
}

__global__ void k_csr_fill(const u64* __restrict__ keys, const u32* __restrict__ vals, i64 H, i64 n, int sh,
                           i32* __restrict__ ptr, i32* __restrict__ idx, i32* __restrict__ rank) {
  ph::pdl_wait();
  ph::pdl_trigger();
  const u64 low = (1ull << sh) - 1;
  for (i64 p = (i64)blockIdx.x * blockDim.x + threadIdx.x; p < H; p += (i64)gridDim.x * blockDim.x) {
    const u64 k = keys[p];
    const i64 s = (i64)(k >> sh);
    idx[p] = (i32)(k & low);
    rank[p] = (i32)vals[p];
    const i64 prev = p ? (i64)(keys[p - 1] >> sh) : -1;
    for (i64 v = prev + 1; v <= s; ++v) ptr[v] = (i32)p;
    if (p == H - 1)
      for (i64 v = s + 1; v <= n; ++v) ptr[v] = (i32)H;
  }
}

// ---- adjacency without a sort of all half-edges ----------------------------------------
// Degrees are counted (the counter's old value is the half-edge's slot in its
// row), scanned, the half-edges (neighbour << 32 | 2 rank + side) scattered to
// their rows, and each row sorted where it lies: three passes over memory
// instead of a radix sort's two per digit. Slots come from atomics, in any
// order; the keys of a row differ (the side bit tells a self-loop's two), so
// the sorted row is the same whatever it was.
// Radix sort -> this form: 20,000 vertices, 48,000 edges 57 -> 30 us; 1500,
// 158,000 68 -> 42; 50,000, 300,000 109 -> 47; 200,000, 330,000 134 -> 35;
// 186,000, 11M 3242 -> 944 (the row sorts' 64-bit exchanges; else bound by the
// atomics' and the scattered stores' sectors).
constexpr int CSR_NT = 256;
constexpr int CSR_WARP = 1024;    // entries a warp sorts in its registers
constexpr int CSR_BIG_NT = 1024;
constexpr int CSR_BLOCK = 16384;  // entries a block sorts in shared memory
constexpr int CSR_RANGE = 32768;  // neighbours a block counts at a time in a longer row
constexpr int CSR_FEW = 32;       // entries of one neighbour that a thread puts in order
constexpr int CSR_RUN = 4096;     // and that a warp does
constexpr u64 CSR_NONE = ~0ull;
// half-edges: fewer are sorted by one cluster in less time than these six or
// seven launches (16,000 edges 25 us by the sort, 36 us here; 24,000: 30, 31;
// 48,000: 45, 30)
constexpr i64 CSR_MIN = 48 * 1024;

__device__ __forceinline__ i32 csr_rank(u64 half) { return (i32)((u32)half >> 1); }

// A place in v's row, by a whole warp (v < 0: none). Where most lanes hold the
// vertex of the lane before them (edges of one vertex in a run), lanes of one
// vertex count together: the atomics of one address are served one by one.
__device__ __forceinline__ int csr_place(i32 v, i32* __restrict__ cnt) {
  const int lane = threadIdx.x & 31;
  const i32 up = __shfl_up_sync(0xffffffffu, v, 1);
  if (__popc(__ballot_sync(0xffffffffu, lane > 0 && v == up)) < 16) return v >= 0 ? atomicAdd(&cnt[v], 1) : 0;
  const u32 same = __match_any_sync(0xffffffffu, v);
  const int first = __ffs(same) - 1;
  int at = 0;
  if (lane == first && v >= 0) at = atomicAdd(&cnt[v], __popc(same));
  return __shfl_sync(0xffffffffu, at, first) + __popc(same & lanemask_lt());
}

__global__ void k_csr_count(const i32* __restrict__ ei, const i32* __restrict__ ej, i64 E, i32* __restrict__ cnt,
                            int2* __restrict__ slot) {
  ph::pdl_wait();
  ph::pdl_trigger();
  const i64 first = (i64)blockIdx.x * blockDim.x + threadIdx.x - (threadIdx.x & 31);
  for (i64 e0 = first; e0 < E; e0 += (i64)gridDim.x * blockDim.x) {
    const i64 e = e0 + (threadIdx.x & 31);
    const int a = csr_place(e < E ? ei[e] : -1, cnt), b = csr_place(e < E ? ej[e] : -1, cnt);
    if (e < E) slot[e] = make_int2(a, b);
  }
}

__global__ void k_csr_scatter(const i32* __restrict__ ei, const i32* __restrict__ ej, i64 E,
                              const i32* __restrict__ ptr, const int2* __restrict__ slot, u64* __restrict__ half) {
  ph::pdl_wait();
  ph::pdl_trigger();
  for (i64 e = (i64)blockIdx.x * blockDim.x + threadIdx.x; e < E; e += (i64)gridDim.x * blockDim.x) {
    const i32 i = ei[e], j = ej[e];
    const int2 at = slot[e];
    half[ptr[i] + at.x] = (u64)(u32)j << 32 | (u64)(2 * e);
    half[ptr[j] + at.y] = (u64)(u32)i << 32 | (u64)(2 * e + 1);
  }
}

// bitonic sort of len2 (a power of two) keys by threads t of T
template <typename Sync>
__device__ __forceinline__ void csr_bitonic(u64* key, int len2, int t, int T, Sync sync) {
  for (int k = 2; k <= len2; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int p = t; p < len2 / 2; p += T) {
        const int a = 2 * p - (p & (j - 1)), b = a + j;  // a without bit j, b with it
        const u64 x = key[a], y = key[b];
        if ((x > y) == ((a & k) == 0)) {
          key[a] = y;
          key[b] = x;
        }
      }
      sync();
    }
}

__device__ __forceinline__ void csr_order(u64& lo, u64& hi, bool up) {
  const u64 a = lo, b = hi;
  const bool swap = (a > b) == up;
  lo = swap ? b : a;
  hi = swap ? a : b;
}

// One row of up to 32 K entries by a warp: a bitonic network over K registers
// a lane (entry lane K + k), whose steps inside a lane need no shuffle, then
// through the warp's shared memory (a pad word a lane) to coalesced stores.
template <int K>
__device__ __noinline__ void csr_warp_row(const u64* __restrict__ half, int len, i32* __restrict__ idx,
                                          i32* __restrict__ rank, u64* buf) {
  const int lane = threadIdx.x & 31;
  u64 x[K];
#pragma unroll
  for (int k = 0; k < K; ++k) x[k] = k * 32 + lane < len ? half[k * 32 + lane] : CSR_NONE;
  // runs of K: alternately up and down, the last stage by lane
#pragma unroll
  for (int size = 2; size <= K; size <<= 1)
#pragma unroll
    for (int j = size >> 1; j > 0; j >>= 1)
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (!(k & j)) csr_order(x[k], x[k + j], size < K ? !(k & size) : !(lane & 1));
  for (int m = 2; m <= 32; m <<= 1) {  // runs of m lanes
    const bool up = !(lane & m);
    for (int o = m >> 1; o > 0; o >>= 1) {
      const bool small = !(lane & o) == up;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const u64 y = __shfl_xor_sync(0xffffffffu, x[k], o);
        x[k] = (x[k] < y) == small ? x[k] : y;
      }
    }
#pragma unroll
    for (int j = K >> 1; j > 0; j >>= 1)
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (!(k & j)) csr_order(x[k], x[k + j], up);
  }
#pragma unroll
  for (int k = 0; k < K; ++k) buf[lane * (K + 1) + k] = x[k];
  __syncwarp();
  for (int p = lane; p < len; p += 32) {
    const u64 y = buf[(p / K) * (K + 1) + p % K];
    idx[p] = (i32)(y >> 32);
    rank[p] = csr_rank(y);
  }
  __syncwarp();
}

// a row of up to 32 entries: each key's place is the count of smaller ones
__device__ __forceinline__ void csr_short_row(const u64* __restrict__ half, int len, i32* __restrict__ idx,
                                              i32* __restrict__ rank) {
  const int lane = threadIdx.x & 31;
  const u64 x = lane < len ? half[lane] : CSR_NONE;
  int at = 0;
  for (int k = 0; k < len; ++k) at += __shfl_sync(0xffffffffu, x, k) < x;
  if (lane < len) {
    idx[at] = (i32)(x >> 32);
    rank[at] = csr_rank(x);
  }
}

// Short rows, for an average of up to 8 a row: up to 8 entries by 8 lanes, four
// rows a warp at once, up to 32 by the warp; longer ones are listed.
__global__ void __launch_bounds__(CSR_NT) k_csr_short(const u64* __restrict__ half, const i32* __restrict__ ptr, i64 n,
                                                      i32* __restrict__ idx, i32* __restrict__ rank,
                                                      i32* __restrict__ list, i32* __restrict__ nlist) {
  ph::pdl_wait();
  ph::pdl_trigger();
  const int lane = threadIdx.x & 31, l8 = lane & 7;
  const i64 stride = ((i64)gridDim.x * CSR_NT >> 5) * 4;
  for (i64 v0 = (((i64)blockIdx.x * CSR_NT + threadIdx.x) >> 5) * 4; v0 < n; v0 += stride) {
    const i64 v = v0 + (lane >> 3);
    const int s = v < n ? ptr[v] : 0, len = v < n ? ptr[v + 1] - s : 0;
    const bool mine = len <= 8 && l8 < len;
    const u64 x = mine ? half[s + l8] : CSR_NONE;
    int at = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) at += __shfl_sync(0xffffffffu, x, k, 8) < x;
    if (mine) {
      idx[s + at] = (i32)(x >> 32);
      rank[s + at] = csr_rank(x);
    }
    if (l8 == 0 && len > 32) list[atomicAdd(nlist, 1)] = (i32)v;
    for (u32 todo = __ballot_sync(0xffffffffu, l8 == 0 && len > 8 && len <= 32); todo; todo &= todo - 1) {
      const int from = __ffs(todo) - 1;
      const int rs = __shfl_sync(0xffffffffu, s, from), rl = __shfl_sync(0xffffffffu, len, from);
      csr_short_row(half + rs, rl, idx + rs, rank + rs);
    }
  }
}

// A warp a row of up to CSR_WARP entries: those listed, or (no list) all n;
// longer ones are listed for k_csr_big, in one list from both its ends.
__global__ void __launch_bounds__(CSR_NT) k_csr_rows(const u64* __restrict__ half, const i32* __restrict__ ptr, i64 n,
                                                     const i32* __restrict__ list, const i32* __restrict__ nlist,
                                                     i32* __restrict__ idx, i32* __restrict__ rank,
                                                     i32* __restrict__ big, i32* __restrict__ nbig,
                                                     i32* __restrict__ longs, i32* __restrict__ nlongs) {
  ph::pdl_wait();
  ph::pdl_trigger();
  extern __shared__ u64 key[];
  u64* buf = key + (size_t)(threadIdx.x >> 5) * (CSR_WARP + 32);
  const i64 count = list ? *nlist : n, stride = (i64)gridDim.x * CSR_NT >> 5;
  for (i64 r = ((i64)blockIdx.x * CSR_NT + threadIdx.x) >> 5; r < count; r += stride) {
    const i64 v = list ? list[r] : r;
    const int s = ptr[v], len = ptr[v + 1] - s;
    if (len <= 32)
      csr_short_row(half + s, len, idx + s, rank + s);
    else if (len <= 64)
      csr_warp_row<2>(half + s, len, idx + s, rank + s, buf);
    else if (len <= 128)
      csr_warp_row<4>(half + s, len, idx + s, rank + s, buf);
    else if (len <= 256)
      csr_warp_row<8>(half + s, len, idx + s, rank + s, buf);
    else if (len <= 512)
      csr_warp_row<16>(half + s, len, idx + s, rank + s, buf);
    else if (len <= CSR_WARP)
      csr_warp_row<32>(half + s, len, idx + s, rank + s, buf);
    else if ((threadIdx.x & 31) == 0) {
      if (len <= CSR_BLOCK) big[atomicAdd(nbig, 1)] = (i32)v;
      else longs[-atomicAdd(nlongs, 1)] = (i32)v;
    }
  }
}

// The entries of one row whose neighbours are in [lo, lo + CSR_RANGE), to their
// places, by a block: counted, with those of smaller neighbours, and placed from
// the counters' scan; the entries of one neighbour (repeated edges) are then put
// in rank order: a few by a thread, up to CSR_RUN by a warp, more by the block,
// since an edge may be given any number of times and one thread's moves grow
// with its square.
__device__ void csr_range(const u64* __restrict__ half, int s, int len, i64 lo, i32* cnt, i32* __restrict__ idx,
                          i32* __restrict__ rank) {
  __shared__ int sums[32];
  __shared__ int before_lo, pick, run[2];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  for (int k = t; k < CSR_RANGE; k += CSR_BIG_NT) cnt[k] = 0;
  if (t == 0) before_lo = 0;
  __syncthreads();
  int below = 0;
#pragma unroll 4
  for (int p = t; p < len; p += CSR_BIG_NT) {
    const i64 w = (i64)(half[s + p] >> 32) - lo;
    below += w < 0;
    if (w >= 0 && w < CSR_RANGE) atomicAdd(&cnt[w], 1);
  }
  below = __reduce_add_sync(0xffffffffu, below);
  if (lane == 0 && below) atomicAdd(&before_lo, below);
  __syncthreads();
  // each thread's CSR_RANGE / CSR_BIG_NT counters, the threads' sums, then starts in place of counts
  constexpr int PER = CSR_RANGE / CSR_BIG_NT;
  int sum = 0;
  for (int k = 0; k < PER; ++k) sum += cnt[t * PER + k];
  int incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) sums[warp] = incl;
  __syncthreads();
  const int done = s + before_lo;
  int before = 0;
  for (int w = 0; w < warp; ++w) before += sums[w];
  int at = done + before + incl - sum;
  for (int k = 0; k < PER; ++k) {
    const int c = cnt[t * PER + k];
    cnt[t * PER + k] = at;
    at += c;
  }
  __syncthreads();
#pragma unroll 4
  for (int p = t; p < len; p += CSR_BIG_NT) {
    const u64 x = half[s + p];
    const i64 w = (i64)(x >> 32) - lo;
    if (w >= 0 && w < CSR_RANGE) {
      const int o = atomicAdd(&cnt[w], 1);
      idx[o] = (i32)(x >> 32);
      rank[o] = csr_rank(x);
    }
  }
  __syncthreads();
  // cnt[w] is now the end of w's entries, which are put in rank order
  static_assert(PER == 32, "a bit a counter");
  u32 many = 0;  // the thread's neighbours left to the block
  for (int k = 0; k < PER; ++k) {
    const int w = t * PER + k, end = cnt[w], start = w ? cnt[w - 1] : done;
    if (end - start <= CSR_FEW)
      for (int a = start + 1; a < end; ++a) {
        const i32 x = rank[a];
        int b = a;
        for (; b > start && rank[b - 1] > x; --b) rank[b] = rank[b - 1];
        rank[b] = x;
      }
    many |= (end - start > CSR_RUN ? 1u : 0u) << k;
    for (u32 todo = __ballot_sync(0xffffffffu, end - start > CSR_FEW && end - start <= CSR_RUN); todo; todo &= todo - 1) {
      const int l = __ffs(todo) - 1;
      const int rs = __shfl_sync(0xffffffffu, start, l), re = __shfl_sync(0xffffffffu, end, l);
      bitonic_group(rank + rs, re - rs, lane, 32, [] { __syncwarp(); });
    }
  }
  while (__syncthreads_or(many != 0)) {
    if (many) pick = t;  // one of them
    __syncthreads();
    if (pick == t) {
      const int w = t * PER + __ffs(many) - 1;
      many &= many - 1;
      run[0] = w ? cnt[w - 1] : done;
      run[1] = cnt[w];
    }
    __syncthreads();
    bitonic_group(rank + run[0], run[1] - run[0], t, CSR_BIG_NT, [] { __syncthreads(); });
  }
}

// Rows beyond CSR_WARP: a block a row in shared memory up to CSR_BLOCK entries
// (big); longer ones (longs, descending from the list's end) by counting, a
// block a range of CSR_RANGE neighbours, so that one long row is shared by many
// blocks (no row is too long). One vertex joined to 2,000,000 others: 0.56 ms
// by the radix sort, 38 by one block a row, 0.66 this way and with k_csr_count's
// joint counts; 40 joined to 99,000 each: 1.05, 3.04, 0.50.
__global__ void __launch_bounds__(CSR_BIG_NT) k_csr_big(const u64* __restrict__ half, const i32* __restrict__ ptr,
                                                        i64 n, i32* __restrict__ idx, i32* __restrict__ rank,
                                                        const i32* __restrict__ big, const i32* __restrict__ nbig,
                                                        const i32* __restrict__ longs,
                                                        const i32* __restrict__ nlongs) {
  ph::pdl_wait();
  ph::pdl_trigger();
  extern __shared__ u64 key[];
  const int t = threadIdx.x;
  for (int r = blockIdx.x; r < *nbig; r += gridDim.x) {
    const i32 v = big[r];
    const int s = ptr[v], len = ptr[v + 1] - s;
    int len2 = 2 * CSR_WARP;
    while (len2 < len) len2 <<= 1;
    for (int k = t; k < len2; k += CSR_BIG_NT) key[k] = k < len ? half[s + k] : CSR_NONE;
    __syncthreads();
    csr_bitonic(key, len2, t, CSR_BIG_NT, [] { __syncthreads(); });
    for (int k = t; k < len; k += CSR_BIG_NT) {
      idx[s + k] = (i32)(key[k] >> 32);
      rank[s + k] = csr_rank(key[k]);
    }
    __syncthreads();
  }
  const i64 ranges = (n + CSR_RANGE - 1) / CSR_RANGE, items = *nlongs * ranges;
  for (i64 q = blockIdx.x; q < items; q += gridDim.x) {
    const i32 v = longs[-(q / ranges)];
    csr_range(half, ptr[v], ptr[v + 1] - ptr[v], (q % ranges) * CSR_RANGE, reinterpret_cast<i32*>(key), idx, rank);
    __syncthreads();
  }
}

__global__ void k_sqrt(const float* __restrict__ in, float* __restrict__ out, i64 n) {
  ph::pdl_wait();
  ph::pdl_trigger();
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x)
    out[i] = __fsqrt_rn(in[i]);
}

inline int grid_for(i64 n, int nt = 256) { return (int)std::max<i64>(1, std::min<i64>((n + nt - 1) / nt, 148 * 16)); }

}  // namespace
}  // namespace ph

using namespace ph;

extern "C" int ph_edges_enumerate(const float* pts, int64_t n, int32_t d, float thr_sq, int32_t* out_i,
                                  int32_t* out_j, float* out_dsq, int64_t capacity,
                                  unsigned long long* d_count, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (n < 0 || d <= 0 || capacity < 0 || !d_count) return PH_ERR_ARG;
  if (n >= (int64_t(1) << 31)) return PH_ERR_OVERFLOW;
  ph::zero_async(d_count, sizeof(unsigned long long), s);
  if (n >= 2) {
    const i64 nt = (n + ET - 1) / ET;
    const i64 tiles = nt * (nt + 1) / 2;
    if (tiles >= (int64_t(1) << 31)) return PH_ERR_OVERFLOW;
    ph_cloud_seg seg{};
    seg.n = (int32_t)n;
    seg.d = d;
    seg.thr_sq = thr_sq;
    ph::count_launch();
    ph::launch_pdl(k_edges, dim3((unsigned)tiles), dim3(ENT), 0, s, pts, nullptr, 1, seg, out_i, out_j, out_dsq, capacity, d_count);
  }
  PH_CHECK_LAUNCH();
  return PH_OK;
}

extern "C" int64_t ph_cloud_tiles(int64_t n) {
  if (n < 2) return 0;
  const i64 nt = (n + ET - 1) / ET;
  return nt * (nt + 1) / 2;
}

extern "C" int ph_batch_edges_enumerate(const float* pts, const ph_cloud_seg* segs, int32_t nsegs,
                                        int64_t ntiles, int32_t* out_i, int32_t* out_j, float* out_dsq,
                                        int64_t capacity, unsigned long long* d_count, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (nsegs < 0 || ntiles < 0 || capacity < 0 || !d_count) return PH_ERR_ARG;
  if (ntiles >= (int64_t(1) << 31)) return PH_ERR_OVERFLOW;
  ph::zero_async(d_count, sizeof(unsigned long long), s);
  if (nsegs > 0 && ntiles > 0) {
    ph::count_launch();
    ph::launch_pdl(k_edges, dim3((unsigned)ntiles), dim3(ENT), 0, s, pts, segs, nsegs, ph_cloud_seg{}, out_i, out_j, out_dsq, capacity,
                                             d_count);
  }
  PH_CHECK_LAUNCH();
  return PH_OK;
}

extern "C" size_t ph_edges_sort_workspace_bytes(int64_t E) {
  return Carve::need((size_t)E * 8) + Carve::need((size_t)E * 4) + radix_sort_workspace_bytes(E);
}

extern "C" int ph_edges_sort(const int32_t* in_i, const int32_t* in_j, const float* in_dsq, int64_t E,
                             int64_t n, int32_t* out_i, int32_t* out_j, float* out_dsq, void* workspace,
                             size_t workspace_bytes, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (E < 0 || E >= (int64_t(1) << 31)) return PH_ERR_OVERFLOW;
  if (E == 0) return PH_OK;
  const int rc = ph::cluster_sort_edges(in_i, in_j, in_dsq, E, n, out_i, out_j, out_dsq, s);
  if (rc != ph::CLUSTER_SORT_NA) return rc;
  Carve c(workspace, workspace_bytes);
  u64* keys = c.take<u64>(E);
  u32* vals = c.take<u32>(E);
  void* rws = c.take<char>((i64)radix_sort_workspace_bytes(E));
  if (!keys || !vals || !rws) return PH_ERR_ARG;
  ph::count_launch();
  ph::launch_pdl(k_edge_keys, dim3(grid_for(E)), dim3(256), 0, s, in_i, in_j, in_dsq, E, keys, vals);
  PH_TRY(radix_sort_pairs(keys, vals, E, 0, 64, rws, radix_sort_workspace_bytes(E), s));
  if (n > 92682) {
    ph::count_launch();
    ph::launch_pdl(k_fix_ties, dim3(grid_for(E)), dim3(256), 0, s, keys, vals, in_i, in_j, E, (u64)((n + 31) / 32));
  }
  ph::count_launch();
  ph::launch_pdl(k_gather_edges, dim3(grid_for(E)), dim3(256), 0, s, vals, in_i, in_j, in_dsq, E, out_i, out_j, out_dsq);
  PH_CHECK_LAUNCH();
  return PH_OK;
}

extern "C" size_t ph_vertex_csr_workspace_bytes(int64_t E) {
  return Carve::need((size_t)E * 16) + Carve::need((size_t)E * 8) + radix_sort_workspace_bytes(2 * E);
}

extern "C" int ph_vertex_csr(const int32_t* edge_i, const int32_t* edge_j, int64_t E, int64_t n,
                             int32_t* adj_ptr, int32_t* adj_idx, int32_t* adj_rank, void* workspace,
                             size_t workspace_bytes, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (E < 0 || 2 * E >= (int64_t(1) << 31) || n < 0) return PH_ERR_OVERFLOW;
  if (E == 0) {
    ph::zero_async(adj_ptr, sizeof(int32_t) * (n + 1), s);
    PH_CHECK_LAUNCH();
    return PH_OK;
  }
  Carve c(workspace, workspace_bytes);
  u64* keys = c.take<u64>(2 * E);
  u32* vals = c.take<u32>(2 * E);
  const Carve rest = c;
  void* rws = c.take<char>((i64)radix_sort_workspace_bytes(2 * E));
  if (!keys || !vals || !rws) return PH_ERR_ARG;
  // the counts, the scan's parts and the list of long rows lie where the radix
  // sort's buffers would; vertices far beyond the edges do not fit there
  Carve w = rest;
  i32* cnt = w.take<i32>(n + 4);
  const i64 nlist_big = 2 * E / CSR_WARP + 1;
  i32* big = w.take<i32>(nlist_big);
  void* sws = w.take<char>((i64)scan_workspace_bytes(n));
  i32* list = w.take<i32>(2 * E / 32 + 1);
  if (2 * E >= CSR_MIN && cnt && big && sws && list) {
    if (ph::allow_dynamic_smem((const void*)k_csr_big) != cudaSuccess) {
      PH_CHECK_LAUNCH();
      return PH_ERR_CUDA;
    }
    int2* slot = reinterpret_cast<int2*>(vals);
    i32 *nbig = cnt + n + 1, *nlist = cnt + n + 2, *nlongs = cnt + n + 3, *longs = big + nlist_big - 1;
    ph::zero_async(cnt, sizeof(i32) * (size_t)(n + 4), s);
    ph::count_launch();
    ph::launch_pdl(k_csr_count, dim3(grid_for(E)), dim3(256), 0, s, edge_i, edge_j, E, cnt, slot);
    PH_TRY(scan_exclusive_i32_i32(cnt, adj_ptr, n, sws, scan_workspace_bytes(n), s));
    ph::count_launch();
    ph::launch_pdl(k_csr_scatter, dim3(grid_for(E)), dim3(256), 0, s, edge_i, edge_j, E, (const i32*)adj_ptr,
                   (const int2*)slot, keys);
    const bool sparse = 2 * E <= 8 * n;
    const size_t rows_smem = sizeof(u64) * (CSR_NT / 32) * (CSR_WARP + 32);
    if (ph::allow_dynamic_smem((const void*)k_csr_rows) != cudaSuccess) {
      PH_CHECK_LAUNCH();
      return PH_ERR_CUDA;
    }
    const i64 sms = ph::device_sms();
    if (sparse) {
      ph::count_launch();
      ph::launch_pdl(k_csr_short, dim3((unsigned)std::min<i64>((n + CSR_NT / 8 - 1) / (CSR_NT / 8), sms * 8)),
                     dim3(CSR_NT), 0, s, (const u64*)keys, (const i32*)adj_ptr, n, adj_idx, adj_rank, list, nlist);
    }
    const i64 rows = sparse ? std::min<i64>(n, 2 * E / 33) : n;
    ph::count_launch();
    ph::launch_pdl(k_csr_rows, dim3((unsigned)std::max<i64>(1, std::min<i64>((rows + CSR_NT / 32 - 1) / (CSR_NT / 32), sms * 2))),
                   dim3(CSR_NT), rows_smem, s, (const u64*)keys, (const i32*)adj_ptr, n,
                   (const i32*)(sparse ? list : nullptr), (const i32*)nlist, adj_idx, adj_rank, big, nbig,
                   longs, nlongs);
    // (not bounded by n: few vertices may share a long row's ranges, or have one edge many times)
    const i64 big_rows = 2 * E / (CSR_WARP + 1);
    ph::count_launch();
    ph::launch_pdl(k_csr_big, dim3((unsigned)std::max<i64>(1, std::min<i64>(big_rows, sms))),
                   dim3(CSR_BIG_NT), sizeof(u64) * CSR_BLOCK, s, (const u64*)keys, (const i32*)adj_ptr, n, adj_idx,
                   adj_rank, (const i32*)big, (const i32*)nbig, (const i32*)longs, (const i32*)nlongs);
    PH_CHECK_LAUNCH();
    return PH_OK;
  }
  // sort only the key bits a vertex pair needs: 2 x bits(n - 1), in whole bytes
  int sh = 1;
  while (sh < 32 && (int64_t(1) << sh) < n) ++sh;
  const int end_bit = std::min(64, ((2 * sh + 7) / 8) * 8);
  ph::count_launch();
  ph::launch_pdl(k_half_keys, dim3(grid_for(E)), dim3(256), 0, s, edge_i, edge_j, E, sh, keys, vals);
  PH_TRY(radix_sort_pairs(keys, vals, 2 * E, 0, end_bit, rws, radix_sort_workspace_bytes(2 * E), s));
  ph::count_launch();
  ph::launch_pdl(k_csr_fill, dim3(grid_for(2 * E)), dim3(256), 0, s, keys, vals, 2 * E, n, sh, adj_ptr, adj_idx, adj_rank);
  PH_CHECK_LAUNCH();
  return PH_OK;
}

extern "C" int ph_sqrt_f32(const float* in, float* out, int64_t count, void* stream) {
  if (count < 0) return PH_ERR_ARG;
  if (count == 0) return PH_OK;
  ph::count_launch();
  ph::launch_pdl(k_sqrt, dim3(grid_for(count)), dim3(256), 0, (cudaStream_t)stream, in, out, count);
  PH_CHECK_LAUNCH();
  return PH_OK;
}
