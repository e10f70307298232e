// Threshold estimation kernels (reference: threshold.py:20-200).
//
// auto_threshold needs the k-th nearest-neighbour distance of every point
// and a linear-interpolation quantile of those distances; enclosing_radius
// needs min over points of the max distance to any point. Both are
// all-pairs scans with squared distances accumulated in dimension order with
// fused multiply-adds (the same arithmetic as the edge kernel). The reference
// uses torch.cdist, whose matrix-product formula rounds differently, so the
// thresholds agree within a tolerance, not bit for bit.
//
// Two forms of the k-NN scan, for a single cloud or every cloud of a batch
// (segment table; a block finds its cloud from the per-cloud offsets of
// 128-point query blocks):
//  * top buffer (k <= 64): a block takes 32 queries against tiles of 128
//    candidates, a thread 4 x 8 pairs in registers, coordinates copied
//    dimension-major into shared memory in chunks of 12 dimensions (any d),
//    one chunk ahead (cp.async). A distance below its query's bound goes to
//    the query's buffer in shared memory; after the 1st, 4th, 16th, 64th ...
//    tile, and when it fills, a warp cuts a buffer to its k smallest values,
//    the largest of which is the new bound. Candidates in no order beat the
//    bound k ln(n / k) times, so the scan is the distances' arithmetic: two
//    instructions a coordinate for two pairs (sub.f32x2, fma.f32x2).
//    20,011 x 10, k = 20: 7.5 ms as one query a thread with a sorted list in
//    local memory, 0.95 ms this way (0.24 ms of it are the distances'
//    instructions at full issue; the selection and the cuts take about half);
//    the enclosing radius on the same tiles 1.30 -> 0.50 ms. Packed
//    instructions against scalar ones: 0.50 against 0.58 ms;
//  * radix select: any k, any d. A block takes 32 queries and finds each
//    query's k-th smallest squared distance bit by bit: four passes over all
//    candidates, each pass a 256-bin histogram per query (shared-memory
//    atomics) of the next 8 bits among the distances that share the bits
//    found so far. Coordinates are staged in 32-dimension chunks, so d is
//    unbounded; the four passes recompute the distances instead of storing
//    n per query.
// The reference's _tiled_knn (threshold.py:133-176) keeps a running top-k of
// cdist tiles; it clamps k to n - 1 and excludes the point itself
// (duplicates of it count, at distance 0), as both forms do.
#include <algorithm>

#include "prim.cuh"

namespace ph {
namespace {

constexpr int KN_NT = 128;   // queries per query block of the offsets
constexpr int KN_MAXK = 64;  // largest k of the top buffer

constexpr int KT_NT = 128;   // threads of a tile block (top buffer and enclosing)
constexpr int KT_QB = 32;    // queries per block
constexpr int KT_TC = 128;   // candidates per tile
constexpr int KT_DC = 12;    // dimensions per staged chunk
// buffered distances per query, by k: a cut leaves k and a tile brings up to
// KT_TC. The smaller buffer lets five blocks share an SM (20,000 queries are
// 4.2 blocks an SM: all resident); with the larger k it would be cut at every
// tile
constexpr int KT_SMALL_K = 32, KT_SMALL_CAP = 192, KT_CAP = 320;
static_assert(KT_SMALL_CAP >= KT_SMALL_K + KT_TC && KT_CAP >= KN_MAXK + KT_TC, "a tile fits a buffer that was cut");

constexpr int KS_NT = 256;           // threads of a select / enclosing block
constexpr int KS_QB = 32;            // queries per select / enclosing block
constexpr int KS_TC = 64;            // candidates per tile
constexpr int KS_DC = 32;            // dimensions per staged chunk
constexpr int KS_R = KS_TC / (KS_NT / KS_QB);  // candidates per thread per tile (8)
constexpr int KS_SUB = KN_NT / KS_QB;          // select blocks per 128-point query block (4)

__device__ __forceinline__ int seg_of_block(const i64* __restrict__ off, int nsegs, i64 x) {
  int lo = 0, hi = nsegs - 1;  // last s with off[s] <= x
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= x) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// the cloud a query block belongs to: single cloud when segs is null
struct CloudView {
  const float* pts;
  i64 n;
  int d;
  i64 qblk;     // 128-point query block within the cloud
  i64 out_off;  // output index of the cloud's first point
};

__device__ __forceinline__ CloudView cloud_view(const float* pts, i64 n, int d, const ph_cloud_seg* segs, int nsegs,
                                                const i64* qb_off, i64 block128) {
  CloudView v;
  if (!segs) {
    v.pts = pts;
    v.n = n;
    v.d = d;
    v.qblk = block128;
    v.out_off = 0;
    return v;
  }
  const int c = seg_of_block(qb_off, nsegs, block128);
  const ph_cloud_seg sg = segs[c];
  v.pts = pts + sg.pt_off;
  v.n = sg.n;
  v.d = sg.d;
  v.qblk = block128 - qb_off[c];
  v.out_off = sg.vbase;
  return v;
}

// ---- tile scan: 32 queries against tiles of 128 candidates -----------------------------
// One sub.f32x2 gives the differences of a query (twice in a register pair)
// with two candidates and one fma.f32x2 adds their squares: the roundings of
// __fsub_rn and __fmaf_rn, coordinate by coordinate.
struct PairTile {
  alignas(16) float q[2][KT_DC][KT_QB];
  alignas(16) float c[2][KT_DC][KT_TC + 4];
};

__device__ __forceinline__ u64 sub2(u64 a, u64 b) {
  u64 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
  u64 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ u64 twice(float x) {
  u64 r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void copy4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((u32)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// Scans all candidates: pairs(j0, acc) by every thread for each tile with the
// squared distances of queries q0 + 4 (t % 8) + a to candidates j0 + 8 (t / 8)
// + b in acc[a][b], a < 4, b < 8 (of no meaning past the cloud's end). The
// threads are synchronised between the calls.
template <typename F>
__device__ __forceinline__ void scan_tiles(PairTile& sh, const float* __restrict__ pts, i64 n, int d, i64 q0,
                                           F&& pairs) {
  const int t = threadIdx.x, tq = 4 * (t & 7), tc = 8 * (t >> 3);
  const bool whole = d <= KT_DC;  // one chunk: the queries are staged once
  // `count` rows from row r0 on, dimensions [d0, d0 + dc), to dst[k][row], the
  // threads along the rows so that the loads coalesce
  auto copy = [&](float* dst, int pitch, i64 r0, int count, int d0) {
    const int dc = min(KT_DC, d - d0), rows = KT_NT / dc, left = KT_NT - rows * dc;
    int r = t / dc, k = t - r * dc;
    const int end = (int)min((i64)count, n - r0);
    const float* p = pts + (r0 + r) * d + d0 + k;
    const i64 step = (i64)rows * d + left;
    while (r < end) {
      copy4(dst + k * pitch + r, p);
      r += rows;
      k += left;
      p += step;
      if (k >= dc) {
        k -= dc;
        ++r;
        p += d - dc;
      }
    }
  };
  auto stage = [&](int buf, i64 j0, int d0, bool queries) {
    copy(&sh.c[buf][0][0], KT_TC + 4, j0, KT_TC, d0);
    if (queries) copy(&sh.q[buf][0][0], KT_QB, q0, KT_QB, d0);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  stage(0, 0, 0, true);
  int buf = 0;
  for (i64 j0 = 0; j0 < n; j0 += KT_TC) {
    u64 s[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int h = 0; h < 4; ++h) s[a][h] = 0;
    for (int d0 = 0; d0 < d; d0 += KT_DC) {
      const bool last = d0 + KT_DC >= d;
      const i64 jn = last ? j0 + KT_TC : j0;
      if (jn < n) {
        stage(buf ^ 1, jn, last ? 0 : d0 + KT_DC, !whole);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
      } else {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
      __syncthreads();
      const float* q = &sh.q[whole ? 0 : buf][0][tq];
      const float* c = &sh.c[buf][0][tc];
      const int dc = min(KT_DC, d - d0);
#pragma unroll 4
      for (int k = 0; k < dc; ++k) {
        const float4 qf = *reinterpret_cast<const float4*>(q + k * KT_QB);
        const ulonglong2 c01 = *reinterpret_cast<const ulonglong2*>(c + k * (KT_TC + 4));
        const ulonglong2 c23 = *reinterpret_cast<const ulonglong2*>(c + k * (KT_TC + 4) + 4);
        const u64 qv[4] = {twice(qf.x), twice(qf.y), twice(qf.z), twice(qf.w)}, cv[4] = {c01.x, c01.y, c23.x, c23.y};
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            const u64 df = sub2(qv[a], cv[h]);
            s[a][h] = fma2(df, df, s[a][h]);
          }
      }
      __syncthreads();  // the stage is free for the copies after the next
      buf ^= 1;
    }
    float acc[4][8];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        acc[a][2 * h] = __uint_as_float((u32)s[a][h]);
        acc[a][2 * h + 1] = __uint_as_float((u32)(s[a][h] >> 32));
      }
    pairs(j0, acc);
  }
}

// The k smallest of a query's m > k buffered values (m <= 32 PER) to the
// buffer's front, by one warp; returns the k-th smallest. Non-negative floats
// order as their bits: the value is found bit by bit between the extremes.
template <int PER>
__device__ __forceinline__ float cut_values(float* buf, int m, int k) {
  const int lane = threadIdx.x & 31;
  u32 v[PER], lo = 0xffffffffu, hi = 0;
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    v[p] = lane + 32 * p < m ? __float_as_uint(buf[lane + 32 * p]) : 0xffffffffu;
    lo = min(lo, v[p]);
    if (lane + 32 * p < m) hi = max(hi, v[p]);
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  while (lo < hi) {  // the smallest value with k values at or below it
    const u32 mid = lo + ((hi - lo) >> 1);
    int c = 0;
#pragma unroll
    for (int p = 0; p < PER; ++p) c += v[p] <= mid;
    if (__reduce_add_sync(0xffffffffu, c) >= k) hi = mid;
    else lo = mid + 1;
  }
  // what is below it, and of its equals as many as make up k
  int c = 0;
#pragma unroll
  for (int p = 0; p < PER; ++p) c += v[p] < lo;
  int equal = k - __reduce_add_sync(0xffffffffu, c), at = 0;
  __syncwarp();
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    const u32 below = __ballot_sync(0xffffffffu, v[p] < lo), same = __ballot_sync(0xffffffffu, v[p] == lo);
    const u32 lt = lanemask_lt();
    if (v[p] < lo) buf[at + __popc(below & lt)] = __uint_as_float(v[p]);
    at += __popc(below);
    const int eq = min(equal, __popc(same));
    if (v[p] == lo && __popc(same & lt) < eq) buf[at + __popc(same & lt)] = __uint_as_float(lo);
    at += eq;
    equal -= eq;
  }
  __syncwarp();
  return __uint_as_float(lo);
}

template <int CAP>
__device__ __noinline__ float cut_buffer(float* buf, int m, int k) {
  if (m <= 96) return cut_values<3>(buf, m, k);
  return cut_values<CAP / 32>(buf, m, k);
}

template <int CAP>
struct KnnSmem {
  PairTile tile;
  float buf[KT_QB][CAP];
  int cnt[KT_QB];
  alignas(16) float bound[KT_QB];
};

template <int CAP>
__global__ void __launch_bounds__(KT_NT) k_knn_top(const float* __restrict__ pts_all, i64 n1, int d1,
                                                  const ph_cloud_seg* __restrict__ segs, int nsegs,
                                                  const i64* __restrict__ qb_off, int kreq, float* __restrict__ out) {
  ph::pdl_wait();
  ph::pdl_trigger();
  extern __shared__ __align__(16) unsigned char kt_smem[];
  KnnSmem<CAP>& sm = *reinterpret_cast<KnnSmem<CAP>*>(kt_smem);
  auto& buf = sm.buf;
  auto& cnt = sm.cnt;
  auto& bound = sm.bound;
  const CloudView cv = cloud_view(pts_all, n1, d1, segs, nsegs, qb_off, blockIdx.x / (KN_NT / KT_QB));
  const i64 n = cv.n;
  const int d = cv.d, k = (int)min((i64)kreq, n - 1);
  const i64 q0 = cv.qblk * KN_NT + (i64)(blockIdx.x % (KN_NT / KT_QB)) * KT_QB;
  if (q0 >= n) return;  // the whole block is past the cloud's end (uniform)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tq = 4 * (threadIdx.x & 7), tc = 8 * (threadIdx.x >> 3);
  const float inf = __int_as_float(0x7f800000);
  if (threadIdx.x < KT_QB) {
    cnt[threadIdx.x] = 0;
    bound[threadIdx.x] = inf;
  }
  i64 tile = 0;
  // (the scan synchronises before the first call: counts and bounds are set)
  scan_tiles(sm.tile, cv.pts, k >= 1 ? n : 0, d, q0, [&](i64 j0, float (&acc)[4][8]) {
    if (j0 + KT_TC > n || (j0 < q0 + KT_QB && q0 < j0 + KT_TC)) {  // points past the end, the query itself
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          const i64 j = j0 + tc + b;
          if (j >= n || j == q0 + tq + a) acc[a][b] = inf;
        }
    }
    const float4 tau4 = *reinterpret_cast<const float4*>(&bound[tq]);
    const float tau[4] = {tau4.x, tau4.y, tau4.z, tau4.w};
    // a place in the buffer for all a thread has for a query at once: the four
    // atomics are in flight together
    int c[4], total = 0;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      c[a] = 0;
#pragma unroll
      for (int b = 0; b < 8; ++b) c[a] += acc[a][b] < tau[a];
      total += c[a];
    }
    if (total) {
      int at[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) at[a] = c[a] ? atomicAdd(&cnt[tq + a], c[a]) : 0;
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 8; ++b)
          if (acc[a][b] < tau[a]) buf[tq + a][at[a]++] = acc[a][b];
    }
    ++tile;
    __syncthreads();
    const bool step = (tile & (tile - 1)) == 0 && (tile & 0x5555555555555555ll) != 0;
    for (int q = warp; q < KT_QB; q += KT_NT / 32) {
      const int m = cnt[q];
      if (m <= k || !(step || m > CAP - KT_TC)) continue;
      const float t = cut_buffer<CAP>(buf[q], m, k);
      if (lane == 0) {
        cnt[q] = k;
        bound[q] = t;
      }
    }
  });
  __syncthreads();
  for (int q = warp; q < KT_QB; q += KT_NT / 32) {
    if (q0 + q >= n) break;
    float t = inf;  // fewer than k distances are finite
    const int m = cnt[q];
    if (m > k) {
      t = cut_buffer<CAP>(buf[q], m, k);
    } else if (m == k && k >= 1) {
      t = 0.0f;
      for (int p = lane; p < m; p += 32) t = fmaxf(t, buf[q][p]);
      t = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(t)));
    }
    if (lane == 0) out[cv.out_off + q0 + q] = k >= 1 ? __fsqrt_rn(t) : 0.0f;
  }
}

// ---- chunked distance tile (select) ---------------------------------------------------
// Thread t owns query lane ql = t % 32 and candidates cg + 8 r (r < KS_R) of
// the tile, cg = t / 32 (one value per warp, so candidate reads are
// broadcasts); acc[r] receives the squared distance accumulated over all d
// dimensions in order.
struct TileSmem {
  float qs[KS_DC][KS_QB];
  float cs[KS_TC][KS_DC + 1];
};

__device__ __forceinline__ void tile_distances(const float* __restrict__ pts, i64 n, int d, i64 q0, i64 j0,
                                               TileSmem& sh, float (&acc)[KS_R]) {
  const int t = threadIdx.x, ql = t & (KS_QB - 1), cg = t / KS_QB;
#pragma unroll
  for (int r = 0; r < KS_R; ++r) acc[r] = 0.0f;
  for (int d0 = 0; d0 < d; d0 += KS_DC) {
    const int dc = min(KS_DC, d - d0);
    __syncthreads();
    for (int idx = t; idx < KS_QB * dc; idx += KS_NT) {
      const int qq = idx / dc, kk = idx - qq * dc;
      const i64 g = q0 + qq;
      sh.qs[kk][qq] = g < n ? pts[g * d + d0 + kk] : 0.0f;
    }
    for (int idx = t; idx < KS_TC * dc; idx += KS_NT) {
      const int cc = idx / dc, kk = idx - cc * dc;
      const i64 g = j0 + cc;
      sh.cs[cc][kk] = g < n ? pts[g * d + d0 + kk] : 0.0f;
    }
    __syncthreads();
    for (int kk = 0; kk < dc; ++kk) {
      const float qv = sh.qs[kk][ql];
#pragma unroll
      for (int r = 0; r < KS_R; ++r) {
        const float df = __fsub_rn(qv, sh.cs[cg + r * (KS_NT / KS_QB)][kk]);
        acc[r] = __fmaf_rn(df, df, acc[r]);
      }
    }
  }
}

// ---- radix select: any k, any d --------------------------------------------------------
__global__ void __launch_bounds__(KS_NT) k_knn_select(const float* __restrict__ pts_all, i64 n1, int d1,
                                                     const ph_cloud_seg* __restrict__ segs, int nsegs,
                                                     const i64* __restrict__ qb_off, int kreq,
                                                     float* __restrict__ out) {
  ph::pdl_wait();
  ph::pdl_trigger();
  __shared__ TileSmem sh;
  __shared__ u32 hist[KS_QB][256];
  __shared__ u32 prefix[KS_QB];
  __shared__ u32 rem[KS_QB];
  const CloudView cv = cloud_view(pts_all, n1, d1, segs, nsegs, qb_off, blockIdx.x / KS_SUB);
  const i64 n = cv.n;
  const int k = (int)min((i64)kreq, n - 1);
  const i64 q0 = cv.qblk * KN_NT + (i64)(blockIdx.x % KS_SUB) * KS_QB;
  if (q0 >= n) return;  // the whole block is past the cloud's end (uniform)
  const int t = threadIdx.x, ql = t & (KS_QB - 1), cg = t / KS_QB;
  const i64 qi = q0 + ql;
  if (t < KS_QB) {
    prefix[t] = 0;
    rem[t] = (u32)max(k, 1);
  }
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = 24 - 8 * pass;  // the bits this pass decides: [shift, shift + 8)
    for (int idx = t; idx < KS_QB * 256; idx += KS_NT) (&hist[0][0])[idx] = 0;
    for (i64 j0 = 0; j0 < n; j0 += KS_TC) {
      float acc[KS_R];
      tile_distances(cv.pts, n, cv.d, q0, j0, sh, acc);  // its first barrier orders the clears above
      if (qi < n && k >= 1) {
        const u32 pre = prefix[ql];
#pragma unroll
        for (int r = 0; r < KS_R; ++r) {
          const i64 j = j0 + cg + r * (KS_NT / KS_QB);
          const u32 b = __float_as_uint(acc[r]);
          const bool same = ((u64)b >> (shift + 8)) == (u64)pre;  // pass 0: both 0
          if (j < n && j != qi && same) atomicAdd(&hist[ql][(b >> shift) & 255u], 1u);
        }
      }
    }
    __syncthreads();
    if (t < KS_QB) {  // the bin that holds the rem-th smallest among the matching values
      u32 r = rem[t], p = prefix[t];
      int b = 0;
      for (; b < 255; ++b) {
        const u32 c = hist[t][b];
        if (r <= c) break;
        r -= c;
      }
      prefix[t] = (p << 8) | (u32)b;
      rem[t] = r;
    }
    __syncthreads();
  }
  if (t < KS_QB && qi < n) out[cv.out_off + qi] = k >= 1 ? __fsqrt_rn(__uint_as_float(prefix[t])) : 0.0f;
}

// ---- enclosing radius: any d --------------------------------------------------------------
__global__ void __launch_bounds__(KT_NT) k_enclosing(const float* __restrict__ pts, i64 n, int d,
                                                    unsigned int* __restrict__ best_bits) {
  ph::pdl_wait();
  ph::pdl_trigger();
  __shared__ PairTile sh;
  __shared__ u32 far[KT_QB];
  const i64 q0 = (i64)blockIdx.x * KT_QB;
  const int tq = 4 * (threadIdx.x & 7);
  if (threadIdx.x < KT_QB) far[threadIdx.x] = 0;
  float mx[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  scan_tiles(sh, pts, n, d, q0, [&](i64 j0, float (&acc)[4][8]) {
    const int have = (int)min((i64)8, n - j0 - 8 * (threadIdx.x >> 3));
    if (have < 8) {  // the last tile
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 8; ++b)
          if (b >= have) acc[a][b] = 0.0f;
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 8; ++b) mx[a] = fmaxf(mx[a], acc[a][b]);
  });
  __syncthreads();
#pragma unroll
  for (int a = 0; a < 4; ++a) atomicMax(&far[tq + a], __float_as_uint(mx[a]));
  __syncthreads();
  if (threadIdx.x < KT_QB && q0 + threadIdx.x < n)
    atomicMin(best_bits, __float_as_uint(__fsqrt_rn(__uint_as_float(far[threadIdx.x]))));
}

// torch.quantile (linear): rank = q * (n - 1) in float32, lerp between the
// neighbouring order statistics with torch's two-sided lerp formula.
__global__ void k_quantile(const u64* __restrict__ sorted_bits, i64 n, float qf, float* out) {
  ph::pdl_wait();
  ph::pdl_trigger();
  const float rank = __fmul_rn(qf, (float)(n - 1));
  i64 lo = (i64)rank;
  const float w = __fsub_rn(rank, (float)lo);
  i64 hi = (i64)ceilf(rank);
  lo = lo < 0 ? 0 : (lo > n - 1 ? n - 1 : lo);
  hi = hi < 0 ? 0 : (hi > n - 1 ? n - 1 : hi);
  const float a = __uint_as_float((u32)(sorted_bits[lo] >> 32));
  const float b = __uint_as_float((u32)(sorted_bits[hi] >> 32));
  float r;
  if (fabsf(w) < 0.5f) r = __fadd_rn(a, __fmul_rn(w, __fsub_rn(b, a)));
  else r = __fsub_rn(b, __fmul_rn(__fsub_rn(b, a), __fsub_rn(1.0f, w)));
  *out = r;
}

__global__ void k_float_keys(const float* __restrict__ v, i64 n, u64* __restrict__ keys, u32* __restrict__ vals) {
  ph::pdl_wait();
  ph::pdl_trigger();
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
    u32 b = __float_as_uint(v[i]);
    b = (b & 0x80000000u) ? ~b : (b | 0x80000000u);  // order-preserving for all floats
    keys[i] = (u64)b << 32;
    vals[i] = (u32)i;
  }
}

__global__ void k_unflip(u64* __restrict__ keys, i64 n) {
  ph::pdl_wait();
  ph::pdl_trigger();
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
    u32 b = (u32)(keys[i] >> 32);
    b = (b & 0x80000000u) ? (b & 0x7fffffffu) : ~b;
    keys[i] = (u64)b << 32;
  }
}

__global__ void k_enclosing_init(unsigned int* bits) {
  ph::pdl_wait();
  ph::pdl_trigger();
  *bits = 0x7f800000u;  // +inf
}

__global__ void k_bits_to_float(const unsigned int* bits, float* out) {
  ph::pdl_wait();
  ph::pdl_trigger();
  *out = __uint_as_float(*bits);
}

inline int grid_for(i64 n, int nt = 256) {
  return (int)std::max<i64>(1, std::min<i64>((n + nt - 1) / nt, 148 * 16));
}

}  // namespace

// k-NN of a single cloud (segs null) or of every cloud of a batch: the top
// buffer where it applies, the radix select otherwise. nqb: 128-point query blocks.
int knn_kth_launch(const float* pts, i64 n, int d, const ph_cloud_seg* segs, int nsegs, const i64* qb_off, i64 nqb,
                   int k, float* out, cudaStream_t s) {
  if (nqb <= 0) return PH_OK;
  if (k <= KN_MAXK) {
    const bool small = k <= KT_SMALL_K;
    const auto kernel = small ? k_knn_top<KT_SMALL_CAP> : k_knn_top<KT_CAP>;
    if (ph::allow_dynamic_smem((const void*)kernel) != cudaSuccess) {
      PH_CHECK_LAUNCH();
      return PH_ERR_CUDA;
    }
    ph::count_launch();
    ph::launch_pdl(kernel, dim3((unsigned)(nqb * (KN_NT / KT_QB))), dim3(KT_NT),
                   small ? sizeof(KnnSmem<KT_SMALL_CAP>) : sizeof(KnnSmem<KT_CAP>), s, pts, n, d, segs, nsegs, qb_off,
                   k, out);
  } else {
    ph::count_launch();
    ph::launch_pdl(k_knn_select, dim3((unsigned)(nqb * KS_SUB)), dim3(KS_NT), 0, s, pts, n, d, segs, nsegs, qb_off,
                   k, out);
  }
  PH_CHECK_LAUNCH();
  return PH_OK;
}

}  // namespace ph

using namespace ph;

extern "C" int ph_knn_kth(const float* pts, int64_t n, int32_t d, int32_t k, float* out, void* stream) {
  if (n < 0 || d <= 0 || k < 1 || (n > 0 && k > n - 1)) return PH_ERR_ARG;
  if (n == 0) return PH_OK;
  return knn_kth_launch(pts, n, d, nullptr, 0, nullptr, (n + KN_NT - 1) / KN_NT, k, out, (cudaStream_t)stream);
}

extern "C" int ph_batch_knn_kth(const float* pts, const ph_cloud_seg* segs, int32_t nsegs, const int64_t* qb_off,
                                int64_t nqb, int32_t max_d, int32_t k, float* out, void* stream) {
  if (nsegs < 1 || nqb < 0 || max_d < 1 || k < 1) return PH_ERR_ARG;
  return knn_kth_launch(pts, 0, 0, segs, nsegs, qb_off, nqb, k, out, (cudaStream_t)stream);
}

extern "C" size_t ph_quantile_workspace_bytes(int64_t n) {
  return Carve::need((size_t)n * 8) + Carve::need((size_t)n * 4) + radix_sort_workspace_bytes(n);
}

extern "C" int ph_quantile_f32(const float* values, int64_t n, double q, float* d_out, void* workspace,
                               size_t workspace_bytes, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (n <= 0 || !(q >= 0.0 && q <= 1.0)) return PH_ERR_ARG;
  Carve c(workspace, workspace_bytes);
  u64* keys = c.take<u64>(n);
  u32* vals = c.take<u32>(n);
  void* rws = c.take<char>((i64)radix_sort_workspace_bytes(n));
  if (!keys || !vals || !rws) return PH_ERR_ARG;
  ph::count_launch();
  ph::launch_pdl(k_float_keys, dim3(grid_for(n)), dim3(256), 0, s, values, n, keys, vals);
  PH_TRY(radix_sort_pairs(keys, vals, n, 32, 64, rws, radix_sort_workspace_bytes(n), s));
  ph::count_launch();
  ph::launch_pdl(k_unflip, dim3(grid_for(n)), dim3(256), 0, s, keys, n);
  ph::count_launch();
  ph::launch_pdl(k_quantile, dim3(1), dim3(1), 0, s, keys, n, (float)q, d_out);
  PH_CHECK_LAUNCH();
  return PH_OK;
}

extern "C" size_t ph_enclosing_radius_workspace_bytes(int64_t n) {
  (void)n;
  return Carve::need(sizeof(unsigned int));
}

extern "C" int ph_enclosing_radius(const float* pts, int64_t n, int32_t d, float* d_out, void* workspace,
                                   size_t workspace_bytes, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (n <= 0 || d <= 0) return PH_ERR_ARG;
  Carve c(workspace, workspace_bytes);
  unsigned int* bits = c.take<unsigned int>(1);
  if (!bits) return PH_ERR_ARG;
  ph::count_launch();
  ph::launch_pdl(k_enclosing_init, dim3(1), dim3(1), 0, s, bits);
  ph::count_launch();
  ph::launch_pdl(k_enclosing, dim3((unsigned)((n + KT_QB - 1) / KT_QB)), dim3(KT_NT), 0, s, pts, n, d, bits);
  ph::count_launch();
  ph::launch_pdl(k_bits_to_float, dim3(1), dim3(1), 0, s, bits, d_out);
  PH_CHECK_LAUNCH();
  return PH_OK;
}
