// Edge enumeration of large clouds in few dimensions (d <= NEAR_MAX_D): the
// points are put in the order of a grid, so that blocks of 128 consecutive
// points are compact, and only pairs of blocks whose bounding boxes come
// within the threshold of each other are enumerated, with the exact chain of
// ph_edges_enumerate (k_edges): the same edges with the same dist^2 bits.
//
// Reference: kernels/edge_kernel.py:23-224. The direct kernel and the
// tensor-core screen look at all n(n-1)/2 pairs; here a sparse cloud costs a
// few blocks' worth of pairs a block, and a dense one (threshold near the
// cloud's size) what the direct kernel costs.
//
// The box test is conservative: the chain C < thr implies a true squared
// distance below thr (1 + (d + 3) 2^-24), and a pair's distance is no less than
// its boxes'; their gap is taken in FP32, wrong by less than (d + 2) 2^-24
// relative, against thr (1 + 2^-16) + 2^-120. Points with coordinates that are
// not finite lie in any cell; a NaN coordinate leaves its block's box to the
// other points (its own distances are NaN, never an edge), an infinite one
// widens it (a gap of NaN keeps the pair of blocks).
#include <algorithm>
#include <climits>

#include "edges.cuh"

namespace ph {
namespace {

constexpr int NR_NT = 256;
constexpr u32 FULL = 0xffffffffu;

// order-preserving unsigned image of a float
__device__ __forceinline__ u32 ordered(float f) {
  const u32 b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float unordered(u32 u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// box[2 k] = ~least, box[2 k + 1] = largest coordinate k of the finite ones, as
// their ordered images (zero on entry)
__global__ void k_near_box(const float* __restrict__ pts, i64 n, int d, u32* __restrict__ box) {
  ph::pdl_wait();
  ph::pdl_trigger();
  u32 lo[NEAR_MAX_D], hi[NEAR_MAX_D];
#pragma unroll
  for (int k = 0; k < NEAR_MAX_D; ++k) lo[k] = hi[k] = 0u;
  for (i64 p = (i64)blockIdx.x * NR_NT + threadIdx.x; p < n; p += (i64)gridDim.x * NR_NT)
#pragma unroll
    for (int k = 0; k < NEAR_MAX_D; ++k)
      if (k < d) {
        const float x = pts[p * d + k];
        if (fabsf(x) < INFINITY) {
          lo[k] = max(lo[k], ~ordered(x));
          hi[k] = max(hi[k], ordered(x));
        }
      }
#pragma unroll
  for (int k = 0; k < NEAR_MAX_D; ++k)
    if (k < d) {
      lo[k] = __reduce_max_sync(FULL, lo[k]);
      hi[k] = __reduce_max_sync(FULL, hi[k]);
      if ((threadIdx.x & 31) == 0) {
        atomicMax(&box[2 * k], lo[k]);
        atomicMax(&box[2 * k + 1], hi[k]);
      }
    }
}

// the cell of a point: `bits` bits a dimension of its place in the box,
// interleaved (Z order)
__device__ __forceinline__ u32 cell_of(const float* __restrict__ x, int d, int bits, const u32* __restrict__ box) {
  const int side = 1 << bits;
  u32 cell = 0;
#pragma unroll
  for (int k = 0; k < NEAR_MAX_D; ++k)
    if (k < d) {
      const float lo = unordered(~box[2 * k]), hi = unordered(box[2 * k + 1]);
      const float f = (x[k] - lo) / (hi - lo) * (float)side;
      // NaN and what lies outside end up in the border cells
      const int c = f > 0.0f ? (f < (float)side ? (int)f : side - 1) : 0;
      for (int b = 0; b < bits; ++b) cell |= (u32)((c >> b) & 1) << (b * d + k);
    }
  return cell;
}

__global__ void k_near_count(const float* __restrict__ pts, i64 n, int d, int bits, const u32* __restrict__ box,
                             u32* __restrict__ cell, i32* __restrict__ cnt) {
  ph::pdl_wait();
  ph::pdl_trigger();
  for (i64 p = (i64)blockIdx.x * NR_NT + threadIdx.x; p < n; p += (i64)gridDim.x * NR_NT) {
    const u32 c = cell_of(pts + p * d, d, bits, box);
    cell[p] = c;
    atomicAdd(&cnt[c], 1);
  }
}

// points and their numbers in cell order (any order within a cell)
__global__ void k_near_place(const float* __restrict__ pts, i64 n, int d, const u32* __restrict__ cell,
                             const i32* __restrict__ off, i32* __restrict__ cursor, float* __restrict__ out,
                             i32* __restrict__ perm) {
  ph::pdl_wait();
  ph::pdl_trigger();
  for (i64 p = (i64)blockIdx.x * NR_NT + threadIdx.x; p < n; p += (i64)gridDim.x * NR_NT) {
    const u32 c = cell[p];
    const i64 at = off[c] + atomicAdd(&cursor[c], 1);
    perm[at] = (i32)p;
    for (int k = 0; k < d; ++k) out[at * d + k] = pts[p * d + k];
  }
}

// bounding box of every block of ET points, a warp each: lo[k], hi[k]
__global__ void k_near_blocks(const float* __restrict__ pts, i64 n, int d, i64 nt, float* __restrict__ boxes) {
  ph::pdl_wait();
  ph::pdl_trigger();
  const int lane = threadIdx.x & 31;
  for (i64 b = ((i64)blockIdx.x * NR_NT + threadIdx.x) >> 5; b < nt; b += ((i64)gridDim.x * NR_NT) >> 5)
    for (int k = 0; k < d; ++k) {
      float lo = INFINITY, hi = -INFINITY;
      for (i64 p = b * ET + lane; p < min(n, (b + 1) * ET); p += 32) {
        lo = fminf(lo, pts[p * d + k]);
        hi = fmaxf(hi, pts[p * d + k]);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(FULL, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(FULL, hi, o));
      }
      if (lane == 0) {
        boxes[(2 * k) * nt + b] = lo;
        boxes[(2 * k + 1) * nt + b] = hi;
      }
    }
}

// The pairs of blocks I <= J whose boxes come within the threshold: a warp a
// row I, a lane a column, the pairs appended to the list.
__global__ void k_near_pairs(const float* __restrict__ boxes, i64 nt, int d, float thr_sq, int2* __restrict__ list,
                             unsigned long long* __restrict__ count) {
  ph::pdl_wait();
  ph::pdl_trigger();
  const int lane = threadIdx.x & 31;
  const float bound = thr_sq * (1.0f + 0x1p-16f) + 0x1p-120f;
  for (i64 I = ((i64)blockIdx.x * NR_NT + threadIdx.x) >> 5; I < nt; I += ((i64)gridDim.x * NR_NT) >> 5) {
    float lo[NEAR_MAX_D], hi[NEAR_MAX_D];
#pragma unroll
    for (int k = 0; k < NEAR_MAX_D; ++k)
      if (k < d) {
        lo[k] = boxes[(2 * k) * nt + I];
        hi[k] = boxes[(2 * k + 1) * nt + I];
      }
    for (i64 J0 = I; J0 < nt; J0 += 32) {
      const i64 J = J0 + lane;
      bool near = false;
      if (J < nt) {
        float sum = 0.0f;
#pragma unroll
        for (int k = 0; k < NEAR_MAX_D; ++k)
          if (k < d) {
            const float a = boxes[(2 * k) * nt + J] - hi[k], b = lo[k] - boxes[(2 * k + 1) * nt + J];
            const float gap = a > 0.0f ? a : (b > 0.0f ? b : (a <= 0.0f && b <= 0.0f ? 0.0f : NAN));
            sum += gap * gap;
          }
        near = !(sum > bound);
      }
      const u32 m = __ballot_sync(FULL, near);
      if (!m) continue;
      unsigned long long at = 0;
      if (lane == 0) at = atomicAdd(count, (unsigned long long)__popc(m));
      at = __shfl_sync(FULL, at, 0);
      if (near) list[at + __popc(m & lanemask_lt())] = make_int2((int)I, (int)J);
    }
  }
}

// the listed pairs of blocks, taken from a common counter
__global__ void __launch_bounds__(ENT, 2)
    k_edges_near(const float* __restrict__ pts, i64 n, int d, float thr_sq, const i32* __restrict__ perm,
                 const int2* __restrict__ list, const unsigned long long* __restrict__ npairs,
                 unsigned long long* __restrict__ next, i32* __restrict__ oi, i32* __restrict__ oj,
                 float* __restrict__ od, i64 cap, unsigned long long* __restrict__ count) {
  ph::pdl_wait();
  ph::pdl_trigger();
  __shared__ EdgeTile sh;
  __shared__ unsigned long long take;
  const unsigned long long total = *npairs;
  for (;;) {
    __syncthreads();  // the last tile's stage and `take` are free
    if (threadIdx.x == 0) take = atomicAdd(next, 1ull);
    __syncthreads();
    const unsigned long long q = take;
    if (q >= total) break;
    const int2 ij = list[q];
    const i64 i0 = (i64)ij.x * ET, j0 = (i64)ij.y * ET;
    edge_tile(sh, pts, n, d, thr_sq, i0, j0, cap, count, [&](unsigned long long at, i64 gi, i64 gj, float dsq) {
      const i32 a = perm[gi], b = perm[gj];
      oi[at] = min(a, b);
      oj[at] = max(a, b);
      od[at] = dsq;
    });
  }
}

inline int grid_for(i64 n, int nt = NR_NT) {
  return (int)std::max<i64>(1, std::min<i64>((n + nt - 1) / nt, 148 * 8));
}

// bits a dimension of the grid: two points a cell or more on average
int near_bits(i64 n, int d) {
  int b = 1;
  while ((b + 1) * d <= 18 && (int64_t(1) << ((b + 1) * d)) <= n / 2) ++b;
  return b;
}

}  // namespace

size_t edges_near_workspace_bytes(i64 n, int d) {
  const i64 nt = (n + ET - 1) / ET, cells = i64(1) << (near_bits(n, d) * d);
  return Carve::need(2 * sizeof(unsigned long long) + 2 * NEAR_MAX_D * sizeof(u32)) + Carve::need(n * sizeof(u32)) +
         Carve::need(2 * cells * sizeof(i32)) + Carve::need((cells + 1) * sizeof(i32)) +
         Carve::need(n * d * sizeof(float)) + Carve::need(n * sizeof(i32)) + Carve::need(2 * d * nt * sizeof(float)) +
         Carve::need((size_t)(nt * (nt + 1) / 2) * sizeof(int2)) + Carve::need(scan_workspace_bytes(cells));
}

int edges_near(const float* pts, i64 n, int d, float thr_sq, i32* oi, i32* oj, float* od, i64 cap,
               unsigned long long* d_count, void* ws, size_t ws_bytes, cudaStream_t s) {
  if (n < 2 || d < 1 || d > NEAR_MAX_D) return PH_ERR_ARG;
  const i64 nt = (n + ET - 1) / ET;
  const int bits = near_bits(n, d);
  const i64 cells = i64(1) << (bits * d);
  Carve c(ws, ws_bytes);
  // pairs of blocks listed, taken; the box
  unsigned long long* ctr = c.take<unsigned long long>(2 + NEAR_MAX_D);
  u32* box = reinterpret_cast<u32*>(ctr + 2);
  u32* cell = c.take<u32>(n);
  i32* cnt = c.take<i32>(2 * cells);  // points a cell, and the cursors
  i32* off = c.take<i32>(cells + 1);
  float* sorted = c.take<float>(n * d);
  i32* perm = c.take<i32>(n);
  float* boxes = c.take<float>(2 * d * nt);
  int2* list = c.take<int2>(nt * (nt + 1) / 2);
  void* sws = c.take<char>((i64)scan_workspace_bytes(cells));
  if (!ctr || !cell || !cnt || !off || !sorted || !perm || !boxes || !list || !sws) return PH_ERR_ARG;
  ph::zero_async(cnt, 2 * cells * sizeof(i32), s, ctr, (2 + NEAR_MAX_D) * sizeof(unsigned long long));
  ph::zero_async(d_count, sizeof(unsigned long long), s);
  ph::count_launch();
  ph::launch_pdl(k_near_box, dim3(grid_for(n)), dim3(NR_NT), 0, s, pts, n, d, box);
  ph::count_launch();
  ph::launch_pdl(k_near_count, dim3(grid_for(n)), dim3(NR_NT), 0, s, pts, n, d, bits, (const u32*)box, cell, cnt);
  PH_TRY(scan_exclusive_i32_i32(cnt, off, cells, sws, scan_workspace_bytes(cells), s));
  ph::count_launch();
  ph::launch_pdl(k_near_place, dim3(grid_for(n)), dim3(NR_NT), 0, s, pts, n, d, (const u32*)cell, (const i32*)off,
                 cnt + cells, sorted, perm);
  ph::count_launch();
  ph::launch_pdl(k_near_blocks, dim3(grid_for(nt * 32)), dim3(NR_NT), 0, s, (const float*)sorted, n, d, nt, boxes);
  ph::count_launch();
  ph::launch_pdl(k_near_pairs, dim3(grid_for(nt * 32)), dim3(NR_NT), 0, s, (const float*)boxes, nt, d, thr_sq, list,
                 ctr);
  ph::count_launch();
  ph::launch_pdl(k_edges_near, dim3((unsigned)std::min<i64>(nt * (nt + 1) / 2, 2 * ph::device_sms())), dim3(ENT), 0, s,
                 (const float*)sorted, n, d, thr_sq, (const i32*)perm, (const int2*)list,
                 (const unsigned long long*)ctr, ctr + 1, oi, oj, od, cap, d_count);
  PH_CHECK_LAUNCH();
  return PH_OK;
}

}  // namespace ph
