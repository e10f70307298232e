// The direct edge kernels' tile (edges.cu, edges_near.cu).
#pragma once
#include "prim.cuh"

namespace ph {

constexpr int ET = 128;  // points per tile side
constexpr int EK = 16;   // dimensions per shared-memory chunk
constexpr int ENT = 256;

// Edge kernels of a single cloud (pipeline.cu chooses, with the figures).
constexpr int NEAR_MAX_D = 4;               // dimensions of the grid order
constexpr i64 NEAR_MAX_N = i64(1) << 21;    // points: the list of block pairs then takes 1 GiB at most
size_t edges_near_workspace_bytes(i64 n, int d);
int edges_near(const float* pts, i64 n, int d, float thr_sq, i32* oi, i32* oj, float* od, i64 cap,
               unsigned long long* d_count, void* ws, size_t ws_bytes, cudaStream_t s);

struct EdgeTile {
  alignas(16) float x[EK][ET];
  alignas(16) float y[EK][ET];
};

// Pairs gi < gj < n of points i0 + [0, ET) and j0 + [0, ET) with a squared
// distance (chain in dimension order, one fused multiply-add a step) below
// thr_sq: counted, and emit(position, gi, gj, dsq) for those below cap. By a
// block of ENT threads, 8 x 8 pairs each in registers. The least of a thread's
// 64 distances is compared first (three-input minima): without a hit in the
// warp, the usual case, no pair is looked at again.
template <typename F>
__device__ __forceinline__ void edge_tile(EdgeTile& sh, const float* __restrict__ pts, i64 n, int d, float thr_sq,
                                          i64 i0, i64 j0, i64 cap, unsigned long long* __restrict__ count, F&& emit) {
  constexpr u32 FULL = 0xffffffffu;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[8][8];
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[r][c] = 0.0f;

  for (int k0 = 0; k0 < d; k0 += EK) {
    const int kc = min(EK, d - k0);
    const int tot = ET * kc;
    for (int idx = threadIdx.x; idx < tot; idx += ENT) {
      const int p = idx / kc, k = idx - p * kc;
      const i64 gi = i0 + p, gj = j0 + p;
      sh.x[k][p] = gi < n ? pts[gi * d + k0 + k] : 0.0f;
      sh.y[k][p] = gj < n ? pts[gj * d + k0 + k] : 0.0f;
    }
    __syncthreads();
#pragma unroll 2
    for (int k = 0; k < kc; ++k) {
      const float4 xa = *reinterpret_cast<const float4*>(&sh.x[k][ty * 8]);
      const float4 xb = *reinterpret_cast<const float4*>(&sh.x[k][ty * 8 + 4]);
      const float4 ya = *reinterpret_cast<const float4*>(&sh.y[k][tx * 8]);
      const float4 yb = *reinterpret_cast<const float4*>(&sh.y[k][tx * 8 + 4]);
      const float xv[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
      const float yv[8] = {ya.x, ya.y, ya.z, ya.w, yb.x, yb.y, yb.z, yb.w};
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float df = __fsub_rn(xv[r], yv[c]);
          acc[r][c] = __fmaf_rn(df, df, acc[r][c]);
        }
    }
    __syncthreads();
  }

  float least = INFINITY;
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int c = 0; c < 8; c += 2)
      asm("min.f32 %0, %1, %2, %3;" : "=f"(least) : "f"(least), "f"(acc[r][c]), "f"(acc[r][c + 1]));
  if (!__any_sync(FULL, least < thr_sq)) return;
  // hits of this thread's 8x8 block as a 64-bit mask
  u64 hit = 0;
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const i64 gi = i0 + ty * 8 + r, gj = j0 + tx * 8 + c;
      const bool ok = (gi < gj) && (gj < n) && (acc[r][c] < thr_sq);
      hit |= (u64)ok << (r * 8 + c);
    }
  const int cnt = __popcll(hit);
  if (!__any_sync(FULL, cnt != 0)) return;
  // warp-aggregated reservation
  const int lane = threadIdx.x & 31;
  int incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += y;
  }
  const int wtot = __shfl_sync(FULL, incl, 31);
  unsigned long long base = 0;
  if (lane == 31) base = atomicAdd(count, (unsigned long long)wtot);
  base = __shfl_sync(FULL, base, 31);
  unsigned long long pos = base + (unsigned long long)(incl - cnt);
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      if ((hit >> (r * 8 + c)) & 1ull) {
        if (pos < (unsigned long long)cap) emit(pos, i0 + ty * 8 + r, j0 + tx * 8 + c, acc[r][c]);
        ++pos;
      }
    }
}

}  // namespace ph
