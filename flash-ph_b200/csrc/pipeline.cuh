// Host-side plumbing shared by the native whole-call pipelines (one cloud in
// pipeline.cu, a batch of clouds in batch_pipeline.cu): stream-ordered
// scratch, host readbacks of device counts and statuses, reduction-pool
// sizing and the reduction + rows step.
#pragma once
#include <algorithm>
#include <string>
#include <vector>

#include "prim.cuh"

namespace ph {
namespace pl {

// Stream-ordered allocations released together when the run ends. A call takes
// some 50 buffers, most of them small, and an allocation with its release costs
// the host about a microsecond while a small call's kernels, of 2 to 5 us each,
// wait for their launches: requests of up to ARENA_SMALL bytes share slabs.
// Calls of 211, 500, 4001 and 20,000 points 311 -> 293 us, 577 -> 549, 667 -> 652,
// 685 -> 651.
constexpr size_t ARENA_SMALL = 512 << 10;
constexpr size_t ARENA_SLAB = 4 << 20;
struct Arena {
  cudaStream_t s;
  std::vector<void*> ptrs, slabs;
  char* slab = nullptr;  // the newest slab's unused part
  size_t left = 0;
  bool failed = false;
  // buffers to give back where memory runs out, with the pointer to clear
  // (null: nothing reads them any more)
  struct Spare {
    void* p;
    const i32** slot;
  };
  std::vector<Spare> spares;
  explicit Arena(cudaStream_t st) : s(st) {}
  Arena(const Arena&) = delete;
  Arena& operator=(const Arena&) = delete;
  // null where it is not to be had, spares given back or not (the error is the
  // caller's to report, not the next launch's)
  void* get(size_t bytes) {
    void* p = nullptr;
    if (cudaMallocAsync(&p, bytes, s) == cudaSuccess) return p;
    cudaGetLastError();
    if (spares.empty()) return nullptr;
    for (const Spare& x : spares) {
      ptrs.erase(std::find(ptrs.begin(), ptrs.end(), x.p));
      cudaFreeAsync(x.p, s);
      if (x.slot) *x.slot = nullptr;
    }
    spares.clear();
    if (cudaMallocAsync(&p, bytes, s) == cudaSuccess) return p;
    cudaGetLastError();
    return nullptr;
  }
  void* raw(size_t bytes, std::vector<void*>& kept) {
    void* p = get(bytes);
    if (p) kept.push_back(p);
    else failed = true;
    return p;
  }
  template <typename T>
  T* take(i64 count) {
    const size_t bytes = (size_t)std::max<i64>(count, 1) * sizeof(T);
    if (bytes > ARENA_SMALL) return static_cast<T*>(raw(bytes, ptrs));
    const size_t need = (bytes + 255) & ~size_t(255);
    if (need > left) {
      slab = static_cast<char*>(raw(ARENA_SLAB, slabs));
      left = slab ? ARENA_SLAB : 0;
      if (!slab) return nullptr;
    }
    char* p = slab;
    slab += need;
    left -= need;
    return reinterpret_cast<T*>(p);
  }
  void* bytes(size_t n) { return take<unsigned char>((i64)std::max<size_t>(n, 1)); }
  // A buffer that the call can do without (a table, the first guess of a size):
  // null where it is not to be had, or is over ph_set_optional_buffer_limit,
  // and the call goes on.
  template <typename T>
  T* optional(i64 count) {
    const long long limit = optional_buffer_limit();
    if (limit > 0 && std::max<i64>(count, 1) * (i64)sizeof(T) > limit) return nullptr;
    T* p = take<T>(count);
    if (!p) failed = false;
    return p;
  }
  // p may go where memory runs out (nothing happens to one that lies in a slab)
  void spare(void* p, const i32** slot = nullptr) {
    if (p && std::find(ptrs.begin(), ptrs.end(), p) != ptrs.end()) spares.push_back(Spare{p, slot});
  }
  // hands the buffers to a result, which frees them later
  void release_to(std::vector<void*>& keep) {
    keep.swap(ptrs);
    keep.insert(keep.end(), slabs.begin(), slabs.end());
    ptrs.clear();
    slabs.clear();
    spares.clear();
    left = 0;
  }
  ~Arena() {
    for (void* p : ptrs) cudaFreeAsync(p, s);
    for (void* p : slabs) cudaFreeAsync(p, s);
  }
};

// Small pinned, device-mapped host buffers for count and status readbacks (a
// kernel writes the values into them directly), from a process-wide pool.
struct Slots {
  int64_t* host = nullptr;
  int64_t* dev = nullptr;
  int64_t* seq = nullptr;  // host-side count of readbacks through this buffer
};
Slots take_slots();
void give_slots(const Slots& b);
struct SlotsLease {
  Slots b = take_slots();
  ~SlotsLease() {
    if (b.host) give_slots(b);
  }
};

// Pinned host buffers of any size for bulk readbacks and uploads (per-cloud
// arrays of a batch), from a process-wide pool: cudaHostAlloc can wait for
// the whole device, so buffers are reused rather than allocated per call.
struct Pinned {
  void* host = nullptr;
  size_t bytes = 0;
};
Pinned take_pinned(size_t bytes);
void give_pinned(const Pinned& p);
struct PinnedLease {
  Pinned p;
  explicit PinnedLease(size_t bytes) : p(take_pinned(bytes)) {}
  PinnedLease(const PinnedLease&) = delete;
  PinnedLease& operator=(const PinnedLease&) = delete;
  ~PinnedLease() {
    if (p.host) give_pinned(p);
  }
  template <typename T>
  T* as() const {
    return static_cast<T*>(p.host);
  }
};

// keeps the device's stream-ordered pool from returning memory at every sync
void keep_pool(int dev);
// fp32 of a double, round to nearest even, inf beyond the fp32 range (numpy's float32())
float to_f32(double v);
// records msg for ph_last_error() and returns code
int fail(int code, const std::string& msg);

// Brings count (<= 8) int64 values from the device into the pinned slots and
// waits (spins briefly on a sequence word written after them, then blocks).
int readback(const int64_t* const* src, int count, const Slots& dst, cudaStream_t s);
// One part of a bulk readback: bytes from device src to host dst.
struct Part {
  const void* src;
  void* dst;
  size_t bytes;
};
// Copies every part to pinned host memory (stream-ordered) and waits as
// readback does.
int readback_parts(const Part* parts, int nparts, const Slots& slots, cudaStream_t s);

// reduction pool (int32 entries): initial records (nnz + 4 a column), per-warp
// chunks, reduced columns; bounded by the 33-bit record offsets
constexpr i64 POOL_MAX = (i64(1) << 33) - 1;
i64 pool_capacity(i64 nnz, i64 K);

struct RedOut {
  i32* state;
  i32* piv;
  int64_t* info;
  int64_t* nrows;
};

// One reduction (H1 or H2) of cofacet lists in any order, enqueued on s; span
// as ph_reduce takes it.
int reduce_only(Arena& A, cudaStream_t s, const i32* off, const i32* data, i64 K, i32 col_base, i64 R,
                i32 row_base, i64 span, const uint8_t* skip, const i32* cmf, i64 pool_cap, bool windows_only, int* status,
                RedOut& o);

// The forest of a batch's union graph: a block a cloud where every cloud fits
// one (those that it turns out too slow for by the grid then), else
// ph_boruvka_mst over the union. Edges lie cloud by cloud (e_off); max_n is the
// largest cloud's vertex count; *d_ncomp and *d_left (the clouds left to the
// grid) start at zero; the workspace is ph_boruvka_mst's.
int batch_forest(const i32* edge_i, const i32* edge_j, i64 E, i64 n, const i64* e_off, const ph_cloud_seg* segs,
                 int K, i64 max_n, uint8_t* mst_mask, i32* comp, i64* d_ncomp, int* d_left, int* d_status,
                 void* workspace, size_t workspace_bytes, cudaStream_t s);

// Triangles per cloud of a batch's union graph, of the clouds with want set
// (the others' are zero); max_n is the largest cloud's vertex count; the
// workspace is ph_triangles_total_edges's.
int batch_triangles_total(const i32* edge_i, const i32* edge_j, i64 E, const i32* adj_ptr, i64 n, i64 max_n,
                          const i32* vcloud, const uint8_t* want, const ph_cloud_seg* segs, int K, unsigned long long* d_per,
                          void* workspace, size_t workspace_bytes, cudaStream_t s);

}  // namespace pl
}  // namespace ph
