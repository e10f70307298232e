// The rows of the H1 and H2 reductions: the simplices that can be pivots.
//
// The H1 coboundary matrix has a row per triangle, but most triangles can
// never be the pivot of a reduced column. Write a triangle as (m, w): its
// largest edge m = (a, b) and its third vertex w; the triangles with largest
// edge m are ordered by w. If the link of m holds a vertex x < w joined to w
// by an edge ranked below m, all four faces of {a, b, x, w} exist and the
// other three, (m, x), {a, x, w} and {b, x, w}, come before (m, w). The
// boundary of the tetrahedron's boundary is zero, so the boundary of (m, w)
// is the sum of three earlier boundaries: (m, w) bounds nothing new, it kills
// no H1 class, and by the uniqueness of the pairing it is no pivot of any
// reduction of the coboundary matrix. Its row can be left out: the serial
// algorithm (cohomology_general.py:202-371) only ever meets pivots as lowest
// entries, so with the row gone every step is the same, and pivots, pairs,
// apparent pairs (the first cofacet of a column is a pivot too) and emptied
// columns are unchanged. This test of one tetrahedron per triangle (Bauer's
// zero-persistence apparent pairs, Ripser 2021, in the dimension above) keeps
// 3-6% of the triangles of dense clouds and 10-25% of sparser ones, 1.0-1.6
// rows an edge, so the cofacet rows, their order and the reducer's columns
// shrink by that factor, and only these triangles need storing for H1.
// Measured with the reducer of one addition a step (present calls are faster on
// both sides), all triangles as rows -> these rows: 1501 x 8 Gaussian (6.1M
// triangles, 209K rows) 8.8 -> 2.0 ms a call; 4001-point torus in 3-D (0.94M,
// 90K) 3.8 -> 1.0 ms; a union of 192 clouds of 64-4096 points 119 -> 27 ms;
// 20,000 x 10 at 1.4 (17.6K, 13.4K) unchanged, 0.88 ms.
//
// H2 likewise: a tetrahedron (m, p, q), p < q in m's link, comes after every
// (m, y, .) with y < p, so it is no pivot when the link holds a y < p joined to
// both p and q below m (the five-vertex clique's boundary). 6-13% of the
// tetrahedra of dense clouds remain (331 x 50: 0.44M of 4.9M).
//
// k_links: a group of G lanes an edge. The lanes intersect the ends' adjacency
// rows into the link (its length is the edge's triangle count). Then each lane
// takes a third vertex and all test the link's first vertices together: in a
// dense link an earlier neighbour turns up within a few; the vertices left
// over (the rows, and a few more) are each tested against the rest of the
// link by the whole group. Lookups of an edge's rank go to an n x n rank table
// where that is small and the graph dense (one load, and the lanes share its
// row), to a binary search of the sorted adjacency row elsewhere, four
// searches in flight a lane. G is a warp; in sparse graphs, whose rows hold a
// few entries and whose pass is bound by the latency of its dependent loads,
// eight lanes (four edges a warp in flight), the warp taking an edge of long
// rows (over 64 entries: 155 us for 10^6 edges against 180 at 32 and 210 at
// 16) together. The rows found go to a stash in no order, from which
// k_link_rows places them once the counts are scanned.
//
// k_tet_links: a warp a triangle (m, p). The earlier link vertices joined to p
// go to shared memory; the later ones, q, a lane each, are tetrahedra where
// they are joined to p, and each is tested against the former, by all lanes
// together first and one after another then, as above.
#include <algorithm>
#include <climits>
#include <cmath>
#include <functional>
#include <vector>

#include "arith.cuh"
#include "links.cuh"

namespace ph {
namespace {

constexpr int LK_NT = 256;
constexpr int LK_WARPS = LK_NT / 32;
constexpr int LK_LIST = 768;   // link vertices a warp's groups hold in shared memory
constexpr int LK_HEAVY = 64;   // a row this long is the whole warp's
constexpr int LK_BLOCKS = 4;   // resident blocks an SM
constexpr int LK_CHUNK = 8;    // stash rows a group takes at a time
constexpr u32 FULL = 0xffffffffu;
constexpr i32 NO_RANK = INT_MAX;

// the graph as one warp sees it for an edge: adjacency rows, and the rank
// table of the edge's cloud where there is one
struct Graph {
  const i32* __restrict__ aptr;
  const i32* __restrict__ aidx;
  const i32* __restrict__ arank;
  const char* __restrict__ tab;  // rank of (0, 0), were the table of all vertices; null: no table
  i32 row;                       // bytes of a table row (n <= 16384)

  // The rank at (x, w), col the address of (0, w): one multiply-add and a load.
  // The passes over links are bound by instruction issue (64% of the slots,
  // 770 a dense edge, at 15% L1 and 96% L2 hits), not by the table's bytes.
  // Index arithmetic in 64 bits and single list loads -> this: 1501 points in
  // 8 dimensions 217 -> 202 us, tetrahedra of 331 in 50 214 -> 193 us.
  __device__ __forceinline__ const char* col(i32 w) const { return tab + 4 * (i64)w; }
  __device__ __forceinline__ i32 cell(const char* c, i32 x) const {
    return *reinterpret_cast<const i32*>(c + (i64)x * row);
  }

  // the ranks at key[q] of the adjacency rows [lo[q], hi[q]), NO_RANK where
  // there is no such entry (an empty range: not looked up), searches interleaved
  template <int N>
  __device__ __forceinline__ void search(int (&lo)[N], int (&hi)[N], const i32 (&key)[N], i32 (&r)[N]) const {
    int end[N];
#pragma unroll
    for (int q = 0; q < N; ++q) end[q] = hi[q];
    for (;;) {
      // every load of a level before the first use (no branch between them)
      int mid[N];
      i32 v[N];
      bool more = false;
#pragma unroll
      for (int q = 0; q < N; ++q) {
        mid[q] = midpoint(lo[q], hi[q]);
        more |= lo[q] < hi[q];
      }
      if (!more) break;
#pragma unroll
      for (int q = 0; q < N; ++q) v[q] = lo[q] < hi[q] ? aidx[mid[q]] : INT_MAX;
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const bool up = v[q] < key[q];
        lo[q] = up ? mid[q] + 1 : lo[q];
        hi[q] = up ? hi[q] : min(hi[q], mid[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < N; ++q) r[q] = lo[q] < end[q] && aidx[lo[q]] == key[q] ? arank[lo[q]] : NO_RANK;
  }

  // ranks of the edges (x[q], w), NO_RANK where there is none or ask[q] is false
  template <int N>
  __device__ __forceinline__ void ranks(const i32 (&x)[N], const bool (&ask)[N], i32 w, i32 (&r)[N]) const {
    if (tab) {
      const char* c = col(w);
#pragma unroll
      for (int q = 0; q < N; ++q) r[q] = ask[q] ? cell(c, x[q]) : NO_RANK;
      return;
    }
    int lo[N], hi[N];
    i32 key[N];
#pragma unroll
    for (int q = 0; q < N; ++q) {
      lo[q] = ask[q] ? aptr[x[q]] : 0;
      hi[q] = ask[q] ? aptr[x[q] + 1] : 0;
      key[q] = w;
    }
    search(lo, hi, key, r);
  }

  __device__ __forceinline__ i32 rank(i32 x, i32 w) const {
    const i32 xs[1] = {x};
    const bool ask[1] = {true};
    i32 r[1];
    ranks(xs, ask, w, r);
    return r[0];
  }
};

__device__ __forceinline__ Graph graph_of(const LinkGraph& g, i32 a) {
  Graph r{g.adj_ptr, g.adj_idx, g.adj_rank, nullptr, 0};
  if (!g.table) return r;
  if (!g.table_off) {
    r.tab = reinterpret_cast<const char*>(g.table);
    r.row = (i32)(4 * g.n);
    return r;
  }
  const i32 c = g.vcloud[a];
  const i64 at = g.table_off[c];
  if (at < 0) return r;
  const i64 vb = g.segs[c].vbase;
  r.row = 4 * g.segs[c].n;
  r.tab = reinterpret_cast<const char*>(g.table + at) - vb * r.row - 4 * vb;
  return r;
}

// the group of G lanes of this thread
template <int G>
struct Group {
  u32 mask;  // its lanes
  int lane;  // within the group
  int base;  // its first lane
  __device__ __forceinline__ Group() {
    const int l = threadIdx.x & 31;
    lane = l & (G - 1);
    base = l - lane;
    mask = (G == 32 ? FULL : (1u << (G & 31)) - 1u) << base;
  }
  // which lanes of the group (bit 0 its first)
  __device__ __forceinline__ u32 ballot(bool p) const { return (__ballot_sync(mask, p) & mask) >> base; }
  __device__ __forceinline__ i32 from(i32 v, int l) const { return __shfl_sync(mask, v, base + l); }
  __device__ __forceinline__ void sync() const { __syncwarp(mask); }
  __device__ __forceinline__ u32 below() const { return (1u << lane) - 1u; }
};

// an edge and its two adjacency rows, the shorter first
struct Ends {
  i32 m, a, b;
  int s0, s1, l0, l1;
  bool a_short;
};

__device__ __forceinline__ Ends ends_of(const LinkGraph& g, i32 m, i32 a, i32 b) {
  const int sa = g.adj_ptr[a], ea = g.adj_ptr[a + 1], sb = g.adj_ptr[b], eb = g.adj_ptr[b + 1];
  const bool as = (ea - sa) <= (eb - sb);
  return Ends{m, a, b, as ? sa : sb, as ? ea : eb, as ? sb : sa, as ? eb : ea, as};
}

// entries j, j + 1, ... of a group's list (j a multiple of their number); those
// past its end are whatever the words hold, and are not looked up
__device__ __forceinline__ void list_at(const i32* list, int j, i32 (&x)[4]) {
  const int4 v = *reinterpret_cast<const int4*>(list + j);
  x[0] = v.x;
  x[1] = v.y;
  x[2] = v.z;
  x[3] = v.w;
}
__device__ __forceinline__ void list_at(const i32* list, int j, i32 (&x)[2]) {
  const int2 v = *reinterpret_cast<const int2*>(list + j);
  x[0] = v.x;
  x[1] = v.y;
}

// The rows of an edge in ascending order, up to G at a time: f(mine, lanes, i,
// fa, fb) by the whole group, where the lanes of the mask hold one each, the
// one with link index i and other edges fa, fb. Returns the link's length
// (uniform in the group). `list` is the group's LK_LIST G / 32 words of shared
// memory. count_only: the length alone, no rows.
template <int G, typename F>
__device__ __forceinline__ int edge_rows(const Group<G>& gr, const Graph& g, const Ends& e, i32* list, bool count_only,
                                         F&& f) {
  constexpr int LIST = LK_LIST * G / 32;
  constexpr int U = G == 32 ? 4 : 2;  // row positions, or tests, a lane has in flight
  const int lane = gr.lane;
  const u32 lt = gr.below();
  const i32 m = e.m;
  const u32 end = e.s1;
  const i32* ltab = g.tab ? reinterpret_cast<const i32*>(g.tab + (i64)(e.a_short ? e.b : e.a) * g.row) : nullptr;
  // positions base + lane + G q of the shorter row: the vertex, its edges'
  // ranks, and whether it is in the link (positions past the row's end may
  // pass 2^31: unsigned)
  auto look = [&](u32 base, auto& w, auto& rs, auto& rl, auto& in) {
    constexpr int N = sizeof(w) / sizeof(w[0]);
    int lo[N], hi[N];
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const u32 p = base + lane + G * q;
      rs[q] = p < end ? g.arank[p] : NO_RANK;
      w[q] = p < end ? g.aidx[p] : 0;
    }
    if (ltab) {
#pragma unroll
      for (int q = 0; q < N; ++q) rl[q] = rs[q] < m ? ltab[w[q]] : NO_RANK;
    } else {
#pragma unroll
      for (int q = 0; q < N; ++q) {
        lo[q] = rs[q] < m ? e.l0 : 0;
        hi[q] = rs[q] < m ? e.l1 : 0;
      }
      g.search(lo, hi, w, rl);
    }
#pragma unroll
    for (int q = 0; q < N; ++q) in[q] = rl[q] < m;
  };
  if (e.s1 - e.s0 <= G) {  // a short row: one look, and the lanes go on with what they hold
    i32 w[1], rs[1], rl[1];
    bool in[1];
    look(e.s0, w, rs, rl, in);
    const u32 vb = gr.ballot(in[0]);
    const int nl = __popc(vb), i = __popc(vb & lt);
    if (count_only) return nl;
    if (in[0]) list[i] = w[0];
    gr.sync();
    bool open = in[0];
    for (int j = 0; j + 1 < nl; j += U) {
      if (!gr.ballot(open && j < i)) break;
      i32 x[U], r[U];
      bool ask[U];
      list_at(list, j, x);
#pragma unroll
      for (int q = 0; q < U; ++q) ask[q] = open && j + q < i;
      g.ranks(x, ask, w[0], r);
#pragma unroll
      for (int q = 0; q < U; ++q) open &= r[q] >= m;
    }
    const u32 lanes = gr.ballot(open);
    if (lanes) f(open, lanes, i, e.a_short ? rs[0] : rl[0], e.a_short ? rl[0] : rs[0]);
    gr.sync();  // the list is free for the next edge
    return nl;
  }
  int nl = 0, held = 0;
  u32 stop = end;  // vertices in the link and in the list, row position after the last of the list's
  for (u32 base = e.s0; base < end; base += U * G) {
    i32 w[U], rs[U], rl[U];
    bool in[U];
    look(base, w, rs, rl, in);
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const u32 vb = gr.ballot(in[q]);
      const int cnt = __popc(vb);
      if (stop == end) {
        if (nl + cnt <= LIST) {
          if (in[q]) list[nl + __popc(vb & lt)] = w[q];
          held = nl + cnt;
        } else {
          stop = base + G * q;  // whole groups only: this one and the rest are walked below
        }
      }
      nl += cnt;
    }
  }
  gr.sync();
  if (count_only) return nl;
  for (int base = 0; base < held; base += G) {
    const int i = base + lane;
    const i32 w = i < held ? list[i] : 0;
    bool open = i < held;  // no earlier neighbour found yet
    // the link's vertices from the first on, all lanes together, while that
    // takes fewer steps for the rest than a vertex after another does
    const int top = min(base + G - 1, held - 1);
    int tested = 0;
    u32 left = gr.ballot(open && i > 0);
    while (tested == 0 ? left != 0 : __popc(left) * (base / G + 1) > (top - tested) / U) {
      i32 x[U], r[U];
      bool ask[U];
      list_at(list, tested, x);
#pragma unroll
      for (int q = 0; q < U; ++q) ask[q] = open && tested + q < i;
      g.ranks(x, ask, w, r);
#pragma unroll
      for (int q = 0; q < U; ++q) open &= r[q] >= m;
      tested += U;
      left = gr.ballot(open && i > tested);
    }
    // the rest, one vertex after another by the whole group
    while (left) {
      const int l = __ffs(left) - 1;
      left &= left - 1;
      const i32 wl = list[base + l];
      for (int j = tested; j < base + l; j += G) {
        const bool mine = j + lane < base + l;
        if (gr.ballot(mine && g.rank(wl, list[mine ? j + lane : 0]) < m)) {
          if (lane == l) open = false;
          break;
        }
      }
    }
    const u32 lanes = gr.ballot(open);
    if (lanes) f(open, lanes, i, open ? g.rank(e.a, w) : 0, open ? g.rank(e.b, w) : 0);
  }
  if (nl > held) {  // a link longer than the list: its tail against the list, then against the row
    int at = held;
    for (u32 base = stop; base < end; base += G) {
      i32 w[1], rs[1], rl[1];
      bool in[1];
      look(base, w, rs, rl, in);
      const u32 vb = gr.ballot(in[0]);
      bool open = in[0];
      for (int j = 0; j < held; ++j) {
        if (!gr.ballot(open)) break;
        if (open && g.rank(list[j], w[0]) < m) open = false;
      }
      for (u32 x = stop; open && x < base + lane; ++x) {
        const i32 v = g.aidx[x];
        if (g.arank[x] < m && g.rank(e.a_short ? e.b : e.a, v) < m && g.rank(v, w[0]) < m) open = false;
      }
      gr.sync();
      const u32 lanes = gr.ballot(open);
      if (lanes) f(open, lanes, at + __popc(vb & lt), e.a_short ? rs[0] : rl[0], e.a_short ? rl[0] : rs[0]);
      at += __popc(vb);
    }
  }
  gr.sync();  // the list is free for the next edge
  return nl;
}

// n x n edge ranks, NO_RANK where there is no edge; one block a vertex
__global__ void __launch_bounds__(LK_NT) k_rank_table(LinkGraph g, i32* __restrict__ table) {
  ph::pdl_wait();
  ph::pdl_trigger();
  for (i64 v = blockIdx.x; v < g.n; v += gridDim.x) {
    i64 ld = g.n, at = 0;
    i32 vb = 0;
    if (g.table_off) {
      const i32 c = g.vcloud[v];
      at = g.table_off[c];
      if (at < 0) continue;
      ld = g.segs[c].n;
      vb = (i32)g.segs[c].vbase;
    }
    i32* row = table + at + (v - vb) * ld;
    for (i64 k = threadIdx.x; k < ld; k += LK_NT) row[k] = NO_RANK;
    __syncthreads();
    for (int p = g.adj_ptr[v] + threadIdx.x; p < g.adj_ptr[v + 1]; p += LK_NT) row[g.adj_idx[p] - vb] = g.adj_rank[p];
    __syncthreads();
  }
}

// a batch's tables: offsets of the clouds that get one, -1 for the others, in
// cloud order while the buffer lasts (one warp)
__global__ void k_table_offsets(const ph_cloud_seg* __restrict__ segs, const i64* __restrict__ e_off, int nclouds,
                                i64 cap, i64* __restrict__ off) {
  ph::pdl_wait();
  ph::pdl_trigger();
  const int lane = threadIdx.x & 31;
  i64 used = 0;
  for (int c0 = 0; c0 < nclouds; c0 += 32) {
    const int c = c0 + lane;
    i64 size = 0;
    if (c < nclouds && link_table_pays(segs[c].n, e_off[c + 1] - e_off[c])) size = (i64)segs[c].n * segs[c].n;
    i64 incl = size;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const i64 v = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += v;
    }
    // a cloud past the end of the buffer has none
    const i64 at = used + incl - size;
    if (c < nclouds) off[c] = size && at + size <= cap ? at : -1;
    used += __shfl_sync(FULL, incl, 31);
  }
}

// A group's place in the stash: chunks of LK_CHUNK rows (or of what one call
// brings) taken from the common count, so that a row costs a fraction of an
// atomic; the last one's rest is marked.
template <int G>
struct StashChunk {
  i64 pos = 0, end = 0;

  // where the n <= G rows of one call go: the first `room` of them from pos on,
  // the others from the new chunk on
  template <typename Row>
  __device__ __forceinline__ void put(const Group<G>& gr, const Stash<Row>& st, int n, bool mine, int z,
                                      const Row& row) {
    const int room = (int)min((i64)n, end - pos);
    const int take = max(n - room, LK_CHUNK);
    i64 next = 0;
    if (n > room) {
      if (gr.lane == 0) next = (i64)atomicAdd(&st.totals->stash, (unsigned long long)take);
      next = __shfl_sync(gr.mask, next, gr.base);
    }
    if (mine) {
      const i64 at = z < room ? pos + z : next + (z - room);
      if (at < st.cap) st.rows[at] = row;
    }
    if (n > room) {
      pos = next + (n - room);
      end = next + take;
    } else {
      pos += n;
    }
  }

  template <typename Row>
  __device__ __forceinline__ void finish(const Group<G>& gr, const Stash<Row>& st) {
    for (i64 at = pos + gr.lane; at < min(end, st.cap); at += G) st.rows[at].m = -1;
  }
};

// LIMIT: counts only, once the triangles are over the limit (a variant of its
// own: as an argument it cost the batches' pass 5%)
template <int G, bool LIMIT>
__global__ void __launch_bounds__(LK_NT, LK_BLOCKS) k_links(const i32* __restrict__ ei, const i32* __restrict__ ej, i64 E,
                                                LinkGraph lg, const uint8_t* __restrict__ keep,
                                                const uint8_t* __restrict__ skip, i32* __restrict__ tri_cnt,
                                                i32* __restrict__ row_cnt, i32* __restrict__ len_cnt,
                                                LinkStash stash, i64 limit) {
  ph::pdl_wait();
  ph::pdl_trigger();
  constexpr int PER = 32 / G;  // edges a warp has in flight
  __shared__ __align__(16) i32 lists[LK_WARPS][LK_LIST];
  __shared__ unsigned long long sum[2];
  const Group<G> gr;
  const Group<32> wp;
  const int wl = threadIdx.x >> 5;
  const i64 warp = ((i64)blockIdx.x * LK_NT + threadIdx.x) >> 5;
  const i64 nwarps = ((i64)gridDim.x * LK_NT) >> 5;
  if (threadIdx.x < 2) sum[threadIdx.x] = 0;
  __syncthreads();
  StashChunk<G> chunk;
  StashChunk<32> wchunk;  // of the edges the warp takes together
  i64 ntri = 0, nrow = 0;
  bool over = false;
  auto walk = [&](const auto& grp, auto& ch, const Ends& e, i32* list) {
    const Graph g = graph_of(lg, e.a);
    int k = 0;
    const int nl = edge_rows(grp, g, e, list, LIMIT && over, [&](bool mine, u32 lanes, int i, i32 fa, i32 fb) {
      const int z = __popc(lanes & grp.below()), n = __popc(lanes);
      ch.put(grp, stash, n, mine, z, LinkRow{e.m, k + z, i, fa, fb});
      if (mine) {
        if (!skip[fa]) atomicAdd(&len_cnt[fa], 1);
        if (!skip[fb]) atomicAdd(&len_cnt[fb], 1);
      }
      k += n;
    });
    if (grp.lane == 0) {
      tri_cnt[e.m] = nl;
      row_cnt[e.m] = k;
      if (k && !skip[e.m]) atomicAdd(&len_cnt[e.m], k);
      ntri += nl;
      nrow += k;
    }
  };
  // With a limit, longest edges first (their links are the largest): once the triangles seen
  // so far, brought together every 16 edges, are over the limit, no row is
  // needed, and the rest is only counted. 70,166 points in 3-D with outliers,
  // 1.5M edges, 14.7M triangles (limit 10M): 2510 -> 1895 us, the call 6.67 ->
  // 6.05 ms (6.12 when all triangles were counted an edge without rows).
  int turn = 0;
  for (i64 m0 = warp * PER; m0 < E; m0 += nwarps * PER) {
    if (LIMIT && (++turn & 15) == 0 && !over) {
      for (int o = 16; o > 0; o >>= 1) ntri += __shfl_xor_sync(FULL, ntri, o);
      if (wp.lane == 0)
        over = (i64)(atomicAdd(&stash.totals->triangles, (unsigned long long)ntri) + ntri) > limit;
      over = __shfl_sync(FULL, over, 0);
      ntri = 0;
    }
    i64 m = m0 + gr.base / G;
    if (LIMIT) m = E - 1 - m;
    Ends e{-1, 0, 0, 0, 0, 0, 0, false};
    if (m >= 0 && m < E) {
      const i32 a = ei[m], b = ej[m];
      if (keep && !keep[lg.vcloud[a]]) {  // a cloud already known to be over its limit counts nothing
        if (gr.lane == 0) {
          tri_cnt[m] = 0;
          row_cnt[m] = 0;
        }
      } else {
        e = ends_of(lg, (i32)m, a, b);
      }
    }
    const bool heavy = G < 32 && e.s1 - e.s0 > LK_HEAVY;
    if (e.m >= 0 && !heavy) walk(gr, chunk, e, lists[wl] + (gr.base / G) * (LK_LIST * G / 32));
    if (G < 32) {
      u32 todo = __ballot_sync(FULL, heavy && gr.lane == 0);
      while (todo) {
        const int l = __ffs(todo) - 1;
        todo &= todo - 1;
        const i32 hm = __shfl_sync(FULL, e.m, l);
        walk(wp, wchunk, ends_of(lg, hm, ei[hm], ej[hm]), lists[wl]);
      }
    }
  }
  chunk.finish(gr, stash);
  if (G < 32) wchunk.finish(wp, stash);
  if (ntri) atomicAdd(&sum[0], (unsigned long long)ntri);
  if (nrow) atomicAdd(&sum[1], (unsigned long long)nrow);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (sum[0]) atomicAdd(&stash.totals->triangles, sum[0]);
    if (sum[1]) atomicAdd(&stash.totals->rows, sum[1]);
  }
}

// The rows in their order: row r = row_off[m] + z is edge m's z-th. Each gets
// its largest edge, its index among all triangles (where those are numbered),
// its largest face that is a column, and an entry in the (unsorted) cofacet
// list of each face that is a column.
__global__ void __launch_bounds__(LK_NT) k_link_rows(LinkStash stash, const uint8_t* __restrict__ skip,
                                                     const i64* __restrict__ row_off,
                                                     const i64* __restrict__ tri_off,
                                                     const i32* __restrict__ off, i32* __restrict__ cursor,
                                                     i32 row_base, i64 nrows, i32* __restrict__ row_m,
                                                     i32* __restrict__ row_tri, i32* __restrict__ cmf,
                                                     i32* __restrict__ data, int* status) {
  ph::pdl_wait();
  ph::pdl_trigger();
  const i64 n = min((i64)stash.totals->stash, stash.cap);
  for (i64 k = (i64)blockIdx.x * LK_NT + threadIdx.x; k < n; k += (i64)gridDim.x * LK_NT) {
    const LinkRow x = stash.rows[k];
    if (x.m < 0) continue;
    const i64 r = row_off[x.m] + x.z;
    if (r >= nrows) {  // the counts and the rows disagree: never write past the buffers
      set_status(status, PH_ERR_ARG);
      continue;
    }
    row_m[r] = x.m;
    if (row_tri) {  // -1 where the edge's triangles are not stored (a cloud without H2)
      const i64 t = tri_off[x.m] + x.i;
      row_tri[r] = t < tri_off[x.m + 1] ? (i32)t : -1;
    }
    // m is the largest of the three
    const i32 f[3] = {skip[x.m] ? -1 : x.m, skip[x.fa] ? -1 : x.fa, skip[x.fb] ? -1 : x.fb};
    cmf[r] = f[0] >= 0 ? f[0] : max(f[1], f[2]);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      if (f[q] < 0) continue;
      const i32 pos = off[f[q]] + atomicAdd(&cursor[f[q]], 1);
      if (pos < off[f[q] + 1]) data[pos] = row_base + (i32)r;
      else set_status(status, PH_ERR_ARG);
    }
  }
}

// ---- tetrahedra -------------------------------------------------------------------------
struct TetArgs {
  const i32* tri_m;
  const i32* tri_w;
  const i64* tri_off;
  i64 T;
  const uint8_t* keep;  // per cloud, may be null: the others' tetrahedra are neither counted nor kept
};

__global__ void __launch_bounds__(LK_NT) k_tet_links(LinkGraph lg, TetArgs ta,
                                                     i32* __restrict__ tet_cnt, i32* __restrict__ row_cnt,
                                                     TetStash stash) {
  ph::pdl_wait();
  ph::pdl_trigger();
  constexpr int U = 4;  // lookups a lane has in flight
  __shared__ __align__(16) i32 lists[LK_WARPS][LK_LIST];
  __shared__ unsigned long long sum[2];
  const Group<32> gr;
  const int lane = gr.lane;
  const u32 lt = gr.below();
  i32* list = lists[threadIdx.x >> 5];
  const i64 warp = ((i64)blockIdx.x * LK_NT + threadIdx.x) >> 5;
  const i64 nwarps = ((i64)gridDim.x * LK_NT) >> 5;
  if (threadIdx.x < 2) sum[threadIdx.x] = 0;
  __syncthreads();
  StashChunk<32> chunk;
  i64 ntet = 0, nrow = 0;
  for (i64 t = warp; t < ta.T; t += nwarps) {
    const i32 m = ta.tri_m[t], p = ta.tri_w[t];
    const i64 t0 = ta.tri_off[m], t1 = ta.tri_off[m + 1];
    int tets = 0, rows = 0;
    if (t + 1 < t1 && (!ta.keep || ta.keep[lg.vcloud[p]])) {
      const Graph g = graph_of(lg, p);
      // the earlier vertices of the link joined to p
      int held = 0;
      i64 stop = t;  // link position after the last of those in the list
      for (i64 base = t0; base < t; base += 32) {
        const i32 y = base + lane < t ? ta.tri_w[base + lane] : -1;
        const bool in = y >= 0 && g.rank(p, y) < m;
        const u32 b = gr.ballot(in);
        if (held + __popc(b) > LK_LIST) {
          stop = base;  // the rest is walked below
          break;
        }
        if (in) list[held + __popc(b & lt)] = y;
        held += __popc(b);
      }
      gr.sync();
      for (i64 base = t + 1; base < t1; base += 32) {
        const i64 k = base + lane;
        const i32 q = k < t1 ? ta.tri_w[k] : -1;
        const i32 rpq = q >= 0 ? g.rank(p, q) : NO_RANK;
        const bool tet = rpq < m;
        bool open = tet;
        u32 left = gr.ballot(tet);
        tets += __popc(left);
        int tested = 0;
        while (tested < held && __popc(left) * ((held - tested + 31) / 32) > (tested ? (held - tested) / U : 0)) {
          i32 x[U], r[U];
          bool ask[U];
          list_at(list, tested, x);
#pragma unroll
          for (int u = 0; u < U; ++u) ask[u] = open && tested + u < held;
          g.ranks(x, ask, q, r);
#pragma unroll
          for (int u = 0; u < U; ++u) open &= r[u] >= m;
          tested += U;
          left = gr.ballot(open);
        }
        if (tested < held) {
          while (left) {
            const int l = __ffs(left) - 1;
            left &= left - 1;
            const i32 ql = gr.from(q, l);
            for (int j = tested; j < held; j += 32) {
              const i32 y = list[min(j + lane, held - 1)];
              if (gr.ballot(g.rank(ql, y) < m)) {
                if (lane == l) open = false;
                break;
              }
            }
          }
        }
        for (i64 x = stop; open && x < t; ++x) {  // a list that did not hold them all
          const i32 y = ta.tri_w[x];
          if (g.rank(p, y) < m && g.rank(y, q) < m) open = false;
        }
        gr.sync();
        const u32 lanes = gr.ballot(open);
        if (lanes) {
          const int n = __popc(lanes), z = __popc(lanes & lt);
          chunk.put(gr, stash, n, open, z, TetRow{(i32)t, rows + z, (i32)k, rpq});
          rows += n;
        }
      }
      gr.sync();  // the list is free for the next triangle
    }
    if (lane == 0) {
      if (tet_cnt) tet_cnt[t] = tets;
      row_cnt[t] = rows;
    }
    ntet += tets;
    nrow += rows;
  }
  chunk.finish(gr, stash);
  if (lane == 0) {
    if (ntet) atomicAdd(&sum[0], (unsigned long long)ntet);
    if (nrow) atomicAdd(&sum[1], (unsigned long long)nrow);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (sum[0]) atomicAdd(&stash.totals->triangles, sum[0]);
    if (sum[1]) atomicAdd(&stash.totals->rows, sum[1]);
  }
}

// The kept tetrahedra in their order: row r = row_off[t] + z is the z-th of
// triangle t = (m, p). Each gets its largest edge, its four faces, its largest
// face that is a column, and counts in the cofacet lists of its faces.
__global__ void __launch_bounds__(LK_NT) k_tet_rows(TetStash stash, const i32* __restrict__ ei,
                                                    const i32* __restrict__ ej, TetArgs ta,
                                                    const i32* __restrict__ tfa, const i32* __restrict__ tfb,
                                                    const uint8_t* __restrict__ skip, const i64* __restrict__ row_off,
                                                    i32 face_base, i64 nrows, i32* __restrict__ row_m,
                                                    i32* __restrict__ faces, i32* __restrict__ cmf,
                                                    i32* __restrict__ len_cnt, int* status) {
  ph::pdl_wait();
  ph::pdl_trigger();
  const i64 n = min((i64)stash.totals->stash, stash.cap);
  for (i64 x = (i64)blockIdx.x * LK_NT + threadIdx.x; x < n; x += (i64)gridDim.x * LK_NT) {
    const TetRow row = stash.rows[x];
    if (row.m < 0) continue;
    const i64 t = row.m, k = row.k, r = row_off[t] + row.z;
    if (r >= nrows) {  // the counts and the rows disagree: never write past the buffers
      set_status(status, PH_ERR_ARG);
      continue;
    }
    const i32 m = ta.tri_m[t], p = ta.tri_w[t], q = ta.tri_w[k], rpq = row.r;
    i32 f[4] = {(i32)t, (i32)k, 0, 0};
    // {a, p, q} and {b, p, q}: their largest edge and third vertex
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      const i32 v = side ? ej[m] : ei[m];
      const i32 rp = side ? tfb[t] : tfa[t], rq = side ? tfb[k] : tfa[k];
      const i32 big = max(max(rp, rq), rpq), third = big == rp ? q : (big == rq ? p : v);
      const int lo = (int)ta.tri_off[big], hi = (int)ta.tri_off[big + 1];
      f[2 + side] = lower_bound_i32(ta.tri_w, lo, hi, third);
      if (f[2 + side] >= hi || ta.tri_w[f[2 + side]] != third) {  // cannot happen for a consistent adjacency
        set_status(status, PH_ERR_ARG);
        f[2 + side] = (i32)t;
      }
    }
    row_m[r] = m;
    reinterpret_cast<int4*>(faces)[r] = make_int4(f[0], f[1], f[2], f[3]);
    i32 best = -1;
#pragma unroll
    for (int z = 0; z < 4; ++z)
      if (!skip[f[z]]) {
        best = max(best, face_base + f[z]);
        atomicAdd(&len_cnt[f[z]], 1);
      }
    cmf[r] = best;
  }
}

// the rows' ranks into the cofacet lists of their faces that are columns
__global__ void k_tet_scatter(const i32* __restrict__ faces, i64 entries, const uint8_t* __restrict__ skip,
                              i32 row_base, const i32* __restrict__ off, i32* __restrict__ cursor,
                              i32* __restrict__ data, int* status) {
  ph::pdl_wait();
  ph::pdl_trigger();
  for (i64 x = (i64)blockIdx.x * blockDim.x + threadIdx.x; x < entries; x += (i64)gridDim.x * blockDim.x) {
    const i32 f = faces[x];
    if (skip[f]) continue;
    const i32 pos = off[f] + atomicAdd(&cursor[f], 1);
    if (pos < off[f + 1]) data[pos] = row_base + (i32)(x >> 2);
    else set_status(status, PH_ERR_ARG);
  }
}

inline int grid_for(i64 n, int nt = 256) {
  return (int)std::max<i64>(1, std::min<i64>((n + nt - 1) / nt, 148 * 16));
}

// lanes an edge: eight up to 16 neighbours a vertex on average
inline int lanes_for(i64 E, i64 n) { return E <= 8 * n ? 8 : 32; }

inline int links_grid(i64 E, int lanes) {
  const int per = LK_NT / lanes;
  return (int)std::max<i64>(1, std::min<i64>((E + per - 1) / per, (i64)ph::device_sms() * LK_BLOCKS));
}

}  // namespace

// Room for `rows` rows: what the groups can leave unused of their last chunks
// comes on top.
i64 link_stash_cap(i64 E, i64 n, i64 rows) {
  const int lanes = lanes_for(E, n);
  return rows + (i64)links_grid(E, lanes) * (LK_NT / lanes + LK_WARPS) * LK_CHUNK;
}

i64 link_tables_bound(const int64_t* n, int K, i64 E) {
  std::vector<i64> sizes;
  for (int c = 0; c < K; ++c)
    if (n[c] <= LINK_TABLE_MAX_N) sizes.push_back(n[c]);
  std::sort(sizes.begin(), sizes.end(), std::greater<i64>());
  i64 entries = 0;
  double left = (double)E;
  for (const i64 m : sizes) {
    const double edges = std::sqrt((double)m) * (double)m / 8.0;
    if (left < edges) {  // the next one's share: an upper bound for any smaller ones in its place
      entries += (i64)std::ceil((double)m * (double)m * (left / edges));
      break;
    }
    left -= edges;
    entries += m * m;
  }
  return entries;
}

int link_table(const LinkGraph& g, i32* table, cudaStream_t s) {
  ph::count_launch();
  ph::launch_pdl(k_rank_table, dim3((unsigned)std::min<i64>(g.n, 148 * 8)), dim3(LK_NT), 0, s, g, table);
  PH_CHECK_LAUNCH();
  return PH_OK;
}

int link_table_offsets(const ph_cloud_seg* segs, const i64* e_off, int nclouds, i64 cap, i64* off, cudaStream_t s) {
  ph::count_launch();
  ph::launch_pdl(k_table_offsets, dim3(1), dim3(32), 0, s, segs, e_off, nclouds, cap, off);
  PH_CHECK_LAUNCH();
  return PH_OK;
}

size_t link_count_workspace_bytes(i64 E) { return scan_workspace_bytes(E); }

int link_count(const i32* ei, const i32* ej, i64 E, const LinkGraph& g, const uint8_t* keep, const uint8_t* skip,
               i64 limit, const LinkCounts& o, void* ws, size_t ws_bytes, cudaStream_t s) {
  if (E < 1) return PH_ERR_ARG;
  ph::zero_async(o.len_cnt, sizeof(i32) * E, s, o.cursor, sizeof(i32) * E);
  const int lanes = lanes_for(E, g.n);
  const auto kernel = limit < LLONG_MAX ? (lanes == 8 ? k_links<8, true> : k_links<32, true>)
                                        : (lanes == 8 ? k_links<8, false> : k_links<32, false>);
  ph::count_launch();
  ph::launch_pdl(kernel, dim3(links_grid(E, lanes)), dim3(LK_NT), 0, s, ei, ej, E, g,
                 keep, skip, o.tri_cnt, o.row_cnt, o.len_cnt, o.stash, limit);
  if (o.tri_off) PH_TRY(scan_exclusive_i32_i64(o.tri_cnt, o.tri_off, E, ws, ws_bytes, s));
  PH_TRY(scan_exclusive_i32_i64(o.row_cnt, o.row_off, E, ws, ws_bytes, s));
  PH_TRY(scan_exclusive_i32_i32(o.len_cnt, o.off, E, ws, ws_bytes, s));
  PH_CHECK_LAUNCH();
  return PH_OK;
}

int link_rows(i64 nrows, const uint8_t* skip, const LinkCounts& o, i32 row_base, i32* row_m, i32* row_tri, i32* cmf,
              i32* data, int* status, cudaStream_t s) {
  ph::count_launch();
  ph::launch_pdl(k_link_rows, dim3(grid_for(o.stash.cap, LK_NT)), dim3(LK_NT), 0,
                 s, o.stash, skip, (const i64*)o.row_off, (const i64*)o.tri_off, (const i32*)o.off, o.cursor, row_base,
                 nrows, row_m, row_tri, cmf, data, status);
  PH_CHECK_LAUNCH();
  return PH_OK;
}

// ---- tetrahedra ---------------------------------------------------------------------------
namespace {
inline int tets_grid(i64 T) {
  return (int)std::max<i64>(1, std::min<i64>((T + LK_WARPS - 1) / LK_WARPS, (i64)ph::device_sms() * 8));
}
}  // namespace

i64 tet_stash_cap(i64 T, i64 rows) { return rows + (i64)tets_grid(T) * LK_WARPS * LK_CHUNK; }

int tet_count(const LinkGraph& g, const TetInput& in, const uint8_t* keep, const TetCounts& o, void* ws,
              size_t ws_bytes, cudaStream_t s) {
  if (in.T < 1) return PH_ERR_ARG;
  const TetArgs ta{in.tri_m, in.tri_w, in.tri_off, in.T, keep};
  ph::count_launch();
  ph::launch_pdl(k_tet_links, dim3(tets_grid(in.T)), dim3(LK_NT), 0, s, g, ta, o.tet_cnt, o.row_cnt, o.stash);
  if (o.tet_off) PH_TRY(scan_exclusive_i32_i64(o.tet_cnt, o.tet_off, in.T, ws, ws_bytes, s));
  PH_TRY(scan_exclusive_i32_i64(o.row_cnt, o.row_off, in.T, ws, ws_bytes, s));
  PH_CHECK_LAUNCH();
  return PH_OK;
}

int tet_rows(const i32* ei, const i32* ej, const TetInput& in, const uint8_t* skip, const TetCounts& o, i32 face_base,
             i32 row_base, i64 nrows, i32* row_m, i32* faces, i32* cmf, i32* len_cnt, i32* cursor, i32* off, i32* data,
             void* ws, size_t ws_bytes, int* status, cudaStream_t s) {
  if (in.T < 1) return PH_ERR_ARG;
  const TetArgs ta{in.tri_m, in.tri_w, in.tri_off, in.T, nullptr};
  ph::zero_async(len_cnt, sizeof(i32) * in.T, s, cursor, sizeof(i32) * in.T);
  ph::count_launch();
  ph::launch_pdl(k_tet_rows, dim3(grid_for(o.stash.cap, LK_NT)), dim3(LK_NT), 0, s, o.stash, ei, ej, ta, in.tri_fa,
                 in.tri_fb, skip, (const i64*)o.row_off, face_base, nrows, row_m, faces, cmf, len_cnt, status);
  PH_TRY(scan_exclusive_i32_i32(len_cnt, off, in.T, ws, ws_bytes, s));
  if (nrows > 0) {
    ph::count_launch();
    ph::launch_pdl(k_tet_scatter, dim3(grid_for(4 * nrows, LK_NT)), dim3(LK_NT), 0, s, (const i32*)faces, 4 * nrows,
                   skip, row_base, (const i32*)off, cursor, data, status);
  }
  PH_CHECK_LAUNCH();
  return PH_OK;
}

}  // namespace ph
