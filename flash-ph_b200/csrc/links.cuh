// The simplices that can be pivots of the H1 and H2 reductions (links.cu).
#pragma once
#include "prim.cuh"

namespace ph {

struct LinkTotals {
  unsigned long long triangles;  // all triangles of the edges counted (tetrahedra of the triangles)
  unsigned long long rows;       // those that can be pivots
  unsigned long long stash;      // stash entries taken
};

// a row on its way from the count pass to its place
struct LinkRow {
  i32 m;       // largest edge; -1: an unused entry
  i32 z;       // index among the edge's rows
  i32 i;       // index among the edge's triangles
  i32 fa, fb;  // ranks of the two other edges
};

// a kept tetrahedron likewise
struct TetRow {
  i32 m;  // its first triangle (largest edge, smaller third vertex); -1: unused
  i32 z;  // index among that triangle's kept tetrahedra
  i32 k;  // its second triangle (largest edge, larger third vertex)
  i32 r;  // rank of the edge between the two third vertices
};

// Rows in no order. The count pass writes the first cap of them; where
// totals->stash came out larger it has to be run again with that much room.
template <typename Row>
struct Stash {
  Row* rows;
  i64 cap;
  LinkTotals* totals;  // zero on entry
};
using LinkStash = Stash<LinkRow>;
using TetStash = Stash<TetRow>;

// The sorted adjacency of one cloud (n vertices, segs null) or of a batch's
// union, with an optional table of edge ranks: n x n for one cloud, else the
// table of cloud c at table_off[c] (negative: none).
struct LinkGraph {
  const i32* adj_ptr;
  const i32* adj_idx;
  const i32* adj_rank;
  i64 n;
  const i32* table;
  const i64* table_off;
  const i32* vcloud;
  const ph_cloud_seg* segs;
};

// Whether the rank table pays: it costs a write of 4 n^2 bytes and replaces
// binary searches of ~E deg(G) candidates.
constexpr i64 LINK_TABLE_MAX_N = 16384;  // 1 GiB
__host__ __device__ inline bool link_table_pays(i64 n, i64 E) {
  return n <= LINK_TABLE_MAX_N && 64.0 * (double)E * (double)E > (double)n * (double)n * (double)n;
}

// The most entries that the tables of K clouds can take together, with E edges
// in all: a table of n^2 entries needs a cloud of n^1.5 / 8 edges, so the
// largest clouds first, as far as the edges go.
i64 link_tables_bound(const int64_t* n, int K, i64 E);

// Buffers of the two passes, E entries each (offsets E + 1). tri_off may be
// null where the triangles' numbering is not needed.
struct LinkCounts {
  i32* tri_cnt;
  i32* row_cnt;
  i32* len_cnt;  // cofacet list lengths, by face
  i32* cursor;
  i64* tri_off;
  i64* row_off;
  i32* off;      // cofacet list offsets
  LinkStash stash;
};

i64 link_stash_cap(i64 E, i64 n, i64 rows);
int link_table(const LinkGraph& g, i32* table, cudaStream_t s);
int link_table_offsets(const ph_cloud_seg* segs, const i64* e_off, int nclouds, i64 cap, i64* off, cudaStream_t s);
size_t link_count_workspace_bytes(i64 E);
// counts triangles and rows an edge; clouds with keep[cloud] == 0 count nothing
// (keep may be null); with more than `limit` triangles in all, the rows are not
// complete
int link_count(const i32* ei, const i32* ej, i64 E, const LinkGraph& g, const uint8_t* keep, const uint8_t* skip,
               i64 limit, const LinkCounts& o, void* ws, size_t ws_bytes, cudaStream_t s);
// the nrows rows in order: largest edge, index among all triangles (row_tri
// may be null), largest face not skipped; their entries in the lists of their
// faces
int link_rows(i64 nrows, const uint8_t* skip, const LinkCounts& o, i32 row_base, i32* row_m, i32* row_tri, i32* cmf,
              i32* data, int* status, cudaStream_t s);

// The triangles in their order, T of them: those with largest edge m at
// [tri_off[m], tri_off[m + 1]), third vertices ascending.
struct TetInput {
  const i32 *tri_m, *tri_w, *tri_fa, *tri_fb;
  const i64* tri_off;
  i64 T;
};

// T entries each (offsets T + 1); tet_cnt and tet_off may be null where the
// tetrahedra need no count a triangle.
struct TetCounts {
  i32* tet_cnt;
  i32* row_cnt;
  i64* tet_off;
  i64* row_off;
  TetStash stash;
};

i64 tet_stash_cap(i64 T, i64 rows);
// counts tetrahedra and those that can be pivots; the triangles of clouds with
// keep[cloud] == 0 count nothing (keep may be null). Scans need
// link_count_workspace_bytes(T).
int tet_count(const LinkGraph& g, const TetInput& in, const uint8_t* keep, const TetCounts& o, void* ws,
              size_t ws_bytes, cudaStream_t s);
// the nrows rows in order (largest edge, four faces, largest face not
// skipped), and the cofacet lists of the triangles not skipped
int tet_rows(const i32* ei, const i32* ej, const TetInput& in, const uint8_t* skip, const TetCounts& o, i32 face_base,
             i32 row_base, i64 nrows, i32* row_m, i32* faces, i32* cmf, i32* len_cnt, i32* cursor, i32* off, i32* data,
             void* ws, size_t ws_bytes, int* status, cudaStream_t s);

}  // namespace ph
