// Host side of the adjacency handle: the cleaned lists, and the tables of the
// basin form of the sweep (tfce_basin.cu) built from them.  Plain C++, so that
// it can be compiled and checked without a GPU.
#pragma once

#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <memory>
#include <string>
#include <type_traits>
#include <vector>

#include "host_parallel.h"

namespace tfgb {

constexpr uint32_t kOneWay = 0x80000000u;     // entry whose reverse entry is missing
constexpr uint32_t kIndexMask = 0x7fffffffu;
constexpr int kTile = 4096;                   // vertices per tile at most (12 bits of a packed record)
constexpr int kTileEntries = 120000;          // list entries per tile: pairs are counted in 16 bits
constexpr int kCrossChunk = 1024;             // boundary vertices of a chunk
constexpr uint32_t kOddRow = 0x80000000u;     // in edge_off: the second entries of the row's last words are padding

// An array that starts unwritten: its pages are first touched by the threads
// that fill it.
template <typename T>
class Raw {
 public:
  Raw() = default;
  explicit Raw(int64_t n) : p_(new T[n]), n_(n) {}
  int64_t size() const { return n_; }
  T* data() const { return p_.get(); }
  T& operator[](int64_t i) const {
#ifdef _GLIBCXX_ASSERTIONS
    if (i < 0 || i >= n_) __builtin_trap();
#endif
    return p_[i];
  }

 private:
  std::unique_ptr<T[]> p_;
  int64_t n_ = 0;
};

// Adjacency lists as the kernels read them: sorted, without self entries and
// repeats (which never change the partition), entries whose reverse is missing
// flagged (kOneWay).
struct CleanLists {
  Raw<int64_t> off;      // [V + 1]
  Raw<uint32_t> packed;  // [off[V]]
  bool symmetric = true;
};

// False, with the first bad entry in *error, if an entry is outside the graph or
// its vertex's segment.  offsets are monotone and seg spans [0, V].
inline bool clean_lists(const int64_t* offsets, const int32_t* indices, int32_t V, const std::vector<int64_t>& seg,
                        CleanLists* out, std::string* error) {
  auto segment_of = [&](int64_t v) { return std::upper_bound(seg.begin(), seg.end(), v) - seg.begin() - 1; };
  const int64_t D = offsets[V], blocks = (V + 4095) / 4096;
  out->off = Raw<int64_t>(V + 1);
  Raw<int64_t>& off = out->off;
  off[0] = 0;
  std::vector<int64_t> bad(blocks, -1);
  const Raw<int32_t> idx(D);
  // every list in the place that it came in, and its length (in off[v + 1])
  parallel_for(blocks, D, [&](int64_t k) {
    int64_t v = k * 4096, s = segment_of(v);
    for (; v < std::min<int64_t>(V, (k + 1) * 4096); ++v) {
      while (v >= seg[s + 1]) ++s;
      int32_t* const first = idx.data() + offsets[v];
      int32_t* last = first;
      bool ordered = true;
      for (int64_t e = offsets[v]; e < offsets[v + 1]; ++e) {
        const int32_t u = indices[e];
        if ((u < seg[s] || u >= seg[s + 1]) && bad[k] < 0) bad[k] = e;
        if (u == v) continue;
        ordered = ordered && (last == first || last[-1] < u);
        *last++ = u;
      }
      if (!ordered) {
        std::sort(first, last);
        last = std::unique(first, last);
      }
      off[v + 1] = last - first;
    }
  });
  for (int64_t e : bad) {
    if (e < 0) continue;
    const int64_t v = std::upper_bound(offsets, offsets + V + 1, e) - offsets - 1;
    const bool outside = indices[e] < 0 || indices[e] >= V;
    *error = "adjacency entry " + std::to_string(indices[e]) + " of vertex " + std::to_string(v) +
             (outside ? " outside [0, " + std::to_string(V) + ")" : " crosses segments");
    return false;
  }
  for (int32_t v = 0; v < V; ++v) off[v + 1] += off[v];
  out->packed = Raw<uint32_t>(off[V]);
  std::atomic<bool> two_way{true};
  parallel_for(blocks, D, [&](int64_t k) {
    for (int64_t v = k * 4096; v < std::min<int64_t>(V, (k + 1) * 4096); ++v) {
      const int32_t* const list = idx.data() + offsets[v];
      for (int64_t j = 0; j < off[v + 1] - off[v]; ++j) {
        const int32_t u = list[j];
        const int32_t* const theirs = idx.data() + offsets[u];
        const bool rev = std::binary_search(theirs, theirs + (off[u + 1] - off[u]), static_cast<int32_t>(v));
        out->packed[off[v] + j] = static_cast<uint32_t>(u) | (rev ? 0u : kOneWay);
        if (!rev) two_way = false;
      }
    }
  });
  out->symmetric = two_way;
  return true;
}

struct TileInfo {
  int32_t pos0;    // first list position (a multiple of 32)
  int32_t nv;      // vertices
  int32_t seg;
  int32_t slice0;  // first slice (32 vertices each) of the neighbour and of the edge rows
  int32_t bnd0;    // boundary vertices of the tile: [bnd0, bnd0 + nbnd)
  int32_t nbnd;
  int32_t pair0;   // first pair record
  int32_t in_seg;  // index of the tile in its segment
};

struct ChunkInfo {
  int32_t seg;
  int32_t bnd0, nbnd;  // boundary vertices of the chunk
  int32_t slice0;
  int32_t pair0;       // first crossing-pair record
  int32_t pad;
};

struct SegInfo {
  int32_t tile0, ntiles, chunk0, nchunks;
  int64_t pos0, pair0;  // first entries of the segment's ordered lists
  int64_t basin0;       // basins of one sign of the segments before it at most
};
inline int64_t round_up(int64_t x, int64_t a) { return (x + a - 1) / a * a; }

// An array of the tables' memory.
template <typename T>
struct TableArray {
  T* p = nullptr;
  int64_t n = 0, at = 0;  // entries; bytes before it
  int64_t size() const { return n; }
  T* begin() const { return p; }
  T* end() const { return p + n; }
  T& operator[](int64_t i) const {
#ifdef _GLIBCXX_ASSERTIONS
    if (i < 0 || i >= n) __builtin_trap();
#endif
    return p[i];
  }
};

// What basin_plan_create uploads (in one piece), and the sizes that its
// workspaces follow from.
struct BasinTables {
  TableArray<TileInfo> tiles;
  TableArray<ChunkInfo> chunks;
  TableArray<SegInfo> segs;
  TableArray<int32_t> vert, bnd_vert;
  TableArray<uint32_t> slice_off, nbr, edge_off, edge, cross_off, cross;
  TableArray<uint16_t> bnd_local, bnd_tile;
  std::unique_ptr<char[]> memory;  // not cleared: threads write their parts first
  int64_t bytes = 0;
  int64_t n_pair = 0, n_cpair = 0, n_opair = 0;
  int32_t vmax = 1;    // vertices of the largest segment
  int32_t basins = 1;  // basins of one sign of a segment at most
  int64_t all_basins = 0;  // of one sign of all segments

  template <typename F>
  void each(const F& f) {
    f(tiles), f(chunks), f(segs), f(vert), f(bnd_vert), f(slice_off), f(nbr), f(edge_off), f(edge), f(cross_off), f(cross);
    f(bnd_local), f(bnd_tile);
  }
};

// The tables of cleaned lists (see CleanLists: a repeated entry would outgrow
// its row).  False for graphs that the basin form does not take.
//
// Part of making a handle, so a program that sweeps one map pays for it too.
// Handle and first map of an icosphere L5 / L6 / L7 / a 91 x 109 x 91 mask, 16
// cores: 1.7 / 3.1 / 8.2 / 24 ms, of which the tables take 0.5 / 1.6 / 5 / 19
// (sorted tile by tile, joined by one thread and uploaded table by table: 2.0 /
// 5.1 / 12.5 / 32); swept vertex by vertex, without tables and the lists cleaned
// by one thread, 1.4 / 3.3 / 12.0 / 60.
inline bool build_basin_tables(const CleanLists& lists, const std::vector<int64_t>& seg, BasinTables* out) {
  const Raw<int64_t>& off = lists.off;
  const Raw<uint32_t>& packed = lists.packed;
  const int64_t V = off.size() - 1;
  const int n_seg = static_cast<int>(seg.size()) - 1;
  // Tiles: patches grown breadth first from one vertex, so that few entries
  // cross; a patch that cannot grow goes on from the next free vertex, so that
  // all tiles of a segment but the last are full.  Inside a tile the vertices
  // keep their order, so that the statistic is read in runs.
  const Raw<int32_t> tile_of(V);  // 2 t + 1: in tile t of the segment; 2 t: queued by it last, or kFree
  constexpr int32_t kFree = -2;
  std::vector<std::vector<int32_t>> grown(n_seg);  // vertices of a segment's tiles
  parallel_for(n_seg, V, [&](int64_t s) {
    std::fill(tile_of.data() + seg[s], tile_of.data() + seg[s + 1], kFree);
    std::vector<int32_t> queue(2 * kTile), rim;
    int64_t scan = seg[s], left = seg[s + 1] - seg[s];
    while (left > 0) {
      const int32_t id = static_cast<int32_t>(grown[s].size());
      int32_t members = 0;
      int64_t entries = 0;
      bool full = false;
      size_t rim_at = 0;  // of the free vertices beside the last tile
      while (!full && left > 0) {
        while (rim_at < rim.size() && (tile_of[rim[rim_at]] & 1)) ++rim_at;
        size_t head = 0, tail = 1;
        if (rim_at < rim.size()) {
          queue[0] = rim[rim_at];
        } else {
          while (tile_of[scan] & 1) ++scan;
          queue[0] = static_cast<int32_t>(scan);
        }
        tile_of[queue[0]] = 2 * id;
        for (; head < tail; ++head) {
          const int32_t v = queue[head];
          const int64_t e0 = off[v], e1 = off[v + 1];
          if (members == kTile || (entries > 0 && entries + e1 - e0 > kTileEntries)) {
            full = true;
            break;
          }
          entries += e1 - e0;
          tile_of[v] = 2 * id + 1;
          ++members;
          --left;
          if (tail + (e1 - e0) >= queue.size()) queue.resize(2 * (tail + (e1 - e0)));
          for (int64_t e = e0; e < e1; ++e) {  // (no branches: they would be coin tosses)
            const int32_t u = static_cast<int32_t>(packed[e] & kIndexMask), was = tile_of[u];
            const bool fresh = !(was & 1) & (was < 2 * id);
            tile_of[u] = fresh ? 2 * id : was;
            queue[tail] = u;
            tail += fresh;
          }
        }
        if (full || left == 0) rim.assign(queue.begin() + head, queue.begin() + tail);
      }
      grown[s].push_back(members);
    }
  });
  std::vector<TileInfo> tiles;
  std::vector<SegInfo> segs(n_seg);
  int32_t& vmax = out->vmax;
  int64_t n_vert = 0;
  for (int s = 0; s < n_seg; ++s) {
    vmax = std::max<int32_t>(vmax, static_cast<int32_t>(seg[s + 1] - seg[s]));
    segs[s].tile0 = static_cast<int32_t>(tiles.size());
    segs[s].ntiles = static_cast<int32_t>(grown[s].size());
    if (segs[s].ntiles > 32767) return false;  // tile numbers are 15-bit
    for (int t = 0; t < segs[s].ntiles; ++t) {
      TileInfo ti{};
      ti.seg = s;
      ti.nv = grown[s][t];
      ti.in_seg = t;
      ti.pos0 = static_cast<int32_t>(n_vert);
      n_vert = round_up(n_vert + ti.nv, 32);
      if (n_vert > 0x7fffffffLL) return false;
      tiles.push_back(ti);
    }
  }
  const int nt = static_cast<int>(tiles.size());
  const Raw<int32_t> vert(n_vert);  // (a tile's last slice is filled up with vertex 0)
  // a vertex's place: its tile in the segment, and its index there (12 bits)
  const Raw<int32_t>& place = tile_of;
  parallel_for(n_seg, V, [&](int64_t s) {
    std::vector<int32_t> filled(segs[s].ntiles, 0);
    for (int64_t v = seg[s]; v < seg[s + 1]; ++v) {
      const int32_t t = tile_of[v] >> 1, i = filled[t]++;
      place[v] = t << 12 | i;
      vert[tiles[segs[s].tile0 + t].pos0 + i] = static_cast<int32_t>(v);
    }
    for (int32_t t = 0; t < segs[s].ntiles; ++t) {
      const TileInfo& ti = tiles[segs[s].tile0 + t];
      std::fill(vert.data() + ti.pos0 + ti.nv, vert.data() + round_up(ti.pos0 + ti.nv, 32), 0);
    }
  });
  // entries that basin_cross_kernel takes: to another tile, or one-way
  static_assert(kTile == 1 << 12, "the index in a tile has 12 bits");
  auto crosses = [&](int64_t v, uint32_t entry) { return (entry & kOneWay) || ((place[entry & kIndexMask] ^ place[v]) >> 12) != 0; };
  // rows of neighbours and of pairs of neighbours, by tile
  struct Rows {
    std::vector<uint32_t> nbr, nbr_end, edge, edge_end;
    int64_t n_edges = 0, n_basins = 0;
  };
  std::vector<Rows> rows(nt);
  std::vector<uint8_t> is_bnd(V, 0);
  parallel_for(nt, off[V], [&](int64_t t) {
    const int32_t* const mem = vert.data() + tiles[t].pos0;
    const int nv = tiles[t].nv;
    Rows& r = rows[t];
    // rows of 32 lanes, two entries (4 * index) a lane; padding: the vertex itself
    auto put = [&](std::vector<uint32_t>& out, std::vector<uint32_t>& ends, const std::vector<uint16_t>& list,
                   const std::vector<int32_t>& at, const std::vector<int32_t>& count) {
      size_t words = 0;
      for (int i = 0; i < nv; i += 32) {
        const int width = *std::max_element(count.begin() + i, count.begin() + std::min(nv, i + 32));
        words += static_cast<size_t>((width + 1) / 2) * 32;
        ends.push_back(static_cast<uint32_t>(words) | (width & 1 ? kOddRow : 0u));
      }
      out.resize(words);
      size_t o = 0;
      for (int i = 0; i < nv; i += 32) {
        const int width = *std::max_element(count.begin() + i, count.begin() + std::min(nv, i + 32));
        for (int j = 0; j < width; j += 2)
          for (int v = i; v < i + 32; ++v) {
            const uint32_t self = std::min(v, nv - 1);
            const int c = v < nv ? count[v] : 0;
            const uint32_t x = j < c ? list[at[v] + j] : self, y = j + 1 < c ? list[at[v] + j + 1] : self;
            out[o++] = 4u * x | (4u * y << 16);
          }
      }
    };
    std::vector<int32_t> at(nv + 1, 0), count(nv, 0), held_count(nv, 0);
    for (int i = 0; i < nv; ++i) at[i + 1] = at[i] + static_cast<int32_t>(off[mem[i] + 1] - off[mem[i]]);
    std::vector<uint16_t> near(at[nv]), held(at[nv]);
    auto hold = [&](int v, int u) { held[at[v] + held_count[v]++] = static_cast<uint16_t>(u); };
    for (int i = 0; i < nv; ++i) {
      const int32_t v = mem[i];
      for (int64_t e = off[v]; e < off[v + 1]; ++e) {
        if (crosses(v, packed[e])) {
          __atomic_store_n(&is_bnd[packed[e] & kIndexMask], uint8_t{1}, __ATOMIC_RELAXED);
          __atomic_store_n(&is_bnd[v], uint8_t{1}, __ATOMIC_RELAXED);
          continue;
        }
        const uint16_t u = place[packed[e] & kIndexMask] & (kTile - 1);
        near[at[i] + count[i]++] = u;
        if (u < i) continue;
        // each pair of neighbours once, held by the one that holds fewer so far
        if (held_count[u] < held_count[i]) hold(u, i);
        else hold(i, u);
        ++r.n_edges;
      }
    }
    put(r.nbr, r.nbr_end, near, at, count);
    for (int pass = 0; pass < 4; ++pass)  // even out: a vertex hands one to a neighbour that holds two fewer
      for (int i = 0; i < nv; ++i)
        for (int j = 0; j < held_count[i]; ++j) {
          const int u = held[at[i] + j];
          if (held_count[u] + 1 < held_count[i]) {
            held[at[i] + j] = held[at[i] + --held_count[i]];
            hold(u, i);
          }
        }
    put(r.edge, r.edge_end, held, at, held_count);
    // Basins at most: of vertices that are all neighbours of one another only
    // the highest can start one.  Covered greedily by triples and pairs.
    std::vector<uint8_t> covered(nv, 0);
    for (int i = 0; i < nv; ++i) {
      if (covered[i]) continue;
      covered[i] = 1;
      ++r.n_basins;
      int u = -1, w = -1;
      for (int j = 0; j < count[i] && w < 0; ++j) {
        const int x = near[at[i] + j];
        if (covered[x]) continue;
        if (u < 0) u = x;
        else if (std::find(near.begin() + at[x], near.begin() + at[x] + count[x], u) != near.begin() + at[x] + count[x])
          w = x;
      }
      if (u >= 0) covered[u] = 1;
      if (w >= 0) covered[w] = 1;
    }
  });
  // where the tiles' parts go, and the boundary vertices
  std::vector<int32_t> bnd_vert;
  const Raw<int32_t> bnd_of(V);  // of boundary vertices
  std::vector<uint16_t> bnd_local, bnd_tile;
  std::vector<int64_t> nbr0(nt), edge0(nt), seg_pairs(n_seg, 0), seg_basins(n_seg, 0);
  int64_t &n_pair = out->n_pair, n_nbr = 0, n_edge = 0, n_slice = 0;
  for (int t = 0; t < nt; ++t) {
    TileInfo& ti = tiles[t];
    const Rows& r = rows[t];
    ti.slice0 = static_cast<int32_t>(n_slice);
    ti.bnd0 = static_cast<int32_t>(bnd_vert.size());
    ti.pair0 = static_cast<int32_t>(n_pair);
    nbr0[t] = n_nbr;
    edge0[t] = n_edge;
    n_slice += static_cast<int64_t>(r.nbr_end.size());
    n_nbr += static_cast<int64_t>(r.nbr.size());
    n_edge += static_cast<int64_t>(r.edge.size());
    if (r.n_edges > 65535) return false;  // pairs are counted in 16 bits
    seg_basins[ti.seg] += r.n_basins;
    seg_pairs[ti.seg] += round_up(r.n_edges, 8);  // pairs of basins: at most one per pair of neighbours
    n_pair += round_up(r.n_edges, 8);
    if (n_pair > 0x7fffffffLL || n_nbr >= (1LL << 32) || n_edge >= (1LL << 31)) return false;
    const int32_t* const mem = vert.data() + ti.pos0;
    for (int i = 0; i < ti.nv; ++i) {
      if (!is_bnd[mem[i]]) continue;
      bnd_of[mem[i]] = static_cast<int32_t>(bnd_vert.size());
      bnd_local.push_back(static_cast<uint16_t>(i));
      bnd_vert.push_back(mem[i]);
      bnd_tile.push_back(static_cast<uint16_t>(ti.in_seg));
    }
    ti.nbnd = static_cast<int32_t>(bnd_vert.size()) - ti.bnd0;
  }
  // crossing lists, in chunks of boundary vertices of one segment
  std::vector<ChunkInfo> chunks;
  for (int s = 0; s < n_seg; ++s) {
    segs[s].chunk0 = static_cast<int32_t>(chunks.size());
    if (segs[s].ntiles) {
      const TileInfo& first = tiles[segs[s].tile0];
      const TileInfo& last = tiles[segs[s].tile0 + segs[s].ntiles - 1];
      for (int32_t b0 = first.bnd0; b0 < last.bnd0 + last.nbnd; b0 += kCrossChunk) {
        ChunkInfo c{};
        c.seg = s;
        c.bnd0 = b0;
        c.nbnd = std::min<int32_t>(kCrossChunk, last.bnd0 + last.nbnd - b0);
        chunks.push_back(c);
      }
    }
    segs[s].nchunks = static_cast<int32_t>(chunks.size()) - segs[s].chunk0;
  }
  const int n_chunks = static_cast<int>(chunks.size());
  std::vector<Rows> crows(n_chunks);
  parallel_for(n_chunks, 16 * static_cast<int64_t>(bnd_vert.size()), [&](int64_t c) {
    std::vector<uint32_t> list[32];
    for (int i = 0; i < chunks[c].nbnd; i += 32) {
      size_t width = 0;
      for (int l = 0; l < 32; ++l) {
        list[l].clear();
        if (i + l >= chunks[c].nbnd) continue;
        const int32_t v = bnd_vert[chunks[c].bnd0 + i + l];
        for (int64_t e = off[v]; e < off[v + 1]; ++e)
          if (crosses(v, packed[e])) list[l].push_back(static_cast<uint32_t>(bnd_of[packed[e] & kIndexMask]));
        crows[c].n_edges += static_cast<int64_t>(list[l].size());
        width = std::max(width, list[l].size());
      }
      for (size_t j = 0; j < width; ++j)
        for (int l = 0; l < 32; ++l) {
          const int self = std::min(i + l, chunks[c].nbnd - 1);  // padding: the vertex itself
          crows[c].nbr.push_back(j < list[l].size() ? list[l][j] : static_cast<uint32_t>(chunks[c].bnd0 + self));
        }
      crows[c].nbr_end.push_back(static_cast<uint32_t>(crows[c].nbr.size()));
    }
  });
  std::vector<int64_t> cross0(n_chunks);
  int64_t &n_cpair = out->n_cpair, n_cross = 0, n_cross_slice = 0;
  for (int c = 0; c < n_chunks; ++c) {
    chunks[c].slice0 = static_cast<int32_t>(n_cross_slice);
    chunks[c].pair0 = static_cast<int32_t>(n_cpair);
    cross0[c] = n_cross;
    n_cross_slice += static_cast<int64_t>(crows[c].nbr_end.size());
    n_cross += static_cast<int64_t>(crows[c].nbr.size());
    n_cpair += round_up(crows[c].n_edges, 4);
    seg_pairs[chunks[c].seg] += round_up(crows[c].n_edges, 4);
    if (n_cpair > 0x7fffffffLL || n_cross >= (1LL << 32)) return false;
  }
  int64_t& n_opair = out->n_opair;
  for (int s = 0; s < n_seg; ++s) {
    segs[s].pos0 = seg[s];
    segs[s].pair0 = n_opair;
    segs[s].basin0 = out->all_basins;
    out->all_basins += seg_basins[s];
    n_opair += seg_pairs[s];
  }
  out->basins = static_cast<int32_t>(std::max<int64_t>(1, *std::max_element(seg_basins.begin(), seg_basins.end())));
  // all of it in one piece of memory
  BasinTables& o = *out;
  o.tiles.n = nt;
  o.chunks.n = n_chunks;
  o.segs.n = n_seg;
  o.vert.n = n_vert;
  o.slice_off.n = o.edge_off.n = n_slice + 1;
  o.nbr.n = n_nbr;
  o.edge.n = n_edge;
  o.cross_off.n = n_cross_slice + 1;
  o.cross.n = n_cross;
  o.bnd_vert.n = o.bnd_local.n = o.bnd_tile.n = static_cast<int64_t>(bnd_vert.size());
  o.each([&](auto& a) {
    a.at = o.bytes;
    o.bytes += round_up(a.n * static_cast<int64_t>(sizeof(*a.p)), 256);
  });
  o.memory.reset(new char[o.bytes]);
  o.each([&](auto& a) { a.p = reinterpret_cast<std::remove_reference_t<decltype(a.p)>>(o.memory.get() + a.at); });
  auto copy = [](const auto& from, auto* to) { std::copy(from.begin(), from.end(), to); };
  copy(tiles, o.tiles.p);
  copy(chunks, o.chunks.p);
  copy(segs, o.segs.p);
  std::copy(vert.data(), vert.data() + n_vert, o.vert.p);
  copy(bnd_vert, o.bnd_vert.p);
  copy(bnd_local, o.bnd_local.p);
  copy(bnd_tile, o.bnd_tile.p);
  o.slice_off[0] = o.edge_off[0] = o.cross_off[0] = 0;
  parallel_for(nt + n_chunks, (n_nbr + n_edge + n_cross) / 16, [&](int64_t u) {
    if (u < nt) {
      const Rows& r = rows[u];
      copy(r.nbr, o.nbr.p + nbr0[u]);
      copy(r.edge, o.edge.p + edge0[u]);
      for (size_t i = 0; i < r.nbr_end.size(); ++i) {
        o.slice_off[tiles[u].slice0 + 1 + i] = static_cast<uint32_t>(nbr0[u]) + (r.nbr_end[i] & ~kOddRow);
        o.edge_off[tiles[u].slice0 + 1 + i] = static_cast<uint32_t>(edge0[u]) + r.edge_end[i];
      }
    } else {
      const int64_t c = u - nt;
      copy(crows[c].nbr, o.cross.p + cross0[c]);
      for (size_t i = 0; i < crows[c].nbr_end.size(); ++i)
        o.cross_off[chunks[c].slice0 + 1 + i] = static_cast<uint32_t>(cross0[c]) + crows[c].nbr_end[i];
    }
  });
  return true;
}

}  // namespace tfgb
