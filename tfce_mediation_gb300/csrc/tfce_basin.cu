// Basin form of the batched TFCE sweep: the GB300 replacement of
// tfce_mediation/lib/fast_tfce.hpp:11-95 for every batched launch.
//
// The reference inserts the vertices by decreasing value and joins each to the
// neighbours that were inserted before it.  Here every vertex first points to
// its largest neighbour, inside a tile of up to 4,096 vertices kept in shared
// memory.  Following the pointers gives the vertex's basin, a tree whose
// members are connected from their own activation on.  So the component of a
// vertex at any threshold is the component of its basin, and only the list
// entries that join two different basins need a union: on a smooth map of 164k
// vertices that leaves 2.5k basins and 15k pairs per sign, of 164k vertices
// and 983k entries, and the union-find state of a sweep fits in shared memory.
//
//   basin_max_kernel    segment maxima of +x and -x
//   basin_tile_kernel   one CTA per (map, tile), both signs at once (their
//                       vertices are disjoint): activation steps, basins, and
//                       the pairs of basins that neighbours join
//   basin_cross_kernel  the pairs that cross a tile boundary
//   basin_offset_kernel where each tile's entries go in the segment's lists
//   basin_order_kernel  the segment's lists, ordered by (sign, step)
//   basin_sweep_kernel  one CTA per (map, sign, segment): threshold steps over
//                       the lists, union-find over basins
//   basin_walk_kernel   vertex values of the reference's float accumulation
//
// Measured on one GB300 against the vertex-by-vertex sweep that batched
// launches ran before (its state, 5 MB an item, was walked at random in DRAM):
// 512 maps x 2 hemispheres x +/- of the L7 icosphere, smooth: 21.9 -> 4.35 ms
// (tile 2.25, sweep 1.37, order 0.38, cross 0.18, max 0.11); unsmoothed noise,
// 128 maps: 10.1 -> 2.75 ms; 48 maps of 242k voxels, 26 neighbours, E = 0.5: 9.8
// -> 1.17 ms; one map: 4.64 -> 0.39 ms.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <map>
#include <memory>

#include "basin.cuh"
#include "basin_tables.h"
#include "sweep_common.cuh"

namespace tfgb {

constexpr int kTileThreads = 512;
constexpr int kPerThread = kTile / kTileThreads;
constexpr int kBuckets = 256;          // sign * 128 + step
constexpr int kTab = kBuckets + 2;     // bucket starts and the total
constexpr uint32_t kNegative = 0x80000000u, kPositive = 0x40000000u;  // sign of a vertex of a tile
constexpr uint32_t kRoot = 0x80000000u;
constexpr uint32_t kExtent = 0x00ffffffu;
constexpr int kPairTable = 2048;       // slots for the distinct pairs of basins of a tile
constexpr int kCrossTable = 1024;      // the same for a chunk of boundary vertices
constexpr int kProbes = 12;            // slots tried
constexpr int kQueue = 96;              // neighbours that wait in a warp's queue: 31 and two rows' worth
constexpr int kCrossThreads = 256;
constexpr int kCrossPer = 4;
constexpr int kCrossRows = 4;           // rows of neighbours whose loads are in flight together
constexpr int kCrossQueue = 64;         // 31 and a row's worth
static_assert(kCrossChunk == kCrossThreads * kCrossPer, "a CTA takes a chunk");
constexpr int kMaxSweepThreads = 1024;
constexpr int kSmBytes = 226 * 1024;   // shared memory of an SM's sweeps together
constexpr int kSweepBytes = 4352;      // of a sweep besides its state
constexpr int kFindLimit = 1 << 26;
constexpr int kAhead = 4;              // pairs of events that a thread of the sweep loads a step ahead
constexpr uint32_t kNone = 0xffffffffu;
constexpr int kReady = 1 << 30;         // in a class's counter: the first of the sweep's launches sees the lists

struct Node {
  float inc;
  uint32_t next;
};

enum SweepMode { kMaxima = 0, kPotential = 1, kNodes = 2 };

struct BasinArgs {
  // request
  const float* stats;
  int64_t map_stride;
  int32_t n_maps, signs, n_seg;
  const float* vdensity;
  float* out_max;
  float* out_maps;
  int32_t out_mode;
  int64_t n_vertices;
  const int32_t* thr_group;
  const float* seg_H;
  const int64_t* seg_off;
  const int32_t* seg_rank;
  int32_t* err;
  // plan
  const TileInfo* tiles;
  const ChunkInfo* chunks;
  const SegInfo* segs;
  const int32_t* vert;        // vertex of a list position
  const uint32_t* slice_off;  // first row entry of a slice; the next slice's ends it
  const uint32_t* nbr;        // two neighbours each (4 * index in the tile), 32 lanes a row
  const uint32_t* edge_off;   // the same for the rows that hold each pair of neighbours once
  const uint32_t* edge;
  const uint16_t* bnd_local;  // boundary vertex: its index in its tile
  const int32_t* bnd_vert;    // its vertex
  const uint16_t* bnd_tile;   // its tile in the segment
  const uint32_t* cross_off;  // slices of the crossing lists
  const uint32_t* cross;      // boundary vertices, 32 lanes a row
  const double* const* seg_pow;  // extent^E, or NULL for E == 1
  int32_t n_tiles, n_chunks, n_bnd;
  // workspace
  uint32_t* seg_max;    // [maps][2][n_seg] bits of max(0, max)
  int32_t* counter;     // items taken and, of the queued ones, there are: by class (2 * class, 2 * class + 1)
  uint32_t* ev;         // vertices of a tile by bucket: bucket << 24, index in the tile << 12, basin
  uint32_t* pairs;      // pairs of basins of a tile: bucket << 24, 12 bits each
  uint2* cpairs;        // crossing pairs: tile << 16 | 4 bits of the bucket << 12 | basin, twice
  uint16_t* tab_ev;     // [map][tile][kTab] first entry of every bucket, and their number
  uint16_t* tab_pair;
  uint32_t* tab_cross;  // [map][chunk][kBuckets]
  uint32_t* n_pairs;    // [map][tile] and, after them, [map][chunk]
  uint16_t* n_basin;    // [map][tile][2]
  uint2* bnd;           // [map][boundary vertex] {float bits, basin | step << 16}
  uint32_t* off_ev;     // [map][tile][kBuckets]: entries of earlier tiles in the bucket
  uint32_t* off_pair;
  uint32_t* off_cross;  // [map][chunk][kBuckets]
  uint32_t* base_of;    // [map][tile][2] first basin number of the tile
  uint32_t* start_ev;   // [map][seg][kTab] bucket starts of the ordered lists
  uint32_t* start_pair;
  uint32_t* n_basins;   // [map][seg][2]
  void* ev_out;         // ordered: basin of an active vertex (16 bits, or 32 beyond the shared state)
  void* pair_out;       // ordered: pairs of basins (2 x 16 or 2 x 32 bits)
  int32_t* ord;         // ordered: vertex
  double* base;         // ordered: potential of the component before the vertex joined
  uint32_t* vnode;      // ordered: first node of the vertex
  Node* nodes;          // [maps][signs][node_cap]; a segment's from basin0 * kMaxSteps: step * basins + basin
  uint32_t* part_max;   // [items] encoded maximum
  uint32_t* n_steps;    // [items]
  int64_t pos_per_map, pair_per_map, cpair_per_map, opair_per_map;
  int64_t node_cap;
  char* state;
  int64_t state_bytes;
  int32_t* queue;       // [2][n_items] items of the middle and of the large class
  int32_t n_items;
  int32_t most_first;   // basins of an item of the small class
  int32_t most_mid;     // of the middle class: all state in shared memory too
  int32_t mid;          // the launch takes the middle class
  int32_t first_class;  // and is the first of the classes' launches
  int32_t most_narrow;  // basins of an item whose state (but the lists) is in shared memory
};

// The kernels of a call on few tiles are launched without waiting for one
// another's end (programmatic dependent launch): each begins with this, which
// waits for the one before, and lets the next one's CTAs start beside the last
// of its own.  Up to a tile per SM a call gains 10 us (one map of 2,562 vertices
// 214 -> 204 us, of 163,842 503 -> 490); launches that fill the chip lose 1 %
// (the waiting CTAs' room) and go out plainly, where this does nothing.
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ---------------------------------------------------------------------------
__device__ inline float seg_maximum(const BasinArgs& a, int64_t map, int sgn, int seg) {
  return __uint_as_float(a.seg_max[(map * 2 + sgn) * a.n_seg + seg]);
}

// the maximum that the threshold table of (map, sign, segment) starts from
__device__ inline float table_maximum(const BasinArgs& a, int64_t map, int sgn, int seg) {
  if (!a.thr_group) return seg_maximum(a, map, sgn, seg);
  const int32_t g = a.thr_group[seg];
  float m = 0.0f;
  for (int s = 0; s < a.n_seg; ++s)
    if (a.thr_group[s] == g) m = fmaxf(m, seg_maximum(a, map, sgn, s));
  return m;
}

// Activation step: the first i with x > T[i] (strict, fast_tfce.hpp:41), or L,
// by comparing, from a guess on.
__device__ __noinline__ int step_beside(float x, const float* T, int L, int i) {
  if (L == 0 || !(x > T[L - 1])) return L;
  i = max(0, min(i, L - 1));
  while (i > 0 && x > T[i - 1]) --i;
  while (!(x > T[i])) ++i;  // ends at L - 1
  return i;
}

// The same from the place of x between the thresholds, in steps: T falls by dT
// a step up to float rounding, which adds up to less than 4e-4 of a step over
// the table, so away from a threshold by 1e-3 of a step the place gives the
// step.  inv = 100 / tmx, or 0 for tables that are not the usual 100 or 101
// steps of a normal float (every x is then compared).  place: 1 .. 4095, larger
// the further x is above its threshold.
__device__ inline int step_of(float x, const float* T, int L, float tmx, float inv, uint32_t* place) {
  constexpr float kInt = 12582912.0f;  // 1.5 * 2^23: adding it rounds to an integer, in the low bits
  const float q = (tmx - x) * inv;
  const float t = (q - 0.5f) + kInt;
  const float f = q - (t - kInt);
  int i = __float_as_int(t) - 0x4b400000;
  *place = __float_as_uint(fmaf(-4094.0f, __saturatef(f), 4095.0f) + kInt) & 0xfffu;
  if (f > 1e-3f && f < 0.999f) return min(i + 1, L);
  return step_beside(x, T, L, i);
}

__device__ inline float step_scale(float tmx, int L) {
  return (L >= 100 && L <= 101 && tmx > 1e-30f && tmx < 1e30f) ? __fdiv_rn(100.0f, tmx) : 0.0f;
}

// Block-wide exclusive scan of kBuckets counters by the first 256 threads:
// start[b], start[kBuckets] = total.  Ends with a barrier.
__device__ inline void scan_buckets(int* cnt, int* wsum) {
  const int t = threadIdx.x, lane = t & 31;
  int v = 0, inc = 0;
  if (t < kBuckets) {
    v = cnt[t];
    inc = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    if (lane == 31) wsum[t >> 5] = inc;
  }
  __syncthreads();
  if (t < kBuckets) {
    int before = 0;
    for (int w = 0; w < (t >> 5); ++w) before += wsum[w];
    cnt[t] = before + inc - v;
    if (t == kBuckets - 1) cnt[kBuckets] = before + inc;
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// Maxima of +x and -x of every (map, segment), finite values, at least 0.
__global__ void __launch_bounds__(256) basin_max_kernel(BasinArgs a, int32_t parts) {
  after_previous();
  __shared__ float red[32];
  const int64_t b = blockIdx.x;
  const int part = static_cast<int>(b % parts);
  const int seg = static_cast<int>((b / parts) % a.n_seg);
  const int64_t map = b / parts / a.n_seg;
  const int64_t v0 = a.seg_off[seg], n = a.seg_off[seg + 1] - v0;
  const int64_t per = (n + parts - 1) / parts;
  const int64_t lo = v0 + part * per, hi = min(v0 + n, lo + per);
  const float* x = a.stats + map * a.map_stride;
  float mp = 0.0f, mn = 0.0f;
  for (int64_t v = lo + threadIdx.x; v < hi; v += 256) {
    const float xv = x[v];
    if (isfinite(xv)) {
      mp = fmaxf(mp, xv);
      mn = fmaxf(mn, -xv);
    }
  }
  mp = block_max(mp, red);
  mn = block_max(mn, red);
  if (threadIdx.x == 0) {
    if (mp > 0.0f) atomicMax(a.seg_max + (map * 2) * a.n_seg + seg, __float_as_uint(mp));
    if (mn > 0.0f) atomicMax(a.seg_max + (map * 2 + 1) * a.n_seg + seg, __float_as_uint(mn));
  }
}

// ---------------------------------------------------------------------------
// Activation steps, basins and pairs of basins of one tile of one map.
//
// A vertex is one 32-bit word in shared memory: sign, 127 - step, place inside
// the step (12 bits) and 4095 - index (12 bits).  Words of one sign order the
// tile's vertices by step, then by value, then by index, without ties, so the
// neighbour to point to is a running maximum and carries its own index; a
// neighbour of the other sign is negative after the sign is taken out, an
// inactive one 0.  Any order that keeps the steps gives the same components
// (two-way entries; one-way ones are left to basin_cross_kernel).  Once a
// vertex's root is known its word becomes sign, 128 - step, root, and every
// pair of neighbours with different roots is a pair of basins, joined at the
// later step of the two.
//
// Bound by instruction issue (3.3 of 4 a cycle; 430 warp instructions per 32
// vertices of a mesh: keys 71, neighbours 81, pointers 71, pairs 154, sort 53):
// 2.25 ms for 512 maps x 2 L7.  The pairs' test reads the class of both words at
// once, and rows of an odd width leave their last halves out (198 for the pairs
// before).
__global__ void __launch_bounds__(kTileThreads, 4) basin_tile_kernel(BasinArgs a) {
  after_previous();
  __shared__ uint32_t key[kTile];
  __shared__ __align__(16) uint16_t lab[kTile];  // pointer, then root (2 * index in the tile)
  uint32_t* const table = reinterpret_cast<uint32_t*>(lab);  // distinct pairs, once lab is done with
  static_assert(kPairTable * sizeof(uint32_t) <= sizeof(lab), "the table takes lab's place");
  __shared__ uint16_t rk[kTile];   // basin number of a root
  __shared__ float sT[2][kMaxSteps];
  __shared__ int cnt[kBuckets + 1], pcnt[kBuckets], wsum[8];
  __shared__ float4 sTab[2];  // maximum, steps per unit, step count
  __shared__ int nroots[2], npairs;
  __shared__ uint32_t sQueue[kTileThreads / 32 * kQueue];
  const int tile = blockIdx.x % a.n_tiles;
  const int64_t map = blockIdx.x / a.n_tiles;
  const TileInfo ti = a.tiles[tile];
  const int tid = threadIdx.x, lane = tid & 31;
  const float* x = a.stats + map * a.map_stride;
  const int32_t* vert = a.vert + ti.pos0;

  float xv[kPerThread];
#pragma unroll
  for (int k = 0; k < kPerThread; ++k) {
    const int v = tid + k * kTileThreads;
    xv[k] = (v < ti.nv) ? x[vert[v]] : 0.0f;
  }
  if (tid < 2) {
    const int sgn = tid;
    const float m = (sgn < a.signs) ? table_maximum(a, map, sgn, ti.seg) : 0.0f;
    const int L = threshold_table(m, sT[sgn], a.err);
    sTab[sgn] = make_float4(m, step_scale(m, L), __int_as_float(L), 0.0f);
    nroots[sgn] = 0;
    npairs = 0;
  }
  if (tid < kBuckets) cnt[tid] = pcnt[tid] = 0;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kPerThread; ++k) {
    const int v = tid + k * kTileThreads;
    const int sgn = xv[k] < 0.0f;
    uint32_t w = 0;
    if ((__float_as_uint(xv[k]) & 0x7fffffffu) - 1u < 0x7f7fffffu) {  // finite, and not 0
      const float4 tab = sTab[sgn];
      const int L = __float_as_int(tab.z);
      uint32_t place;
      const int st = step_of(fabsf(xv[k]), sT[sgn], L, tab.x, tab.y, &place);
      if (st < L) w = (static_cast<uint32_t>(127 - st) << 24) | (place << 12) | static_cast<uint32_t>(4095 - v);
      if (sgn) w = 0u - w;
    }
    if (v < ti.nv) key[v] = w;
  }
  __syncthreads();

  auto at = [&](uint32_t offset) { return *reinterpret_cast<const uint32_t*>(reinterpret_cast<const char*>(key) + offset); };
  // the largest neighbour (the smallest, for the negative sign)
#pragma unroll 4
  for (int k = 0; k < kPerThread; ++k) {
    const int v = tid + k * kTileThreads;
    if (v < ti.nv) {
      const uint32_t* so = a.slice_off + ti.slice0 + (v >> 5);
      const uint32_t o1 = so[1];
      const int kv = static_cast<int>(key[v]);
      int hi = kv, lo = kv;
#pragma unroll 3
      for (uint32_t o = so[0] + lane; o < o1; o += 32) {
        const uint32_t two = a.nbr[o];
        const int x0 = static_cast<int>(at(two & 0xffffu)), x1 = static_cast<int>(at(two >> 16));
        hi = max(max(hi, x0), x1);
        lo = min(min(lo, x0), x1);
      }
      const int best = kv < 0 ? -lo : hi;
      lab[v] = static_cast<uint16_t>(8190 - 2 * (best & 0xfff));
    }
  }
  __syncthreads();
  // Follow the pointers, two hops at a time (a root points to itself; a stored
  // root shortens the walks that pass it; keys grow along them, so they end);
  // number the basins.
#pragma unroll 2
  for (int k = 0; k < kPerThread; ++k) {
    const int v = tid + k * kTileThreads;
    const int kv = (v < ti.nv) ? static_cast<int>(key[v]) : 0;
    if (kv) {
      auto up = [&](uint32_t o) { return *reinterpret_cast<volatile uint16_t*>(reinterpret_cast<char*>(lab) + o); };
      uint32_t r = up(2 * v);
      for (;;) {
        const uint32_t n = up(r);
        r = up(n);
        if (r == n) break;
      }
      *reinterpret_cast<volatile uint16_t*>(lab + v) = static_cast<uint16_t>(r);
      r >>= 1;
      const int sgn = kv < 0;
      const uint32_t code = (static_cast<uint32_t>(abs(kv)) >> 24) + 1u;  // 128 - step
      atomicAdd(&cnt[sgn * kMaxSteps + kMaxSteps - code], 1);
      key[v] = (sgn ? kNegative : kPositive) | (code << 12) | r;
      if (r == static_cast<uint32_t>(v)) rk[v] = static_cast<uint16_t>(atomicAdd(&nroots[sgn], 1));
    }
  }
  __syncthreads();
  for (int i = tid; i < kPairTable; i += kTileThreads) table[i] = 0u;
  scan_buckets(cnt, wsum);
  const int64_t row = map * a.n_tiles + tile;
  if (tid <= kBuckets) a.tab_ev[row * kTab + tid] = static_cast<uint16_t>(cnt[tid]);
  // A pair of basins matters at the first step that joins it: the table keeps
  // {pair, 128 - step} words and their maximum per pair.  A pair that finds no
  // slot is written down as it comes (joining two basins again changes nothing).
  uint32_t* pr = a.pairs + map * a.pair_per_map + ti.pair0;
  auto emit = [&](uint32_t e) {
    const uint32_t i = e >> 20, j = (e >> 8) & 0xfffu;
    const uint32_t b = (key[i] >> 31) * kMaxSteps + kMaxSteps - (e & 0xffu);
    atomicAdd(&pcnt[b], 1);
    pr[atomicAdd(&npairs, 1)] = (b << 24) | (static_cast<uint32_t>(rk[i]) << 12) | rk[j];
  };
  // the neighbours of different roots wait in a queue of the warp until there
  // are 32 for a full round
  uint32_t* const queue = sQueue + (tid >> 5) * kQueue;
  int nq = 0;
  auto insert = [&](int q) {
    const uint32_t w = at(queue[q] >> 16), u = at(queue[q] & 0xffffu);
    const uint32_t i = w & 0xfffu, j = u & 0xfffu;
    const uint32_t e = (min(i, j) << 20) | (max(i, j) << 8) | (min(u & 0xff000u, w & 0xff000u) >> 12);
    uint32_t h = ((e >> 8) * 2654435761u) >> 21;
    static_assert(kPairTable == 1 << 11, "the hash gives 11 bits");
    for (int t = 0;; ++t) {
      uint32_t cur = *reinterpret_cast<volatile uint32_t*>(table + h);
      if (cur == 0u) cur = atomicCAS(&table[h], 0u, e);
      if (cur == 0u || (cur ^ e) < 256u) {
        if (cur != 0u && cur < e) atomicMax(&table[h], e);
        break;
      }
      if (t == kProbes) {
        emit(e);
        break;
      }
      h = (h + 1) & (kPairTable - 1);
    }
  };
  const uint32_t below = (1u << lane) - 1u;
  for (int k = 0; k < kPerThread; ++k) {
    const int v = tid + k * kTileThreads;
    if (v - lane >= ti.nv) break;
    const uint32_t w = (v < ti.nv) ? key[v] : 0u, sign = w & (kPositive | kNegative);
    const uint32_t* so = a.edge_off + ti.slice0 + (v >> 5);
    const uint32_t end = so[1], o1 = end & ~kOddRow;
    // neighbours of the same sign with another root
    auto check = [&](uint32_t off) {
      const uint32_t u = at(off);
      const bool hit = (u & sign) && ((u ^ w) & 0xfffu);
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (hit) queue[nq + __popc(m & below)] = (static_cast<uint32_t>(v) << 18) | off;
      nq += __popc(m);
    };
    for (uint32_t o = (so[0] & ~kOddRow) + lane; o < o1; o += 32) {
      const uint32_t two = a.edge[o];
      check(two & 0xffffu);
      if (!(end & kOddRow) || o + 32 < o1) check(two >> 16);
      while (nq >= 32) {
        __syncwarp();
        insert(nq - 32 + lane);
        nq -= 32;
        __syncwarp();
      }
    }
  }
  __syncwarp();
  if (lane < nq) insert(lane);
  // boundary vertices, for the pairs that cross tiles
  for (int q = tid; q < ti.nbnd; q += kTileThreads) {
    const int i = ti.bnd0 + q;
    const uint32_t w = key[a.bnd_local[i]];
    a.bnd[map * a.n_bnd + i] = make_uint2(w ? __float_as_uint(x[a.bnd_vert[i]]) : 0u,
                                          w ? (rk[w & 0xfffu] | ((kMaxSteps - ((w >> 12) & 0xffu)) << 16)) : kNone);
  }
  __syncthreads();
  for (int i = tid; i < kPairTable; i += kTileThreads)
    if (table[i]) emit(table[i]);
  // the vertices in order of their buckets, in place of the keys
  uint32_t rec[kPerThread];
#pragma unroll
  for (int k = 0; k < kPerThread; ++k) {
    const int v = tid + k * kTileThreads;
    rec[k] = (v < ti.nv) ? key[v] : 0u;
  }
  const int n_ev = cnt[kBuckets];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kPerThread; ++k) {
    if (rec[k] == 0u) continue;
    const uint32_t b = (rec[k] >> 31) * kMaxSteps + kMaxSteps - ((rec[k] >> 12) & 0xffu);
    key[atomicAdd(&cnt[b], 1)] = (b << 24) | (static_cast<uint32_t>(tid + k * kTileThreads) << 12) | rk[rec[k] & 0xfffu];
  }
  __syncthreads();
  uint32_t* ev = a.ev + map * a.pos_per_map + ti.pos0;
  for (int p = tid; p < n_ev; p += kTileThreads) ev[p] = key[p];
  if (tid < kBuckets) a.tab_pair[row * kBuckets + tid] = static_cast<uint16_t>(pcnt[tid]);
  if (tid < 2) a.n_basin[row * 2 + tid] = static_cast<uint16_t>(nroots[tid]);
  if (tid == 2) a.n_pairs[row] = npairs;
}

// Pairs that cross a tile boundary, and one-way entries: every boundary vertex
// with the distinct basins of its listed neighbours that precede it by value
// (ties by smaller vertex, the reference's insertion order).  Bound by
// instructions on voxel graphs (97k boundary vertices a map, 13 rows each);
// inserting row by row, with a few lanes each, 48 maps took 331 us, with full
// rounds from a queue 247.
__global__ void __launch_bounds__(kCrossThreads) basin_cross_kernel(BasinArgs a) {
  after_previous();
  __shared__ int cnt[kBuckets], total;
  __shared__ unsigned long long table[kCrossTable];  // {tile << 12 | basin, twice} << 8 | 128 - step
  // pairs wait in a queue of the warp until there are 32 for a full round
  __shared__ unsigned long long sQueue[kCrossThreads / 32 * kCrossQueue];
  const int chunk = blockIdx.x % a.n_chunks;
  const int64_t map = blockIdx.x / a.n_chunks;
  const ChunkInfo ci = a.chunks[chunk];
  const int tid = threadIdx.x, lane = tid & 31;
  const uint2* rec = a.bnd + map * a.n_bnd;
  cnt[tid] = 0;
  if (tid == 0) total = 0;
  for (int i = tid; i < kCrossTable; i += kCrossThreads) table[i] = 0;
  __syncthreads();
  uint2* out = a.cpairs + map * a.cpair_per_map + ci.pair0;
  // sign of a pair: that of its basins, in the top bit of the first
  auto emit = [&](unsigned long long e) {
    const uint32_t i = static_cast<uint32_t>(e >> 36), j = static_cast<uint32_t>(e >> 8) & 0xfffffffu;
    const uint32_t b = (i >> 27) * kMaxSteps + kMaxSteps - static_cast<uint32_t>(e & 0xffu);
    atomicAdd(&cnt[b], 1);
    out[atomicAdd(&total, 1)] = make_uint2(((i << 4) & 0x7fff0000u) | ((b >> 4) << 12) | (i & 0xfffu),
                                           ((j << 4) & 0x7fff0000u) | ((b & 15u) << 12) | (j & 0xfffu));
  };
  unsigned long long* const queue = sQueue + (tid >> 5) * kCrossQueue;
  int nq = 0;
  auto insert = [&](unsigned long long e) {
    uint32_t h = static_cast<uint32_t>(((e >> 8) * 0x9e3779b97f4a7c15ull) >> 54);
    static_assert(kCrossTable == 1 << 10, "the hash gives 10 bits");
    for (int t = 0;; ++t) {
      unsigned long long cur = *reinterpret_cast<volatile unsigned long long*>(&table[h]);
      if (cur == 0) cur = atomicCAS(&table[h], 0ull, e);
      if (cur == 0 || (cur ^ e) < 256) {
        if (cur != 0 && cur < e) atomicMax(&table[h], e);
        break;
      }
      if (t == kProbes) {
        emit(e);
        break;
      }
      h = (h + 1) & (kCrossTable - 1);
    }
  };
  for (int k = 0; k < kCrossPer; ++k) {
    const int q = tid + k * kCrossThreads;
    if (q - lane >= ci.nbnd) break;
    const uint2 me = q < ci.nbnd ? rec[ci.bnd0 + q] : make_uint2(0u, kNone);
    const bool active = me.y != kNone;
    if (!__any_sync(0xffffffffu, active)) continue;
    const int vme = active ? a.bnd_vert[ci.bnd0 + q] : 0;
    const uint32_t s = me.x & 0x80000000u;
    const uint32_t mine = (static_cast<uint32_t>(active ? a.bnd_tile[ci.bnd0 + q] : 0) << 12) | (me.y & 0xfffu);
    const int own = active ? static_cast<int>(me.x ^ s) : 0x7fffffff;
    const uint32_t code = kMaxSteps - (me.y >> 16);
    const int sl = ci.slice0 + (q >> 5);
    uint32_t last = mine;  // (a one-way entry may lead to the vertex's own basin, which is no pair)
    const uint32_t o1 = a.cross_off[sl + 1];
    for (uint32_t o = a.cross_off[sl] + lane; o < o1; o += 32 * kCrossRows) {
      uint32_t ub[kCrossRows];
      uint2 r[kCrossRows];
#pragma unroll
      for (int j = 0; j < kCrossRows; ++j) ub[j] = o + 32 * j < o1 ? a.cross[o + 32 * j] : 0xffffffffu;
#pragma unroll
      for (int j = 0; j < kCrossRows; ++j) r[j] = ub[j] != 0xffffffffu ? rec[ub[j]] : make_uint2(s, kNone);
#pragma unroll
      for (int j = 0; j < kCrossRows; ++j) {
        if (o - lane + 32 * j >= o1) break;
        const int w = static_cast<int>(r[j].x ^ s);
        bool hit = w > own || (w == own && active && a.bnd_vert[ub[j]] < vme);
        uint32_t other = 0;
        if (hit) {
          other = (static_cast<uint32_t>(a.bnd_tile[ub[j]]) << 12) | (r[j].y & 0xfffu);
          hit = other != last && other != mine;
          if (hit) last = other;
        }
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (hit) {
          const unsigned long long pair =
              (static_cast<unsigned long long>(min(mine, other) | (s >> 4)) << 28) | max(mine, other);
          queue[nq + __popc(m & ((1u << lane) - 1u))] = (pair << 8) | code;
        }
        nq += __popc(m);
        if (nq >= 32) {
          __syncwarp();
          insert(queue[nq - 32 + lane]);
          nq -= 32;
          __syncwarp();
        }
      }
    }
  }
  __syncwarp();
  if (lane < nq) insert(queue[lane]);
  __syncthreads();
  for (int i = tid; i < kCrossTable; i += kCrossThreads)
    if (table[i]) emit(table[i]);
  __syncthreads();
  a.tab_cross[(map * a.n_chunks + chunk) * kBuckets + tid] = static_cast<uint32_t>(cnt[tid]);
  if (tid == 0) a.n_pairs[(int64_t)a.n_maps * a.n_tiles + map * a.n_chunks + chunk] = total;
}

// Where each tile's entries go: per bucket, the entries of the tiles (and
// chunks) before it, and the bucket starts of the segment's lists; first basin
// number of every tile.  One CTA per (map, segment), one thread per bucket.
__global__ void __launch_bounds__(kBuckets) basin_offset_kernel(BasinArgs a) {
  after_previous();
  __shared__ int tot[kBuckets + 1], wsum[8];
  const int seg = blockIdx.x % a.n_seg;
  const int64_t map = blockIdx.x / a.n_seg;
  const SegInfo si = a.segs[seg];
  const int b = threadIdx.x;
  const int64_t row0 = map * a.n_tiles + si.tile0, crow0 = map * a.n_chunks + si.chunk0;
  const int64_t out = (map * a.n_seg + seg) * kTab;
  uint32_t run = 0;
#pragma unroll 8
  for (int t = 0; t < si.ntiles; ++t) {
    const uint16_t* start = a.tab_ev + (row0 + t) * kTab + b;
    a.off_ev[(row0 + t) * kBuckets + b] = run - start[0];  // for a place in the tile's own order
    run += static_cast<uint32_t>(start[1]) - start[0];
  }
  tot[b] = run;
  __syncthreads();
  scan_buckets(tot, wsum);
  a.start_ev[out + b] = tot[b];
  if (b == 0) a.start_ev[out + kBuckets] = tot[kBuckets];
  run = 0;
#pragma unroll 8
  for (int t = 0; t < si.ntiles; ++t) {
    const uint32_t n = a.tab_pair[(row0 + t) * kBuckets + b];
    a.off_pair[(row0 + t) * kBuckets + b] = run;
    run += n;
  }
#pragma unroll 4
  for (int c = 0; c < si.nchunks; ++c) {
    const uint32_t n = a.tab_cross[(crow0 + c) * kBuckets + b];
    a.off_cross[(crow0 + c) * kBuckets + b] = run;
    run += n;
  }
  __syncthreads();
  tot[b] = run;
  __syncthreads();
  scan_buckets(tot, wsum);
  a.start_pair[out + b] = tot[b];
  if (b == 0) a.start_pair[out + kBuckets] = tot[kBuckets];
  if (b < 64) {  // one warp per sign
    const int lane = b & 31, sgn = b >> 5;
    uint32_t before = 0;
    for (int t0 = 0; t0 < si.ntiles; t0 += 32) {
      const uint32_t v = (t0 + lane < si.ntiles) ? a.n_basin[(row0 + t0 + lane) * 2 + sgn] : 0u;
      uint32_t inc = v;
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
      }
      if (t0 + lane < si.ntiles) a.base_of[(row0 + t0 + lane) * 2 + sgn] = before + inc - v;
      before += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) {
      a.n_basins[(map * a.n_seg + seg) * 2 + sgn] = before;
      if (sgn < a.signs && before > static_cast<uint32_t>(a.most_first)) {
        const int large = before > static_cast<uint32_t>(a.most_mid);
        a.queue[large * a.n_items + atomicAdd(a.counter + 2 * large + 3, 1)] =
            static_cast<int32_t>((map * a.signs + sgn) * a.n_seg + seg);
      }
    }
  }
}

// The segment's ordered lists, with basin numbers of the whole segment: 16
// bits a basin where the sweep keeps its state in shared memory, else 32.  One
// CTA per (map, tile) and (map, chunk).  The order within a bucket is free.
// A tile's vertices are in order already, so the segment's list is written in
// runs.  Bound by the latency of a CTA's loads (512 maps x 2 L7: 525 us with the
// sort in here, 387 with all loads issued before the first is used).
template <bool kOrder>
__global__ void __launch_bounds__(kTileThreads, 4) basin_order_kernel(BasinArgs a) {
  after_previous();
  __shared__ uint32_t to_ev[kBuckets], to_pair[kBuckets];
  const int units = a.n_tiles + a.n_chunks;
  const int unit = blockIdx.x % units;
  const int64_t map = blockIdx.x / units;
  const int tid = threadIdx.x;
  const bool is_tile = unit < a.n_tiles;
  const int chunk = unit - a.n_tiles;
  const int seg = is_tile ? a.tiles[unit].seg : a.chunks[chunk].seg;
  const SegInfo si = a.segs[seg];
  const int64_t srow = (map * a.n_seg + seg) * kTab;
  const uint32_t* nbs = a.n_basins + (map * a.n_seg + seg) * 2;
  const bool wide0 = nbs[0] > (uint32_t)a.most_narrow, wide1 = nbs[1] > (uint32_t)a.most_narrow;
  // the second sign's 16-bit entries start where its 32-bit ones would
  const uint32_t ev1 = a.start_ev[srow + kMaxSteps], pr1 = a.start_pair[srow + kMaxSteps];
  const int64_t po = map * a.opair_per_map + si.pair0;
  if (is_tile) {
    const TileInfo ti = a.tiles[unit];
    const int64_t row = map * a.n_tiles + unit;
    const uint32_t* ev = a.ev + map * a.pos_per_map + ti.pos0;
    uint32_t rec[kPerThread];  // all loads at once: a CTA lives for little more than their latency
#pragma unroll
    for (int k = 0; k < kPerThread; ++k) {
      const int p = tid + k * kTileThreads;
      rec[k] = p < ti.nv ? ev[p] : 0u;
    }
    if (tid < kBuckets) {
      to_ev[tid] = a.start_ev[srow + tid] + a.off_ev[row * kBuckets + tid];
      to_pair[tid] = a.start_pair[srow + tid] + a.off_pair[row * kBuckets + tid];
    }
    const uint32_t base0 = a.base_of[row * 2], base1 = a.base_of[row * 2 + 1];
    const int n_pr = static_cast<int>(a.n_pairs[row]);
    const int n_ev = a.tab_ev[row * kTab + kBuckets];
    const uint32_t* pr = a.pairs + map * a.pair_per_map + ti.pair0;
    uint32_t first = 0;
    if (tid < n_pr) first = pr[tid];
    __syncthreads();
    const int64_t eo = map * a.n_vertices + si.pos0;
    uint32_t* ev32 = reinterpret_cast<uint32_t*>(a.ev_out) + eo;
    uint16_t* ev16 = reinterpret_cast<uint16_t*>(a.ev_out) + 2 * eo;
#pragma unroll
    for (int k = 0; k < kPerThread; ++k) {
      const int p = tid + k * kTileThreads;
      if (p >= n_ev) break;
      const uint32_t r = rec[k];
      const uint32_t bk = r >> 24, d = to_ev[bk] + p;
      const bool neg = bk >= kMaxSteps;
      const uint32_t id = (neg ? base1 : base0) + (r & 0xfffu);
      if (neg ? wide1 : wide0) ev32[d] = id;
      else ev16[d + (neg ? ev1 : 0u)] = static_cast<uint16_t>(id);
      if (kOrder) a.ord[eo + d] = a.vert[ti.pos0 + ((r >> 12) & 0xfffu)];
    }
    for (int p = tid; p < n_pr; p += kTileThreads) {
      const uint32_t r = p == tid ? first : pr[p];
      const uint32_t bk = r >> 24;
      const uint32_t d = atomicAdd(&to_pair[bk], 1u);
      const bool neg = bk >= kMaxSteps;
      const uint32_t base = neg ? base1 : base0;
      const uint32_t i = base + ((r >> 12) & 0xfffu), j = base + (r & 0xfffu);
      if (neg ? wide1 : wide0) reinterpret_cast<uint2*>(a.pair_out)[po + d] = make_uint2(i, j);
      else reinterpret_cast<uint32_t*>(a.pair_out)[2 * po + (neg ? pr1 : 0u) + d] = (i << 16) | j;
    }
  } else {
    const ChunkInfo ci = a.chunks[chunk];
    const int64_t row = map * a.n_chunks + chunk;
    if (tid < kBuckets) to_pair[tid] = a.start_pair[srow + tid] + a.off_cross[row * kBuckets + tid];
    const uint32_t* base = a.base_of + (map * a.n_tiles + si.tile0) * 2;
    const int n = static_cast<int>(a.n_pairs[(int64_t)a.n_maps * a.n_tiles + row]);
    __syncthreads();
    const uint2* pr = a.cpairs + map * a.cpair_per_map + ci.pair0;
    for (int p = tid; p < n; p += kTileThreads) {
      const uint2 r = pr[p];
      const uint32_t bk = (((r.x >> 12) & 15u) << 4) | ((r.y >> 12) & 15u);
      const uint32_t d = atomicAdd(&to_pair[bk], 1u);
      const int sgn = bk >= kMaxSteps;
      const uint32_t i = base[(r.x >> 16) * 2 + sgn] + (r.x & 0xfffu), j = base[(r.y >> 16) * 2 + sgn] + (r.y & 0xfffu);
      if (sgn ? wide1 : wide0) reinterpret_cast<uint2*>(a.pair_out)[po + d] = make_uint2(i, j);
      else reinterpret_cast<uint32_t*>(a.pair_out)[2 * po + (sgn ? pr1 : 0u) + d] = (i << 16) | j;
    }
  }
}

// ---------------------------------------------------------------------------
// Threshold steps of one (map, sign, segment).  Bound by latency: a step is a
// chain of a few hundred dependent instructions on shared memory, and 100
// steps follow one another (about 2 us a step alone on an SM), so what counts
// is how many sweeps an SM holds.  The union-find state of an item's basins is
// private to the CTA: in shared memory, or (more basins than fit) in the CTA's
// slot of global memory, read and written at CTA scope.
//
// Arrays of that state, addressed in the shared window (kShared) or in global
// memory; every access is one explicit instruction on the state space, which
// the threads of the CTA order with barriers or read through atomics.
template <bool kShared, typename T>
struct StateArray {
  using Base = typename std::conditional<kShared, uint32_t, char*>::type;
  Base base;
  __device__ Base at(uint32_t i) const { return base + i * static_cast<uint32_t>(sizeof(T)); }
  __device__ T ld(uint32_t i) const {
    if constexpr (kShared) {
      if constexpr (sizeof(T) == 2) {
        uint16_t v;
        asm volatile("ld.relaxed.cta.shared.u16 %0, [%1];" : "=h"(v) : "r"(at(i)) : "memory");
        return v;
      } else if constexpr (sizeof(T) == 4) {
        uint32_t v;
        asm volatile("ld.relaxed.cta.shared.u32 %0, [%1];" : "=r"(v) : "r"(at(i)) : "memory");
        return v;
      } else {
        double v;
        asm volatile("ld.relaxed.cta.shared.f64 %0, [%1];" : "=d"(v) : "r"(at(i)) : "memory");
        return v;
      }
    } else if constexpr (sizeof(T) == 2) {
      uint16_t v;
      asm volatile("ld.relaxed.cta.global.u16 %0, [%1];" : "=h"(v) : "l"(glob(i)) : "memory");
      return v;
    } else if constexpr (sizeof(T) == 4) {
      uint32_t v;
      asm volatile("ld.relaxed.cta.global.u32 %0, [%1];" : "=r"(v) : "l"(glob(i)) : "memory");
      return v;
    } else {
      double v;
      asm volatile("ld.relaxed.cta.global.f64 %0, [%1];" : "=d"(v) : "l"(glob(i)) : "memory");
      return v;
    }
  }
  __device__ void st(uint32_t i, T v) const {
    if constexpr (kShared) {
      if constexpr (sizeof(T) == 2) asm volatile("st.relaxed.cta.shared.u16 [%0], %1;" ::"r"(at(i)), "h"(v) : "memory");
      else if constexpr (sizeof(T) == 4)
        asm volatile("st.relaxed.cta.shared.u32 [%0], %1;" ::"r"(at(i)), "r"(v) : "memory");
      else asm volatile("st.relaxed.cta.shared.f64 [%0], %1;" ::"r"(at(i)), "d"(v) : "memory");
    } else if constexpr (sizeof(T) == 2) {
      asm volatile("st.relaxed.cta.global.u16 [%0], %1;" ::"l"(glob(i)), "h"(v) : "memory");
    } else if constexpr (sizeof(T) == 4) {
      asm volatile("st.relaxed.cta.global.u32 [%0], %1;" ::"l"(glob(i)), "r"(v) : "memory");
    } else {
      asm volatile("st.relaxed.cta.global.f64 [%0], %1;" ::"l"(glob(i)), "d"(v) : "memory");
    }
  }
  __device__ uint32_t cas(uint32_t i, uint32_t expect, uint32_t v) const {
    uint32_t old;
    if constexpr (kShared)
      asm volatile("atom.relaxed.cta.shared.cas.b32 %0, [%1], %2, %3;" : "=r"(old) : "r"(at(i)), "r"(expect), "r"(v) : "memory");
    else
      asm volatile("atom.relaxed.cta.global.cas.b32 %0, [%1], %2, %3;" : "=r"(old) : "l"(glob(i)), "r"(expect), "r"(v) : "memory");
    return old;
  }
  __device__ uint32_t add(uint32_t i, uint32_t v) const {
    uint32_t old;
    if constexpr (kShared)
      asm volatile("atom.relaxed.cta.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(at(i)), "r"(v) : "memory");
    else
      asm volatile("atom.relaxed.cta.global.add.u32 %0, [%1], %2;" : "=r"(old) : "l"(glob(i)), "r"(v) : "memory");
    return old;
  }
  // old, or `none` where `on` is false (a predicate, not a branch)
  __device__ uint32_t add_if(bool on, uint32_t i, uint32_t v, uint32_t none) const {
    uint32_t old = none;
    if constexpr (kShared)
      asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %3, 0;\n@p atom.relaxed.cta.shared.add.u32 %0, [%1], %2;\n}"
                   : "+r"(old) : "r"(at(i)), "r"(v), "r"(static_cast<uint32_t>(on)) : "memory");
    else if (on) old = add(i, v);
    return old;
  }
  __device__ void max_with(uint32_t i, uint32_t v) const {
    if constexpr (kShared) asm volatile("red.relaxed.cta.shared.max.u32 [%0], %1;" ::"r"(at(i)), "r"(v) : "memory");
    else asm volatile("red.relaxed.cta.global.max.u32 [%0], %1;" ::"l"(glob(i)), "r"(v) : "memory");
  }

 private:
  __device__ char* glob(uint32_t i) const { return (char*)base + (size_t)i * sizeof(T); }
};

// Where a sweep keeps its state: all in shared memory; the lists of live basins
// in global memory (read in order, a step's entries at a time); all global.
enum StateKind { kAllShared = 0, kListsGlobal = 1, kAllGlobal = 2 };

// A basin's word is its parent, or while it is a root kRoot, its age (127 - the
// step it started at, 0 before; 7 bits) and its extent (24 bits).  The older
// root takes the younger one in, ties by number, which keeps the trees flat:
// a large component's root stays, and what it takes in points to it at once.
// Ages only grow, and a root is linked by a CAS on the word that it was
// compared with, so the order along parents is strict and walks end.
template <int kMode, int kKind>
struct BasinState {
  static constexpr bool kShared = kKind != kAllGlobal;
  using W = typename std::conditional<kMode == kPotential, double, uint32_t>::type;
  using Idx = typename std::conditional<kShared, uint16_t, uint32_t>::type;
  StateArray<kShared, W> w;  // maxima: largest float sum (bits); potentials: sum before step `last`, or offset to the parent
  StateArray<kShared, uint32_t> word;
  StateArray<kKind == kAllShared, Idx> list0;  // potentials: a root's `last`; else live basins; they are packed from one list to the other
  StateArray<kKind == kAllShared, Idx> list1;
  __device__ BasinState(char* smem, char* global, uint32_t n) {
    if constexpr (kShared) w.base = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    else w.base = global;
    word.base = w.at(0) + n * static_cast<uint32_t>(sizeof(W));
    if constexpr (kKind == kListsGlobal) list0.base = global;
    else list0.base = word.base + n * 4u;
    list1.base = list0.base + n * static_cast<uint32_t>(sizeof(Idx));
  }
};
constexpr int state_bytes_per_basin(int mode, int kind) {
  return (mode == kPotential ? 12 : 8) + (kind == kListsGlobal ? 0 : (mode == kPotential ? 1 : 2) * (kind == kAllGlobal ? 4 : 2));
}

// One hop of a walk from x, whose word is w (not a root's); kHalve points x to
// its grandparent.
template <bool kHalve, typename Words>
__device__ inline void hop(const Words& word, uint32_t& x, uint32_t& w) {
  const uint32_t up = word.ld(w);
  if (kHalve && !(up & kRoot)) word.st(x, up);
  x = w;
  w = up;
}

// Roots of x and y, whose words are wx and wy, a hop of both at a time; kHalve
// points x and y themselves to them (halving the path at each hop instead made
// a hop 130 cycles of a lone warp, half of which are this: with the predicated
// adds below 2.92 -> 2.72 ms for 2 x 1024 items of an L7 surface).
template <bool kHalve, typename Words>
__device__ inline void find_two(const Words& word, uint32_t& x, uint32_t& wx, uint32_t& y, uint32_t& wy) {
  const uint32_t x0 = x, y0 = y, x1 = wx, y1 = wy;
  while (!(wx & wy & kRoot)) {
    if (!(wx & kRoot)) {
      x = wx;
      wx = word.ld(x);
    }
    if (!(wy & kRoot)) {
      y = wy;
      wy = word.ld(y);
    }
  }
  if (kHalve && !(x1 & kRoot) && x != x1) word.st(x0, x);
  if (kHalve && !(y1 & kRoot) && y != y1) word.st(y0, y);
}

// Root of x, and its word.
template <bool kHalve, typename Words>
__device__ inline uint32_t find_basin(const Words& word, uint32_t x, uint32_t& w) {
  w = word.ld(x);
  while (!(w & kRoot)) hop<kHalve>(word, x, w);
  return x;
}
template <bool kHalve, typename Words>
__device__ inline uint32_t find_basin(const Words& word, uint32_t x) {
  uint32_t w;
  return find_basin<kHalve>(word, x, w);
}

__device__ inline int add_shared(uint32_t at, int v) {
  int old;
  asm volatile("atom.relaxed.cta.shared.add.s32 %0, [%1], %2;" : "=r"(old) : "r"(at), "r"(v) : "memory");
  return old;
}
__device__ inline int load_shared(uint32_t at) {
  int v;
  asm volatile("ld.relaxed.cta.shared.s32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
  return v;
}
__device__ inline void store_shared(uint32_t at, int v) {
  asm volatile("st.relaxed.cta.shared.s32 [%0], %1;" ::"r"(at), "r"(v) : "memory");
}

// Potentials.  A component that keeps its extent from step a to step b gains
// extent^E * (HH_a + .. + HH_b-1), so a root's sum is brought up to a step only
// where its extent changes: it holds the sum before step `last`, and what it
// gained since follows from the sums of HH from a step to the end (small to
// large, so that late steps keep their precision).  Adding every live
// component's increment at every step, in double, took 5,000 of a step's 8,200
// cycles (6k basins, unsmoothed): two additions or conversions per SM and cycle.
// 256 such items: 654 -> 363 us.
__device__ inline double brought_up(double sum, const double* pw, const float* HH, const double* rest, uint32_t word,
                                    int from, int to) {
  const uint32_t ext = word & kExtent;
  if (ext == 0u || from == to) return sum;
  // an extent as a double, by way of a float, off the double pipe
  const uint32_t u = __float_as_uint(static_cast<float>(ext));
  const double power = pw ? pw[ext] : __hiloint2double(static_cast<int>((u >> 3) + 0x38000000u), static_cast<int>(u << 29));
  double gain = rest[from] - rest[to];
  if (!isfinite(rest[from])) {  // a threshold whose power overflows: added up as it comes
    gain = 0.0;
    for (int i = from; i < to; ++i) gain += static_cast<double>(HH[i]);
  }
  return fma(power, gain, sum);
}

// rest[i] of a table of L steps, by one warp.
__device__ inline void sum_rest(const float* HH, int L, double* rest) {
  constexpr int kPer = kMaxSteps / 32;
  const int lane = threadIdx.x & 31;
  double sum[kPer], later = 0.0;
#pragma unroll
  for (int k = kPer - 1; k >= 0; --k) {
    const int i = lane * kPer + k;
    later += i < L ? static_cast<double>(HH[i]) : 0.0;
    sum[k] = later;
  }
  double mine = later;  // of this lane's steps and all later ones
  for (int o = 1; o < 32; o <<= 1) {
    const double v = __shfl_down_sync(0xffffffffu, mine, o);
    if (lane + o < 32) mine += v;
  }
  const double beyond = __shfl_down_sync(0xffffffffu, mine, 1);
#pragma unroll
  for (int k = 0; k < kPer; ++k) rest[lane * kPer + k] = sum[k] + (lane < 31 ? beyond : 0.0);
  if (lane == 31) rest[kMaxSteps] = 0.0;
}

struct SweepShared {
  float T[kMaxSteps], HH[kMaxSteps];
  int ev[kMaxSteps + 1], pair[kMaxSteps + 1];  // first entries of the steps
  float red[32];
  double rest[kMaxSteps + 1];  // potentials: sum of HH from a step to the last
  int L, item, n_basins;
  int n_live[3];  // by packs modulo 3: the list's, the packed one's, and one being cleared
};

__device__ inline uint32_t enc_float(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ inline float dec_float(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

template <int kMode, int kKind>
__device__ __forceinline__ void sweep_item(const BasinArgs& a, SweepShared& S, char* smem, char* global, int64_t map,
                                           int sgn, int seg, int64_t item) {
  constexpr bool kNarrow = kKind != kAllGlobal;
  constexpr bool kHalve = kMode != kPotential;  // a linked root's parent is what its offset refers to
  const SegInfo si = a.segs[seg];
  const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31, wbase = tid - lane;
  const int nb = S.n_basins, L = S.L;
  BasinState<kMode, kKind> st(smem, global, nb);
  const int64_t eo = map * a.n_vertices + si.pos0, po = map * a.opair_per_map + si.pair0;
  const int e1 = sgn ? S.ev[0] : 0, p1 = sgn ? S.pair[0] : 0;
  // events are read two at a time, at even places: entry q of the list is at
  // place q + e1 (16 bits) or q (32 bits)
  const uint32_t* ev16 = reinterpret_cast<const uint32_t*>(a.ev_out) + eo;
  const uint32_t* ev32 = reinterpret_cast<const uint32_t*>(a.ev_out) + eo;
  const int shift = kNarrow ? e1 : 0;
  const uint32_t* pair16 = reinterpret_cast<const uint32_t*>(a.pair_out) + 2 * po + p1;
  const uint2* pair32 = reinterpret_cast<const uint2*>(a.pair_out) + po;
  // the two events at the even place p, as far as they are in [lo, hi)
  using Two = typename std::conditional<kNarrow, uint32_t, uint2>::type;
  auto load_two = [&](int p, int lo, int hi) -> Two {
    if constexpr (kNarrow) {
      (void)lo;
      return p < hi ? ev16[p >> 1] : 0u;
    } else {
      return make_uint2(p >= lo && p < hi ? ev32[p] : 0u, p + 1 >= lo && p + 1 < hi ? ev32[p + 1] : 0u);
    }
  };
  auto split = [](const Two& t) -> uint2 {
    if constexpr (kNarrow) return make_uint2(t & 0xffffu, t >> 16);
    else return t;
  };
  auto load_pair = [&](int q) -> uint2 {
    if constexpr (kNarrow) {
      const uint32_t r = pair16[q];
      return make_uint2(r >> 16, r & 0xffffu);
    } else {
      return pair32[q];
    }
  };
  const double* pw = a.seg_pow[seg];
  for (int i = tid; i < nb; i += nth) {
    st.word.st(i, kRoot);
    st.w.st(i, 0);
    if constexpr (kMode == kPotential) st.list0.st(i, 0);
  }
  if (kMode == kPotential && tid < 32) sum_rest(S.HH, L, S.rest);
  if (tid == 0) S.n_live[0] = S.n_live[1] = S.n_live[2] = 0;
  __syncthreads();
  Node* nodes = (kMode == kNodes) ? a.nodes + (map * a.signs + sgn) * a.node_cap + si.basin0 * kMaxSteps : nullptr;
  // the thread's first entries of a step are loaded a step ahead
  int ev0 = S.ev[0], ev_end = S.ev[1], pr0 = S.pair[0], pr_end = S.pair[1];
  Two next_ev[kAhead] = {};
  uint2 next_pair = make_uint2(0, 0);
  ev0 += shift;
  ev_end += shift;
  auto load_step = [&](int lo, int hi) {
#pragma unroll
    for (int k = 0; k < kAhead; ++k) next_ev[k] = load_two((lo & ~1) + 2 * (tid + k * nth), lo, hi);
  };
  if (L > 0) {
    load_step(ev0, ev_end);
    if (pr0 + tid < pr_end) next_pair = load_pair(pr0 + tid);
  }
  // the list of live basins, the other one, and their counters and a spare one
  auto live = st.list0, other = st.list1;
  // potential of root r, whose word is given, before step i
  auto potential = [&](uint32_t r, uint32_t word, int i) -> double {
    if constexpr (kMode == kPotential) return brought_up(st.w.ld(r), pw, S.HH, S.rest, word, st.list0.ld(r), i);
    return 0.0;
  };
  uint32_t n_live = static_cast<uint32_t>(__cvta_generic_to_shared(&S.n_live[0])), n_next = n_live + 4, n_spare = n_live + 8;

  for (int i = 0; i < L; ++i) {
    Two my_ev[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) my_ev[k] = next_ev[k];
    const uint2 my_pair = next_pair;
    const int ev2 = S.ev[min(i + 2, kMaxSteps)] + shift, pr2 = S.pair[min(i + 2, kMaxSteps)];
    if (i + 1 < L) {
      load_step(ev_end, ev2);
      if (pr_end + tid < pr2) next_pair = load_pair(pr_end + tid);
    }
    if (ev_end > ev0) {
      // (1) join the basins of the step's pairs, one pair per thread at a time;
      // a warp's walks and links go in rounds, all lanes together.  A thread
      // keeps the root that it linked until all pairs are through.  Then roots
      // stand still, and its extent and its sum go to the one that it ended
      // under, once per warp for those that share the first lane's (potentials:
      // it keeps its offset to that one).  Handed over link by link, the many
      // that a large component takes in waited for one another at its word
      // (96 voxel items of a 91 x 109 x 91 mask: 532 -> 423 us; 256 items of
      // L6 surfaces: 283 -> 219 us).
      for (int q0 = pr0; q0 < pr_end; q0 += nth) {
        const int q = q0 + tid;
        uint32_t x = 0, y = 0;
        bool open = q < pr_end;
        bool linked = false;
        uint32_t low = 0, ext = 0;
        if (q0 + wbase < pr_end) {
          uint32_t px = kRoot, py = kRoot;
          if (open) {
            const uint2 r = (q0 == pr0) ? my_pair : load_pair(q);
            x = r.x;
            y = r.y;
            px = st.word.ld(x);
            py = st.word.ld(y);
          }
          for (int it = 0; it < kFindLimit; ++it) {
            find_two<kHalve>(st.word, x, px, y, py);
            __syncwarp();
            open = open && x != y;
            if (open) {
              const uint32_t ax = px >> 24, ay = py >> 24;
              const bool x_up = ax != ay ? ax > ay : x < y;
              const uint32_t was = x_up ? py : px;
              low = x_up ? y : x;
              if (st.word.cas(low, was, x_up ? x : y) == was) {
                open = false;
                linked = true;
                ext = was & kExtent;
              }
            }
            if (!__any_sync(0xffffffffu, open)) break;
            px = py = kRoot;
            if (open) {
              px = st.word.ld(x);
              py = st.word.ld(y);
            }
          }
          if (open) set_err(a.err, kDevLoopLimit);
        }
        __syncthreads();
        if constexpr (kMode == kPotential) {
          uint32_t r = 0, was_r = 0;
          double sum_r = 0.0;
          if (linked) {
            r = find_basin<kHalve>(st.word, low, was_r);
            sum_r = potential(r, was_r, i);
            st.w.st(low, potential(low, ext, i) - sum_r);
            st.word.st(low, r);
          }
          __syncthreads();
          // the first to change r's extent brings its sum up to this step
          if (linked && ext && st.word.add(r, ext) == was_r) {
            st.w.st(r, sum_r);
            st.list0.st(r, i);
          }
          __syncthreads();  // vertices climb by these
        } else {
          linked = linked && ext;
          const unsigned m = __ballot_sync(0xffffffffu, linked);
          if (m) {
            const uint32_t r = linked ? find_basin<kHalve>(st.word, low) : 0;
            uint32_t sum = 0;
            if (kMode == kMaxima && linked) sum = st.w.ld(low);
            __syncwarp();
            const int first = __ffs(m) - 1;
            const uint32_t r0 = __shfl_sync(0xffffffffu, r, first);
            const bool same = linked && r == r0;
            const uint32_t all_ext = __reduce_add_sync(0xffffffffu, same ? ext : 0u);
            const uint32_t all_sum = kMode == kMaxima ? __reduce_max_sync(0xffffffffu, same ? sum : 0u) : 0u;
            if (lane == first) {
              ext = all_ext;
              sum = all_sum;
            }
            if (lane == first || (linked && !same)) {
              st.word.add(r, ext);
              if constexpr (kMode == kMaxima) st.w.max_with(r, sum);
            }
          }
          if (q0 + nth < pr_end) __syncthreads();
        }
      }
      // the step's vertices join their component
      auto count_two = [&](int p, const Two& t) {
        const uint2 two = split(t);
        uint32_t x = two.x, y = two.y;
        const bool on_x = p >= ev0 && p < ev_end, on_y = p + 1 >= ev0 && p + 1 < ev_end;
        uint32_t root_x = kRoot, root_y = kRoot;  // potentials: the roots' words and sums
        double sum_x = 0.0, sum_y = 0.0;
        if constexpr (kMode == kPotential) {
          auto climb = [&](uint32_t& r, uint32_t& word, double& now, int q) {
            double sum = 0.0;
            for (word = st.word.ld(r); !(word & kRoot); word = st.word.ld(r)) {
              sum += st.w.ld(r);
              r = word;
            }
            now = potential(r, word, i);
            a.base[eo + q - shift] = sum + now;
          };
          if (on_x) climb(x, root_x, sum_x, p);
          if (on_y) climb(y, root_y, sum_y, p + 1);
          __syncthreads();
        } else {
          uint32_t wx = kRoot, wy = kRoot;
          if (on_x) wx = st.word.ld(x);
          if (on_y) wy = st.word.ld(y);
          find_two<kHalve>(st.word, x, wx, y, wy);
        }
        if constexpr (kMode == kNodes) {
          if (on_x) a.vnode[eo + p - shift] = i * nb + x;
          if (on_y) a.vnode[eo + p + 1 - shift] = i * nb + y;
        }
        __syncwarp();
        // those that share the first lane's component are added at once
        const uint32_t r0 = __shfl_sync(0xffffffffu, x, 0);
        const unsigned sx = __ballot_sync(0xffffffffu, on_x && x == r0), sy = __ballot_sync(0xffffffffu, on_y && y == r0);
        const bool leads = lane == __ffs(sx | sy) - 1;
        const uint32_t was_0 = st.word.add_if(leads, r0, __popc(sx) + __popc(sy), kExtent);
        const uint32_t was_x = st.word.add_if(on_x && x != r0, x, 1u, kExtent);
        const uint32_t was_y = st.word.add_if(on_y && y != r0, y, 1u, kExtent);
        // a component's first vertices: it goes live, with its age
        const bool new_0 = !(was_0 & kExtent), new_x = !(was_x & kExtent), new_y = !(was_y & kExtent);
        if constexpr (kMode == kPotential) {
          // the first to change a root's extent brings its sum up to this step
          auto renew = [&](uint32_t r, uint32_t was, double sum) {
            st.w.st(r, sum);
            st.list0.st(r, i);
            if (!(was & kExtent)) st.word.add(r, static_cast<uint32_t>(kMaxSteps - 1 - i) << 24);
          };
          const bool by_x = on_x && x == r0;
          if (leads && was_0 == (by_x ? root_x : root_y)) renew(r0, was_0, by_x ? sum_x : sum_y);
          if (on_x && x != r0 && was_x == root_x) renew(x, was_x, sum_x);
          if (on_y && y != r0 && was_y == root_y) renew(y, was_y, sum_y);
          __syncthreads();
        } else if (new_0 || new_x || new_y) {
          int at = add_shared(n_live, int(new_0) + int(new_x) + int(new_y));
          const uint32_t age = static_cast<uint32_t>(kMaxSteps - 1 - i) << 24;
          if (new_0) {
            live.st(at++, r0);
            st.word.add(r0, age);
          }
          if (new_x) {
            live.st(at++, x);
            st.word.add(x, age);
          }
          if (new_y) {
            live.st(at, y);
            st.word.add(y, age);
          }
        }
      };
      const int even = ev0 & ~1;
      const int ahead = kMode == kPotential ? 0 : wbase;  // the potentials' rounds have barriers
#pragma unroll
      for (int k = 0; k < kAhead; ++k)
        if (even + 2 * (ahead + k * nth) < ev_end) count_two(even + 2 * (tid + k * nth), my_ev[k]);
      for (int p0 = even + 2 * kAhead * nth; p0 + 2 * ahead < ev_end; p0 += 2 * nth)
        count_two(p0 + 2 * tid, load_two(p0 + 2 * tid, ev0, ev_end));
      if (kMode != kPotential) __syncthreads();
    }
    if constexpr (kMode != kPotential) {
      // (3) every live component adds its increment.  Linked ones drop out of
      // the list when it is packed, every eighth step.
      const float HH = S.HH[i];
      const int n = load_shared(n_live);
      const bool pack = (i & 7) == 7;
      // (float)(extent^E * HH): one double product, one rounding
      // (fast_tfce.hpp:77); for E == 1 the double product of an integer below
      // 2^24 and a float is exact, so a float product rounds alike
      auto increment = [&](uint32_t word) {
        const uint32_t ext = word & kExtent;
        return pw ? __double2float_rn(__dmul_rn(pw[ext], static_cast<double>(HH))) : __fmul_rn(static_cast<float>(ext), HH);
      };
      auto grow = [&](uint32_t c, float inc) {
        if constexpr (kMode == kMaxima) st.w.st(c, __float_as_uint(__fadd_rn(__uint_as_float(st.w.ld(c)), inc)));
        if constexpr (kMode == kNodes) nodes[(int64_t)i * nb + c] = Node{inc, c};
      };
      // nodes: a component that was linked at this step leads on to the one that
      // it is part of now (before, it led on to itself).  A node's place follows
      // from its step and basin, so that vertices know theirs as they join (a
      // pass of its own for them cost a quarter of the sweep: 414 -> 342 us)
      auto lead_on = [&](uint32_t c) {
        if constexpr (kMode == kNodes) {
          if (i > 0) nodes[(int64_t)(i - 1) * nb + c].next = find_basin<kHalve>(st.word, c);
        }
      };
      if (!pack) {
        for (int q = tid; q < n; q += nth) {
          const uint32_t c = live.ld(q);
          const uint32_t word = st.word.ld(c);
          if (word & kRoot) grow(c, increment(word));
          else lead_on(c);
        }
      } else {
        for (int q0 = wbase; q0 < n; q0 += nth) {
          const int q = q0 + lane;
          bool root = false;
          uint32_t c = 0;
          if (q < n) {
            c = live.ld(q);
            const uint32_t word = st.word.ld(c);
            root = word & kRoot;
            if (root) grow(c, increment(word));
            else lead_on(c);
          }
          const unsigned m = __ballot_sync(0xffffffffu, root);
          int at = 0;
          if (lane == 0 && m) at = add_shared(n_next, __popc(m));
          at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
          if (root) other.st(at, c);
        }
      }
      if (tid == 0 && pack) store_shared(n_spare, 0);  // the list before this one's: read before the last barrier
      __syncthreads();
      if (pack) {
        auto l = live;
        live = other;
        other = l;
        const uint32_t c = n_live;
        n_live = n_next;
        n_next = n_spare;
        n_spare = c;
      }
    }
    ev0 = ev_end;
    ev_end = ev2;
    pr0 = pr_end;
    pr_end = pr2;
  }

  // largest scaled value (pyfunc.py:116-118); vertices that never became
  // active count as 0
  const float scale = __fdiv_rn(seg_maximum(a, map, sgn, seg), 100.0f);
  const int64_t Vs = a.seg_off[seg + 1] - a.seg_off[seg];
  float best = (L == 0 || S.ev[L] - S.ev[0] < Vs) ? __fmul_rn(0.0f, scale) : -INFINITY;
  if (Vs == 0) best = -INFINITY;
  if constexpr (kMode == kMaxima) {
    const int n = load_shared(n_live);
    for (int q = tid; q < n; q += nth) best = fmaxf(best, __fmul_rn(__uint_as_float(st.w.ld(live.ld(q))), scale));
  }
  if constexpr (kMode == kPotential) {
    for (int r = tid; r < nb; r += nth) {
      const uint32_t word = st.word.ld(r);
      if (word & kRoot) st.w.st(r, potential(r, word, L));
    }
    __syncthreads();
    float* omap = a.out_maps ? a.out_maps + (map * a.signs + sgn) * a.n_vertices : nullptr;
    const int end = L ? S.ev[L] : 0;
    for (int q = S.ev[0] + tid; q < end; q += nth) {
      uint32_t r;
      if constexpr (kNarrow) r = reinterpret_cast<const uint16_t*>(ev16)[q + shift];
      else r = ev32[q];
      double sum = st.w.ld(r);
      for (int it = 0; it < kFindLimit; ++it) {
        const uint32_t p = st.word.ld(r);
        if (p & kRoot) break;
        r = p;
        sum += st.w.ld(r);
      }
      sum -= a.base[eo + q];
      const int64_t v = a.ord[eo + q];
      if (a.out_mode == 2 && omap) sum += static_cast<double>(omap[v]);
      const float val0 = __double2float_rn(sum);
      float val = __fmul_rn(val0, scale);
      if (a.vdensity) val = __fmul_rn(val, a.vdensity[v]);
      if (omap) omap[v] = (a.out_mode == 2) ? val0 : val;
      best = fmaxf(best, val);
    }
  }
  if constexpr (kMode != kNodes) {
    best = block_max(best, S.red);
    if (tid == 0 && a.out_max) a.out_max[item] = (best == -INFINITY) ? 0.0f : best;
  } else {
    if (tid == 0) {
      a.n_steps[item] = L;
      a.part_max[item] = enc_float(best);
    }
  }
}

// One launch per class of items: those of up to most_first basins, those of up
// to most_mid (a queue; all their state in shared memory too, with fewer CTAs
// per SM), and (kLarge) the rest, one CTA per SM with as much shared memory as
// there is.  The launches go out largest class first and do not wait for one
// another: a class's CTAs take the room that the one before leaves.  The end of
// each launch waits for the one before, so that what follows the last of them
// follows all.
template <int kMode, bool kLarge>
__global__ void __launch_bounds__(kLarge ? kMaxSweepThreads : 512, kLarge ? 1 : 2) basin_sweep_kernel(BasinArgs a) {
  __shared__ SweepShared S;
  extern __shared__ __align__(16) char dyn[];
  const int tid = threadIdx.x, nth = blockDim.x;
  // The lists are visible to the launch that waits for the kernel before it.  The
  // launches beside it start after it has let them, and before that it adds
  // kReady to their counters, a release that their first item's acquire meets;
  // a CTA that does not find it waits for the launch before its own.  (A word of
  // its own, released by every CTA and acquired before the first item, made a
  // call of three classes 10 us longer.)
  if (a.first_class) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (blockIdx.x == 0) {
      if (tid < 2 && tid < (kLarge ? 2 : a.mid))
        asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(a.counter + 2 * tid), "r"(kReady) : "memory");
      __syncthreads();
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  } else {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  }
  const int cls = kLarge ? 2 : a.mid;
  int32_t* const counter = a.counter + 2 * cls;
  const int32_t* const queue = a.queue + (kLarge ? a.n_items : 0);
  bool ready = a.first_class;
  for (;;) {
    if (tid == 0) {
      int32_t at;
      if (ready) at = atomicAdd(counter, 1);
      else asm volatile("atom.acquire.gpu.global.add.s32 %0, [%1], 1;" : "=r"(at) : "l"(counter) : "memory");
      S.item = at;
    }
    __syncthreads();
    if (!ready && !(S.item & kReady)) asm volatile("griddepcontrol.wait;" ::: "memory");
    ready = true;
    const int n_items = cls ? counter[1] : a.n_items;
    const int qi = S.item & (kReady - 1);
    if (qi >= n_items) break;
    int64_t out;  // (map * signs + sign) * n_seg + segment
    if (cls) {
      out = queue[qi];
    } else {
      const int per_seg = a.n_items / a.n_seg;  // largest segments first
      out = a.seg_rank ? (int64_t)(qi % per_seg) * a.n_seg + a.seg_rank[qi / per_seg] : qi;
    }
    const int seg = static_cast<int>(out % a.n_seg);
    const int ms = static_cast<int>(out / a.n_seg);
    const int sgn = ms % a.signs;
    const int64_t map = ms / a.signs;
    const int64_t ss = map * a.n_seg + seg;
    const int nb = static_cast<int>(a.n_basins[ss * 2 + sgn]);
    if (!cls && nb > a.most_first) {
      __syncthreads();
      continue;
    }
    for (int i = tid; i <= kMaxSteps; i += nth) {
      S.ev[i] = static_cast<int>(a.start_ev[ss * kTab + sgn * kMaxSteps + i]);
      S.pair[i] = static_cast<int>(a.start_pair[ss * kTab + sgn * kMaxSteps + i]);
    }
    if (tid == 0) {
      S.n_basins = nb;
      S.L = threshold_table(table_maximum(a, map, sgn, seg), S.T, a.err);
    }
    __syncthreads();
    for (int i = tid; i < S.L; i += nth) S.HH[i] = pow_h(S.T[i], a.seg_H[seg]);
    __syncthreads();
    if (!kLarge) {
      sweep_item<kMode, kAllShared>(a, S, dyn, nullptr, map, sgn, seg, out);
    } else {
      char* slot = a.state + blockIdx.x * a.state_bytes;
      if (nb <= a.most_narrow) sweep_item<kMode, kListsGlobal>(a, S, dyn, slot, map, sgn, seg, out);
      else sweep_item<kMode, kAllGlobal>(a, S, dyn, slot, map, sgn, seg, out);
    }
    __syncthreads();
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Fills out_maps for the vertices that never become active: 0 scaled and
// weighted as the others are.
__global__ void basin_fill_kernel(BasinArgs a) {
  after_previous();
  const int64_t V = a.n_vertices, n = (int64_t)a.n_maps * a.signs * V;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    float val = 0.0f;
    if (a.vdensity) val = __fmul_rn(val, a.vdensity[i % V]);
    a.out_maps[i] = val;
  }
}

// Vertex values in the reference's arithmetic: the increments of the vertex's
// component from its own step on, added in float in threshold order
// (fast_tfce.hpp:72-84), along the chain of nodes.
__global__ void __launch_bounds__(256) basin_walk_kernel(BasinArgs a) {
  after_previous();
  __shared__ float red[32];
  const int ms = blockIdx.y / a.n_seg, seg = blockIdx.y % a.n_seg;
  const int sgn = ms % a.signs;
  const int64_t map = ms / a.signs;
  const int64_t item = blockIdx.y;
  const uint32_t* start = a.start_ev + (map * a.n_seg + seg) * kTab + sgn * kMaxSteps;
  const int lo = static_cast<int>(start[0]), hi = static_cast<int>(start[kMaxSteps]);
  const int64_t eo = map * a.n_vertices + a.segs[seg].pos0;
  const Node* nodes = a.nodes + ms * a.node_cap + a.segs[seg].basin0 * kMaxSteps;
  const uint32_t nb = a.n_basins[(map * a.n_seg + seg) * 2 + sgn], L = a.n_steps[item];
  const float scale = __fdiv_rn(seg_maximum(a, map, sgn, seg), 100.0f);
  float* omap = a.out_maps ? a.out_maps + (int64_t)ms * a.n_vertices : nullptr;
  float best = -INFINITY;
  for (int q = lo + blockIdx.x * 256 + threadIdx.x; q < hi; q += gridDim.x * 256) {
    const int64_t v = a.ord[eo + q];
    float acc = (a.out_mode == 2 && omap) ? omap[v] : 0.0f;
    const uint32_t id = a.vnode[eo + q];
    uint32_t c = id % nb;
    for (uint32_t i = id / nb; i < L; ++i) {
      const Node nd = nodes[(int64_t)i * nb + c];
      acc = __fadd_rn(acc, nd.inc);
      c = nd.next;
    }
    float val = __fmul_rn(acc, scale);
    if (a.vdensity) val = __fmul_rn(val, a.vdensity[v]);
    if (omap) omap[v] = (a.out_mode == 2) ? acc : val;
    best = fmaxf(best, val);
  }
  if (a.out_max) {
    best = block_max(best, red);
    if (threadIdx.x == 0 && best > -INFINITY) atomicMax(a.part_max + item, enc_float(best));
  }
}

__global__ void basin_max_out_kernel(BasinArgs a) {
  after_previous();
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < a.n_items; q += gridDim.x * blockDim.x) {
    const float best = dec_float(a.part_max[q]);
    a.out_max[q] = (best == -INFINITY) ? 0.0f : best;
  }
}

__global__ void basin_power_kernel(double* out, int64_t n, float E) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = extent_power(static_cast<int32_t>(i), E);
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
struct BasinPlan {
  int device = 0, sms = 0;
  int32_t n_seg = 0, vmax = 0;
  int32_t basins = 0;  // of one sign of a segment at most
  int64_t V = 0, n_pos = 0, n_pair = 0, n_cpair = 0, n_opair = 0;
  int32_t n_tiles = 0, n_chunks = 0, n_bnd = 0;
  char* tables = nullptr;  // those below, in one piece
  TileInfo* tiles = nullptr;
  ChunkInfo* chunks = nullptr;
  SegInfo* segs = nullptr;
  int32_t* vert = nullptr;
  uint32_t* slice_off = nullptr;
  uint32_t* nbr = nullptr;
  uint32_t* edge_off = nullptr;
  uint32_t* edge = nullptr;
  uint16_t* bnd_local = nullptr;
  int32_t* bnd_vert = nullptr;
  uint16_t* bnd_tile = nullptr;
  uint32_t* cross_off = nullptr;
  uint32_t* cross = nullptr;
  const double** seg_pow = nullptr;
  std::map<float, double*> powers;  // extent^E tables (read through seg_pow)
  int64_t all_basins = 0;  // of one sign of all segments
  char* ws = nullptr;
  int64_t ws_bytes = 0;
  // Once a capture has been seen, a buffer that is replaced by a larger one is
  // kept until the plan goes: captured launches use it.  Growth is geometric.
  bool captured = false;
  int64_t launched = 0;  // kernels
  std::vector<void*> retired;
};

namespace {

// workspace of a launch of M maps
struct Layout {
  int64_t head, ev, pairs, cpairs, tab_ev, tab_pair, tab_cross, n_pairs, queue, n_basin, bnd, off_ev, off_pair, off_cross, base_of,
      start_ev, start_pair, n_basins, ev_out, pair_out, ord, base, vnode, nodes, part, total;
};

Layout layout_of(const BasinPlan* p, int64_t M, int signs, int mode, int64_t node_cap) {
  Layout l{};
  int64_t o = 0;
  auto take = [&](int64_t bytes) {
    const int64_t at = o;
    o += round_up(bytes, 256);
    return at;
  };
  l.head = take(256 + M * 2 * p->n_seg * 4);
  l.ev = take(M * p->n_pos * 4);
  l.pairs = take(M * p->n_pair * 4);
  l.cpairs = take(M * p->n_cpair * 8);
  l.tab_ev = take(M * p->n_tiles * kTab * 2);
  l.tab_pair = take(M * p->n_tiles * kBuckets * 2);
  l.tab_cross = take(M * p->n_chunks * kBuckets * 4);
  l.n_pairs = take(M * (p->n_tiles + p->n_chunks) * 4);
  l.queue = take(2 * M * signs * p->n_seg * 4);
  l.n_basin = take(M * p->n_tiles * 2 * 2);
  l.bnd = take(M * p->n_bnd * 8);
  l.off_ev = take(M * p->n_tiles * kBuckets * 4);
  l.off_pair = take(M * p->n_tiles * kBuckets * 4);
  l.off_cross = take(M * p->n_chunks * kBuckets * 4);
  l.base_of = take(M * p->n_tiles * 2 * 4);
  l.start_ev = take(M * p->n_seg * kTab * 4);
  l.start_pair = take(M * p->n_seg * kTab * 4);
  l.n_basins = take(M * p->n_seg * 2 * 4);
  l.ev_out = take(M * p->V * 4);
  l.pair_out = take(M * p->n_opair * 8);
  if (mode != kMaxima) l.ord = take(M * p->V * 4);
  if (mode == kPotential) l.base = take(M * p->V * 8);
  if (mode == kNodes) {
    l.vnode = take(M * p->V * 4);
    l.nodes = take(M * signs * node_cap * 8);
    l.part = take(2 * M * signs * p->n_seg * 4);
  }
  l.total = o;
  return l;
}

constexpr int64_t kWorkspaceBudget = 8LL << 30;  // maps are swept in as many launches as this asks for
constexpr size_t kPowersKept = 16;  // tables of extent^E that a handle holds on to besides those in use

int64_t node_capacity(const BasinPlan* p) { return p->all_basins * kMaxSteps; }

constexpr int64_t kAskAtOnce = 256LL << 20;  // a workspace that is asked for without a look at free memory (20 us)
constexpr int64_t kStateBudget = 2LL << 30;  // state in global memory of the CTAs of the large class

// tuning knob: the largest workspace that is asked for, in MB
int64_t most_workspace() {
  const char* env = std::getenv("TFCE_SWEEP_WORKSPACE_MB");
  return env ? static_cast<int64_t>(std::max(0, std::atoi(env))) << 20 : INT64_MAX;
}

// A workspace of at least `bytes`.  An outgrown one goes first, or, if a capture
// may have taken its address, with the plan.
int ensure_ws(BasinPlan* p, int64_t bytes, int64_t most) {
  if (p->ws_bytes >= bytes) return TFCE_OK;
  if (bytes > most) {
    set_error("sweep workspace of %lld bytes: more than TFCE_SWEEP_WORKSPACE_MB", static_cast<long long>(bytes));
    return TFCE_ENOMEM;
  }
  int64_t want = std::max(bytes, std::min({2 * p->ws_bytes, most, kWorkspaceBudget}));
  if (p->ws && !p->captured) {
    TFGB_CUDA(cudaDeviceSynchronize());
    cudaFree(p->ws);
    p->ws = nullptr;
    p->ws_bytes = 0;
  }
  char* fresh = nullptr;
  cudaError_t e = cudaMalloc(&fresh, want);
  if (e == cudaErrorMemoryAllocation && want > bytes) {
    cudaGetLastError();
    e = cudaMalloc(&fresh, want = bytes);
  }
  if (e != cudaSuccess) cudaGetLastError();
  TFGB_CUDA(e);
  if (p->ws) p->retired.push_back(p->ws);
  p->ws = fresh;
  p->ws_bytes = want;
  return TFCE_OK;
}

int mode_of(const BasinRequest& r) {
  const bool values = r.vdensity || r.out_maps;
  if (!values && !r.potentials) return kMaxima;  // equal to the float sums bit for bit
  return r.exact ? kNodes : kPotential;
}

// Threads, shared memory and grid of a sweep launch.
struct SweepShape {
  int threads, basins, smem, grid;
};

// tuning knob: fewer CTAs in flight
int most_ctas() {
  const char* env = std::getenv("TFCE_SWEEP_MAX_CTAS");
  return env ? std::max(0, std::atoi(env)) : 0;
}

// The launches of `items` sweeps.  A step of a sweep has about vmax / 128
// entries and is bound by latency, so an SM holds as many items as there are.
// Up to one per SM: as many threads as the steps fill, and all the shared
// memory.  Up to two: CTAs of 512 threads with half of it.  More: CTAs of 256
// threads, four per SM with the state of 4,096 basins each (dense; a smooth map
// of 164k vertices has 3k per sign), and the items with more of them in two per
// SM (256 unsmoothed items of 38k vertices, 5k basins each: one per SM with
// 1,024 threads 894 us, two 654 us).  The classes run beside one another: 320
// items of two surfaces and a voxel skeleton took 353 + 313 us in turn, 390 so.
SweepShape shape_of(const BasinPlan* p, int per_basin, int per_sm, int basins, int most_threads) {
  SweepShape s{};
  s.threads = 128;
  while (s.threads < most_threads && s.threads * 128 < p->vmax) s.threads *= 2;
  s.basins = std::min({basins, (kSmBytes / per_sm - kSweepBytes) / per_basin, p->basins});
  s.smem = s.basins * per_basin;
  const int fit = std::min(1024 / s.threads, kSmBytes / (s.smem + kSweepBytes));
  s.grid = p->sms * (per_sm == 1 ? 1 : std::max(per_sm, fit));
  if (const int cap = most_ctas()) s.grid = std::min(s.grid, cap);
  return s;
}

SweepShape first_shape(const BasinPlan* p, int mode, int64_t items, bool dense) {
  const int per_basin = state_bytes_per_basin(mode, kAllShared);
  const int per_sm = items <= p->sms ? 1 : (items <= 2 * p->sms || !dense) ? 2 : 4;
  return shape_of(p, per_basin, per_sm, per_sm == 4 ? 4096 : 65535, per_sm == 4 ? 256 : 512);
}

// Launches, `chain`: as one of a chain (see after_previous).
template <typename Kernel, typename... Args>
cudaError_t launch_after(bool chain, Kernel kern, dim3 grid, int threads, int smem, cudaStream_t st, const Args&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = chain ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

template <int kMode, bool kLarge>
int launch_sweep_kernel(BasinArgs& a, const SweepShape& s, bool first, bool chain, cudaStream_t st) {
  auto* kern = basin_sweep_kernel<kMode, kLarge>;
  TFGB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmBytes - kSweepBytes));
  a.first_class = first;
  TFGB_CUDA(launch_after(chain || !first, kern, dim3(s.grid), s.threads, s.smem, st, a));
  return TFCE_OK;
}

template <int kMode>
int launch_sweeps(BasinArgs& a, const SweepShape& first, const SweepShape& mid, const SweepShape& large,
                  bool chain, cudaStream_t st) {
  int rc = TFCE_OK;
  if (large.grid) rc = launch_sweep_kernel<kMode, true>(a, large, true, chain, st);
  a.mid = 1;
  if (!rc && mid.grid) rc = launch_sweep_kernel<kMode, false>(a, mid, !large.grid, chain, st);
  a.mid = 0;
  if (!rc) rc = launch_sweep_kernel<kMode, false>(a, first, !large.grid && !mid.grid, chain, st);
  return rc;
}

}  // namespace

int basin_resident_items(const BasinPlan* p, bool dense) {
  return first_shape(p, kMaxima, int64_t{1} << 30, dense).grid;
}

int basin_plan_create(const CleanLists& lists, const std::vector<int64_t>& seg, BasinPlan** out) {
  *out = nullptr;
  BasinTables t;
  if (!build_basin_tables(lists, seg, &t)) return TFCE_OK;
  struct Destroy {
    void operator()(BasinPlan* plan) const { basin_plan_destroy(plan); }
  };
  std::unique_ptr<BasinPlan, Destroy> own(new BasinPlan());
  BasinPlan* const p = own.get();
  cudaGetDevice(&p->device);
  cudaDeviceGetAttribute(&p->sms, cudaDevAttrMultiProcessorCount, p->device);
  p->n_seg = static_cast<int32_t>(seg.size()) - 1;
  p->vmax = t.vmax;
  p->basins = t.basins;
  p->all_basins = t.all_basins;
  p->V = seg.back();
  p->n_pos = static_cast<int64_t>(t.vert.size());
  p->n_pair = t.n_pair;
  p->n_cpair = t.n_cpair;
  p->n_opair = t.n_opair;
  p->n_tiles = static_cast<int32_t>(t.tiles.size());
  p->n_chunks = static_cast<int32_t>(t.chunks.size());
  p->n_bnd = static_cast<int32_t>(t.bnd_vert.size());
  const int64_t pow_at = t.bytes;  // the segments' tables of extent^E: none yet
  TFGB_CUDA(cudaMalloc(&p->tables, t.bytes + p->n_seg * sizeof(double*)));
  TFGB_CUDA(cudaMemcpy(p->tables, t.memory.get(), t.bytes, cudaMemcpyHostToDevice));
  TFGB_CUDA(cudaMemset(p->tables + pow_at, 0, p->n_seg * sizeof(double*)));
  auto on_device = [&](const auto& a, auto*& d) { d = reinterpret_cast<std::remove_reference_t<decltype(d)>>(p->tables + a.at); };
  on_device(t.tiles, p->tiles);
  on_device(t.chunks, p->chunks);
  on_device(t.segs, p->segs);
  on_device(t.vert, p->vert);
  on_device(t.slice_off, p->slice_off);
  on_device(t.nbr, p->nbr);
  on_device(t.edge_off, p->edge_off);
  on_device(t.edge, p->edge);
  on_device(t.bnd_local, p->bnd_local);
  on_device(t.bnd_vert, p->bnd_vert);
  on_device(t.bnd_tile, p->bnd_tile);
  on_device(t.cross_off, p->cross_off);
  on_device(t.cross, p->cross);
  p->seg_pow = reinterpret_cast<const double**>(p->tables + pow_at);
  *out = own.release();
  return TFCE_OK;
}

int64_t basin_launched(const BasinPlan* p) { return p ? p->launched : 0; }

void basin_plan_destroy(BasinPlan* p) {
  if (!p) return;
  int dev = 0;
  cudaGetDevice(&dev);
  cudaSetDevice(p->device);
  cudaFree(p->tables);
  for (auto& kv : p->powers) cudaFree(kv.second);
  for (void* d : p->retired) cudaFree(d);
  cudaFree(p->ws);
  cudaSetDevice(dev);
  delete p;
}

int basin_plan_set_exponents(BasinPlan* p, const float* E) {
  const OnDevice on(p->device);
  std::vector<const double*> rows(p->n_seg, nullptr);
  for (int s = 0; s < p->n_seg; ++s) {
    if (E[s] == 1.0f) continue;
    auto it = p->powers.find(E[s]);
    if (it == p->powers.end()) {
      double* d = nullptr;
      const int64_t n = (int64_t)p->vmax + 1;
      TFGB_CUDA(cudaMalloc(&d, n * sizeof(double)));
      basin_power_kernel<<<static_cast<unsigned>(std::min<int64_t>((n + 255) / 256, 1216)), 256>>>(d, n, E[s]);
      cudaError_t e = cudaGetLastError();
      if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);
      if (e != cudaSuccess) cudaFree(d);  // a table that is not filled is not kept
      TFGB_CUDA(e);
      it = p->powers.emplace(E[s], d).first;
    }
    rows[s] = it->second;
  }
  TFGB_CUDA(cudaMemcpy(p->seg_pow, rows.data(), rows.size() * sizeof(double*), cudaMemcpyHostToDevice));
  if (p->powers.size() > kPowersKept) {  // those of earlier exponents, once nothing reads them
    TFGB_CUDA(cudaDeviceSynchronize());
    for (auto it = p->powers.begin(); it != p->powers.end();) {
      if (std::find(rows.begin(), rows.end(), it->second) != rows.end()) {
        ++it;
      } else {
        cudaFree(it->second);
        it = p->powers.erase(it);
      }
    }
  }
  return TFCE_OK;
}

bool basin_takes(const BasinPlan* p, const BasinRequest& r) {
  if (!p) return false;
  const int mode = mode_of(r);
  const int64_t cap = mode == kNodes ? node_capacity(p) : 0;
  return layout_of(p, 1, r.signs, mode, cap).total <= kWorkspaceBudget;
}

int basin_sweep(BasinPlan* p, const BasinRequest& r, cudaStream_t st, bool* refused) {
  *refused = false;
  const int mode = mode_of(r);
  const int64_t cap = mode == kNodes ? node_capacity(p) : 0;
  const int64_t one = layout_of(p, 1, r.signs, mode, cap).total;
  SweepShape first{}, mid{}, large{};
  int first_ctas = 0, mid_ctas = 0, large_ctas = 0;
  int64_t per = 0, state = 0;
  Layout lay{};
  // launches of equal size, of as many maps as `room` holds; the bytes they take
  auto divide = [&](int64_t room) {
    int64_t most = std::max<int64_t>(1, room / one);
    most = std::min<int64_t>(most, std::max<int64_t>(1, 0x7fffffffLL / std::max(1, p->n_tiles + p->n_chunks)));
    if (mode == kNodes)  // one grid row of the walk per item
      most = std::min<int64_t>(most, std::max<int64_t>(1, 65535 / ((int64_t)r.signs * p->n_seg)));
    const int64_t launches = (r.n_maps + most - 1) / most;
    per = (r.n_maps + launches - 1) / launches;

    const int64_t items_max = per * r.signs * p->n_seg;
    first = first_shape(p, mode, items_max, r.dense);
    mid = large = SweepShape{};
    const int per_basin = state_bytes_per_basin(mode, kAllShared), per_basin_large = state_bytes_per_basin(mode, kListsGlobal);
    first_ctas = first.grid;
    mid_ctas = large_ctas = 0;
    state = 0;
    mid.basins = first.basins;
    if (items_max > 2 * p->sms && r.dense && first.basins < p->basins) {
      mid = shape_of(p, per_basin, 2, 65535, 512);
      mid_ctas = mid.grid;
    }
    if (mid.basins < p->basins) {
      large.threads = kMaxSweepThreads;
      large.basins = std::min({(kSmBytes - kSweepBytes) / per_basin_large, 65535, p->basins});
      large.smem = large.basins * per_basin_large;
      large_ctas = p->sms;
      if (const int cap_ctas = most_ctas()) large_ctas = std::min(large_ctas, cap_ctas);
      state = round_up((int64_t)p->basins * state_bytes_per_basin(mode, kAllGlobal), 256);
      large_ctas = static_cast<int>(
          std::min<int64_t>({large_ctas, items_max, std::max<int64_t>(1, std::min(room, kStateBudget) / state)}));
    }
    lay = layout_of(p, per, r.signs, mode, cap);
    return lay.total + large_ctas * state;
  };
  // A call that has to grow the workspace asks for no more than half of the
  // memory that there is for it (one map's is always asked for), and for less
  // when that is refused; a captured one makes do with what it finds.
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &capturing) != cudaSuccess) cudaGetLastError();
  p->captured = p->captured || capturing != cudaStreamCaptureStatusNone;
  const int64_t knob = most_workspace();
  int64_t budget = std::min(kWorkspaceBudget, knob), need = divide(budget);
  auto least = [&] { return per == 1 && large_ctas <= 1; };
  auto less = [&] { need = divide(budget = std::min(budget, per * one + large_ctas * state) / 2); };
  if (need > p->ws_bytes) {
    int64_t limit = p->ws_bytes;
    if (capturing == cudaStreamCaptureStatusNone) {
      limit = std::max(limit, kAskAtOnce);
      size_t unused = 0, total = 0;
      if (need > limit) {
        if (cudaMemGetInfo(&unused, &total) != cudaSuccess) cudaGetLastError();
        limit = std::max(limit, (static_cast<int64_t>(unused) + (p->captured ? 0 : p->ws_bytes)) / 2);
      }
    }
    while (need > limit && !least()) less();
    for (;;) {
      const int rc = ensure_ws(p, need, knob);
      if (rc == TFCE_OK) break;
      *refused = rc == TFCE_ENOMEM;
      if (rc != TFCE_ENOMEM || least()) return rc;
      less();
    }
    *refused = false;
  }

  BasinArgs a{};
  a.map_stride = r.map_stride;
  a.signs = r.signs;
  a.n_seg = p->n_seg;
  a.vdensity = r.vdensity;
  a.out_mode = r.out_mode;
  a.n_vertices = p->V;
  a.thr_group = r.thr_group;
  a.seg_H = r.d_H;
  a.seg_off = r.d_seg_off;
  a.seg_rank = r.seg_rank;
  a.err = r.err;
  a.tiles = p->tiles;
  a.chunks = p->chunks;
  a.segs = p->segs;
  a.vert = p->vert;
  a.slice_off = p->slice_off;
  a.nbr = p->nbr;
  a.edge_off = p->edge_off;
  a.edge = p->edge;
  a.bnd_local = p->bnd_local;
  a.bnd_vert = p->bnd_vert;
  a.bnd_tile = p->bnd_tile;
  a.cross_off = p->cross_off;
  a.cross = p->cross;
  a.seg_pow = p->seg_pow;
  a.n_tiles = p->n_tiles;
  a.n_chunks = p->n_chunks;
  a.n_bnd = p->n_bnd;
  a.counter = reinterpret_cast<int32_t*>(p->ws + lay.head);
  a.seg_max = reinterpret_cast<uint32_t*>(p->ws + lay.head + 256);
  auto at = [&](auto*& ptr, int64_t o) { ptr = reinterpret_cast<std::remove_reference_t<decltype(ptr)>>(p->ws + o); };
  at(a.ev, lay.ev);
  at(a.pairs, lay.pairs);
  at(a.cpairs, lay.cpairs);
  at(a.tab_ev, lay.tab_ev);
  at(a.tab_pair, lay.tab_pair);
  at(a.tab_cross, lay.tab_cross);
  at(a.n_pairs, lay.n_pairs);
  at(a.queue, lay.queue);
  at(a.n_basin, lay.n_basin);
  at(a.bnd, lay.bnd);
  at(a.off_ev, lay.off_ev);
  at(a.off_pair, lay.off_pair);
  at(a.off_cross, lay.off_cross);
  at(a.base_of, lay.base_of);
  at(a.start_ev, lay.start_ev);
  at(a.start_pair, lay.start_pair);
  at(a.n_basins, lay.n_basins);
  a.ev_out = p->ws + lay.ev_out;
  a.pair_out = p->ws + lay.pair_out;
  at(a.ord, lay.ord);
  at(a.base, lay.base);
  at(a.vnode, lay.vnode);
  at(a.nodes, lay.nodes);
  at(a.part_max, lay.part);
  a.n_steps = a.part_max + per * r.signs * p->n_seg;
  a.pos_per_map = p->n_pos;
  a.pair_per_map = p->n_pair;
  a.cpair_per_map = p->n_cpair;
  a.opair_per_map = p->n_opair;
  a.node_cap = cap;
  a.state = p->ws + lay.total;
  a.state_bytes = state;
  a.most_first = first.basins;
  a.most_mid = mid.basins;
  a.most_narrow = std::max(mid.basins, large.basins);
  for (int64_t m0 = 0; m0 < r.n_maps; m0 += per) {
    const int64_t M = std::min(per, r.n_maps - m0);
    a.n_maps = static_cast<int32_t>(M);
    a.stats = r.stats + m0 * r.map_stride;
    a.out_max = r.out_max ? r.out_max + m0 * r.signs * p->n_seg : nullptr;
    a.out_maps = r.out_maps ? r.out_maps + m0 * r.signs * p->V : nullptr;
    a.n_items = static_cast<int32_t>(M * r.signs * p->n_seg);
    const bool chain = M * p->n_tiles <= p->sms;
    TFGB_CUDA(cudaMemsetAsync(p->ws + lay.head, 0, 256 + M * 2 * p->n_seg * 4, st));
    // a block per (map, segment) reads about 8k values or, with many maps, all of a segment
    const int64_t pairs_ms = M * p->n_seg;
    const int64_t parts = std::max<int64_t>(
        1, std::min<int64_t>((p->vmax + 8191) / 8192, (8 * p->sms + pairs_ms - 1) / pairs_ms));
    basin_max_kernel<<<static_cast<unsigned>(pairs_ms * parts), 256, 0, st>>>(a, static_cast<int32_t>(parts));
    p->launched += 3 + (a.out_maps && r.out_mode == 1) + (p->n_tiles > 0) + (p->n_chunks > 0) +
                   (p->n_tiles + p->n_chunks > 0) + (mid_ctas > 0) + (large_ctas > 0) +
                   (mode == kNodes ? 1 + (a.out_max != nullptr) : 0);
    if (a.out_maps && r.out_mode == 1) {
      const int64_t n = M * r.signs * p->V;
      TFGB_CUDA(launch_after(chain, basin_fill_kernel, dim3(static_cast<unsigned>(std::min<int64_t>((n + 255) / 256, p->sms * 16))),
                             256, 0, st, a));
    }
    if (p->n_tiles)
      TFGB_CUDA(launch_after(chain, basin_tile_kernel, dim3(static_cast<unsigned>(M * p->n_tiles)), kTileThreads, 0, st, a));
    if (p->n_chunks)
      TFGB_CUDA(launch_after(chain, basin_cross_kernel, dim3(static_cast<unsigned>(M * p->n_chunks)), kCrossThreads, 0, st, a));
    TFGB_CUDA(launch_after(chain, basin_offset_kernel, dim3(static_cast<unsigned>(pairs_ms)), kBuckets, 0, st, a));
    const unsigned units = static_cast<unsigned>(M * (p->n_tiles + p->n_chunks));
    if (units)
      TFGB_CUDA(launch_after(chain, mode == kMaxima ? basin_order_kernel<false> : basin_order_kernel<true>, dim3(units),
                             kTileThreads, 0, st, a));
    TFGB_CUDA(cudaGetLastError());
    first.grid = std::min(first_ctas, a.n_items);
    mid.grid = std::min(mid_ctas, a.n_items);
    large.grid = std::min(large_ctas, a.n_items);
    int e;
    if (mode == kMaxima) e = launch_sweeps<kMaxima>(a, first, mid, large, chain, st);
    else if (mode == kPotential) e = launch_sweeps<kPotential>(a, first, mid, large, chain, st);
    else e = launch_sweeps<kNodes>(a, first, mid, large, chain, st);
    if (e) return e;
    if (mode == kNodes) {
      const dim3 g(static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>((p->vmax + 255) / 256, 1024))),
                   static_cast<unsigned>(a.n_items));
      TFGB_CUDA(launch_after(chain, basin_walk_kernel, g, 256, 0, st, a));
      if (a.out_max)
        TFGB_CUDA(launch_after(chain, basin_max_out_kernel, dim3(static_cast<unsigned>((a.n_items + 255) / 256)), 256, 0, st, a));
      TFGB_CUDA(cudaGetLastError());
    }
  }
  return TFCE_OK;
}

}  // namespace tfgb
