"""The host tables of an adjacency handle (csrc/basin_tables.h), compiled by the
host compiler with its checks of vector accesses on (and the address sanitizer
where the compiler has one): lists with repeated entries, one-way entries, tile
remainders.  Every pair of neighbours of a tile is held once, every entry that
leaves its tile or lacks its reverse is in a crossing list, and nothing else is."""
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tfce_mediation_gb300", "csrc")

PROGRAM = r"""
#include "basin_tables.h"
#include <cstdio>
using namespace tfgb;

int main(int, char** argv) {
  FILE* f = fopen(argv[1], "rb");
  int64_t V, n_seg, D;
  auto get = [&](void* p, size_t bytes) { if (bytes && fread(p, 1, bytes, f) != bytes) exit(3); };
  get(&V, 8), get(&n_seg, 8), get(&D, 8);
  std::vector<int64_t> offsets(V + 1), seg(n_seg + 1);
  std::vector<int32_t> indices(D);
  get(offsets.data(), 8 * (V + 1)), get(seg.data(), 8 * (n_seg + 1)), get(indices.data(), 4 * D);
  CleanLists c;
  std::string error;
  if (!clean_lists(offsets.data(), indices.data(), static_cast<int32_t>(V), seg, &c, &error)) return puts(error.c_str()), 0;
  for (int64_t v = 0; v < V; ++v)
    for (int64_t e = c.off[v]; e < c.off[v + 1]; ++e)
      printf("list %d %d %d\n", (int)v, (int)(c.packed[e] & kIndexMask), (int)(c.packed[e] >> 31));
  BasinTables t;
  if (!build_basin_tables(c, seg, &t)) return puts("no tables"), 0;
  printf("basins %d 0\n", t.basins);
  for (int64_t i = 0; i < t.tiles.size(); ++i) {
    const TileInfo ti = t.tiles[i];
    for (int v = 0; v < ti.nv; ++v) {
      printf("vertex %d %d\n", t.vert[ti.pos0 + v], (int)i);
      const int s = ti.slice0 + (v >> 5);
      auto rows = [&](const char* name, const auto& off, const auto& of) {
        for (uint32_t o = (off[s] & ~kOddRow) + (v & 31); o < (off[s + 1] & ~kOddRow); o += 32)
          for (uint32_t u : {(of[o] & 0xffffu) >> 2, of[o] >> 18})
            if ((int)u != v) printf("%s %d %d\n", name, t.vert[ti.pos0 + v], t.vert[ti.pos0 + u]);
      };
      rows("near", t.slice_off, t.nbr);
      rows("held", t.edge_off, t.edge);
    }
  }
  for (const ChunkInfo& ci : t.chunks)
    for (int q = 0; q < ci.nbnd; ++q) {
      const int s = ci.slice0 + (q >> 5);
      for (uint32_t o = t.cross_off[s] + (q & 31); o < t.cross_off[s + 1]; o += 32)
        if ((int)t.cross[o] != ci.bnd0 + q) printf("cross %d %d\n", t.bnd_vert[ci.bnd0 + q], t.bnd_vert[t.cross[o]]);
    }
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("tables")
    (d / "t.cpp").write_text(PROGRAM)
    base = [cxx, "-std=c++17", "-O1", "-g", "-pthread", "-D_GLIBCXX_ASSERTIONS", "-I", CSRC, str(d / "t.cpp"), "-o"]
    for extra in (["-fsanitize=address,undefined", "-fno-sanitize-recover=all"], []):
        exe = str(d / ("t%d" % len(extra)))
        if subprocess.run(base + [exe] + extra, capture_output=True).returncode == 0:
            break
    else:
        subprocess.run(base + [exe], check=True)
    return exe


def _tables(program, tmp_path, lists=None, csr=None, seg=None):
    if csr is None:
        csr = np.cumsum([0] + [len(x) for x in lists]), [u for x in lists for u in x]
    off, idx = np.asarray(csr[0], np.int64), np.asarray(csr[1], np.int32)
    V = len(off) - 1
    seg = np.asarray([0, V] if seg is None else seg, np.int64)
    path = tmp_path / "graph"
    path.write_bytes(np.asarray([V, len(seg) - 1, len(idx)], np.int64).tobytes() + off.tobytes() + seg.tobytes() +
                     idx.tobytes())
    r = subprocess.run([program, str(path)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    out = {}
    for line in r.stdout.splitlines():
        name, *rest = line.split()
        out.setdefault(name, []).append(tuple(int(x) for x in rest))
    return off, idx, out


def _check(off, idx, out):
    V = len(off) - 1
    rows = np.repeat(np.arange(V), np.diff(off))
    entries = sorted({(int(v), int(u)) for v, u in zip(rows, idx) if u != v})
    have = set(entries)
    assert out.get("list", []) == [(v, u, int((u, v) not in have)) for v, u in entries]
    tile = dict(out["vertex"])
    assert len(out["vertex"]) == len(tile) == V
    inside = [(v, u) for v, u in entries if (u, v) in have and tile[v] == tile[u]]
    assert sorted(out.get("near", [])) == inside
    held = [(min(p), max(p)) for p in out.get("held", [])]
    assert sorted(held) == [(v, u) for v, u in inside if v < u]
    assert sorted(out.get("cross", [])) == sorted(have - set(inside))
    return tile


@pytest.mark.parametrize("lists", [
    [[1, 1, 1, 1], [0]],
    [[1] * 40, [0]],
    [[2, 3], [2, 3, 4, 4], [0, 1, 3], [0, 1, 2], [1]],  # the receiving vertex is its tile's last
    [[1, 1, 1, 1, 2], [0, 2], [1, 0, 3], [2]],          # and an inner one
    [[0, 0, 1, 1], [1, 1]],                             # one-way, self entries
    [[], [2, 2, 2], []],
])
def test_repeated_entries_count_once(program, tmp_path, lists):
    _check(*_tables(program, tmp_path, lists))


@pytest.mark.parametrize("V", [1, 31, 33, 4096, 4097, 9001])
def test_every_pair_once_with_one_sided_repeats(program, tmp_path, V):
    rng = np.random.default_rng(V)
    i = np.arange(V)
    both = np.concatenate([np.stack([i, (i + d) % V], 1) for d in (1, 2, 37)])
    both = np.concatenate([both, both[:, ::-1]])
    pairs = np.concatenate([both[rng.random(len(both)) > 0.1]] + [both[rng.random(len(both)) > 0.7]] * 3)
    pairs = pairs[rng.permutation(len(pairs))]
    pairs = pairs[np.argsort(pairs[:, 0], kind="stable")]
    off = np.cumsum(np.r_[0, np.bincount(pairs[:, 0], minlength=V)])
    tile = _check(*_tables(program, tmp_path, csr=(off, pairs[:, 1])))
    assert len(set(tile.values())) == -(-V // 4096)


def test_bad_entries_are_named(program, tmp_path):
    for lists, seg, want in (([[1], [0, 5]], None, "entry 5 of vertex 1 outside [0, 2)"),
                             ([[1], [0], [-1]], None, "entry -1 of vertex 2 outside [0, 3)"),
                             ([[1], [0]], [0, 1, 2], "entry 1 of vertex 0 crosses segments")):
        off = np.cumsum([0] + [len(x) for x in lists]).astype(np.int64)
        seg = np.asarray([0, len(lists)] if seg is None else seg, np.int64)
        path = tmp_path / "graph"
        path.write_bytes(np.asarray([len(lists), len(seg) - 1, off[-1]], np.int64).tobytes() + off.tobytes() +
                         seg.tobytes() + np.asarray([u for x in lists for u in x], np.int32).tobytes())
        r = subprocess.run([program, str(path)], capture_output=True, text=True)
        assert want in r.stdout


THROWS = r"""
#include "host_parallel.h"
#include <cstdio>
#include <new>

int main() {
  std::atomic<int64_t> calls{0};
  for (int64_t work : {int64_t{0}, int64_t{1} << 30})
    try {
      tfgb::parallel_for(100000, work, [&](int64_t i) {
        ++calls;
        if (i % 1000 == 999) throw std::bad_alloc();
      });
      return 1;
    } catch (const std::bad_alloc&) {
    }
  if (calls >= 200000) return 2;
  int64_t sum = 0;
  tfgb::parallel_for(0, 1 << 30, [&](int64_t) { ++sum; });
  return sum ? 3 : 0;
}
"""


def test_out_of_memory_on_a_thread_reaches_the_caller(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host compiler")
    (tmp_path / "t.cpp").write_text(THROWS)
    exe = str(tmp_path / "t")
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(tmp_path / "t.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe]).returncode == 0
