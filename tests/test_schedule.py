"""The order in which a packed launch hands out its tiles (csrc/schedule.cuh), run on the CPU: the header
is compiled with the 32 lanes of a warp as threads and compared with a plain restatement (no GPU)."""
import os
import random
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HARNESS = r"""
#include <algorithm>
#include <barrier>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>
#define __device__
#define __forceinline__ inline
#define __restrict__
using std::max; using std::min;
struct Dim { int x; };
thread_local Dim threadIdx;
static std::barrier<> gate(32);
static int slot[32];
template <typename F> static int meet(int v, F f) {
  slot[threadIdx.x] = v; gate.arrive_and_wait();
  int r = f(); gate.arrive_and_wait(); return r;
}
static int __reduce_add_sync(unsigned, int v) { return meet(v, [] { int s = 0; for (int x : slot) s += x; return s; }); }
static int __reduce_max_sync(unsigned, int v) { return meet(v, [] { return *std::max_element(slot, slot + 32); }); }
static unsigned __ballot_sync(unsigned, bool v) {
  return (unsigned)meet(v, [] { unsigned m = 0; for (int i = 0; i < 32; ++i) m |= (slot[i] ? 1u : 0u) << i; return (int)m; });
}
static int __shfl_sync(unsigned, int v, int src) { return meet(v, [=] { return slot[src & 31]; }); }
static int __popc(unsigned v) { return __builtin_popcount(v); }
static int __ffs(unsigned v) { return __builtin_ffs((int)v); }
#include "schedule.cuh"
using namespace b200attn;
// argv: tile max_tiles heads causal kv_bytes equal len...; prints the grid, then "b head level n_tiles" per item
int main(int argc, char** argv) {
  auto num = [&](int i) { return atoll(argv[i]); };
  const int tile = num(1), max_tiles = num(2), heads = num(3), batch = argc - 7;
  std::vector<int32_t> cu(1, 0);
  for (int i = 7; i < argc; ++i) cu.push_back(cu.back() + (int)num(i));
  PackedGrid g = packed_grid(batch, cu.back(), heads, num(4) != 0, num(5));
  if (num(6) && equal_lengths(batch, cu.back(), (int)num(7))) g.equal = ((int)num(7) + tile - 1) / tile;
  const int items = (int)packed_tiles_bound(batch, cu.back(), tile, max_tiles) * heads;
  printf("%d %d %d %d %d\n", g.seqs, g.n_chunks, g.heads, g.equal, (int)tight_grid(batch, cu.back(), tile, max_tiles));
  auto lane = [&](int l) {
    threadIdx.x = l;
    for (int i = 0; i < items; ++i) {
      PackedItem it = {-1, -1, -1, -1};
      bool there = true;
      if (g.equal > 0) equal_item(g, batch, heads, i, it);
      else there = packed_item(g, cu.data(), batch, tile, max_tiles, heads, i, it);
      if (l == 0) { if (there) printf("%d %d %d %d\n", it.b, it.head, it.level, it.n_tiles); else printf("-\n"); }
    }
  };
  std::vector<std::thread> warp;
  for (int l = 0; l < 32; ++l) warp.emplace_back(lane, l);
  for (auto& t : warp) t.join();
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("schedule")
    (d / "harness.cpp").write_text(HARNESS)
    exe = d / "harness"
    subprocess.check_call(["g++", "-std=c++20", "-O1", "-pthread", "-I", os.path.join(ROOT, "tritonops_b200", "csrc"),
                           "-o", str(exe), str(d / "harness.cpp")])

    def call(lens, heads, causal, tile=256, max_tiles=1 << 20, kv_bytes=2048, equal=False):
        args = [tile, max_tiles, heads, int(causal), kv_bytes, int(equal), *lens]
        out = subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True, check=True).stdout.split("\n")
        return [int(x) for x in out[0].split()], [tuple(map(int, x.split())) for x in out[1:] if x and x != "-"]
    return call


def _batches():
    rng = random.Random(3)
    yield [1], 1, 1 << 20
    yield [700, 0, 256, 257, 1, 0, 511], 12, 1 << 20        # heads that do not fill groups of eight
    yield [700, 0, 256, 257, 1, 0, 511], 8, 2               # cut at two tiles
    yield [1500, 600], 9, 1 << 20
    yield [rng.randint(0, 600) for _ in range(40)], 1, 1 << 20      # more sequences than lanes


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("kv_bytes", [2048, 1 << 16])       # chunks of many sequences, and of one or a few
def test_every_tile_once_and_the_heaviest_first(run, causal, kv_bytes):
    for lens, heads, max_tiles in _batches():
        (seqs, n_chunks, group, _, _), items = run(lens, heads, causal, max_tiles=max_tiles, kv_bytes=kv_bytes)
        tiles = [min(-(-n // 256), max_tiles) for n in lens]
        assert sorted(i[:3] for i in items) == sorted((b, h, t) for b, n in enumerate(tiles) for h in range(heads)
                                                      for t in range(n))
        assert all(n == tiles[b] for b, _, _, n in items) and seqs * n_chunks >= len(lens)
        # within a chunk of sequences and a group of heads no tile comes before a heavier one
        last = None
        for b, h, level, n in items:
            at, weight = (b // seqs, h // group), (level if causal else n)
            if last is not None and last[0] == at:
                assert weight <= last[1], (lens, heads, at)
            elif last is not None:
                assert at > last[0]
            last = (at, weight)


def test_head_groups_are_of_one_size(run):
    for heads, want in [(1, 1), (8, 8), (9, 5), (12, 6), (16, 8), (28, 7), (40, 8)]:
        assert run([1], heads, True)[0][2] == want


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("batch,n,heads,kv_bytes", [(1, 1500, 9, 2048), (5, 600, 12, 2048), (7, 256, 8, 1 << 17), (40, 257, 1, 2048)])
def test_equal_lengths_are_handed_out_in_the_same_order(run, causal, batch, n, heads, kv_bytes):
    grid, items = run([n] * batch, heads, causal, max_tiles=-(-n // 256), kv_bytes=kv_bytes)
    fast, same = run([n] * batch, heads, causal, max_tiles=-(-n // 256), kv_bytes=kv_bytes, equal=True)
    assert grid[3] == 0 and fast[3] == -(-n // 256)
    assert same == items
    # other lengths of the same sum are not taken for equal ones
    if batch > 1:
        assert run([n - 1] + [n] * (batch - 2) + [n + 1], heads, causal, equal=True)[0][3] == 0


def test_which_grids_are_tight(run):
    """Longest 3000: four sequences of that length, of half that length, one among short ones."""
    for lens, want in [([3000] * 4, 1), ([3000, 1600, 1500, 1400], 1), ([3000, 100, 100, 100], 0)]:
        assert run(lens, 1, True, max_tiles=12)[0][4] == want
