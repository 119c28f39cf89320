// Which tile of which sequence a CTA of a packed (varlen) launch works on.
//
// The launch is one CTA per (sequence, head, tile that exists) plus a few that find nothing to do:
// sum_b ceil(len_b / tile) <= total / tile + batch, a bound the host knows without reading the
// lengths back, where a grid of batch x (tiles of the longest sequence) is mostly empty CTAs for
// ragged batches and needs the longest length on the host.  Order: sequences are taken in chunks
// (PackedGrid::seqs, at most 32: one per lane), inside a chunk heads in groups of at most kSchedHeads,
// inside that the heaviest tiles of all its sequences first, heads fastest.  Causal tiles grow with
// their level (how many tiles of its own sequence are lighter); without a mask all tiles of a sequence
// weigh the same, so there the longest sequence comes first.  The groups are of one size (12 heads as
// 6 + 6, not 8 + 4: the heaviest tiles of a small last group would start behind the lightest of the
// one before it).  The chunk is small enough for the K / V of a head group to stay in L2 while its
// CTAs are resident.
// (Forward, graph-replayed, before these two rules -> with them: 12 heads, causal, 5000 + 2 x 500 tokens
// 97.3 -> 78.9 us, 4 x 4096 tokens 203 -> 190; not causal, 12 heads, six of up to 3000 tokens 96.5 -> 66.5.)
// (12 sequences of 37 to 3000 tokens, 32 / 8 heads, forward: 349 us with a grid of batch x longest,
// 340 us so.  A training step over 9 sequences of 100 to 2500 tokens, 64-wide heads: 197 us; 227 us
// with a grid of batch x total / tile, the other way not to need the longest length on the host.)
#pragma once
#include <stdint.h>

namespace b200attn {

constexpr int kSchedHeads = 8;          // heads scheduled together, at most
constexpr int kSchedMaxChunks = 8;      // sequence chunks a CTA may have to look through
constexpr int kSchedMaxBatch = 32 * kSchedMaxChunks;
constexpr long long kSchedL2Bytes = 32LL << 20;   // K + V bytes of a head group of a chunk

struct PackedGrid {
  int seqs;        // sequences per chunk; 0: not a packed launch
  int n_chunks;
  int heads;       // heads scheduled together
  int by_length;   // the weight of a tile is its sequence's length, not its level
  int equal;       // tiles of every sequence where the host knows that all are of one length, else 0
};

struct PackedItem {
  int b, head, level, n_tiles;   // n_tiles: tiles of sequence b
};

// kv_bytes: K + V bytes of one token for kSchedHeads heads
inline PackedGrid packed_grid(int batch, long long total_tokens, int heads, bool causal, long long kv_bytes) {
  const long long per_seq = (total_tokens / batch + 1) * kv_bytes;
  long long seqs = kSchedL2Bytes / per_seq;
  const long long least = (batch + kSchedMaxChunks - 1) / kSchedMaxChunks;
  if (seqs < least) seqs = least;
  if (seqs < 1) seqs = 1;
  if (seqs > 32) seqs = 32;
  if (seqs > batch) seqs = batch;
  PackedGrid g;
  g.seqs = (int)seqs;
  g.n_chunks = (int)((batch + seqs - 1) / seqs);
  const int groups = (heads + kSchedHeads - 1) / kSchedHeads;
  g.heads = (heads + groups - 1) / groups;
  g.by_length = causal ? 0 : 1;
  g.equal = 0;
  return g;
}

// All lengths are max_seqlen when they add up to batch x max_seqlen.
inline bool equal_lengths(int batch, long long total_tokens, int max_seqlen) {
  return (long long)batch * max_seqlen == total_tokens;
}
// Does a grid of batch x tiles of the longest sequence hold few tiles that do not exist (fewer than 3
// for 4 that may)?  Then a CTA is better off finding its place from its number: looking it up takes
// about a microsecond, an empty CTA about half of one.
inline bool tight_grid(int batch, long long total_tokens, int tile, int max_tiles) {
  return 4LL * batch * max_tiles <= 7 * (total_tokens / tile + batch);
}

// upper bound on the number of tiles of all sequences (each of them cut at max_tiles tiles)
inline long long packed_tiles_bound(int batch, long long total_tokens, int tile, int max_tiles) {
  const long long by_total = total_tokens / tile + batch, by_max = (long long)batch * max_tiles;
  return by_total < by_max ? by_total : by_max;
}

// Item `idx` of a launch of g.equal tiles of every sequence: the order packed_item gives, without a look
// at the lengths.
__device__ __forceinline__ void equal_item(const PackedGrid g, int batch, int heads, int idx, PackedItem& out) {
  const int b0 = idx / (g.seqs * g.equal * heads) * g.seqs;
  const int n = min(g.seqs, batch - b0);
  idx -= b0 * g.equal * heads;
  const int per_group = n * g.equal * g.heads;
  const int grp = idx / per_group;
  const int in_grp = idx - grp * per_group;
  const int g_heads = min(g.heads, heads - grp * g.heads);
  const int rank = in_grp / g_heads;
  out.head = grp * g.heads + in_grp - rank * g_heads;
  out.level = g.equal - 1 - rank / n;
  out.b = b0 + rank % n;
  out.n_tiles = g.equal;
}

// Item `idx` of the launch; false when there are fewer.  Executed by whole converged warps.
__device__ __forceinline__ bool packed_item(const PackedGrid g, const int32_t* cu, int batch, int tile,
                                            int max_tiles, int heads, int idx, PackedItem& out) {
  const int lane = threadIdx.x & 31;
  auto tiles_of = [&](int c) {   // of this lane's sequence in chunk c
    const int b = c * g.seqs + lane;
    if (lane >= g.seqs || b >= batch) return 0;
    const int len = cu[b + 1] - cu[b];
    return len > 0 ? min((len - 1) / tile + 1, max_tiles) : 0;
  };
  int np = 0, b0 = 0, total = 0;
  bool found = false;
  if (g.n_chunks == 1) {
    np = tiles_of(0);
    total = __reduce_add_sync(0xffffffffu, np);
    found = idx < total * heads;
  } else {
    int n[kSchedMaxChunks];      // (all loads in flight at once)
#pragma unroll
    for (int c = 0; c < kSchedMaxChunks; ++c) n[c] = c < g.n_chunks ? tiles_of(c) : 0;
#pragma unroll
    for (int c = 0; c < kSchedMaxChunks; ++c) {
      if (!found && c < g.n_chunks) {
        const int sum = __reduce_add_sync(0xffffffffu, n[c]);
        if (idx < sum * heads) { np = n[c]; b0 = c * g.seqs; total = sum; found = true; }
        else idx -= sum * heads;
      }
    }
  }
  if (!found) return false;
  const int per_group = total * g.heads;
  const int grp = idx / per_group;
  const int in_grp = idx - grp * per_group;
  const int g_heads = min(g.heads, heads - grp * g.heads);
  const int rank = in_grp / g_heads;               // heaviest first, over the sequences of the chunk
  out.head = grp * g.heads + in_grp - rank * g_heads;
  if (g.seqs == 1) {                               // one sequence: its tiles from the heaviest down
    out.level = total - 1 - rank;
    out.b = b0;
    out.n_tiles = total;
    return true;
  }
  // the level of that rank: the largest L with more than `rank` tiles at levels >= L (by_length: with
  // more than `rank` tiles in sequences of more than L tiles)
  int lo = 0, hi = __reduce_max_sync(0xffffffffu, np);      // C(lo) > rank, C(hi) = 0
  int above = 0;                                             // C(hi)
  const int slope = g.by_length ? 0 : 1;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    const int cnt = __reduce_add_sync(0xffffffffu, np > mid ? np - mid * slope : 0);
    if (cnt > rank) lo = mid; else { hi = mid; above = cnt; }
  }
  int nth = rank - above;                                    // among the sequences with a tile at this level
  out.level = lo;
  bool there = np > lo;
  if (g.by_length) {     // among the tiles of the sequences of just this many (hi = lo + 1), the last of each first
    there = np == hi;
    const int n = __popc(__ballot_sync(0xffffffffu, there)), down = nth / n;
    out.level = hi - 1 - down;
    nth -= down * n;
  }
  const unsigned at = __ballot_sync(0xffffffffu, there);
  const bool mine = there && __popc(at & ((1u << lane) - 1u)) == nth;
  const int src = __ffs(__ballot_sync(0xffffffffu, mine)) - 1;
  out.b = b0 + src;
  out.n_tiles = __shfl_sync(0xffffffffu, np, src);
  return true;
}

}  // namespace b200attn
