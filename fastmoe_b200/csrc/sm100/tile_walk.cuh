// Which parts of which output tiles a CTA pair of a persistent grouped GEMM works on.
//
// T tiles on P pairs take ceil(T / P) rounds, and a last round of few tiles leaves most of the chip
// idle.  The full rounds are dealt out tile by tile, in turn, which keeps tiles that run at the same time
// next to each other.  Where cutting pays (dealt_tiles), the T mod P tiles left are one sequence of K
// blocks, cut into equal pieces, one per pair, but no more pieces than leave each `cost_kb` K blocks on
// average (at least one per tile).  A piece begins with the end of one tile and ends with the beginning of
// another, or lies inside one.  The pair that has a tile's first K block owns the tile; the others hand it
// their sums through global memory.  A pair meets the part it does not own first and the part for which it
// has to collect the rest last: nobody waits before handing over, so every wait ends whatever order the
// pairs run in, and an owner hardly waits.  The cut depends on the offsets alone: equal calls add in equal
// order.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace fmoe {

struct WalkPart {
  int group;
  int tile;         // in the group
  int kb0, kb1;     // K blocks [kb0, kb1) of num_kb
  int num_kb;
  int last_piece;   // kb0 == 0: the pieces after this pair's up to this one hold the rest of the tile
};

// Tiles dealt out in turn.  All of them unless cutting saves more than the `cost_kb` K blocks of time
// that a pair spends on handing its sum over and on collecting another.
__host__ __device__ inline int dealt_tiles(int tiles, int units, int pairs, int cost_kb) {
  const int rest = tiles % pairs;
  if (cost_kb <= 0 || rest == 0) return tiles;
  const long idle = static_cast<long>(pairs - rest) * units / tiles;   // K blocks that nobody works on
  if (idle <= static_cast<long>(cost_kb) * pairs) return tiles;
  return tiles - rest;
}

// `tiles` and `units` are exclusive prefixes over the groups ([num_groups + 1]) of the tiles and of
// their K blocks.  Every role of a kernel walks the same parts.
class TileWalk {
 public:
  // cost_kb: see dealt_tiles; 0: no tile is cut.
  __host__ __device__ TileWalk(const int* tiles, const int* units, int num_groups, int pair, int pairs, int cost_kb)
      : tiles_(tiles), units_(units), groups_(num_groups), pairs_(pairs), next_(pair) {
    const int total = tiles[num_groups];
    dealt_ = dealt_tiles(total, units[num_groups], pairs, cost_kb);
    if (dealt_ == total) return;
    const int g = find(tiles, dealt_);
    first_ = units[g] + (dealt_ - tiles[g]) * blocks(g);
    len_ = units[num_groups] - first_;
    const int left = total - dealt_;
    pieces_ = len_ / cost_kb;   // no shorter than that on average
    if (pieces_ < left) pieces_ = left;
    if (pieces_ > pairs) pieces_ = pairs;
    if (pair < pieces_) {
      at_ = begin(pair);
      end_ = begin(pair + 1);
    }
  }

  __host__ __device__ bool next(WalkPart& p) {
    if (next_ < dealt_) {
      p.group = find(tiles_, next_);
      p.tile = next_ - tiles_[p.group];
      p.num_kb = blocks(p.group);
      p.kb0 = 0;
      p.kb1 = p.num_kb;
      p.last_piece = -1;
      next_ += pairs_;
      return true;
    }
    if (at_ >= end_) return false;
    p.group = find(units_, first_ + at_);
    p.num_kb = blocks(p.group);
    const int local = first_ + at_ - units_[p.group];
    p.tile = local / p.num_kb;
    p.kb0 = local - p.tile * p.num_kb;
    const int left = end_ - at_;
    p.kb1 = p.num_kb - p.kb0 < left ? p.num_kb : p.kb0 + left;
    p.last_piece = p.kb0 == 0 && p.kb1 < p.num_kb ? piece_of(at_ + p.num_kb - 1) : -1;
    at_ += p.kb1 - p.kb0;
    return true;
  }

 private:
  // The group whose range of the prefix contains `value`; groups without tiles have none.
  __host__ __device__ int find(const int* prefix, int value) const {
    int lo = 0, hi = groups_;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (prefix[mid] <= value) lo = mid; else hi = mid;
    }
    return lo;
  }
  __host__ __device__ int blocks(int g) const { return (units_[g + 1] - units_[g]) / (tiles_[g + 1] - tiles_[g]); }
  __host__ __device__ int begin(int q) const { return static_cast<int>(static_cast<long>(len_) * q / pieces_); }
  __host__ __device__ int piece_of(int u) const {
    int q = static_cast<int>(static_cast<long>(u) * pieces_ / len_);
    while (q + 1 < pieces_ && begin(q + 1) <= u) ++q;
    while (begin(q) > u) --q;
    return q;
  }

  const int* tiles_;
  const int* units_;
  int groups_, pairs_;
  int next_;            // next dealt tile
  int dealt_ = 0;
  int first_ = 0;       // K blocks before tile `dealt_`
  int len_ = 0;         // K blocks from there on
  int pieces_ = 1;
  int at_ = 0, end_ = 0;
};

}  // namespace fmoe
