// Work split of the persistent CG on CSR values in place (cg_persist.cu):
// tiles of whole node rows, tiles of whole Schwarz block rows, and contiguous
// tile ranges per CTA.  Host code without CUDA types, so that its bounds can
// be tested on the CPU.
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

namespace hoefem {

// Operator tile: nodes [n0, n0 + nn), whose adjacency entries (and 3 x 3
// blocks, 9 values each) are [o0, o0 + nblk) of the pattern.
struct alignas(16) PcgTile {
  int n0, nn, o0, nblk;
};

// Schwarz tile: rows [row0, row0 + rows) of one dim x dim block whose values
// start at `src` (elements) and whose node list starts at `o`.
struct alignas(16) PcgSwTile {
  long long src;
  int o, dim, row0, rows, pad0, pad1;
};

constexpr int PCG_MAX_TILE_NODES = 16;  // bounds a tile's row offsets in a stage
constexpr int PCG_MAX_SUB_NODES = 32;   // bounds a subdomain's node list in a stage, and its rows in three per lane
constexpr int PCG_SW_ROWS = 8;          // Schwarz rows reduced together

// Bytes of the 16-byte granules that cover [begin, end) bytes, not reaching
// past `limit` bytes (the array's whole granules); `head` gets the offset of
// `begin` in the first granule.
struct PcgSpan {
  long long from;
  int bytes, head;
};
#ifdef __CUDACC__
__host__ __device__
#endif
inline PcgSpan pcg_span(long long begin, long long end, long long limit) {
  PcgSpan s;
  s.from = begin & ~15LL;
  long long to = (end + 15) & ~15LL;
  if (to > limit) to = limit;
  s.bytes = (int)(to > s.from ? to - s.from : 0);
  s.head = (int)(begin - s.from);
  return s;
}

// Packs consecutive nodes into tiles of at most cap_bytes of values and
// PCG_MAX_TILE_NODES nodes, a multiple of `group` where there are more; every
// node's rows must fit a tile.  False if one does not.
inline bool pcg_op_tiles(const std::vector<int>& adj_off, long long nv, int vsize, long long cap_bytes, int group,
                         std::vector<PcgTile>& tiles, int& max_blk) {
  tiles.clear();
  max_blk = 0;
  const long long cap_blk = cap_bytes / (9LL * vsize);
  for (long long a = 0; a < nv;) {
    const int o0 = adj_off[a];
    long long e = a;
    while (e < nv && e - a < PCG_MAX_TILE_NODES && (long long)adj_off[e + 1] - o0 <= cap_blk) ++e;
    if (e == a) return false;
    if (e < nv && e - a > group) e -= (e - a) % group;
    const int nblk = adj_off[e] - o0;
    tiles.push_back(PcgTile{(int)a, (int)(e - a), o0, nblk});
    max_blk = std::max(max_blk, nblk);
    a = e;
  }
  return true;
}

// Splits every subdomain block into tiles of at most cap_bytes and a multiple
// of PCG_SW_ROWS rows (the last tile of a block may have fewer).
inline bool pcg_sw_tiles(const std::vector<int64_t>& sub_off, int vsize, long long cap_bytes,
                         std::vector<PcgSwTile>& tiles) {
  tiles.clear();
  long long base = 0;
  for (size_t s = 0; s + 1 < sub_off.size(); ++s) {
    const int dim = 3 * (int)(sub_off[s + 1] - sub_off[s]);
    long long rows = dim ? cap_bytes / ((long long)dim * vsize) : 0;
    if (rows >= PCG_SW_ROWS) rows -= rows % PCG_SW_ROWS;
    if (dim && rows < 1) return false;
    for (int r = 0; r < dim; r += (int)rows)
      tiles.push_back(PcgSwTile{base + (long long)r * dim, (int)sub_off[s], dim, r, (int)std::min<long long>(rows, dim - r),
                                0, 0});
    base += (long long)dim * dim;
  }
  return true;
}

// Contiguous ranges of G CTAs with nearly equal weight: CTA c gets the items
// [off[c], off[c + 1]).
inline std::vector<int> pcg_ranges(const std::vector<long long>& weight, int G) {
  long long total = 0;
  for (long long w : weight) total += w;
  std::vector<int> off(G + 1, 0);
  long long sum = 0;
  size_t k = 0;
  for (int c = 0; c < G; ++c) {
    off[c] = (int)k;
    const long long target = total * (c + 1) / G;
    // an item goes to the CTA in which its middle falls
    while (k < weight.size() && 2 * sum + weight[k] <= 2 * target) sum += weight[k++];
  }
  off[G] = (int)weight.size();
  return off;
}

}  // namespace hoefem
