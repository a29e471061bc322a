// Properties of the persistent CG's work split (csrc/pcg_layout.h): tiles
// cover every node row and every Schwarz row once and in order, fit their
// stages with their 16-byte granules, stay inside the arrays, and the CTA
// ranges are contiguous and balanced.
#include <cstdio>
#include <random>

#include "pcg_layout.h"

using namespace hoefem;

#define CHECK(c)                                             \
  do {                                                       \
    if (!(c)) {                                              \
      std::printf("line %d: %s\n", __LINE__, #c);            \
      return 1;                                              \
    }                                                        \
  } while (0)

static long long align16(long long b) { return (b + 15) & ~15LL; }

int main() {
  std::mt19937 rng(7);
  for (int rep = 0; rep < 400; ++rep) {
    const int nv = 1 + (int)(rng() % 900), vsize = rep & 1 ? 4 : 8, dmax = 1 + (int)(rng() % 125);
    std::vector<int> off(nv + 1, 0);
    long long maxrow = 0;
    for (int a = 0; a < nv; ++a) {
      const int d = rng() % 5 ? 1 + (int)(rng() % dmax) : (rng() % 3 ? 1 : 0);
      off[a + 1] = off[a] + d;
      maxrow = std::max<long long>(maxrow, 9LL * vsize * d);
    }
    const long long cap = std::max<long long>(maxrow, 768 + rng() % 6000);
    std::vector<PcgTile> t;
    int max_blk = 0;
    CHECK(pcg_op_tiles(off, nv, vsize, cap, rep % 3 ? 4 : 8, t, max_blk));
    const long long val_stage = align16(cap + 32), adj_stage = std::max<long long>(align16(4LL * max_blk + 16), 160);
    const long long val_limit = (9LL * off[nv] * vsize) & ~15LL;
    int a = 0;
    std::vector<long long> w;
    for (const PcgTile& k : t) {
      CHECK(k.n0 == a && k.nn >= 1 && k.nn <= PCG_MAX_TILE_NODES);
      CHECK(k.o0 == off[a] && k.o0 + k.nblk == off[a + k.nn] && k.nblk <= max_blk);
      a += k.nn;
      const long long vb = 9LL * k.o0 * vsize, ve = 9LL * (k.o0 + k.nblk) * vsize;
      const PcgSpan v = pcg_span(vb, ve, val_limit);
      CHECK(v.from % 16 == 0 && v.bytes % 16 == 0 && v.from + v.bytes <= 9LL * off[nv] * vsize);
      CHECK(v.from + v.head == vb && v.bytes <= val_stage && v.head + (ve - vb) <= val_stage);
      // what the bulk copy leaves out is less than one granule, at the array's end
      CHECK(v.from + v.bytes >= ve || (ve == 9LL * off[nv] * vsize && ve - val_limit < 16));
      const PcgSpan j = pcg_span(4LL * k.o0, 4LL * (k.o0 + k.nblk), 1LL << 62);
      CHECK(j.bytes <= adj_stage && j.from + j.bytes <= 4LL * off[nv] + 16 && j.head == 4 * (k.o0 & 3));
      const PcgSpan o = pcg_span(4LL * k.n0, 4LL * (k.n0 + k.nn + 1), 1LL << 62);
      CHECK(o.bytes <= 160 && o.from + o.bytes <= 4LL * (nv + 1) + 16 && o.head == 4 * (k.n0 & 3));
      w.push_back(ve - vb + 64);
    }
    CHECK(a == nv);
    for (int G : {1, 7, 148}) {
      const std::vector<int> r = pcg_ranges(w, G);
      CHECK((int)r.size() == G + 1 && r[0] == 0 && r[G] == (int)w.size());
      long long total = 0, biggest = 0;
      for (long long x : w) total += x, biggest = std::max(biggest, x);
      for (int c = 0; c < G; ++c) {
        CHECK(r[c] <= r[c + 1]);
        long long sum = 0;
        for (int k = r[c]; k < r[c + 1]; ++k) sum += w[k];
        CHECK(sum <= total / G + biggest + 1);
      }
    }
    // a row longer than a tile is refused
    if (maxrow > 9LL * vsize) CHECK(!pcg_op_tiles(off, nv, vsize, maxrow - 1, 4, t, max_blk));
    // Schwarz rows
    std::vector<int64_t> so(1, 0);
    const int ns = (int)(rng() % 40);
    for (int s = 0; s < ns; ++s) so.push_back(so.back() + 1 + rng() % 27);
    std::vector<PcgSwTile> st;
    const long long scap = std::max<long long>(768, cap);
    CHECK(pcg_sw_tiles(so, vsize, scap, st));
    long long src = 0;
    size_t k = 0;
    for (int s = 0; s < ns; ++s) {
      const int dim = 3 * (int)(so[s + 1] - so[s]);
      for (int r = 0; r < dim; ++k) {
        CHECK(k < st.size() && st[k].src == src && st[k].o == so[s] && st[k].dim == dim && st[k].row0 == r);
        CHECK(st[k].rows >= 1 && r + st[k].rows <= dim && (long long)st[k].rows * dim * vsize <= scap);
        const PcgSpan v = pcg_span(src * vsize, (src + (long long)st[k].rows * dim) * vsize, 1LL << 62);
        CHECK(v.bytes <= align16(scap + 32));
        r += st[k].rows;
        src += (long long)st[k].rows * dim;
      }
    }
    CHECK(k == st.size());
  }
  std::printf("ok\n");
  return 0;
}
