// tk_split.h -- work splits of the kernels: which units, rows or jobs a CTA's tile
// holds.  Plain integer arithmetic, also compiled for the host, where the tests run
// it.
#pragma once

#ifdef __CUDACC__
#define TK_HD __host__ __device__ __forceinline__
#else
#define TK_HD inline
#endif

namespace tk {

// k_ntt_mma: whole tiles of W units (8 polynomials each) are dealt round robin, tile k
// of CTA c being the (k G + c)-th of the batch; the units left over, less than a tile
// per CTA, are split evenly into a last, short tile each.  So CTAs differ by at most
// one unit, and the launch moves through the batch as one front, upwards in the
// forward and downwards in the inverse: an inverse after a forward on the same
// memory starts on what was written last and is still in L2 (126 MB): ntt then invntt
// in place, us in a long loop, 200,000 polynomials (102 MB) 89.9 -> 83.5, 262,144
// 100.8 -> 97.5; one run of units per CTA before.
template <int W, bool kDown>
struct FrontTiles {
  int nunits, G, cta, whole, left0, nlast;

  TK_HD FrontTiles(int units, int ctas, int c) : nunits(units), G(ctas), cta(c) {
    whole = nunits / (G * W);
    const int left = nunits - whole * G * W;
    left0 = (int)((long long)cta * left / G);
    nlast = (int)((long long)(cta + 1) * left / G) - left0;
  }
  TK_HD int tiles() const { return whole + (nlast > 0); }            // of this CTA
  TK_HD int units(int k) const { return k < whole ? W : nlast; }     // of its tile k
  TK_HD int unit0(int k) const {                                     // the first of them
    const int i = k < whole ? (k * G + cta) * W : whole * G * W + left0;
    return kDown ? nunits - i - units(k) : i;
  }
};

// The tcgen05 kernels: whole tiles round robin, the same fronts.
TK_HD int front_tile_count(int ntiles, int G, int cta) { return (ntiles - 1 - cta) / G + 1; }
TK_HD int front_tile(int ntiles, int G, int cta, int k, bool down) {
  const int t = k * G + cta;
  return down ? ntiles - 1 - t : t;
}

// k_matvec_tiles, tiles of a launch of kind `units` (4, 2 or 1): 8-row shared-memory
// units, rows of the batch and jobs per tile.  k = 3: 24 rows, the smallest whole
// number of both jobs and units, or, with units = 1, two jobs in six rows of one unit
// (six-row TMA boxes).
TK_HD constexpr int tile_units(int k, int units) { return k == 3 && units > 1 ? 3 : units; }
TK_HD constexpr int tile_box_rows(int k, int units) { return k == 3 && units == 1 ? 6 : 8; }
TK_HD constexpr int tile_rows(int k, int units) {
  return tile_units(k, units) * tile_box_rows(k, units);
}
TK_HD constexpr int tile_jobs(int k, int units) { return tile_rows(k, units) / k; }

}  // namespace tk
