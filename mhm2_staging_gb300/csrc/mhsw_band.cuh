// mhsw_band.cuh -- how far an alignment that reaches its score can drift from the end cell's
// diagonal: the bounds the begin searches size their bands and boxes with.
#pragma once
#include "mhsw_types.h"

namespace mhsw {

// Rows the first search covers: twice the diagonal steps the score needs at least, and slack.
__host__ __device__ __forceinline__ int band_first_cap(int S, int mt, int M2) {
  const long long tt = 2ll * S / (mt > 0 ? mt : 1) + 16;
  return (int)(tt < M2 ? tt : M2);
}

// Total gap length g (inserted plus deleted cells) of an alignment that scores S with at
// most dmax diagonal steps.  Each diagonal step scores at most match, and g gap cells in
// r >= 1 runs cost r*gO + (g - r)*gE >= g*min(gO, gE) + max(gO - gE, 0), so
// g*min(gO, gE) + max(gO - gE, 0) <= dmax*match - S (g = 0 when that leaves no room for
// one gap cell).  (dmax <= 65000 and match <= 127 keep the product inside 32 bits.)
__host__ __device__ __forceinline__ int gap_cells_bound(int dmax, int S, const Scoring &sc) {
  const int gmin = sc.gap_open < sc.gap_extend ? sc.gap_open : sc.gap_extend;
  const int g1 = gmin > 0 ? gmin : 1;
  const int slack = dmax * sc.match - S - (sc.gap_open > sc.gap_extend ? sc.gap_open - sc.gap_extend : 0);
  return slack < g1 ? 0 : slack / g1;
}

// Total gap length any alignment reaching the score within the first t rows can have:
// its diagonal steps D <= min(t, N2).
__host__ __device__ __forceinline__ int band_gap_bound(int t, int N2, int S, const Scoring &sc) {
  return gap_cells_bound(t < N2 ? t : N2, S, sc);
}

// How far such an alignment can drift from the end cell's diagonal to either side.  I
// vertical gap cells (a row each, no column) leave at most t - I diagonal steps:
// S <= (t - I)*match - I*gmin - c, c = max(gO - gE, 0) once, so
// I <= (t*match - S - c) / (match + gmin); likewise J horizontal gap cells leave at most
// N2 - J, so J <= (N2*match - S - c) / (match + gmin).  Both are at most the total g.  A
// band over columns [row - L, row - L + W) holds every such alignment when I <= L and
// J <= W - 1 - L.
__host__ __device__ __forceinline__ void band_sides(int t, int N2, int S, const Scoring &sc, int &I, int &J) {
  const int g = band_gap_bound(t, N2, S, sc);
  const int gmin = sc.gap_open < sc.gap_extend ? sc.gap_open : sc.gap_extend;
  const int mg = sc.match + (gmin > 0 ? gmin : 1);
  const int c = sc.gap_open > sc.gap_extend ? sc.gap_open - sc.gap_extend : 0;
  const int st = t * sc.match - S - c, sn = N2 * sc.match - S - c;
  I = st < mg ? 0 : st / mg;
  J = sn < mg ? 0 : sn / mg;
  if (I > g) I = g;
  if (J > g) J = g;
}

// Whether the warp-per-pair begin kernel (mhsw_short.cu) takes a search: its rows, columns and
// score fit that kernel's tile and keys.
constexpr int kWarpBeginRows = 512, kWarpBeginCols = 2048, kWarpBeginScore = 4000;
__host__ __device__ __forceinline__ bool warp_begin(int M2, int N2, int S, const Scoring &sc) {
  if (M2 > kWarpBeginRows || S > kWarpBeginScore) return false;
  int I, J;
  band_sides(M2, N2, S, sc, I, J);
  return (M2 + J < N2 ? M2 + J : N2) <= kWarpBeginCols;
}

}  // namespace mhsw
