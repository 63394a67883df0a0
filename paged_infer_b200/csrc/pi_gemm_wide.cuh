// How the wide GEMM (pi_gemm_wide.cu) is cut over the CTAs: plain integer code, for host and device.
#pragma once

#include <cstddef>

#ifndef __CUDACC__
#define __host__
#define __device__
#endif

namespace pi_wide {

constexpr int kRows = 128;       // weight rows of a tile
constexpr int kCols = 64;        // activation rows of a tile
constexpr int kBlock = 64;       // K elements of a block
constexpr int kMinPart = 4;      // a share's end closer than this many blocks to a tile's end moves there
constexpr int kMaxShare = 8;     // CTAs per tile at most, on average
constexpr int kMaxHolders = 16;  // CTAs that can hold parts of one tile

// Tiles in order (row tile, column tile), K blocks innermost, all in one line; CTA i takes [cut_at(i), cut_at(i + 1)).
struct Cut {
  int tiles, mtiles, nkb, ctas;
};

__host__ __device__ inline Cut make_cut(int N, int M, int K, int sms) {
  Cut c;
  c.mtiles = (M + kCols - 1) / kCols;
  c.tiles = (N + kRows - 1) / kRows * c.mtiles;
  c.nkb = (K + kBlock - 1) / kBlock;
  int share = c.nkb / (2 * kMinPart);   // a part is worth its prologue and its parking from eight blocks on
  if (share < 1) share = 1;
  if (share > kMaxShare) share = kMaxShare;
  c.ctas = (long long)c.tiles * share < sms ? c.tiles * share : sms;
  return c;
}

__host__ __device__ inline int cut_at(const Cut& c, int i) {
  const int pos = (int)((long long)c.tiles * c.nkb * i / c.ctas), r = pos % c.nkb;
  if (r < kMinPart) return pos - r;
  if (c.nkb - r < kMinPart) return pos + (c.nkb - r);
  return pos;
}

// The CTAs that hold parts of `tile`, of which `cta` is one: their slots among the parked tiles (2 per CTA: its first tile,
// its last) in order, how many, and the first of them, whose ticket counter the tile uses.  A CTA is first of one shared
// tile at most: the one its share ends in.
__host__ __device__ inline int holders(const Cut& c, int cta, int tile, int* slots, int* first_cta) {
  const int begin = tile * c.nkb, end = begin + c.nkb;
  int j = cta;
  while (j > 0 && cut_at(c, j) > begin) --j;
  int n = 0;
  for (int a = cut_at(c, j); j < c.ctas && a < end; ++j) {
    const int b = cut_at(c, j + 1);
    if (b > begin && b > a) {
      if (n == 0) *first_cta = j;
      if (n < kMaxHolders) slots[n] = j * 2 + (a >= begin ? 0 : 1);
      ++n;
    }
    a = b;
  }
  return n;
}

__host__ __device__ inline size_t ticket_bytes(int sms) { return ((size_t)sms * sizeof(int) + 255) / 256 * 256; }

}  // namespace pi_wide
