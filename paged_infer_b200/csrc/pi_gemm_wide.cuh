// How the wide GEMM (pi_gemm_wide.cu) is cut over the CTAs, how it waits, which calls take it and in what scratch: plain code, for
// host (with or without a CUDA compiler) and device.
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

// A bounded wait.  `*weight` is what a poll counts: 0 while the kernel ahead still runs (those polls are not this launch's), then
// 1, and the whole limit once a wait of the CTA has run out, so that from then on a wait ends with its first poll that fails:
// however many K blocks are left, what a CTA still has to do are its tickets.  (With a comparison of its own for that the loop
// answers later: 2 % of a launch.)
constexpr int kPollLimit = 1 << 21, kGivenUp = kPollLimit;
template <class Done>
__device__ inline bool wait_for(Done done, const volatile int* weight) {
  for (int spin = 0; spin < kPollLimit;) {
    if (done()) return true;
    spin += *weight;
  }
  return false;
}

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

// Which kernel a call takes, of two that both could: true for this one.  Times in us, device, matrices out of HBM, both sides
// measured over 32..28672 rows, 1024..28672 columns and batches of 5 to 512, activations split by a launch of their own.
// The CUDA-core kernel takes 4 and 0.37 per million weights and pass over four activation rows (0.44 where one CTA of it fills
// an SM); rows too long for four in shared memory make passes over two (0.30) or one (0.18).
// On a full grid this one with the split takes 13 and 0.5 per million weights for up to 64 activation rows: the lines cross where
// a million weights times (3 passes - 4) reach 70.  2048 x 2048, 32 rows (84) 18.5 and 16.2, 16 rows (34) 10.9 and 15.0;
// 11264 x 2048, 8 rows (46) 22.8 and 24.3, 16 rows (185) 41.5 and 25.0; 24000 x 5600, 5 rows (269) 104 and 75.
// Few rows of many columns leave it few CTAs with long shares: 8, a microsecond per 1600 columns for the split (twice that beyond
// 16384, where a row leaves the registers) and 0.55 per K block of a share.  32 x 28672, 256 rows 54 and 96; 128 x 28672,
// 32 rows 39 and 68; 2048 x 28672, 5 rows 82 and 100.  Near a draw (1.2) the first line decides.
// Where a model hands planes from projection to projection there is no split and the lines cross lower: six layers of hidden 2048
// and a head, all on this one, 589 instead of 632 for 5 sequences, 644 instead of 683 for 16.
inline bool worth(size_t rows, size_t cols, int M, int sms, size_t smem) {
  int group = M >= 4 ? 4 : M >= 2 ? 2 : 1;
  while (group > 1 && group * cols * sizeof(float) > smem) group >>= 1;
  if (group * cols * sizeof(float) > smem) return true;   // the CUDA-core kernel has no room for a row
  const double mega = 1e-6 * (double)rows * (double)cols, fours = (M - 1) / 4 + 1, passes = (M - 1) / group + 1;
  if (mega * (3 * fours - 4) < 70) return false;
  const double cores = 4 + mega * passes * (group == 1 ? 0.18 : group == 2 ? 0.30 : cols > 7000 ? 0.44 : 0.37);
  const Cut c = make_cut((int)rows, M, (int)cols, sms);
  const double tensor = 8 + (double)cols / (cols > 16384 ? 800 : 1600) + 0.55 * c.tiles * c.nkb / c.ctas;
  return 1.2 * cores > tensor;
}

// Scratch for the activations of a launch: three 16-bit planes and a factor per row.
inline size_t planes_bytes(size_t rows, size_t cols) { return 3 * rows * cols * 2 + rows * sizeof(float) + 256; }

// Activation rows that pass through the scratch at once, from the sizes of the call alone, so that a row's sums do not depend on
// what a context has done before: all of them up to the limit, else equal portions of whole tiles.  The limit keeps the scratch
// at 1024 rows and 256 MiB; 1024 rows are 16 tiles, beside whose products another reading of the matrix does not show.
constexpr int kPortion = 1024;
constexpr size_t kPlanesLimit = (size_t)256 << 20;
inline int portion_limit(size_t cols) {
  const size_t fit = (kPlanesLimit - 256) / (3 * cols * 2 + sizeof(float)) / kCols * kCols;
  return (int)(fit < (size_t)kPortion ? fit : (size_t)kPortion);
}
inline int portion_rows(int M, size_t cols) {
  const int limit = portion_limit(cols);
  if (M <= limit) return M;
  const int n = (M - 1) / limit + 1;
  return ((M - 1) / n + kCols) / kCols * kCols;
}

__host__ __device__ inline size_t ticket_bytes(int sms) { return ((size_t)sms * sizeof(int) + 255) / 256 * 256; }

}  // namespace pi_wide
