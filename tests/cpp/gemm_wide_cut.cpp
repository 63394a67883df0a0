// The cut and the scratch of the GEMM for bf16 weights (csrc/pi_gemm_wide.cuh), without a GPU.  Prints "ok <name>" per group; exit code 0 only
// if every check held.
#include <cstdio>
#include <random>
#include <vector>

#include "../../paged_infer_b200/csrc/pi_gemm_wide.cuh"

using namespace pi_wide;

static int failures = 0;
#define CHECK(cond)                                                 \
  do {                                                              \
    if (!(cond)) {                                                  \
      std::printf("FAILED %s:%d: %s\n", __FILE__, __LINE__, #cond); \
      ++failures;                                                   \
    }                                                               \
  } while (0)

// Every K block of every tile belongs to one CTA; the holders of a tile agree on slots, order and counter; no two tiles share a
// parking slot or a counter.
static void cut() {
  std::mt19937 rng(1);
  auto between = [&](int lo, int hi) { return (int)(lo + rng() % (unsigned)(hi - lo + 1)); };
  for (int round = 0; round < 1500; ++round) {
    const int sms = round % 3 ? 148 : between(1, 160), big = round % 5 == 0;
    const Cut c = make_cut(between(32, big ? 40000 : 3000), between(5, big ? 1300 : 200), 8 * between(1, round % 7 == 0 ? 16384 : 700), sms);
    CHECK(c.ctas >= 1 && c.ctas <= sms && cut_at(c, 0) == 0 && cut_at(c, c.ctas) == c.tiles * c.nkb);
    std::vector<int> counter(c.ctas, -1), slot(2 * c.ctas, -1);
    std::vector<std::vector<int>> seen(c.tiles);
    for (int i = 0; i < c.ctas; ++i) {
      const int pos0 = cut_at(c, i), pos1 = cut_at(c, i + 1);
      CHECK(pos0 <= pos1);
      for (int pos = pos0; pos < pos1;) {
        const int tile = pos / c.nkb, first = tile * c.nkb, end = first + c.nkb < pos1 ? first + c.nkb : pos1;
        if (pos != first || end != first + c.nkb) {   // a part
          const int mine = i * 2 + (pos0 >= first ? 0 : 1);
          CHECK(slot[mine] == -1);
          slot[mine] = tile;
          int slots[kMaxHolders], j0 = -1;
          const int n = holders(c, i, tile, slots, &j0);
          CHECK(n >= 2 && n <= kMaxHolders && j0 >= 0 && j0 < c.ctas);
          CHECK(counter[j0] == -1 || counter[j0] == tile);
          counter[j0] = tile;
          std::vector<int> all(slots, slots + n);
          bool holds = false;
          for (int k = 0; k < n; ++k) {
            holds = holds || all[k] == mine;
            CHECK(k == 0 || all[k] / 2 > all[k - 1] / 2);
          }
          CHECK(holds && (seen[tile].empty() || seen[tile] == all));
          seen[tile] = all;
        } else {
          CHECK(seen[tile].empty());
        }
        pos = end;
      }
    }
    for (int t = 0; t < c.tiles; ++t)
      for (int s : seen[t]) CHECK(slot[s] == t);   // whoever is last reads what that CTA parked for this tile
  }
  std::printf("ok cut\n");
}

// Every call passes through the scratch that was laid out for its matrix, whatever its batch: equal portions of whole tiles.
static void portions() {
  const int Ms[] = {1, 5, 63, 64, 65, 512, 640, 1023, 1024, 1025, 2048, 2049, 100000, 1 << 20, 2147483647};
  for (size_t cols = 8; cols <= 131072; cols += cols < 4096 ? 8 : 1016) {
    const int limit = portion_limit(cols);
    CHECK(limit >= kCols && limit <= kPortion && limit % kCols == 0);
    CHECK(planes_bytes(limit, cols) <= kPlanesLimit);
    for (int M : Ms) {
      const int step = portion_rows(M, cols);
      CHECK(step >= 1 && step <= limit && step <= M);
      CHECK(step == M || step % kCols == 0);
      const long long n = ((long long)M + step - 1) / step;
      CHECK(n <= ((long long)M + limit - 1) / limit);
      CHECK(planes_bytes(step, cols) <= planes_bytes(M < limit ? M : limit, cols));
    }
  }
  std::printf("ok portions\n");
}

// A CTA of many blocks whose products stop coming: one wait runs out, every later one costs a single poll.
static void giving_up() {
  volatile int weight = 1;
  const int limit = kPollLimit, blocks = 2000, reached = 37;
  int done = 0, polls = 0;
  for (int it = 0; it < blocks; ++it) {   // the epilogue walks on to its tickets
    if (wait_for([&] { ++polls; return it < reached; }, &weight) && weight != kGivenUp)
      ++done;
    else
      weight = kGivenUp;
  }
  CHECK(done == reached && polls == reached + limit + (blocks - reached - 1));
  weight = polls = 0;                     // polls ahead of the dependency do not count
  CHECK(wait_for([&] { weight = ++polls > 3 * limit; return polls == 3 * limit + 7; }, &weight));
  weight = 1;
  polls = 0;                              // another warp gives up meanwhile
  CHECK(!wait_for([&] { weight = ++polls == 9 ? kGivenUp : 1; return false; }, &weight) && polls == 9);
  std::printf("ok giving up\n");
}

// The dispatch line against both sides as measured (us): the chosen side is never more than a quarter slower than the other.
static void dispatch() {
  const struct { int rows, cols, M; double cores, tensor; } seen[] = {
      {32, 1024, 512, 4.4, 16.3},       {32, 16384, 64, 15.8, 36.7},     {32, 16384, 256, 31.9, 40.3},     {32, 28672, 64, 24.8, 70.3},
      {32, 28672, 128, 39.0, 71.2},     {32, 28672, 256, 53.8, 96.0},    {64, 5632, 512, 24.1, 25.2},      {128, 2048, 64, 9.7, 16.8},
      {128, 8192, 512, 67.5, 30.0},     {128, 28672, 5, 14.3, 65.3},     {128, 28672, 32, 39.0, 68.0},     {128, 28672, 64, 81.2, 73.4},
      {128, 28672, 512, 336.5, 116.0},  {256, 2048, 512, 33.3, 19.4},    {256, 8192, 128, 38.3, 27.2},     {512, 1024, 64, 6.9, 15.3},
      {512, 4096, 64, 18.2, 21.9},      {512, 4096, 512, 111.4, 30.0},   {1024, 2048, 32, 10.8, 15.9},     {1024, 2048, 128, 32.5, 18.3},
      {1024, 8192, 5, 20.6, 23.4},      {1024, 8192, 64, 67.5, 27.9},    {2048, 2048, 16, 10.9, 15.0},     {2048, 2048, 32, 18.5, 16.2},
      {2048, 5632, 8, 16.2, 20.8},      {2048, 5632, 24, 33.4, 22.4},    {2560, 2048, 16, 14.1, 15.4},     {2560, 2048, 24, 18.5, 16.0},
      {4096, 4096, 5, 18.7, 23.8},      {4096, 4096, 16, 32.1, 26.7},    {11264, 2048, 8, 22.8, 24.3},     {11264, 2048, 12, 33.7, 24.6},
      {2048, 28672, 5, 82.3, 100.4},    {2048, 28672, 16, 175.3, 101.3}, {24000, 5600, 5, 104.4, 75.1},    {28672, 4096, 8, 91.1, 67.3}};
  for (const auto& s : seen) {
    const bool tensor = worth(s.rows, s.cols, s.M, 148, 232448 - 2048);
    const double took = tensor ? s.tensor : s.cores, other = tensor ? s.cores : s.tensor;
    if (took > 1.25 * other) std::printf("FAILED %d x %d, %d rows: %.1f taken, %.1f not\n", s.rows, s.cols, s.M, took, other), ++failures;
  }
  CHECK(worth(40, 65536, 5, 148, 232448 - 2048));   // rows that the CUDA-core kernel refuses
  std::printf("ok dispatch\n");
}

int main() {
  cut();
  dispatch();
  portions();
  giving_up();
  if (!failures) std::printf("all ok\n");
  return failures != 0;
}
