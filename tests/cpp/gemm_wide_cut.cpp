// The scratch of the GEMM for bf16 weights (csrc/pi_gemm_wide.cuh), without a GPU.  Prints "ok <name>" per group; exit code 0 only
// if every check held.
#include <cstdio>

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

int main() {
  portions();
  giving_up();
  if (!failures) std::printf("all ok\n");
  return failures != 0;
}
