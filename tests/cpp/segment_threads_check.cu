// Threads of a search BVH segment's block (csrc/sbr_prep.cuh).  Host code only.
// Exit status 0: a level with a long segment never gives it one warp, and levels
// of short ones do.
#include <cstdio>

#include "sbr_prep.cuh"

int main() {
  int bad = 0;
  auto want = [&bad](int mean, int longest, int threads) {
    const int got = sbr::prep::segment_threads(mean, longest);
    if (got != threads) {
      std::printf("mean %d, longest %d: %d threads, not %d\n", mean, longest, got, threads);
      ++bad;
    }
  };
  want(580000, 580000, 1024);
  want(2049, 9000, 1024);
  want(2048, 9000, 256);
  want(129, 200, 256);
  want(128, 512, 32);
  want(128, 513, 256);
  want(98, 9936, 256);  // 2,028 segments of a scene of 200,000, one with a detailed object
  want(1, 7, 32);
  return bad != 0;
}
