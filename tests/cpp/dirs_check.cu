// The device's launch directions (csrc/sbr_dirs.cuh) against the host's
// subdivision, bit for bit, at the levels given.  Exit status 0: no difference.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "sbr_dirs.cuh"
#include "sbr_host.h"

int main(int argc, char** argv) {
  int bad = 0;
  for (int i = 1; i < argc; ++i) {
    const int level = std::atoi(argv[i]);
    std::vector<double> want, v0;
    std::vector<int> from, mate;
    sbr::icosphere(level, want);
    sbr::icosahedron(v0, from, mate);
    std::vector<double> got(want.size());
    double* v = nullptr;
    int* scratch = nullptr;
    if (cudaMalloc(&v, want.size() * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&scratch, sbr::dirs::scratch_ints(level) * sizeof(int)) != cudaSuccess)
      return 2;
    sbr::dirs::subdivide(level, v0.data(), from.data(), mate.data(), v, scratch, 4, 0);
    if (cudaMemcpy(got.data(), v, got.size() * sizeof(double), cudaMemcpyDeviceToHost) !=
        cudaSuccess)
      return 3;
    const bool same = !std::memcmp(got.data(), want.data(), got.size() * sizeof(double));
    std::printf("level %d: %zu directions %s\n", level, want.size() / 3, same ? "equal" : "DIFFER");
    bad += !same;
    cudaFree(v);
    cudaFree(scratch);
  }
  return bad != 0;
}
