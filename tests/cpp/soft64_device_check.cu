// FP64 operations in integer arithmetic (csrc/sbr_soft64.cuh) as compiled for the
// device, with its own seeds and instructions, against the device's own FP64, bit
// for bit: random and patterned mantissas, values next to products, squares and
// FP32 ties.  Exit status 0: no difference.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "sbr_soft64.cuh"

using namespace sbr;

enum Op { kMul, kDiv, kRcp, kSqrt, kToF32, kFromF32, kFromInt, kOps };
static const char* const kName[kOps] = {"product",  "quotient",          "reciprocal",     "root",
                                        "to FP32", "double of a float", "double of a count"};

struct Report {
  unsigned long long bad[kOps];
  unsigned long long first[kOps];  // the lowest index of a difference
};

// u: arbitrary bits for the conversions.  NaN results count as equal.
__global__ void k_check(const double* a, const double* b, const unsigned long long* u, long long n,
                        Report* rep) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    auto same = [&](int op, double got, double want) {
      if (__double_as_longlong(got) == __double_as_longlong(want) || want != want) return;
      atomicAdd(&rep->bad[op], 1ull);
      atomicMin(&rep->first[op], (unsigned long long)i);
    };
    const double x = a[i], y = b[i];
    same(kMul, soft64::mul(x, y), __dmul_rn(x, y));
    if (y != 0) {
      same(kDiv, soft64::div(x, y), __ddiv_rn(x, y));
      same(kRcp, soft64::rcp(y), __drcp_rn(y));
    }
    same(kSqrt, soft64::sqrt(fabs(x)), __dsqrt_rn(fabs(x)));
    const double z = __longlong_as_double((long long)u[i]);
    same(kToF32, double(soft64::to_f32(x)), double(__double2float_rn(x)));
    same(kToF32, double(soft64::to_f32(z)), double(__double2float_rn(z)));
    const float f = __uint_as_float(unsigned(u[i]));
    same(kFromF32, soft64::from_f32(f), double(f));
    const int k = int((u[i] >> 33) >> (u[i] & 31));
    same(kFromInt, soft64::from_int(k), double(k));
  }
}

int main(int argc, char** argv) {
  const long long n = argc > 1 ? std::atoll(argv[1]) : 1 << 20;
  std::mt19937_64 rng(2);
  auto patterned = [&rng]() {
    uint64_t m = rng() & 0xfffffffffffffull;
    switch (rng() % 8) {
      case 0: m = 0; break;
      case 1: m = 0xfffffffffffffull; break;
      case 2: m &= ~0ull << (rng() % 52); break;
      case 3: m |= (1ull << (rng() % 52)) - 1; break;
      case 4: m = 1ull << (rng() % 52); break;
      case 5: m = 0xfffffffffffffull & ~(1ull << (rng() % 52)); break;
      default: break;
    }
    const uint64_t e = 1023 - 119 + rng() % 218, s = rng() & (1ull << 63);
    return soft64::from_bits(rng() % 64 ? (s | e << 52 | m) : s);
  };
  std::vector<double> a(n), b(n);
  std::vector<unsigned long long> u(n);
  for (long long i = 0; i < n; ++i) {
    a[i] = patterned();
    b[i] = patterned();
    if (a[i] != 0 && b[i] != 0 && i % 3 == 1)  // quotients next to a value
      a[i] = std::nextafter(a[i] * b[i], rng() & 1 ? 1e300 : -1e300);
    if (b[i] != 0 && i % 3 == 2)  // roots next to a value
      a[i] = std::nextafter(b[i] * b[i], rng() & 1 ? 1e300 : 0);
    u[i] = rng();
    if (i & 1) {  // FP32 ties and their neighbours
      u[i] &= ~0x1fffffffull;
      u[i] |= rng() % 3 == 0 ? 0x10000000ull : (rng() & 1 ? 0x0fffffffull : 0x10000001ull);
    }
  }
  double *da = nullptr, *db = nullptr;
  unsigned long long* du = nullptr;
  Report* dr = nullptr;
  Report r = {};
  for (auto& f : r.first) f = ~0ull;
  const size_t bytes = size_t(n) * 8;
  if (cudaMalloc(&da, bytes) || cudaMalloc(&db, bytes) || cudaMalloc(&du, bytes) ||
      cudaMalloc(&dr, sizeof r))
    return 2;
  if (cudaMemcpy(da, a.data(), bytes, cudaMemcpyHostToDevice) ||
      cudaMemcpy(db, b.data(), bytes, cudaMemcpyHostToDevice) ||
      cudaMemcpy(du, u.data(), bytes, cudaMemcpyHostToDevice) ||
      cudaMemcpy(dr, &r, sizeof r, cudaMemcpyHostToDevice))
    return 3;
  k_check<<<1024, 128>>>(da, db, du, n, dr);
  if (cudaMemcpy(&r, dr, sizeof r, cudaMemcpyDeviceToHost)) return 4;
  int bad = 0;
  for (int op = 0; op < kOps; ++op)
    if (r.bad[op]) {
      const size_t i = size_t(r.first[op]);
      std::printf("%s: %llu differences, the first at %a, %a, %llx\n", kName[op], r.bad[op], a[i],
                  b[i], u[i]);
      ++bad;
    }
  std::printf("%lld operands, %d operations differ\n", n, bad);
  return bad != 0;
}
