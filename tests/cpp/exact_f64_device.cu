// Checks the integer-pipe double operations of exact_f64.cuh on the device
// against the device's own IEEE operations, bit for bit.  argv[1]: random cases
// per thread.  Built and run by tests/test_exact_f64_gpu.py.
#include <cstdio>
#include <cstdlib>

#include "exact_f64.cuh"

using namespace om::xf;

struct Report {
  unsigned long long bad;
  int op;
  double a, b, got, want;
};

__device__ uint64_t mix(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__device__ void same(Report *r, int op, double a, double b, double got, double want) {
  if (bits(got) == bits(want) || (got != got && want != want)) return;
  if (atomicAdd(&r->bad, 1ull) == 0) {
    r->op = op;
    r->a = a;
    r->b = b;
    r->got = got;
    r->want = want;
  }
}

__device__ void check(Report *r, double a, double b) {
  same(r, 0, a, b, div(a, b), __ddiv_rn(a, b));
  same(r, 1, a, 0, sqrt_rn(a), __dsqrt_rn(a));
  same(r, 2, a, 0, half(a), __dmul_rn(a, 0.5));
  same(r, 3, a, 0, plus_zero(a), __dadd_rn(0.0, a));
  same(r, 4, a, b, plus_none(a, b), __dadd_rn(a, __dmul_rn(b, 0.0)));
  same(r, 5, a, 0, positive(a), 0.0 < a);
  same(r, 6, a, b, less(a, b), a < b);
  same(r, 7, a, b, lesseq(a, b), a <= b);
  same(r, 8, a, b, absmaller(a, b),
       __dmul_rn(a, b) <= 0.0 ? 0.0 : (fabs(a) < fabs(b) ? a : b));
}

__global__ void random_cases(Report *r, int n) {
  const uint64_t frac = 0x000fffffffffffffull;
  uint64_t x = mix(blockIdx.x * (uint64_t)blockDim.x + threadIdx.x + 1);
  auto rng = [&] { return mix(x += 0x9E3779B97F4A7C15ull); };
  for (int i = 0; i < n; ++i) {
    uint64_t u = rng(), v = rng();
    const int kind = (int)(rng() % 8);
    if (kind < 6) {  // ordinary magnitudes
      u = (u & ~(2047ull << 52)) | (uint64_t)(1003 + rng() % 40) << 52;
      v = (v & ~(2047ull << 52)) | (uint64_t)(1003 + rng() % 40) << 52;
    }
    if (kind == 1) u |= frac >> (rng() % 40), v |= frac >> (rng() % 40);
    if (kind == 2) u &= ~(frac >> (rng() % 40)), v &= ~(frac >> (rng() % 40));
    if (kind == 3) {  // quotients next to exact ones
      const double q = from_bits((rng() & frac) | 1023ull << 52);
      u = bits(__dmul_rn(q, from_bits(v))) + rng() % 3 - 1;
    }
    if (kind == 4) {  // squares and their neighbours
      const double s = from_bits(u);
      u = bits(__dmul_rn(s, s)) + rng() % 3 - 1;
    }
    if (kind == 5) v = rng() & 1 ? u : u ^ 1ull << 63;
    check(r, from_bits(u), from_bits(v));
  }
}

// every pair of n operands, one thread a pair
__global__ void edge_cases(Report *r, const double *v, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n * n) check(r, v[i / n], v[i % n]);
}

int main(int, char **argv) {
  const double inf = HUGE_VAL;
  const double edge[] = {0.0, -0.0, inf, -inf, inf - inf, 1, -1, 2, 3, 4, 5e-324, -5e-324, 1e-2,
                         2.2250738585072014e-308, 1.7976931348623157e308, 0x1.fffffffffffffp0,
                         0x1.fffffffffffffp1, 0x1.0000000000001p0, 0x1.0000000000001p1, 0x1p-480,
                         0x1.fffffffffffffp-481, 0x1p479, 0x1p480, 1e-160, 1e160, -1e200};
  const int n = (int)(sizeof edge / sizeof edge[0]);
  Report *r, h{};
  double *v;
  if (cudaMalloc(&r, sizeof h) != cudaSuccess || cudaMalloc(&v, sizeof edge) != cudaSuccess) return 2;
  cudaMemcpy(r, &h, sizeof h, cudaMemcpyHostToDevice);
  cudaMemcpy(v, edge, sizeof edge, cudaMemcpyHostToDevice);
  edge_cases<<<(n * n + 127) / 128, 128>>>(r, v, n);
  random_cases<<<304, 256>>>(r, std::atoi(argv[1]));
  if (cudaMemcpy(&h, r, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) {
    std::printf("%s\n", cudaGetErrorString(cudaGetLastError()));
    return 2;
  }
  if (h.bad)
    std::printf("%llu differ; operation %d (%a, %a): %a, not %a\n", h.bad, h.op, h.a, h.b, h.got,
                h.want);
  return h.bad != 0;
}
