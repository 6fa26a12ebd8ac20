// Check of the quotients, square roots and comparisons of csrc/fvs_ieee64.cuh
// against the IEEE operations, bit for bit: on the host with FP32 seeds off by
// -2..2 ulp (more than the device's seeds are), or with an argument on the
// device with its own seeds.  Operands: random mantissas, mantissas at both
// ends and with long runs of zeros or ones, equal and neighbouring operands,
// every exponent, and zeros, infinities, NaN and subnormals.  Prints "bad 0"
// and exits 0 when every result agrees.
#include <cmath>
#include <cstdio>
#include <cstdint>
#include <cstring>
#include <limits>

#include "fvs_ieee64.cuh"

using namespace fvs::ieee64;

namespace {

__host__ __device__ uint64_t Mix(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

__host__ __device__ double FromBits(uint64_t b) {
  return Make(static_cast<uint32_t>(b >> 32), static_cast<uint32_t>(b));
}

// operand pair number i
__host__ __device__ void Operands(uint64_t i, double* a, double* b) {
  const uint64_t full = (1ull << 52) - 1;
  uint64_t ma = Mix(3 * i) & full, mb = Mix(3 * i + 1) & full;
  const uint64_t r = Mix(3 * i + 2);
  switch (i % 14) {
  case 1: mb = 0; break;
  case 2: mb = full; break;
  case 3: ma = mb; break;
  case 4: ma = (mb + 1) & full; break;
  case 5: ma = (mb - 1) & full; break;
  case 6: ma &= ~0xFFFFFFFFull; break;
  case 7: mb &= ~((1ull << 40) - 1); break;
  case 8: mb |= (1ull << 40) - 1; break;
  case 9: ma = 0; break;
  case 10: ma = full; break;
  case 11: mb = r & 15; break;
  default: break;
  }
  uint64_t ea = 923 + r % 200, eb = 923 + (r >> 16) % 200;
  if (i % 14 == 12) {
    ea = 513 + r % 1021;
    eb = 513 + (r >> 16) % 1021;
  } else if (i % 14 == 13) {
    ea = r % 2048;
    eb = (r >> 16) % 2048;
  }
  *a = FromBits((r & (1ull << 63)) | (ea << 52) | ma);
  *b = FromBits(((r << 1) & (1ull << 63)) | (eb << 52) | mb);
}

__host__ __device__ bool Same(double x, double y) {
  return Bits(x) == Bits(y) || (x != x && y != y);
}

__host__ __device__ int Wrong(double a, double b) {
  const double c = fabs(a);
#ifdef __CUDA_ARCH__
  const double q = __ddiv_rn(a, b), h = __ddiv_rn(0.5 * a, b), s = __dsqrt_rn(c);
#else
  const double q = a / b, h = 0.5 * a / b, s = std::sqrt(c);
#endif
  int bad = !Same(Div(a, b), q) + !Same(Sqrt(c), s);
  bad += !Same(Div<true>(a, MakeDivisor(b)), h);
  bad += Positive(a) != (a > 0.0);
  bad += Negative(a) != (a < 0.0);
  bad += IsZero(a) != (a == 0.0);
  if (!(a == 0.0 && b == 0.0)) bad += Less(a, b) != (a < b);
  return bad;
}

__global__ void CheckKernel(uint64_t first, int per, unsigned long long* bad) {
  const uint64_t t = first + (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) * per;
  int n = 0;
  for (int k = 0; k < per; ++k) {
    double a, b;
    Operands(t + k, &a, &b);
    n += Wrong(a, b);
  }
  if (n) atomicAdd(bad, static_cast<unsigned long long>(n));
}

}  // namespace

int main(int argc, char**) {
  unsigned long long bad = 0;
  if (argc > 1) {
    unsigned long long* d = nullptr;
    if (cudaMalloc(&d, sizeof *d) != cudaSuccess) return 2;
    cudaMemset(d, 0, sizeof *d);
    CheckKernel<<<4096, 256>>>(1u << 28, 256, d);
    if (cudaMemcpy(&bad, d, sizeof bad, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    cudaFree(d);
  } else {
    const double inf = std::numeric_limits<double>::infinity(), nan = std::nan("");
    const double special[] = {0.0, -0.0, 1.0, -1.0, inf, -inf, nan, -nan, 5e-324, -5e-324,
                              2.2250738585072014e-308, 1.7976931348623157e308, 0x1p-510,
                              -0x1p-511, 0x1p511, 0x1.fffffffffffffp510, 4.0, 2.0, 3.0, 1e-300};
    for (seed_error = -2; seed_error <= 2; ++seed_error) {
      for (uint64_t i = 0; i < 2000000; ++i) {
        double a, b;
        Operands(i, &a, &b);
        bad += Wrong(a, b);
      }
      for (double a : special)
        for (double b : special) bad += Wrong(a, b);
    }
  }
  std::printf("bad %llu\n", bad);
  return bad ? 1 : 0;
}
