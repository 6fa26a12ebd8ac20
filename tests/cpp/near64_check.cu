// Check of the nearly rounded quotients and square roots of
// csrc/fvs_ieee64.cuh (Div<., true>, Sqrt<true>: the fast FP64 flavour, the fast
// cut cells, the exact Riemann solver) against their bounds, 0.57 and 0.75 units
// in the last place, and of quotients that are 53-bit numbers, which have to
// stay exact: on the host with FP32 seeds off by -2..2 ulp (more than the
// device's are), or with an argument on the device with its own.  The distance
// from the exact value comes from the remainders a - q b and a - s s of one FMA,
// exact but for a rounding of 2^-53 of themselves.  Also IsNan.  Prints "bad 0"
// and exits 0 when every bound holds.
#include <cmath>
#include <cstdint>
#include <cstdio>
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

// a unit in the last place of a normal x
__host__ __device__ double Ulp(double x) {
  return FromBits((Bits(x) & kInf) - (uint64_t(52) << 52));
}

__host__ __device__ int Wrong(uint64_t i, float* worst_q, float* worst_s) {
  const uint64_t full = (1ull << 52) - 1, r = Mix(3 * i + 2);
  uint64_t ma = Mix(3 * i) & full, mb = Mix(3 * i + 1) & full;
  switch (i % 8) {
  case 1: mb = 0; break;
  case 2: mb = full; break;
  case 3: ma = (mb + 1) & full; break;
  case 4: ma = (mb - 1) & full; break;
  case 5: ma = full; break;
  case 6: mb = r & 15; break;
  default: break;
  }
  const uint64_t ea = 923 + r % 200, eb = 923 + (r >> 16) % 200;
  const double a = FromBits((ea << 52) | ma);
  const double b = FromBits(((r << 1) & kSign) | (eb << 52) | mb);
  int bad = 0;
  const double q = Div<false, true>(a, MakeDivisor(b));
  const double dq = fabs(fma(-q, b, a) / b) / Ulp(q);
  bad += !(dq <= 0.57);
  const double h = Div<true, true>(a, MakeDivisor(b));
  bad += Bits(h) != Bits(0.5 * q);
  const double s = Sqrt<true>(a);
  const double ds = fabs(fma(-s, s, a)) / (2.0 * s) / Ulp(s);
  bad += !(ds <= 0.75);
  *worst_q = fmaxf(*worst_q, static_cast<float>(dq));
  *worst_s = fmaxf(*worst_s, static_cast<float>(ds));
  // 26-bit factors: their product and its quotient by one of them are exact
  const double c = double((r & 0x3FFFFFF) | 1), d = double((mb & 0x3FFFFFF) | 1);
  bad += Div<false, true>(c * d, MakeDivisor(d)) != c;
  bad += Div<false, true>(b, MakeDivisor(b)) != 1.0;
  bad += Div<false, true>(a, MakeDivisor(1.0)) != a;
  return bad;
}

__global__ void CheckKernel(uint64_t first, int per, unsigned long long* bad) {
  const uint64_t t = first + (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) * per;
  int n = 0;
  float q = 0.0f, s = 0.0f;
  for (int k = 0; k < per; ++k) n += Wrong(t + k, &q, &s);
  if (n) atomicAdd(bad, static_cast<unsigned long long>(n));
  atomicMax(bad + 1, static_cast<unsigned long long>(q * 1e6f));
  atomicMax(bad + 2, static_cast<unsigned long long>(s * 1e6f));
}

}  // namespace

int main(int argc, char**) {
  unsigned long long out[3] = {0, 0, 0};
  if (argc > 1) {
    unsigned long long* d = nullptr;
    if (cudaMalloc(&d, sizeof out) != cudaSuccess) return 2;
    cudaMemset(d, 0, sizeof out);
    CheckKernel<<<4096, 256>>>(1u << 28, 64, d);
    if (cudaMemcpy(out, d, sizeof out, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    cudaFree(d);
  } else {
    for (seed_error = -2; seed_error <= 2; ++seed_error) {
      float q = 0.0f, s = 0.0f;
      for (uint64_t i = 0; i < 2000000; ++i) out[0] += Wrong(i, &q, &s);
      std::printf("seeds off by %d ulp: quotient %.4f, root %.4f ulp\n", seed_error, q, s);
    }
    const double inf = std::numeric_limits<double>::infinity(), nan = std::nan("");
    for (double x : {0.0, -0.0, 1.0, -1.0, inf, -inf, 5e-324, -1.7976931348623157e308})
      out[0] += IsNan(x);
    out[0] += !IsNan(nan) + !IsNan(-nan) + !IsNan(FromBits(kInf + 1)) +
              !IsNan(FromBits(kSign | (kInf + 1)));
  }
  if (argc > 1) std::printf("device: quotient %.4f, root %.4f ulp\n", out[1] * 1e-6, out[2] * 1e-6);
  std::printf("bad %llu\n", out[0]);
  return out[0] ? 1 : 0;
}
