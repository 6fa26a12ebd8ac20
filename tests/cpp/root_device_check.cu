// Check of RecipRoot (csrc/fvs_roots.cuh), x^(-1/n), over the whole range of
// ratios that it takes, 1e-30 < x < 1e30, for n = 3 to 64: on the device with
// the device's FP32 estimate (with an argument), or on the host with the
// host's.  Against the 80- or 128-bit power of the host.
//
// Bound, with u = 2^-53: the power r^n of the estimate carries n - 1 products'
// roundings, so the residual is off by (n - 1) u and the correction by less
// than u; the last FMA rounds by u; the step's remainder, (n + 1) (2 n + 1)
// e^3 / (6 n^3), is below 0.9 u for an estimate with |e| < 8.2e-6 at n = 3
// (the host's; the device's is better): 2.9 u.  An estimate off by 2 FP32 ulp
// more exceeds it.  Prints the largest error in u and exits 1 above the bound.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "fvs_roots.cuh"

using fvs::riemann::Powers;

namespace {

__global__ void RootKernel(Powers pw, const double* x, double* y, int count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) y[i] = pw.RecipRoot(x[i]);
}

}  // namespace

int main(int argc, char**) {
  const bool device = argc > 1;
  const int count = 1 << 17;
  std::vector<double> x(count), y(count);
  double *dx = nullptr, *dy = nullptr;
  if (device && (cudaMalloc(&dx, count * sizeof(double)) != cudaSuccess ||
                 cudaMalloc(&dy, count * sizeof(double)) != cudaSuccess))
    return 2;
  int fail = 0;
  for (int n : {3, 4, 5, 7, 12, 21, 64}) {
    std::mt19937_64 rng(n);
    std::uniform_real_distribution<double> e(-30.0, 30.0);
    const Powers pw(n);
    for (int i = 0; i < count; ++i) {
      // an eighth of the ratios at each end of the range
      const double t = e(rng);
      const double v = i % 8 == 0 ? 29.0 + t / 30.1 : i % 8 == 1 ? -29.0 + t / 30.1 : t;
      x[i] = std::pow(10.0, v);
      if (!pw.Fast(x[i])) x[i] = 1.0;
    }
    if (device) {
      if (cudaMemcpy(dx, x.data(), count * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess)
        return 2;
      RootKernel<<<count / 256, 256>>>(pw, dx, dy, count);
      if (cudaMemcpy(y.data(), dy, count * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess)
        return 2;
    } else {
      for (int i = 0; i < count; ++i) y[i] = pw.RecipRoot(x[i]);
    }
    double worst = 0.0;
    for (int i = 0; i < count; ++i) {
      const long double ref = powl(x[i], -1.0L / n);
      const double err = static_cast<double>(fabsl((y[i] - ref) / ref)) * 0x1p53;
      worst = !(err <= worst) ? err : worst;
    }
    std::printf("n %d worst %.3f u\n", n, worst);
    fail |= !(worst <= 2.9);
  }
  std::printf("fail %d\n", fail);
  return fail;
}
