// Checks the integer-pipe logistic function of device.cuh (exp_neg_fixed, logistic_fixed)
// against long double arithmetic on the host: e^-t, 1/(1+e^-t), e^-t/(1+e^-t) and their
// product, each within half an ulp and the fixed-point error of 2^-56 relative. Arguments:
// both ends of the range, every table step's neighbourhood and random ones over all
// magnitudes.
// Exit status 0 when every result is within its bound; prints the worst otherwise.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>

#include "device.cuh"

using namespace mpsb;

__global__ void evaluate(const double* t, double* out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[4 * i] = fixed64_to_f64(exp_neg_fixed(t[i]));
  logistic_fixed(t[i], out + 4 * i + 1, out + 4 * i + 2, out + 4 * i + 3);
}

int main() {
  std::vector<double> t = {0.0, 0x1p-1074, 0x1p-300, 0x1p-60, 0x1p-58, 0x1p-53, kExpFixedMax,
                           std::nextafter(kExpFixedMax, 0.0)};
  for (int j = 0; j < 256 * 57; ++j) {  // t log2(e) at the table steps
    const double at = j / 256.0 * 0.6931471805599453;
    for (double x : {std::nextafter(at, 0.0), at, std::nextafter(at, 100.0)})
      if (x >= 0.0 && x <= kExpFixedMax) t.push_back(x);
  }
  std::mt19937_64 rng(7);
  std::uniform_real_distribution<double> all(0.0, kExpFixedMax), low(0.0, 3.0), magnitude(-40.0, 5.3);
  for (int i = 0; i < 200000; ++i) {
    t.push_back(all(rng));
    t.push_back(low(rng));
    t.push_back(std::exp2(magnitude(rng)));
  }
  while (t.back() > kExpFixedMax) t.pop_back();
  for (double& x : t)
    if (x > kExpFixedMax) x = kExpFixedMax;
  const int n = int(t.size());
  double *d_t = nullptr, *d_out = nullptr;
  std::vector<double> out(4 * size_t(n));
  if (cudaMalloc(&d_t, n * sizeof(double)) != cudaSuccess) return 2;
  if (cudaMalloc(&d_out, out.size() * sizeof(double)) != cudaSuccess) return 2;
  cudaMemcpy(d_t, t.data(), n * sizeof(double), cudaMemcpyHostToDevice);
  evaluate<<<(n + 255) / 256, 256>>>(d_t, d_out, n);
  if (cudaMemcpy(out.data(), d_out, out.size() * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  cudaFree(d_t);
  cudaFree(d_out);
  const long double bound = 0x1p-53L + 0x1p-56L;
  long double worst[4] = {0, 0, 0, 0};
  for (int i = 0; i < n; ++i) {
    const long double e = expl(-(long double)t[i]);
    const long double want[4] = {e, e / (1 + e), 1 / (1 + e), e / (1 + e) / (1 + e)};
    for (int k = 0; k < 4; ++k) {
      const long double r = fabsl(out[4 * size_t(i) + k] / want[k] - 1);
      if (!(r <= worst[k])) worst[k] = r;
    }
  }
  bool ok = true;
  for (int k = 0; k < 4; ++k) ok = ok && worst[k] <= bound;
  std::printf("%d arguments, worst relative errors %.3Lg %.3Lg %.3Lg %.3Lg, bound %.3Lg\n", n, worst[0],
              worst[1], worst[2], worst[3], bound);
  return ok ? 0 : 1;
}
