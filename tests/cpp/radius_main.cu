// Every Box-Muller radius, that of each of the 2^24 uniforms, against
// sqrt(-2 ln a) in double precision.  Prints "ok" and the largest errors.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <vector>

#include "bd_device.cuh"

__global__ void radii(float* a, float* r) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  a[k] = bd::radius_uniform(k << 8);
  r[k] = bd::box_muller_radius(a[k]);
}

int main() {
  const size_t n = 1u << 24;
  std::vector<float> a(n), r(n);
  float *da, *dr;
  if (cudaMalloc(&da, n * 4) != cudaSuccess || cudaMalloc(&dr, n * 4) != cudaSuccess) return 2;
  radii<<<n / 256, 256>>>(da, dr);
  if (cudaMemcpy(a.data(), da, n * 4, cudaMemcpyDeviceToHost) != cudaSuccess ||
      cudaMemcpy(r.data(), dr, n * 4, cudaMemcpyDeviceToHost) != cudaSuccess)
    return 2;
  double worst_abs = 0.0, worst_rel = 0.0, worst_share = 0.0;
  for (size_t k = 0; k < n; k++) {
    // error of q = -2 ln a: that of the logarithm (2^-22, absolute above 1/2,
    // else relative) times 2 ln 2, and two roundings of q (the constant, the
    // product)
    const double q = -2.0 * std::log((double)a[k]);
    const double eq = (a[k] > 0.5f ? 1.3862943611198906 * std::ldexp(1.0, -22) : q * std::ldexp(1.0, -22)) +
                      q * std::ldexp(1.0, -23);
    // through the root, then the reciprocal root's and the product's errors
    const double exact = std::sqrt(q);
    const double root = std::max(std::sqrt(q + eq) - exact, exact - std::sqrt(std::max(q - eq, 0.0)));
    const double bound = root + std::sqrt(q + eq) * (std::exp2(-22.9) + std::ldexp(1.0, -23)) + 2e-15;
    const double err = std::fabs((double)r[k] - exact);
    if (!(err <= bound)) return printf("a %.9g radius %.9g exact %.9g bound %.3g\n", a[k], r[k], exact, bound), 1;
    worst_abs = std::max(worst_abs, err);
    if (exact > 0.01) worst_rel = std::max(worst_rel, err / exact);
    worst_share = std::max(worst_share, err / bound);
  }
  printf("ok: largest error %.3g, %.3g relative above 0.01, %.2f of the bound\n", worst_abs, worst_rel, worst_share);
  return 0;
}
