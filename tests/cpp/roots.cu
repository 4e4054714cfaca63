// Largest errors of the roots and reciprocals of common.cuh over their ranges,
// in ulps against the host's long double: one line "name ulps" each.
#include <cmath>
#include <cstdio>
#include <random>
#include <string>
#include <vector>

#include "common.cuh"

namespace {

template<class T, class Fn>
__global__ void k_apply(const T* x, T* y, int n, Fn fn) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = fn(x[i]);
}

template<class T, class Fn, class Ref>
void report(const char* name, const std::vector<T>& x, Fn fn, Ref ref) {
  const int n = static_cast<int>(x.size());
  T *dx = nullptr, *dy = nullptr;
  std::vector<T> y(x.size());
  if (cudaMalloc(&dx, sizeof(T) * n) != cudaSuccess ||
      cudaMalloc(&dy, sizeof(T) * n) != cudaSuccess ||
      cudaMemcpy(dx, x.data(), sizeof(T) * n, cudaMemcpyHostToDevice) != cudaSuccess) {
    std::exit(1);
  }
  k_apply<<<(n + 255) / 256, 256>>>(dx, dy, n, fn);
  if (cudaMemcpy(y.data(), dy, sizeof(T) * n, cudaMemcpyDeviceToHost) != cudaSuccess) std::exit(1);
  cudaFree(dx);
  cudaFree(dy);
  long double worst = 0.0L;
  for (int i = 0; i < n; ++i) {
    const long double want = ref(x[i]);
    const T near = static_cast<T>(want);
    const T up = std::nextafter(near, static_cast<T>(INFINITY));
    const long double ulp = static_cast<long double>(up) - static_cast<long double>(near);
    const long double e = std::fabs(static_cast<long double>(y[i]) - want) / ulp;
    if (!(e <= worst)) worst = e;  // also a NaN
  }
  std::printf("%s %.4Lf\n", name, worst);
}

// Magnitudes spread over powers of two, and the numbers around each power.
template<class T>
std::vector<T> spread(int lo, int hi, int n) {
  std::mt19937_64 rng(7);
  std::uniform_real_distribution<double> m(1.0, 2.0), e(lo, hi);
  std::vector<T> x;
  for (int i = 0; i < n; ++i) {
    x.push_back(static_cast<T>(std::ldexp(m(rng), static_cast<int>(std::floor(e(rng))))));
  }
  for (int k = lo + 1; k < hi; ++k) {
    const T p = std::ldexp(T(1), k);
    x.insert(x.end(), {p, std::nextafter(p, T(0)), std::nextafter(p, T(INFINITY))});
  }
  return x;
}

}  // namespace

int main() {
  using LD = long double;
  report("rcp_f64", spread<double>(-1020, 1020, 4000000),
         [] __device__(double x) { return tg::rcp_f64(x); }, [](double x) { return 1.0L / x; });
  report("sqrt_f64", spread<double>(-1020, 1020, 4000000),
         [] __device__(double x) { return tg::sqrt_f64(x); },
         [](double x) { return std::sqrt(static_cast<LD>(x)); });
  report("rcp_newton", spread<float>(-120, 120, 4000000),
         [] __device__(float x) { return tg::rcp_newton(x); }, [](float x) { return 1.0L / x; });
  report("sqrt_newton", spread<float>(-120, 120, 4000000),
         [] __device__(float x) { return tg::sqrt_newton(x); },
         [](float x) { return std::sqrt(static_cast<LD>(x)); });
  // rho(H) over the range of u = 1 + 6 H / cs0^2, with cs0^2 = 6 and rho0 = 1
  // (so that u is exact) and the potentials of densities around rho0.
  tg::PhysDev P{};
  P.xi_is_7 = true;
  P.eos = TG_EOS_TAIT;
  P.xi = 7.0;
  tg::TankDev T{};
  T.rho0 = 1.0;
  T.cs0 = 1.0;
  std::vector<double> H;
  for (const double u : spread<double>(-60, 60, 2000000)) H.push_back((u - 1.0) / 6.0);
  std::mt19937_64 rng(8);
  std::uniform_real_distribution<double> d(-0.15, 1.0);
  for (int i = 0; i < 2000000; ++i) H.push_back(d(rng));
  report("wall_density_f64", H,
         [=] __device__(double h) { return tg::wall_density_f64(P, T, h); },
         [](double h) {
           volatile double t = 6.0 * h;  // rounded as on the device
           const double u = 1.0 + t;
           return std::pow(static_cast<LD>(u), 1.0L / 6.0L);
         });
  // Zero, and squares that are no normal numbers: no larger than the root.
  std::vector<double> tiny = {0.0, 4.9e-324, 1e-320, 1e-310, 2.2250738585072009e-308};
  report("sqrt_f64_tiny", tiny, [] __device__(double x) {
    const double r = tg::sqrt_f64(x);
    return r >= 0.0 && r <= 1.0001 * sqrt(x) ? 1.0 : 0.0;
  }, [](double) { return 1.0L; });
  return 0;
}
