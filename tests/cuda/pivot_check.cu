// The factorizations' pivot reciprocals (sapb_ldlt.cuh) against the IEEE
// quotient 1 / d on the GPU, in FP64 and FP32: over positive and negative d of
// the whole range, the largest error in ulps of the results that
// positive_normal takes; and the d that must not be taken -- not positive,
// subnormal, infinite, NaN, or with a quotient below the normal range.
// Prints per type "<type> max_ulps <u> taken <t> wrong <w>".
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../sap_warp_b200/csrc/sapb_ldlt.cuh"

template <typename T>
__global__ void k(const T* in, T* fast, T* ref, int* taken, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    fast[i] = sapb::pivot<false>(in[i]);
    ref[i] = sapb::pivot<true>(in[i]);
    taken[i] = sapb::positive_normal(fast[i]) ? 1 : 0;
  }
}

template <typename T, typename I>
static int run(const char* name, int lo, int hi, const std::vector<T>& special) {
  std::vector<T> h(special);
  srand(4321);
  for (int i = 0; i < 1 << 20; ++i) {
    const int e = lo + (int)((double)rand() / RAND_MAX * (hi - lo));
    const double m = 1.0 + (double)rand() / RAND_MAX + (double)rand() / RAND_MAX / 1073741824.0;
    h.push_back((T)std::ldexp((T)m, e) * ((rand() & 15) ? T(1) : T(-1)));
  }
  const int n = (int)h.size();
  T *di, *df, *dr;
  int* dt;
  cudaMalloc(&di, n * sizeof(T));
  cudaMalloc(&df, n * sizeof(T));
  cudaMalloc(&dr, n * sizeof(T));
  cudaMalloc(&dt, n * sizeof(int));
  cudaMemcpy(di, h.data(), n * sizeof(T), cudaMemcpyHostToDevice);
  k<T><<<(n + 255) / 256, 256>>>(di, df, dr, dt, n);
  const cudaError_t err = cudaDeviceSynchronize();
  if (err != cudaSuccess) {
    printf("cuda error %s\n", cudaGetErrorString(err));
    return 2;
  }
  std::vector<T> f(n), r(n);
  std::vector<int> t(n);
  cudaMemcpy(f.data(), df, n * sizeof(T), cudaMemcpyDeviceToHost);
  cudaMemcpy(r.data(), dr, n * sizeof(T), cudaMemcpyDeviceToHost);
  cudaMemcpy(t.data(), dt, n * sizeof(int), cudaMemcpyDeviceToHost);
  long long worst = 0, taken = 0, wrong = 0;
  for (int i = 0; i < n; ++i) {
    const bool normal = h[i] > T(0) && std::isnormal(h[i]) && std::isnormal(r[i]);
    if (t[i]) {
      ++taken;
      I a, b;
      memcpy(&a, &f[i], sizeof a);
      memcpy(&b, &r[i], sizeof b);
      const long long u = a > b ? a - b : b - a;
      if (u > worst) worst = u;
      if (!normal) ++wrong;
    } else if (normal && std::fabs(std::ilogb(h[i])) < hi - 4) {
      ++wrong;  // well inside the range, and not taken
    }
  }
  printf("%s max_ulps %lld taken %lld wrong %lld\n", name, worst, taken, wrong);
  return 0;
}

int main() {
  const double inf = INFINITY, nan = NAN;
  if (run<double, int64_t>("fp64", -1074, 1023,
                           {0.0, -0.0, -1.0, -1e-310, 4.9e-324, 1e-310, 2.2e-308, 8e307, DBL_MAX, -DBL_MAX, inf, -inf,
                            nan}))
    return 2;
  return run<float, int32_t>("fp32", -149, 127,
                             {0.0f, -0.0f, -1.0f, -1e-40f, 1.4e-45f, 1e-40f, 1.1e-38f, 1e38f, FLT_MAX, -FLT_MAX,
                              (float)inf, (float)-inf, (float)nan});
}
