// The branch-free scaling of the digit-sliced passes (oz::scaled_plain_fp64)
// against the general one (oz::scaled), on the device, bit for bit, wherever
// oz::plain_pow2 admits it; and oz::scaled on the host against the exact
// value rounded once (a conversion and std::scalbn, exact in that range).
//
// Prints "N values, M differ on the device, K on the host".
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "ev_ozaki.cuh"

using namespace ev;

__global__ void k_compare(const int64_t* acc, const int* pow2, int count, unsigned* differ) {
  const int i = int(blockIdx.x * blockDim.x + threadIdx.x);
  if (i >= count) return;
  const double a = oz::scaled(acc[i], pow2[i]);
  const double b = oz::scaled_plain_fp64(acc[i], uint32_t(pow2[i]) << 20);
  if (__double_as_longlong(a) != __double_as_longlong(b)) atomicAdd(differ, 1u);
}

int main(int argc, char** argv) {
  const bool device = argc > 1 && std::strcmp(argv[1], "device") == 0;
  std::mt19937_64 rng(9);
  std::vector<int64_t> acc;
  std::vector<int> pow2;
  const int lo = -1022, hi = 961;  // the ends of plain_pow2
  if (!oz::plain_pow2(lo, hi) || oz::plain_pow2(lo - 1, hi) || oz::plain_pow2(lo, hi + 1)) {
    std::printf("range\n");
    return 1;
  }
  auto add = [&](int64_t a) {
    const int ends[6] = {lo, lo + 1, hi, hi - 1, 0, lo + int(rng() % uint64_t(hi - lo + 1))};
    for (int p : ends)
      for (int64_t s : {a, -a}) {
        acc.push_back(s);
        pow2.push_back(p);
      }
  };
  add(0);
  for (int b = 0; b < 62; ++b) {
    const int64_t one = int64_t(1) << b;
    for (int64_t a : {one, one - 1, one + 1, one | (one >> 53), one | (one >> 54), (one - 1) ^ 1}) add(a);
    for (int r = 0; r < 400; ++r) {
      const int64_t a = one | int64_t(rng() & uint64_t(one - 1));
      add(a);
      if (b > 54) {  // ties between two doubles, to even and to odd
        const int64_t half = int64_t(1) << (b - 53);
        add((a & ~(2 * half - 1)) | half);
      }
    }
  }
  add((int64_t(1) << 62) - 1);
  const int n = int(acc.size());
  unsigned differ = 0, host = 0;
  for (int i = 0; i < n; ++i) {
    const double a = oz::scaled(acc[i], pow2[i]), b = std::scalbn(double(acc[i]), pow2[i]);
    host += std::memcmp(&a, &b, 8) != 0 && !(a == 0.0 && b == 0.0);
  }
  if (device) {
    int64_t* da = nullptr;
    int* dp = nullptr;
    unsigned* dd = nullptr;
    cudaMalloc(reinterpret_cast<void**>(&da), n * 8);
    cudaMalloc(reinterpret_cast<void**>(&dp), n * 4);
    cudaMalloc(reinterpret_cast<void**>(&dd), 4);
    cudaMemcpy(da, acc.data(), n * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(dp, pow2.data(), n * 4, cudaMemcpyHostToDevice);
    cudaMemset(dd, 0, 4);
    k_compare<<<(n + 255) / 256, 256>>>(da, dp, n, dd);
    if (cudaMemcpy(&differ, dd, 4, cudaMemcpyDeviceToHost) != cudaSuccess) {
      std::printf("device error\n");
      return 1;
    }
  }
  std::printf("%d values, %u differ on the device, %u on the host\n", n, differ, host);
  return differ != 0 || host != 0;
}
