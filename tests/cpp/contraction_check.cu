// ddmath.cuh's quick forms in a translation unit compiled with FMA
// contraction (the default), as k_mixed.cu is: wherever the rounding test
// settles a result, it is the host's double-double series', bit for bit.
// (Where it does not, the device's series runs, whose own last bits may
// gain from contraction.)  argv: count.  Prints the calls, those settled and
// the number of them that differ.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include <cuda_runtime.h>

#include "ddmath.cuh"

using namespace a2c;

__global__ void forms(const double *x, const double *u, int n, double *out, unsigned *settled) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned ok = dd::quick_cr_exp(x[i], out[i]) ? 1u : 0u;
  ok |= (unsigned)dd::quick_cr_exp_both(x[i], out[n + i], out[2 * n + i]) << 1;
  ok |= dd::quick_cr_log(u[i], out[3 * n + i]) ? 8u : 0u;
  ok |= dd::quick_cr_pow(u[i], 2.18860, out[4 * n + i]) ? 16u : 0u;
  settled[i] = ok;
}

int main(int argc, char **argv) {
  if (argc < 2) return 2;
  const int n = std::atoi(argv[1]);
  if (n < 1 || n > (1 << 20)) return 2;
  std::mt19937_64 g(7);
  std::uniform_real_distribution<double> U(0.0, 1.0);
  std::vector<double> x(n), u(n), out(5 * (size_t)n);
  std::vector<unsigned> ok(n);
  for (int i = 0; i < n; ++i) {
    x[i] = i % 2 ? (U(g) - 0.5) * 1300 : (U(g) - 0.5) * std::ldexp(1.0, 4 - (int)(g() % 40));
    u[i] = i % 3 == 0 ? std::exp((U(g) - 0.5) * 200) : i % 3 == 1 ? 60 * U(g) + 0.05 : 1.0 + (U(g) - 0.5) * std::ldexp(1.0, -(int)(g() % 40));
  }
  double *dx = nullptr, *du = nullptr, *dout = nullptr;
  unsigned *dok = nullptr;
  if (cudaMalloc(&dok, sizeof(unsigned) * n) || cudaMalloc(&dx, sizeof(double) * n) || cudaMalloc(&du, sizeof(double) * n) ||
      cudaMalloc(&dout, sizeof(double) * out.size()))
    return 3;
  cudaMemcpy(dx, x.data(), sizeof(double) * n, cudaMemcpyHostToDevice);
  cudaMemcpy(du, u.data(), sizeof(double) * n, cudaMemcpyHostToDevice);
  forms<<<(n + 127) / 128, 128>>>(dx, du, n, dout, dok);
  if (cudaGetLastError() || cudaMemcpy(out.data(), dout, sizeof(double) * out.size(), cudaMemcpyDeviceToHost) ||
      cudaMemcpy(ok.data(), dok, sizeof(unsigned) * n, cudaMemcpyDeviceToHost))
    return 3;
  cudaFree(dok);
  cudaFree(dx);
  cudaFree(du);
  cudaFree(dout);
  long settled = 0, bad = 0;
  for (int i = 0; i < n; ++i) {
    const double up = dd::series_exp(x[i]);
    const double want[5] = {up, up, dd::series_exp(-x[i]), dd::series_log(u[i]), dd::series_pow(u[i], 2.18860)};
    for (int k = 0; k < 5; ++k) {
      if (!(ok[i] >> k & 1u)) continue;
      ++settled;
      bad += out[(size_t)k * n + i] != want[k];
    }
  }
  std::printf("%ld %ld %ld\n", 5L * n, settled, bad);
  return 0;
}
