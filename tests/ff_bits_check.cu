// Test program for the conversions of velo2cycles_gb300/csrc/v2c_ff.cuh that
// avoid FP64 arithmetic (built and run by tests/test_gpu_newton_phases.py).
//   ff_bits_check <in.bin> <out.bin>
// in.bin: int64 n, then n doubles x.  out.bin: n (hi, lo) float pairs of x by
// bit pattern, then n doubles widened from (float)x by bit pattern.
#include <cstdio>
#include <vector>

#include "../velo2cycles_gb300/csrc/v2c_ff.cuh"

using namespace v2c;

__global__ void k_check(const double *x, long n, float2 *pair, double *wide) {
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const ff a = ff_from_double_bits(x[i]);
  pair[i] = make_float2(a.hi, a.lo);
  wide[i] = widen<true>((float)x[i]);
}

int main(int argc, char **argv) {
  if (argc != 3) return 2;
  FILE *f = fopen(argv[1], "rb");
  if (!f) return 3;
  long long n = 0;
  if (fread(&n, 8, 1, f) != 1 || n <= 0 || n > (1 << 24)) return 4;
  std::vector<double> h(n);
  if (fread(h.data(), 8, n, f) != (size_t)n) return 5;
  fclose(f);
  double *d, *w;
  float2 *o;
  if (cudaMalloc(&d, 8 * n) != cudaSuccess || cudaMalloc(&w, 8 * n) != cudaSuccess ||
      cudaMalloc(&o, 8 * n) != cudaSuccess)
    return 6;
  cudaMemcpy(d, h.data(), 8 * n, cudaMemcpyHostToDevice);
  k_check<<<(unsigned)((n + 255) / 256), 256>>>(d, n, o, w);
  std::vector<float2> ho(n);
  if (cudaMemcpy(ho.data(), o, 8 * n, cudaMemcpyDeviceToHost) != cudaSuccess) return 7;
  if (cudaMemcpy(h.data(), w, 8 * n, cudaMemcpyDeviceToHost) != cudaSuccess) return 7;
  FILE *g = fopen(argv[2], "wb");
  if (!g) return 8;
  fwrite(ho.data(), 8, n, g);
  fwrite(h.data(), 8, n, g);
  return fclose(g) ? 9 : 0;
}
