// Sums of runs of floats and of their squares by vg::TripleSum (csrc/vg_internal.cuh), a thread a run:
// sums <in.bin> <out.bin>; in: int32 runs, int32 n, float values[runs][n]; out: double sum, sum of squares,
// whether the squares are in range [runs][3].
#include <cstdio>
#include <vector>

#include "vg_internal.cuh"

__global__ void k_sums(const float* v, int runs, int n, double* out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= runs) return;
  vg::TripleSum s, q;
  for (int i = 0; i < n; ++i) {
    s.add(v[(size_t)t * n + i]);
    q.add_square(v[(size_t)t * n + i]);
  }
  out[3 * t] = s.value();
  out[3 * t + 1] = q.value();
  out[3 * t + 2] = q.in_range();
}

int main(int argc, char** argv) {
  int head[2];
  FILE* f = argc == 3 ? fopen(argv[1], "rb") : nullptr;
  if (!f || fread(head, 4, 2, f) != 2) return 1;
  std::vector<float> v((size_t)head[0] * head[1]);
  if (fread(v.data(), 4, v.size(), f) != v.size()) return 1;
  fclose(f);
  float* dv = nullptr;
  double* dout = nullptr;
  std::vector<double> out(3 * (size_t)head[0]);
  if (cudaMalloc(&dv, v.size() * 4) || cudaMalloc(&dout, out.size() * 8)) return 2;
  if (cudaMemcpy(dv, v.data(), v.size() * 4, cudaMemcpyHostToDevice)) return 2;
  k_sums<<<(head[0] + 127) / 128, 128>>>(dv, head[0], head[1], dout);
  if (cudaMemcpy(out.data(), dout, out.size() * 8, cudaMemcpyDeviceToHost)) return 2;
  f = fopen(argv[2], "wb");
  if (!f || fwrite(out.data(), 8, out.size(), f) != out.size() || fclose(f)) return 1;
  return 0;
}
