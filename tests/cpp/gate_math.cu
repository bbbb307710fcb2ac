// The activations of csrc/gate_math.cuh beside CUDA's own functions.  Arguments: input and output file of fp32 numbers.
// Output: for e^-v, sigmoid, gelu and sqrt(1 - e^(-2 v)) in turn, the header's results and then CUDA's; exit code 1 on a CUDA error.
#include <cstdio>
#include <vector>

#include "common.cuh"
#include "gate_math.cuh"

using namespace kge;

__global__ void gates(const float* in, float* out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float v = in[i], other = in[n - 1 - i];
  auto put = [&](int row, float x) { out[(int64_t)row * n + i] = x; };
  auto first = [](f2 p) { float a, b; upk(p, a, b); return a; };
  const f2 p = pk(v, other), neg = pk(-v, -other);      // the pair's other number must not matter
  put(0, first(exp2_(neg)));
  put(1, expf(-v));
  put(2, first(sigmoid2(p)));
  put(3, 1.f / (1.f + expf(-v)));
  put(4, first(gelu_tanh2(p)));
  put(5, 0.5f * v * (1.f + tanhf(0.79788456080286536f * (v + 0.044715f * v * v * v))));
  put(6, first(complement_root2(neg)));
  put(7, sqrtf(-expm1f(-2.f * v)));
}

int main(int argc, char** argv) {
  if (argc < 3) return 2;
  std::vector<float> h;
  FILE* f = fopen(argv[1], "rb");
  float x;
  while (f && fread(&x, 4, 1, f) == 1) h.push_back(x);
  if (f) fclose(f);
  const int n = (int)h.size();
  float *in = nullptr, *out = nullptr;
  std::vector<float> r((size_t)8 * n);
  if (n == 0 || cudaMalloc(&in, (size_t)n * 4) || cudaMalloc(&out, r.size() * 4) || cudaMemcpy(in, h.data(), (size_t)n * 4, cudaMemcpyHostToDevice)) return 1;
  gates<<<(n + 255) / 256, 256>>>(in, out, n);
  if (cudaGetLastError() || cudaMemcpy(r.data(), out, r.size() * 4, cudaMemcpyDeviceToHost)) return 1;
  f = fopen(argv[2], "wb");
  const bool ok = f && fwrite(r.data(), 4, r.size(), f) == r.size();
  return (f && fclose(f) == 0 && ok) ? 0 : 1;
}
