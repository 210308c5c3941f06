// Both forms of Distribution1D::SetFunction (csrc/cdf.cuh) on the device, over
// the weights of a binary file (test infrastructure).
// usage: cdf_harness <in.f32> <out.f32> <ndist> <stride> <count, or -1>
// in: ndist x stride weights; count < 0: all of them, else the first `count` of one
// distribution, the length then being read on the device. out: the one-block form's
// cdfs and integrals, the three-launch form's, those of the form that the library
// takes (entries at or behind the length: -1).
#include "../../tensorray_b200/csrc/cdf.cuh"
#include <cstdio>
#include <cstdlib>
#include <vector>
using namespace trn;

int main(int argc, char** argv) {
  if (argc != 6) return 2;
  const int ndist = atoi(argv[3]), n = atoi(argv[4]), count = atoi(argv[5]);
  const size_t total = (size_t)ndist * n;
  std::vector<float> w(total), out;
  FILE* f = fopen(argv[1], "rb");
  if (!f || fread(w.data(), sizeof(float), total, f) != total) return 2;
  fclose(f);
  float *func, *cdf, *integral;
  double* part;
  int* len = nullptr;
  if (cudaMalloc(&func, total * 4) || cudaMalloc(&cdf, total * 4) || cudaMalloc(&integral, ndist * 4) ||
      cudaMalloc(&part, sizeof(double) * kCdfChunks * ndist))
    return 3;
  if (count >= 0 && (cudaMalloc(&len, 4) || cudaMemcpy(len, &count, 4, cudaMemcpyHostToDevice))) return 3;
  cudaMemcpy(func, w.data(), total * 4, cudaMemcpyHostToDevice);
  for (int form = 0; form < 3; form++) {
    std::vector<float> a(total, -1.f), b(ndist, -1.f);
    cudaMemcpy(cdf, a.data(), total * 4, cudaMemcpyHostToDevice);
    if (form == 0) {
      k_cdf_small<<<ndist, kCdfChunks>>>(n, len, func, cdf, integral);
    } else if (form == 1) {
      const dim3 g(kCdfChunks / kCdfPerBlock, ndist);
      k_cdf_chunks<false><<<g, 128>>>(n, len, func, cdf, integral, part);
      k_cdf_chunks<true><<<g, 128>>>(n, len, func, cdf, integral, part);
      k_cdf_divide<<<dim3(256, ndist), 256>>>(n, len, cdf, integral);
    } else {
      cdf_launch(ndist, n, len, func, cdf, integral, part, nullptr);
    }
    if (cudaMemcpy(a.data(), cdf, total * 4, cudaMemcpyDeviceToHost) ||
        cudaMemcpy(b.data(), integral, ndist * 4, cudaMemcpyDeviceToHost))
      return 4;
    out.insert(out.end(), a.begin(), a.end());
    out.insert(out.end(), b.begin(), b.end());
  }
  f = fopen(argv[2], "wb");
  if (!f || fwrite(out.data(), sizeof(float), out.size(), f) != out.size()) return 2;
  fclose(f);
  return 0;
}
