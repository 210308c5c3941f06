// Distribution1D::SetFunction (Distribution.cpp:45-58) over n weights: cdf_i =
// (S_i / n) / (S_n / n), with the prefix sums in double in a fixed order: 1024
// chunks, each summed in order, then the chunk sums in order, then the weights
// in order behind their chunk's offset. The order fixes every rounding, so the
// result does not depend on which of the two forms below computes it.
#pragma once
#include "common.cuh"

namespace trn {

constexpr int kCdfChunks = 1024;
constexpr int kCdfPerBlock = 8;    // chunks per block of the three-launch form
constexpr int kCdfTile = 256;      // weights of a chunk staged at a time

struct CdfRange {
  int n, chunk, used;              // weights, weights per chunk, chunks with any
  TRN_D explicit CdfRange(int n_) : n(n_) {
    chunk = max(1, (n + kCdfChunks - 1) / kCdfChunks);
    used = (n + chunk - 1) / chunk;
  }
  TRN_D int begin(int c) const { return min(n, c * chunk); }
};

// sum of part[0, count) in order (the adds are a chain, the loads are not)
TRN_D double cdf_chain(const double* part, int count) {
  double run = 0.0;
  int i = 0;
  for (; i + 8 <= count; i += 8) {
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = part[i + k];
#pragma unroll
    for (int k = 0; k < 8; k++) run += v[k];
  }
  for (; i < count; i++) run += part[i];
  return run;
}

// One block of kCdfChunks threads per distribution: few weights.
static __global__ void __launch_bounds__(kCdfChunks) k_cdf_small(int n_, const int* count, const float* func_all, float* cdf_all,
                                                          float* integral_all) {
  __shared__ double part[kCdfChunks];
  __shared__ float integral;
  const CdfRange r(count ? __ldg(count) : n_);
  const float* func = func_all + (long long)blockIdx.x * n_;
  float* cdf = cdf_all + (long long)blockIdx.x * n_;
  const int tid = threadIdx.x, a = r.begin(tid), b = r.begin(tid + 1);
  double s = 0.0;
  for (int i = a; i < b; i++) s += (double)func[i];
  part[tid] = s;
  __syncthreads();
  if (tid == 0) {
    double run = 0.0;
    int c = 0;
    for (; c + 8 <= r.used; c += 8) {
      double v[8];
#pragma unroll
      for (int k = 0; k < 8; k++) v[k] = part[c + k];
#pragma unroll
      for (int k = 0; k < 8; k++) { part[c + k] = run; run += v[k]; }
    }
    for (; c < r.used; c++) { const double x = part[c]; part[c] = run; run += x; }
  }
  __syncthreads();
  const float inv_size = 1.0f / (float)r.n;
  double run = part[tid];
  for (int i = a; i < b; i++) { run += (double)func[i]; cdf[i] = (float)run * inv_size; }
  __syncthreads();
  if (tid == 0) {
    integral = r.n > 0 ? cdf[r.n - 1] : 0.f;
    integral_all[blockIdx.x] = integral;
  }
  __syncthreads();
  if (integral > 0.f) for (int i = a; i < b; i++) cdf[i] = cdf[i] / integral;
}

// Many weights, in three launches over kCdfChunks / kCdfPerBlock blocks (times
// the distributions): chunk sums; cdf behind the chunk offsets; division by
// the integral. Tiles of the block's chunks pass through shared memory so that
// every access to the arrays is coalesced; one thread per chunk runs its chain
// of double additions, which bounds the first two launches. 150K edge lengths:
// one block alone took 0.12 ms; Scene::Configure of 100K triangles went from
// 0.69 to 0.46 ms with its edge distribution in this form.
template <bool WRITE>
static __global__ void __launch_bounds__(128) k_cdf_chunks(int n_, const int* count, const float* func_all, float* cdf_all,
                                                    float* integral_all, double* part_all) {
  __shared__ float tile[kCdfPerBlock][kCdfTile + 1];
  __shared__ double offset[kCdfPerBlock];
  const CdfRange r(count ? __ldg(count) : n_);
  const float* func = func_all + (long long)blockIdx.y * n_;
  float* cdf = cdf_all + (long long)blockIdx.y * n_;
  double* part = part_all + (long long)blockIdx.y * kCdfChunks;
  const int c0 = blockIdx.x * kCdfPerBlock, tid = threadIdx.x;
  if (c0 >= r.used) return;
  double run = 0.0;
  if (WRITE) {
    if (tid == 0) {
      double s = cdf_chain(part, c0);
      for (int c = 0; c < kCdfPerBlock; c++) { offset[c] = s; s += part[c0 + c]; }
    }
    __syncthreads();
    if (tid < kCdfPerBlock) run = offset[tid];
  }
  const float inv_size = 1.0f / (float)r.n;
  for (int t0 = 0; t0 < r.chunk; t0 += kCdfTile) {
    const int len = min(kCdfTile, r.chunk - t0);
    for (int k = tid; k < kCdfPerBlock * kCdfTile; k += blockDim.x) {
      const int c = k / kCdfTile, e = k % kCdfTile, i = (c0 + c) * r.chunk + t0 + e;
      if (e < len && c0 + c < r.used && i < r.n) tile[c][e] = func[i];
    }
    __syncthreads();
    if (tid < kCdfPerBlock && c0 + tid < r.used) {
      const int end = min(len, r.begin(c0 + tid + 1) - ((c0 + tid) * r.chunk + t0));
      for (int e = 0; e < end; e++) {
        run += (double)tile[tid][e];
        if (WRITE) tile[tid][e] = (float)run * inv_size;
      }
    }
    __syncthreads();
    if (WRITE) {
      for (int k = tid; k < kCdfPerBlock * kCdfTile; k += blockDim.x) {
        const int c = k / kCdfTile, e = k % kCdfTile, i = (c0 + c) * r.chunk + t0 + e;
        if (e < len && c0 + c < r.used && i < r.n) {
          cdf[i] = tile[c][e];
          if (i == r.n - 1) integral_all[blockIdx.y] = tile[c][e];
        }
      }
      __syncthreads();
    }
  }
  if (!WRITE && tid < kCdfPerBlock) part[c0 + tid] = run;
}

static __global__ void k_cdf_divide(int n_, const int* count, float* cdf_all, const float* integral_all) {
  const int n = count ? __ldg(count) : n_;
  const float integral = integral_all[blockIdx.y];
  float* cdf = cdf_all + (long long)blockIdx.y * n_;
  if (!(integral > 0.f)) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) cdf[i] = cdf[i] / integral;
}

// Below this many weights one block per distribution is as fast (its chain of
// 1024 chunk sums is about 5 us either way, and it is one launch).
constexpr int kCdfSmall = 16384;

// Distributions of n weights each at func + v n. With `count`, one
// distribution whose length is on the device (at most n). part: kCdfChunks
// doubles per distribution. Returns the number of launches.
inline int cdf_launch(int ndist, int n, const int* count, const float* func, float* cdf, float* integral, double* part,
                      cudaStream_t st) {
  if (n <= kCdfSmall) {
    k_cdf_small<<<ndist, kCdfChunks, 0, st>>>(n, count, func, cdf, integral);
    return 1;
  }
  const dim3 g(kCdfChunks / kCdfPerBlock, ndist);
  k_cdf_chunks<false><<<g, 128, 0, st>>>(n, count, func, cdf, integral, part);
  k_cdf_chunks<true><<<g, 128, 0, st>>>(n, count, func, cdf, integral, part);
  k_cdf_divide<<<dim3(256, ndist), 256, 0, st>>>(n, count, cdf, integral);
  return 3;
}

}  // namespace trn
