// Global average pooling over a channels-last activation [N, S, C] (S = H * W), 16-bit types, fp32 sums.
// Memory-bound: the forward reads the activation once, the backward writes it once (64 x 3136 x 256 bf16, 103 MB: 16 us each at the copy
// rate).  The library's mean took 29 us, its backward wrote the broadcast in NCHW order (80 us) and the layers in front of it copied
// that to channels-last (114 us).
#include "vec8.cuh"

namespace dl4j {

// One block per image and 64 channels: 8 channel vectors x 32 rows of 128 bytes, four rows in flight per thread.
template <typename T>
__global__ void __launch_bounds__(256)
avgpool_fwd_kernel(const T* __restrict__ x, T* __restrict__ y, int S, int C, float inv) {
  __shared__ float red[32][65];
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
  const int c = blockIdx.x * 64 + tx * 8;
  const T* base = x + (long long)blockIdx.y * S * C + c;
  float a[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) a[j] = 0.f;
  if (c < C) {
    for (int r = ty; r < S; r += 128) {
      Raw8<T> q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (r + 32 * u < S) q[u] = ld_raw8_keep(base + (long long)(r + 32 * u) * C);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (r + 32 * u < S) {
          float v[8];
          unpack8(q[u], v);
#pragma unroll
          for (int j = 0; j < 8; ++j) a[j] += v[j];
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) red[ty][tx * 8 + j] = a[j];
  __syncthreads();
  if (threadIdx.x < 64 && blockIdx.x * 64 + threadIdx.x < C) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 32; ++w) t += red[w][threadIdx.x];
    stf(y + (long long)blockIdx.y * C + blockIdx.x * 64 + threadIdx.x, t * inv);
  }
}

// dx[n, s, c] = dy[n, c] / S
template <typename T>
__global__ void __launch_bounds__(256)
avgpool_bwd_kernel(const T* __restrict__ dy, T* __restrict__ dx, int S, int cv, long long n_vec, float inv) {
  for (long long g = blockIdx.x * 256LL + threadIdx.x; g < n_vec; g += (long long)gridDim.x * 256) {
    int c, px;
    const long long image = div_mod(div_mod(g, cv, c), S, px);
    float v[8];
    Vec8<T>::load(dy + image * (cv * 8LL) + c * 8, v);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] *= inv;
    Vec8<T>::store(dx + g * 8, v);
  }
}

}  // namespace dl4j

using namespace dl4j;

// x / dx [N, S, C] dense, y / dy [N, C] dense, 16-byte aligned, C a multiple of 8; dtype 0 fp16, 1 bf16.
DL4J_API int dl4j_global_avgpool(int backward, const void* in, void* out, int N, int S, int C, int dtype, void* stream) {
  if (N < 1 || S < 1 || C < 8 || C % 8 || N > 65535 || (dtype != 0 && dtype != 1)) return -DL4J_ERR_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const float inv = 1.f / S;
  if (!backward) {
    const dim3 grid((C + 63) / 64, N);
    if (dtype == 1) avgpool_fwd_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>((const __nv_bfloat16*)in, (__nv_bfloat16*)out, S, C, inv);
    else avgpool_fwd_kernel<__half><<<grid, 256, 0, st>>>((const __half*)in, (__half*)out, S, C, inv);
  } else {
    const long long n_vec = (long long)N * S * (C / 8);
    const long long blocks = (n_vec + 255) / 256;
    const int grid = (int)(blocks < 148 * 16 ? blocks : 148 * 16);
    if (dtype == 1) avgpool_bwd_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>((const __nv_bfloat16*)in, (__nv_bfloat16*)out, S, C / 8, n_vec, inv);
    else avgpool_bwd_kernel<__half><<<grid, 256, 0, st>>>((const __half*)in, (__half*)out, S, C / 8, n_vec, inv);
  }
  return (int)cudaGetLastError();
}
