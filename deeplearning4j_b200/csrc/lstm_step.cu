// One LSTM time step for inference (rnnTimeStep, one character at a time): input projection, recurrent projection and cell in one
// launch.  A step moves a few MB at most, so it is bound by launch and latency: the general path runs an input GEMM, a transposed-
// weight check, a state copy and the persistent sequence kernel, whose set-up (resident weights, grid barrier) one step cannot repay.
//
// One block per hidden unit, one warp per gate (order a | f | o | g): the gate's column of W and of RW is contiguous in the 'f'-ordered
// parameters, the lanes split it and keep eight batch rows' partial sums, the columns are re-read from L1 for the next eight rows.
// The weights are the fp32 parameters themselves: no shadow to be stale, no rounding.
// Sums, bias and cell are fp32 throughout; only h is rounded.  h_out may not alias h.
// The same dot product serves a dense layer of a few rows whose width the tensor-core kernels cannot address (a 77-symbol alphabet),
// which took two casts of the parameters and a library product.
// Measured: the line to the sequence kernel stands at lstm_step_supported in ops/native.py.
#include "vec8.cuh"

namespace dl4j {

constexpr int LT_ROWS = 8;

// acc[r] += dot(w[0 .. K), x[row0 + r][0 .. K)), this lane's share; rows past mb repeat the last one
template <typename TW>
__device__ __forceinline__ void lt_dot(const TW* __restrict__ w, const __nv_bfloat16* __restrict__ x, long ldx, int K, int row0, int mb,
                                       int lane, bool vec, float (&acc)[LT_ROWS]) {
  if (vec) {
    for (int k = lane * 8; k < K; k += 256) {
      float a[8];
      Vec8<TW>::load(w + k, a);
#pragma unroll
      for (int r = 0; r < LT_ROWS; ++r) {
        float b[8];
        Vec8<__nv_bfloat16>::load(x + min(row0 + r, mb - 1) * ldx + k, b);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[r] = fmaf(a[j], b[j], acc[r]);
      }
    }
  } else {
    for (int k = lane; k < K; k += 32) {
      const float a = ldf(w + k);
#pragma unroll
      for (int r = 0; r < LT_ROWS; ++r) acc[r] = fmaf(a, __bfloat162float(x[min(row0 + r, mb - 1) * ldx + k]), acc[r]);
    }
  }
}

__global__ void __launch_bounds__(128)
lstm_step_kernel(const __nv_bfloat16* __restrict__ x, long ldx, const float* __restrict__ W, const float* __restrict__ RW,
                 const float* __restrict__ bias, const __nv_bfloat16* __restrict__ h, const float* __restrict__ c,
                 __nv_bfloat16* __restrict__ h_out, float* __restrict__ c_out, int mb, int nIn, int n, int vec_x, int vec_h) {
  __shared__ float z[4][LT_ROWS];
  const int u = blockIdx.x, gate = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long col = (long)gate * n + u;
  const float b = bias ? bias[col] : 0.f;
  for (int row0 = 0; row0 < mb; row0 += LT_ROWS) {
    float acc[LT_ROWS];
#pragma unroll
    for (int r = 0; r < LT_ROWS; ++r) acc[r] = 0.f;
    lt_dot(W + col * nIn, x, ldx, nIn, row0, mb, lane, vec_x, acc);
    lt_dot(RW + col * n, h, n, n, row0, mb, lane, vec_h, acc);
#pragma unroll
    for (int r = 0; r < LT_ROWS; ++r) acc[r] = warp_sum(acc[r]);
    if (lane == 0) {
#pragma unroll
      for (int r = 0; r < LT_ROWS; ++r) z[gate][r] = acc[r] + b;
    }
    __syncthreads();
    const int row = row0 + threadIdx.x;
    if (threadIdx.x < LT_ROWS && row < mb) {
      const float a = tanhf(z[0][threadIdx.x]), f = 1.f / (1.f + expf(-z[1][threadIdx.x])), o = 1.f / (1.f + expf(-z[2][threadIdx.x])),
                  g = 1.f / (1.f + expf(-z[3][threadIdx.x]));
      const float cn = fmaf(f, c[(long)row * n + u], g * a);
      c_out[(long)row * n + u] = cn;
      h_out[(long)row * n + u] = __float2bfloat16(o * tanhf(cn));
    }
    __syncthreads();
  }
}

// y[m, o] = sum_k x[m, k] W[k, o] + b[o], one warp per output column
template <typename TW>
__global__ void __launch_bounds__(128)
linear_small_kernel(const __nv_bfloat16* __restrict__ x, long ldx, const TW* __restrict__ W, const float* __restrict__ bias,
                    __nv_bfloat16* __restrict__ y, int M, int K, int N, int vec) {
  const int col = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (col >= N) return;
  const float b = bias ? bias[col] : 0.f;
  for (int row0 = 0; row0 < M; row0 += LT_ROWS) {
    float acc[LT_ROWS];
#pragma unroll
    for (int r = 0; r < LT_ROWS; ++r) acc[r] = 0.f;
    lt_dot(W + (long)col * K, x, ldx, K, row0, M, lane, vec, acc);
#pragma unroll
    for (int r = 0; r < LT_ROWS; ++r) {
      acc[r] = warp_sum(acc[r]);
      if (lane == r && row0 + r < M) y[(long)(row0 + r) * N + col] = __float2bfloat16(acc[r] + b);
    }
  }
}

}  // namespace dl4j

using namespace dl4j;

static bool lt_aligned(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// x [mb, nIn] bf16 (row stride ldx), W [nIn, 4n] and RW [n, 4n] fp32 column-major ('f'), bias fp32 [4n] or null, h [mb, n] bf16, c [mb, n] fp32.
DL4J_API int dl4j_lstm_step(const void* x, long ldx, const float* W, const float* RW, const float* bias, const void* h, const float* c,
                            void* h_out, float* c_out, int mb, int nIn, int n, void* stream) {
  if (mb < 1 || nIn < 1 || n < 1 || h == h_out) return -DL4J_ERR_BAD_ARG;
  const int vec_x = nIn % 8 == 0 && ldx % 8 == 0 && lt_aligned(x) && lt_aligned(W), vec_h = n % 8 == 0 && lt_aligned(h) && lt_aligned(RW);
  using B = __nv_bfloat16;
  lstm_step_kernel<<<n, 128, 0, (cudaStream_t)stream>>>((const B*)x, ldx, W, RW, bias, (const B*)h, c, (B*)h_out, c_out, mb, nIn, n, vec_x,
                                                        vec_h);
  return (int)cudaGetLastError();
}

// x [M, K] bf16 (row stride ldx), W [K, N] column-major fp32 or bf16, bias fp32 [N] or null, y [M, N] bf16 dense.
DL4J_API int dl4j_linear_small(const void* x, long ldx, const void* W, int w_fp32, const float* bias, void* y, int M, int K, int N,
                               void* stream) {
  if (M < 1 || K < 1 || N < 1) return -DL4J_ERR_BAD_ARG;
  const int vec = K % 8 == 0 && ldx % 8 == 0 && lt_aligned(x) && lt_aligned(W);
  using B = __nv_bfloat16;
  if (w_fp32)
    linear_small_kernel<float><<<(N + 3) / 4, 128, 0, (cudaStream_t)stream>>>((const B*)x, ldx, (const float*)W, bias, (B*)y, M, K, N, vec);
  else
    linear_small_kernel<B><<<(N + 3) / 4, 128, 0, (cudaStream_t)stream>>>((const B*)x, ldx, (const B*)W, bias, (B*)y, M, K, N, vec);
  return (int)cudaGetLastError();
}
