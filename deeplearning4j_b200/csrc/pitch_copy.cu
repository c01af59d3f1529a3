// dst[r, c] = convert(src[r, c]) between row-major matrices of different row pitch: widths off the 8-element grid (a 30522-word
// vocabulary) are laid out once with rows on 16-byte boundaries for the tensor-core kernels, and their gradients packed again.
// Memory-bound.  One of the two sides has unaligned rows, so its accesses are scalar and coalesced (64 bytes per warp and
// instruction, eight per thread in flight); an aligned destination is written in 16-byte pieces.
// 768 x 30522 bf16 to a pitch of 30528 (94 MB moved): 17 - 19 us; the library's strided copy of the transposed gradient took 112 us.
#include "vec8.cuh"

namespace dl4j {

template <typename S, typename D, bool VEC_DST>
__global__ void __launch_bounds__(256)
pitch_copy_kernel(const S* __restrict__ src, D* __restrict__ dst, long rows, int cols, long ld_src, long ld_dst) {
  for (long r = blockIdx.y; r < rows; r += gridDim.y) {
    const S* s = src + r * ld_src;
    D* d = dst + r * ld_dst;
    const int c0 = blockIdx.x * 2048;
    if (VEC_DST) {
      const int c = c0 + threadIdx.x * 8;
      if (c >= cols) continue;
      float v[8];
      const int m = min(8, cols - c);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = j < m ? ldf(s + c + j) : 0.f;
      if (m == 8) Vec8<D>::store(d + c, v);
      else
        for (int j = 0; j < m; ++j) stf(d + c + j, v[j]);
    } else {
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) { const int c = c0 + j * 256 + threadIdx.x; v[j] = c < cols ? ldf(s + c) : 0.f; }
#pragma unroll
      for (int j = 0; j < 8; ++j) { const int c = c0 + j * 256 + threadIdx.x; if (c < cols) stf(d + c, v[j]); }
    }
  }
}

template <typename S, typename D>
static int pitch_run(const void* src, void* dst, long rows, int cols, long ld_src, long ld_dst, cudaStream_t st) {
  const dim3 grid((cols + 2047) / 2048, (unsigned)(rows < 65535 ? rows : 65535));
  const bool vec = (reinterpret_cast<uintptr_t>(dst) & 15) == 0 && (ld_dst * sizeof(D)) % 16 == 0;
  if (vec) pitch_copy_kernel<S, D, true><<<grid, 256, 0, st>>>((const S*)src, (D*)dst, rows, cols, ld_src, ld_dst);
  else pitch_copy_kernel<S, D, false><<<grid, 256, 0, st>>>((const S*)src, (D*)dst, rows, cols, ld_src, ld_dst);
  return (int)cudaGetLastError();
}

}  // namespace dl4j

using namespace dl4j;

// dtypes: 0 fp16, 1 bf16, 2 fp32
DL4J_API int dl4j_pitch_copy(const void* src, int src_dtype, void* dst, int dst_dtype, long rows, int cols, long ld_src, long ld_dst,
                             void* stream) {
  if (rows < 1 || cols < 1) return 0;
  cudaStream_t st = (cudaStream_t)stream;
  using B = __nv_bfloat16;
  switch (src_dtype * 3 + dst_dtype) {
    case 0: return pitch_run<__half, __half>(src, dst, rows, cols, ld_src, ld_dst, st);
    case 4: return pitch_run<B, B>(src, dst, rows, cols, ld_src, ld_dst, st);
    case 6: return pitch_run<float, __half>(src, dst, rows, cols, ld_src, ld_dst, st);
    case 7: return pitch_run<float, B>(src, dst, rows, cols, ld_src, ld_dst, st);
    case 8: return pitch_run<float, float>(src, dst, rows, cols, ld_src, ld_dst, st);
    default: return -DL4J_ERR_BAD_ARG;
  }
}
