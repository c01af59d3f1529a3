// Batch normalisation folded into the convolutions in front of it, for inference: with s = gamma / sqrt(var + eps) per output channel
//     w'[o][tap][i] = w[o][i][tap] * s[o]  (bf16, channels-last)      b'[o] = (b[o] - mean[o]) * s[o] + beta[o]  (fp32)
// for every convolution of a network in one launch: one block per output channel, a device table says which convolution it is in.
// Memory-bound: reads the fp32 weights once, writes them once in bf16 (ResNet-50: 94 + 47 MB, 22 us at the copy rate).  It replaces
// one relayout launch per k x k convolution, seven element-wise launches per batch norm and the pass that applied the result to the
// activations (ResNet-50 at 32 images: 636 launches, 10.3 ms of mostly launch time per call).
#include "common.cuh"

namespace dl4j {

struct BnFoldEntry {                 // element offsets into the flat parameter buffer; -1: absent
  long long w, bias, gamma, beta, mean, stat;
  long long w_out, b_out;            // element offsets into the two outputs
  int O, I, S;                       // S = kH * kW
  int log_std;                       // stat holds log10(standard deviation) instead of the variance
  float eps, gamma_const, beta_const;
  int first_block;
};

__global__ void __launch_bounds__(128)
bn_fold_kernel(const BnFoldEntry* __restrict__ table, const int* __restrict__ block_entry, const float* __restrict__ params,
               __nv_bfloat16* __restrict__ w_out, float* __restrict__ b_out) {
  const BnFoldEntry e = table[block_entry[blockIdx.x]];
  const int o = blockIdx.x - e.first_block;
  const float st = params[e.stat + o];
  const float var = e.log_std ? exp10f(2.f * st) : st;
  const float s = (e.gamma >= 0 ? params[e.gamma + o] : e.gamma_const) * rsqrtf(var + e.eps);
  if (threadIdx.x == 0)
    b_out[e.b_out + o] = ((e.bias >= 0 ? params[e.bias + o] : 0.f) - params[e.mean + o]) * s + (e.beta >= 0 ? params[e.beta + o] : e.beta_const);
  const int n = e.I * e.S;
  const float* w = params + e.w + (long long)o * n;
  __nv_bfloat16* out = w_out + e.w_out + (long long)o * n;
  if (e.S == 1 && (n & 3) == 0 && ((reinterpret_cast<uintptr_t>(w) & 15) | (reinterpret_cast<uintptr_t>(out) & 7)) == 0) {
    for (int i = threadIdx.x * 4; i < n; i += 512) {
      const float4 v = __ldcs(reinterpret_cast<const float4*>(w + i));
      const __nv_bfloat162 a = __floats2bfloat162_rn(v.x * s, v.y * s), b = __floats2bfloat162_rn(v.z * s, v.w * s);
      *reinterpret_cast<uint2*>(out + i) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    }
  } else {                           // the row (a few KB) is read with a stride of S elements: L1 serves the other taps
    for (int g = threadIdx.x; g < n; g += 128) out[g] = __float2bfloat16(w[(g % e.I) * e.S + g / e.I] * s);
  }
}

}  // namespace dl4j

using namespace dl4j;

DL4J_API int dl4j_bn_fold(const void* table, const int* block_entry, int blocks, const float* params, void* w_out, float* b_out, void* stream) {
  if (blocks < 1 || !table || !block_entry || !params || !w_out || !b_out) return -DL4J_ERR_BAD_ARG;
  bn_fold_kernel<<<blocks, 128, 0, (cudaStream_t)stream>>>(reinterpret_cast<const BnFoldEntry*>(table), block_entry, params,
                                                          reinterpret_cast<__nv_bfloat16*>(w_out), b_out);
  return (int)cudaGetLastError();
}
