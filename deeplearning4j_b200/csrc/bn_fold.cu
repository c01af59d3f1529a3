// Batch normalisation folded into the convolutions in front of it, for inference: with s = gamma / sqrt(var + eps) per output channel
//     w'[o][tap][i] = w[o][i][tap] * s[o]  (bf16, channels-last)      b'[o] = (b[o] - mean[o]) * s[o] + beta[o]  (fp32)
// for every convolution of a network in one launch; a device table says which convolution an output channel is in.
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

// One warp per output channel: its chain (table -> statistics and weights -> stores) is three memory latencies long whatever the channel's
// size, so 48 channels are in flight per SM and a lane issues its weight loads before it needs the scale.  k x k kernels go through
// shared memory, read in order and written tap by tap.  ResNet-50 (26560 channels): 44.6 -> 33.4 us; one block per channel had 16 in
// flight, and its strided reads of the k x k rows took ten L1 lines per warp instruction.
constexpr int BF_WARPS = 8;
constexpr int BF_STAGE = 1152;       // floats per warp: 128 input channels of a 3 x 3 kernel

__global__ void __launch_bounds__(32 * BF_WARPS)
bn_fold_kernel(const BnFoldEntry* __restrict__ table, const int* __restrict__ block_entry, int channels, const float* __restrict__ params,
               __nv_bfloat16* __restrict__ w_out, float* __restrict__ b_out) {
  __shared__ float stage[BF_WARPS][BF_STAGE];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ch = blockIdx.x * BF_WARPS + warp;
  if (ch >= channels) return;
  const BnFoldEntry e = table[block_entry[ch]];
  const int o = ch - e.first_block;
  const int n = e.I * e.S;
  const float* w = params + e.w + (long long)o * n;
  __nv_bfloat16* out = w_out + e.w_out + (long long)o * n;
  const float st = params[e.stat + o], gamma = e.gamma >= 0 ? params[e.gamma + o] : e.gamma_const;
  const float bias = e.bias >= 0 ? params[e.bias + o] : 0.f, mean = params[e.mean + o], beta = e.beta >= 0 ? params[e.beta + o] : e.beta_const;
  auto scale = [&] { return gamma * rsqrtf((e.log_std ? exp10f(2.f * st) : st) + e.eps); };
  if (e.S == 1 && (n & 3) == 0 && ((reinterpret_cast<uintptr_t>(w) & 15) | (reinterpret_cast<uintptr_t>(out) & 7)) == 0) {
    for (int i = lane * 4; i < n; i += 512) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i + 128 * u < n) v[u] = __ldcs(reinterpret_cast<const float4*>(w + i + 128 * u));
      const float s = scale();
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i + 128 * u < n) {
          const __nv_bfloat162 a = __floats2bfloat162_rn(v[u].x * s, v[u].y * s), b = __floats2bfloat162_rn(v[u].z * s, v[u].w * s);
          *reinterpret_cast<uint2*>(out + i + 128 * u) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
        }
    }
  } else if (e.S <= BF_STAGE) {
    const int step = BF_STAGE / e.S;                   // input channels per round
    for (int i0 = 0; i0 < e.I; i0 += step) {
      const int cc = min(step, e.I - i0), m = cc * e.S;
      const float* src = w + (long long)i0 * e.S;
#pragma unroll 12
      for (int g = lane; g < m; g += 32) stage[warp][g] = __ldcs(src + g);
      __syncwarp();
      const float s = scale();
      const bool pair = ((e.I | i0 | cc) & 1) == 0 && (reinterpret_cast<uintptr_t>(out) & 3) == 0;
      for (int t = 0; t < e.S; ++t) {
        __nv_bfloat16* dst = out + (long long)t * e.I + i0;
        if (pair) {
          for (int i = lane * 2; i < cc; i += 64) {
            const __nv_bfloat162 a = __floats2bfloat162_rn(stage[warp][i * e.S + t] * s, stage[warp][(i + 1) * e.S + t] * s);
            *reinterpret_cast<__nv_bfloat162*>(dst + i) = a;
          }
        } else {
          for (int i = lane; i < cc; i += 32) dst[i] = __float2bfloat16(stage[warp][i * e.S + t] * s);
        }
      }
      __syncwarp();
    }
  } else {                           // kernels of more than BF_STAGE taps: element by element
    const float s = scale();
    for (int g = lane; g < n; g += 32) out[g] = __float2bfloat16(w[(g % e.I) * e.S + g / e.I] * s);
  }
  if (lane == 0) b_out[e.b_out + o] = (bias - mean) * scale() + beta;
}

}  // namespace dl4j

using namespace dl4j;

DL4J_API int dl4j_bn_fold(const void* table, const int* block_entry, int blocks, const float* params, void* w_out, float* b_out, void* stream) {
  if (blocks < 1 || !table || !block_entry || !params || !w_out || !b_out) return -DL4J_ERR_BAD_ARG;
  bn_fold_kernel<<<(blocks + BF_WARPS - 1) / BF_WARPS, 32 * BF_WARPS, 0, (cudaStream_t)stream>>>(
      reinterpret_cast<const BnFoldEntry*>(table), block_entry, blocks, params, reinterpret_cast<__nv_bfloat16*>(w_out), b_out);
  return (int)cudaGetLastError();
}
