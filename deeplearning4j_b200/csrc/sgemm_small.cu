// fp32 GEMM for problems too small to fill the chip: C = act(A B + bias) in plain fp32 multiply-adds.
//
// The default data type of a network is fp32, and the forward pass of a small one (batch 128, 784-512-512-10) gives a library kernel 16
// to 64 tiles on 148 SMs with the whole reduction as one serial chain, then a ReLU launch.  Here a tile's reduction is split over the
// CTAs of a thread-block cluster; each keeps its partial 64 x 64 tile in its own shared memory and every CTA then adds one slice of it
// from all of them, in rank order, through distributed shared memory: no atomics, no zeroed output, a result that does not depend on
// timing, bias and ReLU applied once at the end.
// 128 x 512 x 784 with bias and ReLU 14.5 us against 19.1, 128 x 512 x 512 8.9 against 14.7, 128 x 10 x 512 5.9 against 13.7 (library
// product + ReLU).  A K step takes a lone CTA 2.6 us, 1.0 of it arithmetic: shared-memory reads and their latency.  16 warps (18.5 us) and
// 8 x 8 results a thread (19.9 us, 254 registers) were slower.
// 256 threads, 4 x 4 results each.
// K steps are double-buffered through registers.  An operand contiguous along K is stored row by row in shared memory, one contiguous
// along its rows K slice by K slice, so that both are filled with coalesced loads and conflict-free stores; which rows or columns a
// thread has follows the layout.
#include "common.cuh"
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace dl4j {

constexpr int SG_T = 64;               // tile edge
constexpr int SG_K = 32;
constexpr int SG_THREADS = 256;
constexpr int SG_LDK = SG_K + 4;       // [row][k] pitch
constexpr int SG_LDR = SG_T + 4;       // [k][row] pitch
constexpr int SG_OP = SG_T * SG_LDK > SG_K * SG_LDR ? SG_T * SG_LDK : SG_K * SG_LDR;

struct SgemmParams {
  const float *A, *B, *bias;
  float* C;
  int M, N, K;
  long a_rs, b_rs;         // pitch of the non-contiguous dimension of A (over m or k) and of B (over n or k)
  long ldc;
  int act;                 // 1: ReLU
};

// One operand's tile: `rows` x K, element (r, k) at base[r * ld + k] (KC) or base[k * ld + r].
template <bool KC>
struct SgOperand {
  __device__ static __forceinline__ void fetch(const float* base, long ld, int row0, int rows, int k0, int k1, float (&v)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = KC ? (threadIdx.x >> 5) + 8 * i : threadIdx.x & 63, k = KC ? threadIdx.x & 31 : (threadIdx.x >> 6) + 4 * i;
      const bool in = row0 + r < rows && k0 + k < k1;
      v[i] = in ? __ldg(KC ? base + (row0 + r) * ld + k0 + k : base + (k0 + k) * ld + row0 + r) : 0.f;
    }
  }
  __device__ static __forceinline__ void stage(float* s, const float (&v)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = KC ? (threadIdx.x >> 5) + 8 * i : threadIdx.x & 63, k = KC ? threadIdx.x & 31 : (threadIdx.x >> 6) + 4 * i;
      s[KC ? r * SG_LDK + k : k * SG_LDR + r] = v[i];
    }
  }
  // this thread's i-th row (t: its coordinate 0 .. 15 along this operand)
  __device__ static __forceinline__ int row(int t, int i) { return KC ? t + 16 * i : t * 4 + i; }
  // four rows x four K values
  __device__ static __forceinline__ void read(const float* s, int t, int k, float (&v)[4][4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 q = *reinterpret_cast<const float4*>(KC ? s + row(t, i) * SG_LDK + k : s + (k + i) * SG_LDR + t * 4);
      if (KC) { v[i][0] = q.x; v[i][1] = q.y; v[i][2] = q.z; v[i][3] = q.w; }
      else { v[0][i] = q.x; v[1][i] = q.y; v[2][i] = q.z; v[3][i] = q.w; }
    }
  }
};

template <bool AK, bool BK>
__global__ void __launch_bounds__(SG_THREADS, 2) sgemm_small_kernel(const SgemmParams p) {
  __shared__ __align__(16) float sm[2][2][SG_OP];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int m0 = blockIdx.y * SG_T, n0 = blockIdx.x * SG_T;
  const int splits = gridDim.z, rank = blockIdx.z;
  const int steps = (p.K + SG_K - 1) / SG_K, per = (steps + splits - 1) / splits;
  const int ks = min(rank * per * SG_K, p.K), ke = min(ks + per * SG_K, p.K);
  const int n_it = (ke - ks + SG_K - 1) / SG_K;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  float va[8], vb[8];
  if (n_it > 0) {
    SgOperand<AK>::fetch(p.A, p.a_rs, m0, p.M, ks, ke, va);
    SgOperand<BK>::fetch(p.B, p.b_rs, n0, p.N, ks, ke, vb);
    SgOperand<AK>::stage(sm[0][0], va);
    SgOperand<BK>::stage(sm[0][1], vb);
  }
  __syncthreads();
  for (int it = 0; it < n_it; ++it) {
    const int buf = it & 1;
    const bool more = it + 1 < n_it;
    if (more) {
      SgOperand<AK>::fetch(p.A, p.a_rs, m0, p.M, ks + (it + 1) * SG_K, ke, va);
      SgOperand<BK>::fetch(p.B, p.b_rs, n0, p.N, ks + (it + 1) * SG_K, ke, vb);
    }
#pragma unroll
    for (int k = 0; k < SG_K; k += 4) {
      float a[4][4], b[4][4];
      SgOperand<AK>::read(sm[buf][0], ty, k, a);
      SgOperand<BK>::read(sm[buf][1], tx, k, b);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i][kk], b[j][kk], acc[i][j]);
    }
    if (more) {
      SgOperand<AK>::stage(sm[buf ^ 1][0], va);
      SgOperand<BK>::stage(sm[buf ^ 1][1], vb);
    }
    __syncthreads();
  }
  // the tile goes through shared memory (the loop ended with a barrier: the operand buffers are free): every CTA of the cluster then
  // finishes one slice of it, adding the ranks in order, with coalesced accesses
  float* mine = &sm[0][0][0];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) mine[SgOperand<AK>::row(ty, i) * SG_T + SgOperand<BK>::row(tx, j)] = acc[i][j];
  if (splits > 1) cg::this_cluster().sync(); else __syncthreads();
  const int n_el = SG_T * SG_T / splits;                        // 4096, 2048, 1024 or 512
#pragma unroll 2
  for (int e = threadIdx.x; e < n_el; e += SG_THREADS) {
    const int idx = rank * n_el + e, m = m0 + idx / SG_T, n = n0 + idx % SG_T;
    if (m >= p.M || n >= p.N) continue;
    float v;
    if (splits > 1) {
      float part[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) part[r] = r < splits ? cg::this_cluster().map_shared_rank(mine, r)[idx] : 0.f;
      v = part[0];
#pragma unroll
      for (int r = 1; r < 8; ++r) v += part[r];
    } else {
      v = mine[idx];
    }
    if (p.bias) v += __ldg(p.bias + n);
    if (p.act == 1) v = relu_f(v);
    p.C[m * p.ldc + n] = v;
  }
  if (splits > 1) cg::this_cluster().sync();                    // nobody leaves while its tile is being read
}

static_assert(4 * SG_OP >= SG_T * SG_T, "the partial tile reuses the operand buffers");

}  // namespace dl4j

using namespace dl4j;

// C[M, N] (row pitch ldc) = act(A B + bias).  A element (m, k) at m * lda + k (a_kc) or k * lda + m; B element (k, n) at
// n * ldb + k (b_kc) or k * ldb + n.  The split is chosen to give about two CTAs per SM, with at least two K steps each.
DL4J_API int dl4j_sgemm_small(const float* A, long lda, int a_kc, const float* B, long ldb, int b_kc, const float* bias, float* C, long ldc,
                              int M, int N, int K, int act, int num_sms, void* stream) {
  if (M < 1 || N < 1 || K < 1) return -DL4J_ERR_BAD_ARG;
  const SgemmParams p{A, B, bias, C, M, N, K, lda, ldb, ldc, act};
  const long tiles = (long)((M + SG_T - 1) / SG_T) * ((N + SG_T - 1) / SG_T);
  const int steps = (K + SG_K - 1) / SG_K;
  int s = 1;
  while (s < 8 && tiles * s * 2 <= 2L * num_sms && steps >= s * 4) s *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((N + SG_T - 1) / SG_T, (M + SG_T - 1) / SG_T, s);
  cfg.blockDim = dim3(SG_THREADS);
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaError_t e;
  if (a_kc && b_kc) e = cudaLaunchKernelEx(&cfg, sgemm_small_kernel<true, true>, p);
  else if (a_kc) e = cudaLaunchKernelEx(&cfg, sgemm_small_kernel<true, false>, p);
  else if (b_kc) e = cudaLaunchKernelEx(&cfg, sgemm_small_kernel<false, true>, p);
  else e = cudaLaunchKernelEx(&cfg, sgemm_small_kernel<false, false>, p);
  return (int)e;
}
