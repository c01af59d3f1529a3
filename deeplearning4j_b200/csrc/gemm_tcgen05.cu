// bf16/fp16 GEMM on the 5th-generation tensor cores: D = act(A·B + bias) (+ residual).
//
// Replaces the reference's cuBLAS call sites and naive SIMT fallbacks
// (libnd4j/include/helpers/cuda/MmulHelper.cu:41-129 usualCudaGemm, :501-517 cublas*gemm) and the
// matmul+addBias+activation sequences of xw_plus_b / relu_layer / DenseLayer.
//
// Structure (one persistent CTA per SM, 320 threads):
//   warp 0      : TMA producer  - cp.async.bulk.tensor tiles of A and B into a multi-stage smem ring
//   warp 1      : MMA issuer    - one elected lane issues tcgen05.mma (128 x BLOCK_N x 16), accumulators
//                                 live in TMEM, double-buffered (2 x BLOCK_N columns) so the epilogue of
//                                 tile i overlaps the main loop of tile i+1
//   warps 2..9  : epilogue      - tcgen05.ld 32 lanes x 32 columns, bias / activation / residual,
//                                 16-byte global stores (or fp32 vector reductions for split-K)
// Operands may be K-major (reduction dimension contiguous) or MN-major (output dimension contiguous),
// which covers forward (X·Wᵀ), data-gradient (dY·W) and weight-gradient (dYᵀ·X) without transposes.
#include "common.cuh"

namespace dl4j {

constexpr int BLOCK_M = 128;
constexpr int BLOCK_K = 64;         // 64 x 2 bytes = one 128-byte swizzle row
constexpr int UMMA_K = 16;
constexpr int GEMM_PAIR_TILE = 512;  // `block_n` of the 256 x 256 tiles on CTA pairs
constexpr int GEMM_EPI_WARPS = 8;   // two per TMEM lane quadrant: they take every second group of 32 columns
constexpr int GEMM_THREADS = 64 + 32 * GEMM_EPI_WARPS;

struct GemmParams {
  int M, N, K;
  long ldc;               // elements
  long ld_aux, ld_res;
  void* C;
  void* aux;              // optional pre-activation output (same dtype as inputs)
  const void* bias;       // optional [N], dtype bias_fp32 ? float : input dtype
  const void* residual;   // optional [M, N] input dtype
  int bias_fp32;
  int out_fp32;           // C is float
  int act;                // 0 none, 1 relu, 2 gelu(erf), 3 gelu(tanh), 4 sigmoid, 5 tanh
  int atomic_out;         // 1: accumulate into fp32 C with vector reductions (split-K / grad accumulation); 2: split s stores its
                          // partial result in slab s of an fp32 [splits, M, ldc] buffer (staged epilogue only)
  int splits;             // split-K factor (>1 requires atomic_out)
  int fmt;                // 0 fp16, 1 bf16
  float alpha;
  int* status;
  int batch1, batch2;     // two batch dimensions (1 when unused); batch index = b2 * batch1 + b1
  long c_stride_b1, c_stride_b2;   // output batch strides in elements
  int tma_store;          // epilogue stages tiles in shared memory and writes them with TMA (needs 16-byte aligned C rows)
  int tma_aux;            // same for the auxiliary pre-activation output
  int bias_mma;           // the bias is added on the tensor core: one extra K=16 step ones[128 x 1] x bias[1 x N] per tile
  int raster_gn;          // tile raster: column-tile groups of this width, column index fastest inside a group
  int relu_last;          // ReLU after the residual has been added (a residual block's output; inference)
  int res_act;            // != 0: `residual` holds pre-activations z and the result is multiplied by act'(z) instead of added to
                          // (the data-gradient GEMM of a layer that feeds an activation writes dz directly)
};

// Tile order.  CTAs that run at the same time take consecutive tile numbers, so the order decides what they share in L2:
// within a group of `gn` column tiles the column index runs fastest, i.e. the CTAs of one wave cover few row panels of A
// (each read from DRAM once and hit in L2 by the other column tiles) and at most gn column panels of B.
__device__ __forceinline__ void tile_coords(int tile, int tiles_m, int tiles_n, int gn, int& mt, int& nt) {
  const int per_group = tiles_m * gn;
  const int g = tile / per_group;
  const int n_base = g * gn;
  const int gw = min(gn, tiles_n - n_base);
  const int r = tile - g * per_group;
  mt = r / gw;
  nt = n_base + (r - mt * gw);
}

// ------------------------------------------------------------------ CTA pairs
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of `local` (a shared::cta address of this CTA) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tmem_alloc2(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish2() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// D[tmem of both CTAs] (+)= A * B over the CTA pair: 256 rows (128 per CTA), N columns (each CTA stages N / 2 of B)
__device__ __forceinline__ void umma2_f16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      :
      : "r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives on the mbarrier at shared::cluster address `bar` once all MMAs issued so far by this thread have completed
__device__ __forceinline__ void umma2_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// a load into this CTA's shared memory that completes on a barrier of either CTA of the pair (shared::cluster address)
__device__ __forceinline__ void tma_load_4d_pair(void* smem_dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

template <int BLOCK_N, bool A_MN, bool B_MN, bool PAIR>
struct GemmSmem {
  static constexpr int A_BYTES = BLOCK_M * BLOCK_K * 2;
  static constexpr int B_COLS = PAIR ? BLOCK_N / 2 : BLOCK_N;      // columns of the tile that this CTA stages
  static constexpr int B_BYTES = B_COLS * BLOCK_K * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = B_COLS == 256 ? 4 : 6;
  static constexpr int EPI_SLAB = 32 * 64;                  // one warp's 32 rows x 32 16-bit columns (fp32: both slabs)
  static constexpr int EPI_BYTES = GEMM_EPI_WARPS * 2 * EPI_SLAB;
  static constexpr int BIAS_BYTES = GEMM_EPI_WARPS * 32 * 4;   // one group of 32 columns per warp
  static constexpr int TOTAL = STAGES * STAGE_BYTES + EPI_BYTES + BIAS_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/;
};

__device__ __forceinline__ float apply_act(float v, int act) {
  switch (act) {
    case 1: return relu_f(v);
    case 2: return gelu_erf(v);
    case 3: return gelu_tanh(v);
    case 4: return sigmoidf_(v);
    case 5: return tanhf(v);
    case 6: return gelu_sigmoid(v);
    default: return v;
  }
}

// v *= act'(z): the activation-gradient factor applied in the epilogue of a data-gradient GEMM.  The GELU forms use one
// tanh.approx per value (sigmoid(y) = 0.5 + 0.5 tanh(y / 2)).
__device__ __forceinline__ float tanh_fast(float x) {
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(x));
  return t;
}
__device__ __forceinline__ float mul_act_grad(float v, float z, int act) {
  switch (act) {
    case 1: return z > 0.f ? v : 0.f;
    case 2: return v * (0.5f * (1.f + erff(z * 0.70710678118654752f)) + z * 0.3989422804014327f * __expf(-0.5f * z * z));
    case 3: {
      const float z2 = z * z;
      const float t = tanh_fast(0.7978845608028654f * z * fmaf(0.044715f, z2, 1.f));
      return v * (fmaf(0.5f, t, 0.5f) + 0.5f * z * (1.f - t * t) * 0.7978845608028654f * fmaf(0.134145f, z2, 1.f));
    }
    case 4: { const float sg = fmaf(0.5f, tanh_fast(0.5f * z), 0.5f); return v * sg * (1.f - sg); }
    case 5: { const float t = tanh_fast(z); return v * (1.f - t * t); }
    case 6: { const float sg = fmaf(0.5f, tanh_fast(0.851f * z), 0.5f); return v * fmaf(1.702f * z * sg, 1.f - sg, sg); }
    default: return v;
  }
}

// Warp-uniform dispatch hoisted out of the element loop.
__device__ __forceinline__ void apply_act32(float (&v)[32], int act) {
  if (act == 1) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = relu_f(v[j]);
  } else if (act == 2) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = gelu_erf(v[j]);
  } else if (act == 3) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = gelu_tanh(v[j]);
  } else if (act == 6) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = gelu_sigmoid(v[j]);
  } else if (act == 4) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = sigmoidf_(v[j]);
  } else if (act == 5) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = tanhf(v[j]);
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = apply_act(v[j], act);
  }
}

template <typename T>
__device__ __forceinline__ float to_f(T v);
template <>
__device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <>
__device__ __forceinline__ float to_f<__half>(__half v) { return __half2float(v); }

__device__ __forceinline__ uint32_t pack2(float a, float b, int fmt) {
  if (fmt == 1) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ float unpack_lo(uint32_t u, int fmt) {
  if (fmt == 1) return __bfloat162float(*reinterpret_cast<__nv_bfloat16*>(&u));
  return __half2float(*reinterpret_cast<__half*>(&u));
}

__device__ __forceinline__ float unpack_hi(uint32_t u, int fmt) {
  uint32_t h = u >> 16;
  if (fmt == 1) return __bfloat162float(*reinterpret_cast<__nv_bfloat16*>(&h));
  return __half2float(*reinterpret_cast<__half*>(&h));
}

// 32 values of a row as four 16-byte units of the 64-byte swizzle, the format decided once
template <bool BF16>
__device__ __forceinline__ void store_row32(uint8_t* row, int sw64, const float (&v)[32]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    constexpr int F = BF16 ? 1 : 0;
    const uint4 u = make_uint4(pack2(v[8 * j], v[8 * j + 1], F), pack2(v[8 * j + 2], v[8 * j + 3], F), pack2(v[8 * j + 4], v[8 * j + 5], F),
                               pack2(v[8 * j + 6], v[8 * j + 7], F));
    *reinterpret_cast<uint4*>(row + ((j ^ sw64) << 4)) = u;
  }
}
template <bool BF16>
__device__ __forceinline__ void unpack_row32(const uint4 (&z)[4], float (&f)[32]) {
  constexpr int F = BF16 ? 1 : 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t w[4] = {z[j].x, z[j].y, z[j].z, z[j].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) { f[8 * j + 2 * e] = unpack_lo(w[e], F); f[8 * j + 2 * e + 1] = unpack_hi(w[e], F); }
  }
}

// bias[col] as float (0 beyond N); the bias vector is fp32 or the operand type
__device__ __forceinline__ float load_bias(const GemmParams& p, int col) {
  if (col >= p.N) return 0.f;
  return p.bias_fp32 ? __ldg(reinterpret_cast<const float*>(p.bias) + col)
                     : unpack_lo((uint32_t)__ldg(reinterpret_cast<const uint16_t*>(p.bias) + col), p.fmt);
}

// FULL: pre-activation output, activations other than ReLU, activation gradients.  The other form knows bias, residual and ReLU only: what an
// epilogue warp executes per 32 columns is then one short run of code.  With both kinds in one kernel, four epilogue warps, the operand
// format looked at for every pair of values and the bias broadcast by shuffles, 32 columns took 310 instructions and 1900 clocks, most of
// them waits for the instruction fetch and for dependent results.  Before / now, us (N = 256 tiles): 200704 x 256 x 64 53 / 33, with fp32
// bias 70 / 41, with residual 156 / 74; 16384 x 3072 x 768 with bias, GELU and pre-activations 99 / 85, with residual 179 / 89.
// PAIR: the two CTAs of a cluster work on one tile of 256 rows.  Each stages its own 128 rows of A and half of B's columns, 32 KB per 64 of K
// instead of 48: what a k-step takes is the time its operands need from L2.  The leader's MMA thread issues tcgen05.mma.cta_group::2 for
// both (each tensor core produces its own 128 rows in its own tensor memory); both CTAs' loads complete on the leader's barrier, commits
// free the stage and announce the accumulator in both CTAs, and both epilogues release the accumulator on the leader's barrier.
// 256 wide / pair, us: 16384 x 3072 x 768 67 / 58, 16384 x 768 x 3072 62 / 57, 16384 x 2304 x 768 51 / 44, 2456 x 30520 x 768 150 / 122,
// 8192 x 8192 x 8192 796 / 768.  With the peer's loads on its own barrier and a thread that forwarded their arrival the form was no faster.
template <int BLOCK_N, bool A_MN, bool B_MN, bool FULL, bool PAIR>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                    const __grid_constant__ CUtensorMap tmap_c, const __grid_constant__ CUtensorMap tmap_aux,
                    const __grid_constant__ CUtensorMap tmap_ones, const __grid_constant__ CUtensorMap tmap_bias,
                    const GemmParams p) {
  using S = GemmSmem<BLOCK_N, A_MN, B_MN, PAIR>;
  constexpr int TILE_M = PAIR ? 2 * BLOCK_M : BLOCK_M;
  constexpr int B_COLS = S::B_COLS;
  constexpr int STAGES = S::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* epi_smem = smem + STAGES * S::STAGE_BYTES;       // 1024-byte aligned (stage sizes are multiples of 1024)
  float* bias_smem = reinterpret_cast<float*>(epi_smem + S::EPI_BYTES);
  uint64_t* bars = reinterpret_cast<uint64_t*>(epi_smem + S::EPI_BYTES + S::BIAS_BYTES);
  uint64_t* full_bar = bars;                    // [STAGES]
  uint64_t* empty_bar = bars + STAGES;          // [STAGES]
  uint64_t* tmem_full = bars + 2 * STAGES;      // [2]
  uint64_t* tmem_empty = bars + 2 * STAGES + 2; // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  const uint32_t rank = PAIR ? cluster_ctarank() : 0u;      // 0: the leader, issues the MMAs
  const int first_work = PAIR ? blockIdx.x >> 1 : blockIdx.x, work_step = PAIR ? gridDim.x >> 1 : gridDim.x;
  const int tiles_m = (p.M + TILE_M - 1) / TILE_M;
  const int tiles_n = (p.N + BLOCK_N - 1) / BLOCK_N;
  const int kb_total = (p.K + BLOCK_K - 1) / BLOCK_K;
  const int kb_per_split = (kb_total + p.splits - 1) / p.splits;
  const int per_batch = tiles_m * tiles_n * p.splits;
  const int num_work = per_batch * p.batch1 * p.batch2;

  if (threadIdx.x == 0) {
    prefetch_tmap(&tmap_a);
    prefetch_tmap(&tmap_b);
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full[i], 1);
      mbar_init(&tmem_empty[i], (PAIR ? 2 : 1) * GEMM_EPI_WARPS);   // one arrive per epilogue warp
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    if constexpr (PAIR) {
      tmem_alloc2(tmem_slot, 2 * BLOCK_N);
      tmem_relinquish2();
    } else {
      tmem_alloc(tmem_slot, 2 * BLOCK_N);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();       // both CTAs' barriers exist before anybody arrives on a remote one
  tc_fence_after();
  pdl_wait_and_release();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      auto expect = [&](uint32_t bytes) {              // of both CTAs of a pair, on the leader's barrier
        if (!PAIR || rank == 0) mbar_expect_tx(&full_bar[stage], PAIR ? 2 * bytes : bytes);
      };
      auto load = [&](void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3) {
        if constexpr (PAIR) tma_load_4d_pair(dst, map, mapa(smem_u32(&full_bar[stage]), 0), c0, c1, c2, c3);
        else tma_load_4d(dst, map, &full_bar[stage], c0, c1, c2, c3);
      };
      for (int w = first_work; w < num_work && ok; w += work_step) {
        const int batch = w / per_batch, wr = w % per_batch;
        const int b1 = batch % p.batch1, b2 = batch / p.batch1;
        const int tile = wr / p.splits, split = wr % p.splits;
        int mt, nt;
        tile_coords(tile, tiles_m, tiles_n, p.raster_gn, mt, nt);
        const int m0 = mt * TILE_M + (int)rank * BLOCK_M, n0 = nt * BLOCK_N + (int)rank * B_COLS;
        const int kb0 = split * kb_per_split;
        const int kb1 = min(kb0 + kb_per_split, kb_total);
        if (p.bias_mma) {
          // bias stage: both operands MN-major with a single valid K row (row 0 = ones / bias, rows 1..15 zero-filled by
          // TMA because the maps' K extent is 1); only the 16 K rows of the one MMA step are written (2 KB per 64-column box
          // at the usual box addresses), so the usual stage layout and descriptors apply
          if (!mbar_wait_bounded(&empty_bar[stage], phase ^ 1, p.status, DL4J_ERR_TIMEOUT_PRODUCER)) { ok = false; break; }
          uint8_t* sa = smem + stage * S::STAGE_BYTES;
          uint8_t* sb = sa + S::A_BYTES;
          expect((BLOCK_M / 64 + B_COLS / 64) * (64 * UMMA_K * 2));
#pragma unroll
          for (int i = 0; i < BLOCK_M / 64; ++i)
            load(sa + i * (64 * BLOCK_K * 2), &tmap_ones, i * 64, 0, 0, 0);
#pragma unroll
          for (int i = 0; i < B_COLS / 64; ++i)
            load(sb + i * (64 * BLOCK_K * 2), &tmap_bias, n0 + i * 64, 0, 0, 0);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_bounded(&empty_bar[stage], phase ^ 1, p.status, DL4J_ERR_TIMEOUT_PRODUCER)) { ok = false; break; }
          uint8_t* sa = smem + stage * S::STAGE_BYTES;
          uint8_t* sb = sa + S::A_BYTES;
          expect(S::STAGE_BYTES);
          const int k0 = kb * BLOCK_K;
          if (!A_MN) {
            load(sa, &tmap_a, k0, m0, b1, b2);
          } else {
#pragma unroll
            for (int i = 0; i < BLOCK_M / 64; ++i)
              load(sa + i * (64 * BLOCK_K * 2), &tmap_a, m0 + i * 64, k0, b1, b2);
          }
          if (!B_MN) {
            load(sb, &tmap_b, k0, n0, b1, b2);
          } else {
#pragma unroll
            for (int i = 0; i < B_COLS / 64; ++i)
              load(sb + i * (64 * BLOCK_K * 2), &tmap_b, n0 + i * 64, k0, b1, b2);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      if constexpr (PAIR)              // every commit of the leader has arrived here before this CTA may go
        for (int i = 0; i < STAGES; ++i) {
          mbar_wait_bounded(&empty_bar[stage], phase ^ 1, p.status, DL4J_ERR_TIMEOUT_PRODUCER);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = make_idesc(p.fmt, A_MN ? 1 : 0, B_MN ? 1 : 0, TILE_M, BLOCK_N);
      auto mma = [&](uint32_t d, uint64_t a, uint64_t b, uint32_t id, uint32_t accumulate) {
        if constexpr (PAIR) umma2_f16(d, a, b, id, accumulate);
        else umma_f16(d, a, b, id, accumulate);
      };
      auto commit = [&](uint64_t* bar) {
        if constexpr (PAIR) {
          umma2_commit(mapa(smem_u32(bar), 0));
          umma2_commit(mapa(smem_u32(bar), 1));
        } else {
          umma_commit(bar);
        }
      };
      // K-major: 8-row groups are 1024 B apart (SBO); MN-major: 64-element column blocks are one
      // TMA box apart (LBO = 64 rows x 128 B) and 8-row K groups 1024 B apart (SBO).
      constexpr uint32_t LBO_A = A_MN ? 64 * BLOCK_K * 2 : 16, LBO_B = B_MN ? 64 * BLOCK_K * 2 : 16;
      constexpr uint32_t KSTEP_A = A_MN ? UMMA_K * 128 : UMMA_K * 2, KSTEP_B = B_MN ? UMMA_K * 128 : UMMA_K * 2;
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      bool ok = true;
      for (int w = first_work; w < num_work && ok; w += work_step, ++it) {
        const int split = (w % per_batch) % p.splits;
        const int kb0 = split * kb_per_split;
        const int kb1 = min(kb0 + kb_per_split, kb_total);
        const int buf = it & 1;
        const uint32_t acc_phase = (it >> 1) & 1;
        if (!mbar_wait_bounded(&tmem_empty[buf], acc_phase ^ 1, p.status, DL4J_ERR_TIMEOUT_MMA)) { ok = false; break; }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + buf * BLOCK_N;
        if (p.bias_mma) {
          // accumulator := ones[128 x 16] * bias[16 x BLOCK_N] (only K row 0 is non-zero): every row starts at the bias
          if (!mbar_wait_bounded(&full_bar[stage], phase, p.status, DL4J_ERR_TIMEOUT_MMA)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * S::STAGE_BYTES);
          const uint32_t sb = sa + S::A_BYTES;
          mma(tmem_d, make_smem_desc_sw128(sa, 64 * BLOCK_K * 2, 1024), make_smem_desc_sw128(sb, 64 * BLOCK_K * 2, 1024),
                   make_idesc(p.fmt, 1, 1, TILE_M, BLOCK_N), 0u);
          commit(&empty_bar[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_bounded(&full_bar[stage], phase, p.status, DL4J_ERR_TIMEOUT_MMA)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * S::STAGE_BYTES);
          const uint32_t sb = sa + S::A_BYTES;
          const uint64_t da = make_smem_desc_sw128(sa, LBO_A, 1024);
          const uint64_t db = make_smem_desc_sw128(sb, LBO_B, 1024);
#pragma unroll
          for (int k = 0; k < BLOCK_K / UMMA_K; ++k) {
            mma(tmem_d, da + ((uint64_t)(k * KSTEP_A) >> 4), db + ((uint64_t)(k * KSTEP_B) >> 4), idesc,
                     (kb > kb0 || k > 0 || p.bias_mma) ? 1u : 0u);
          }
          commit(&empty_bar[stage]);   // frees the smem stage once these MMAs have read it
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        commit(&tmem_full[buf]);       // accumulator ready for the epilogue
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..9)
    const int q = warp & 3;                 // TMEM lane quadrant this warp may access
    const int c_first = ((warp - 2) >> 2) * 32;
    int it = 0;
    bool ok = true;
    auto release = [&](int buf) {           // the accumulator has been read
      if constexpr (PAIR) mbar_arrive_cluster(mapa(smem_u32(&tmem_empty[buf]), 0));
      else mbar_arrive(&tmem_empty[buf]);
    };
    for (int w = first_work; w < num_work && ok; w += work_step, ++it) {
      const int batch = w / per_batch, wr = w % per_batch;
      const long c_off = (long)(batch % p.batch1) * p.c_stride_b1 + (long)(batch / p.batch1) * p.c_stride_b2;
      const int tile = wr / p.splits, split = wr % p.splits;
      int mt, nt;
      tile_coords(tile, tiles_m, tiles_n, p.raster_gn, mt, nt);
      const int m0 = mt * TILE_M + (int)rank * BLOCK_M, n0 = nt * BLOCK_N;
      const int kb0 = split * kb_per_split;
      const bool has_k = kb0 < min(kb0 + kb_per_split, kb_total);
      const int buf = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1;
      const bool lead_split = split == 0;
      // lane L of the warp fetches bias[col0 + L] one group ahead of its use (first group here, before the wait for the
      // accumulator), and the group is broadcast through the warp's own 32 floats: no load latency inside the tile loop
      const bool use_bias = p.bias != nullptr && lead_split && !p.bias_mma;
      float bias_cur = use_bias ? load_bias(p, n0 + c_first + lane) : 0.f;
      // the residual's 64 bytes of this thread's row likewise travel one group ahead (rows 16-byte aligned, whole groups)
      const bool use_res = p.residual != nullptr && lead_split && m0 + q * 32 + lane < p.M;
      const uint16_t* res_row = reinterpret_cast<const uint16_t*>(p.residual) + (long)(m0 + q * 32 + lane) * p.ld_res + n0;
      const bool res_vec = use_res && p.tma_store && (reinterpret_cast<uintptr_t>(res_row) & 15) == 0;
      uint4 rz[4];
      auto load_res = [&](int c) {
        if (res_vec && c < BLOCK_N && n0 + c + 32 <= p.N) {
#pragma unroll
          for (int j = 0; j < 4; ++j) rz[j] = *reinterpret_cast<const uint4*>(res_row + c + 8 * j);
        }
      };
      load_res(c_first);
      if (!mbar_wait_bounded(&tmem_full[buf], acc_phase, p.status, DL4J_ERR_TIMEOUT_EPILOGUE)) { ok = false; break; }
      tc_fence_after();
      const int row = m0 + q * 32 + lane;
      const bool row_ok = row < p.M;
      const uint32_t taddr_row = tmem_base + buf * BLOCK_N + ((uint32_t)(q * 32) << 16);
      if (p.tma_store) {
        // -------- staged epilogue: registers -> swizzled smem slab (32 rows x 64 B, fp32 128 B, per warp) -> TMA store / reduce
        const int b1 = batch % p.batch1, b2 = p.atomic_out == 2 ? split : batch / p.batch1;
        uint8_t* ring = epi_smem + (warp - 2) * (2 * S::EPI_SLAB);
        float* my_bias = bias_smem + (warp - 2) * 32;
        const bool rescale = !has_k || p.alpha != 1.0f;
        const bool want_aux = FULL && p.aux != nullptr && p.tma_aux;
        const bool two_slabs = want_aux || p.out_fp32;        // an iteration fills both slabs: every earlier store must have been read
        int ring_idx = 0;
#pragma unroll 1
        for (int c = c_first; c < BLOCK_N; c += 64) {
          const int col0 = n0 + c;
          if (col0 >= p.N) break;                                     // warp-uniform
          uint32_t r[32];
          tmem_ld_32x32(taddr_row + c, r);
          tmem_ld_wait();
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
          if (rescale) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = has_k ? v[j] * p.alpha : 0.0f;
          }
          if (use_bias) {
            my_bias[lane] = bias_cur;
            __syncwarp();
            bias_cur = load_bias(p, col0 + 64 + lane);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float4 b4 = reinterpret_cast<const float4*>(my_bias)[j];
              v[4 * j] += b4.x; v[4 * j + 1] += b4.y; v[4 * j + 2] += b4.z; v[4 * j + 3] += b4.w;
            }
          }
          if (lane == 0) { if (two_slabs) bulk_wait_read<0>(); else bulk_wait_read<1>(); }
          __syncwarp();
          uint8_t* slab_out = ring + (p.out_fp32 ? 0 : want_aux ? S::EPI_SLAB : ring_idx * S::EPI_SLAB);
          const int sw64 = (lane >> 1) & 3;                           // 64-byte swizzle: 16-byte unit ^ (row / 2 % 4)
          if constexpr (FULL) {
            if (want_aux) {
              if (p.fmt == 1) store_row32<true>(ring + lane * 64, sw64, v);
              else store_row32<false>(ring + lane * 64, sw64, v);
            }
            if (p.act != 0) apply_act32(v, p.act);
          } else if (p.act == 1) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = relu_f(v[j]);
          }
          if (use_res) {
            if (res_vec && col0 + 32 <= p.N) {
              float z[32];
              if (p.fmt == 1) unpack_row32<true>(rz, z);
              else unpack_row32<false>(rz, z);
              if (FULL && p.res_act) {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = mul_act_grad(v[j], z[j], p.res_act);
              } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] += z[j];
              }
              load_res(c + 64);
            } else {
              const uint16_t* rs = res_row + c;
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (col0 + j < p.N) {
                  const float z = unpack_lo((uint32_t)rs[j], p.fmt);
                  v[j] = FULL && p.res_act ? mul_act_grad(v[j], z, p.res_act) : v[j] + z;
                }
            }
          }
          if (p.relu_last) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = relu_f(v[j]);
          }
          if (p.out_fp32) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              *reinterpret_cast<float4*>(slab_out + lane * 128 + ((j ^ (lane & 7)) << 4)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          } else if (p.fmt == 1) {
            store_row32<true>(slab_out + lane * 64, sw64, v);
          } else {
            store_row32<false>(slab_out + lane * 64, sw64, v);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            const int r0 = m0 + q * 32;
            if (r0 < p.M) {
              if (want_aux) tma_store_4d(&tmap_aux, ring, col0, r0, b1, b2);
              if (p.atomic_out == 1) tma_reduce_add_4d(&tmap_c, slab_out, col0, r0, b1, b2);
              else tma_store_4d(&tmap_c, slab_out, col0, r0, b1, b2);
            }
            bulk_commit();
          }
          ring_idx ^= 1;
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) release(buf);
        continue;
      }
#pragma unroll 1
      for (int c = c_first; c < BLOCK_N; c += 64) {
        const int col0 = n0 + c;
        if (col0 >= p.N) break;             // warp-uniform
        uint32_t r[32];
        tmem_ld_32x32(taddr_row + c, r);
        tmem_ld_wait();
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = has_k ? __uint_as_float(r[j]) * p.alpha : 0.0f;
        const bool full_chunk = col0 + 32 <= p.N;
        if (p.bias != nullptr && lead_split && !p.bias_mma) {
          if (p.bias_fp32) {
            const float* b = reinterpret_cast<const float*>(p.bias) + col0;
#pragma unroll
            for (int j = 0; j < 32; ++j) if (full_chunk || col0 + j < p.N) v[j] += __ldg(b + j);
          } else if (p.fmt == 1) {
            const __nv_bfloat16* b = reinterpret_cast<const __nv_bfloat16*>(p.bias) + col0;
#pragma unroll
            for (int j = 0; j < 32; ++j) if (full_chunk || col0 + j < p.N) v[j] += __bfloat162float(b[j]);
          } else {
            const __half* b = reinterpret_cast<const __half*>(p.bias) + col0;
#pragma unroll
            for (int j = 0; j < 32; ++j) if (full_chunk || col0 + j < p.N) v[j] += __half2float(b[j]);
          }
        }
        if (row_ok) {
          if (p.aux != nullptr) {
            uint16_t* a = reinterpret_cast<uint16_t*>(p.aux) + (long)row * p.ld_aux + col0;
            if (full_chunk && ((reinterpret_cast<uintptr_t>(a) & 15) == 0)) {
#pragma unroll
              for (int j = 0; j < 32; j += 8) {
                uint4 u = make_uint4(pack2(v[j], v[j + 1], p.fmt), pack2(v[j + 2], v[j + 3], p.fmt),
                                     pack2(v[j + 4], v[j + 5], p.fmt), pack2(v[j + 6], v[j + 7], p.fmt));
                *reinterpret_cast<uint4*>(a + j) = u;
              }
            } else {
              for (int j = 0; j < 32 && col0 + j < p.N; ++j) a[j] = (uint16_t)(pack2(v[j], 0.f, p.fmt) & 0xffff);
            }
          }
          if (p.act != 0) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = apply_act(v[j], p.act);
          }
          if (p.residual != nullptr && lead_split) {
            const uint16_t* rs = reinterpret_cast<const uint16_t*>(p.residual) + (long)row * p.ld_res + col0;
            if (full_chunk && ((reinterpret_cast<uintptr_t>(rs) & 15) == 0)) {
#pragma unroll
              for (int j = 0; j < 32; j += 8) {
                const uint4 u = *reinterpret_cast<const uint4*>(rs + j);
                const float z8[8] = {unpack_lo(u.x, p.fmt), unpack_hi(u.x, p.fmt), unpack_lo(u.y, p.fmt), unpack_hi(u.y, p.fmt),
                                     unpack_lo(u.z, p.fmt), unpack_hi(u.z, p.fmt), unpack_lo(u.w, p.fmt), unpack_hi(u.w, p.fmt)};
#pragma unroll
                for (int e = 0; e < 8; ++e) v[j + e] = p.res_act ? mul_act_grad(v[j + e], z8[e], p.res_act) : v[j + e] + z8[e];
              }
            } else {
              for (int j = 0; j < 32 && col0 + j < p.N; ++j) {
                const float z = unpack_lo((uint32_t)rs[j], p.fmt);
                v[j] = p.res_act ? mul_act_grad(v[j], z, p.res_act) : v[j] + z;
              }
            }
          }
          if (p.relu_last) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = relu_f(v[j]);
          }
          if (p.out_fp32) {
            float* o = reinterpret_cast<float*>(p.C) + c_off + (long)row * p.ldc + col0;
            const bool al = full_chunk && ((reinterpret_cast<uintptr_t>(o) & 15) == 0);
            if (p.atomic_out) {
              if (al) {
#pragma unroll
                for (int j = 0; j < 32; j += 4)
                  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(o + j), "f"(v[j]), "f"(v[j + 1]),
                               "f"(v[j + 2]), "f"(v[j + 3]) : "memory");
              } else {
                for (int j = 0; j < 32 && col0 + j < p.N; ++j) atomicAdd(o + j, v[j]);
              }
            } else if (al) {
#pragma unroll
              for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4*>(o + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
            } else {
              for (int j = 0; j < 32 && col0 + j < p.N; ++j) o[j] = v[j];
            }
          } else {
            uint16_t* o = reinterpret_cast<uint16_t*>(p.C) + c_off + (long)row * p.ldc + col0;
            if (full_chunk && ((reinterpret_cast<uintptr_t>(o) & 15) == 0)) {
#pragma unroll
              for (int j = 0; j < 32; j += 8) {
                uint4 u = make_uint4(pack2(v[j], v[j + 1], p.fmt), pack2(v[j + 2], v[j + 3], p.fmt),
                                     pack2(v[j + 4], v[j + 5], p.fmt), pack2(v[j + 6], v[j + 7], p.fmt));
                *reinterpret_cast<uint4*>(o + j) = u;
              }
            } else {
              for (int j = 0; j < 32 && col0 + j < p.N; ++j) o[j] = (uint16_t)(pack2(v[j], 0.f, p.fmt) & 0xffff);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) release(buf);
    }
    if (lane == 0) bulk_wait<0>();          // staged tiles must have left shared memory before the CTA exits
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();   // the partner's shared and tensor memory stay until the pair is done
  if (warp == 1) {
    tc_fence_after();
    if constexpr (PAIR) tmem_dealloc2(tmem_base, 2 * BLOCK_N);
    else tmem_dealloc(tmem_base, 2 * BLOCK_N);
  }
}

}  // namespace dl4j

// =============================================================================== host side
using namespace dl4j;

static int encode_2d(CUtensorMap* map, const void* base, uint64_t inner, uint64_t outer, uint64_t row_stride_bytes,
                     uint32_t box_inner, uint32_t box_outer, uint64_t nb1 = 1, uint64_t nb2 = 1, uint64_t sb1_bytes = 0,
                     uint64_t sb2_bytes = 0, CUtensorMapDataType dt = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                     CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B) {
  dl4j_PFN_encodeTiled enc = dl4j_get_encode_tiled();
  if (!enc) return -1;
  // rank-4 map {inner, outer, batch1, batch2}; unit batch dims get a harmless 16-byte-multiple stride
  if (sb1_bytes == 0) sb1_bytes = row_stride_bytes * outer;
  if (sb2_bytes == 0) sb2_bytes = sb1_bytes * nb1;
  cuuint64_t dims[4] = {inner, outer, nb1, nb2};
  cuuint64_t strides[3] = {row_stride_bytes, sb1_bytes, sb2_bytes};
  cuuint32_t box[4] = {box_inner, box_outer, 1, 1};
  cuuint32_t es[4] = {1, 1, 1, 1};
  CUresult r = enc(map, dt, 4, const_cast<void*>(base), dims, strides, box, es,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)r;
}

// 128 ones in each operand format: the A operand of the bias step
#define DL4J_REP8(x) x, x, x, x, x, x, x, x
#define DL4J_REP128(x) DL4J_REP8(DL4J_REP8(x)), DL4J_REP8(DL4J_REP8(x))
static __device__ __align__(128) uint16_t g_ones_bf16[128] = {DL4J_REP128(0x3F80)};
static __device__ __align__(128) uint16_t g_ones_f16[128] = {DL4J_REP128(0x3C00)};

template <int BLOCK_N, bool A_MN, bool B_MN, bool FULL, bool PAIR = false>
static int launch_gemm(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const CUtensorMap& tx,
                       const CUtensorMap& tones, const CUtensorMap& tbias, const GemmParams& p, int grid, int dev, cudaStream_t stream) {
  using S = GemmSmem<BLOCK_N, A_MN, B_MN, PAIR>;
  auto kern = gemm_tcgen05_kernel<BLOCK_N, A_MN, B_MN, FULL, PAIR>;
  static SmemLimit limit;
  const cudaError_t e = raise_smem_limit((const void*)kern, dev, S::TOTAL, limit);
  if (e != cudaSuccess) return (int)e;
  return (int)launch_dependent_clusters(kern, dim3(grid), dim3(GEMM_THREADS), S::TOTAL, stream, PAIR ? 2 : 1, ta, tb, tc, tx, tones, tbias, p);
}

// C[M,N] = act(alpha * A·B + bias) (+ residual)
//   a_mn = 0: A stored [M, K] (row stride lda);  a_mn = 1: A stored [K, M] (row stride lda)
//   b_mn = 0: B stored [N, K] (row stride ldb);  b_mn = 1: B stored [K, N] (row stride ldb)
// Alignment contract (checked): base pointers 16-byte aligned, lda/ldb multiples of 8 elements.
static int gemm_impl(const void* A, const void* B, void* C, void* aux, const void* bias, const void* residual, int M,
                     int N, int K, long lda, long ldb, long ldc, long ld_aux, long ld_res, int a_mn, int b_mn, int fmt,
                     int bias_fp32, int out_fp32, int act, int atomic_out, int splits, float alpha, int block_n,
                     int num_sms, void* stream_, int batch1, int batch2, const long* a_bs, const long* b_bs,
                     const long* c_bs) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) || (lda & 7) || (ldb & 7)) return -DL4J_ERR_BAD_ARG;
  if (splits < 1) splits = 1;
  if (splits > 1 && !(atomic_out && out_fp32)) return -DL4J_ERR_BAD_ARG;
  int dev = 0;
  cudaGetDevice(&dev);
  GemmParams p;
  p.M = M; p.N = N; p.K = K; p.ldc = ldc; p.ld_aux = ld_aux; p.ld_res = ld_res; p.C = C; p.aux = aux; p.bias = bias;
  // `act` carries two ids: bits 0-7 the forward activation applied to the result, bits 8-15 an activation whose derivative at
  // `residual` multiplies the result (then `residual` is not added); bit 16 applies ReLU after the residual
  p.residual = residual; p.bias_fp32 = bias_fp32; p.out_fp32 = out_fp32; p.act = act & 0xff; p.res_act = (act >> 8) & 0xff;
  p.relu_last = (act >> 16) & 1;
  if (p.res_act && (!residual || p.act || p.relu_last)) return -DL4J_ERR_BAD_ARG;
  p.atomic_out = atomic_out;
  p.splits = splits; p.fmt = fmt; p.alpha = alpha; p.status = dl4j_status_word(dev);
  p.batch1 = batch1; p.batch2 = batch2; p.c_stride_b1 = c_bs[0]; p.c_stride_b2 = c_bs[1];
  if ((a_bs[0] & 7) || (a_bs[1] & 7) || (b_bs[0] & 7) || (b_bs[1] & 7)) return -DL4J_ERR_BAD_ARG;
  const uint64_t nb1 = batch1, nb2 = batch2;
  const bool pair = block_n == GEMM_PAIR_TILE;
  if (block_n != 128 && block_n != 256) block_n = 256;
  CUtensorMap ta, tb;
  int r;
  if (!a_mn) r = encode_2d(&ta, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, BLOCK_K, BLOCK_M, nb1, nb2, a_bs[0] * 2, a_bs[1] * 2);
  else       r = encode_2d(&ta, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda * 2, 64, BLOCK_K, nb1, nb2, a_bs[0] * 2, a_bs[1] * 2);
  if (r) return r > 0 ? -1000 - r : r;
  if (!b_mn) r = encode_2d(&tb, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb * 2, BLOCK_K, (uint32_t)(pair ? 128 : block_n), nb1, nb2, b_bs[0] * 2, b_bs[1] * 2);
  else       r = encode_2d(&tb, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb * 2, 64, BLOCK_K, nb1, nb2, b_bs[0] * 2, b_bs[1] * 2);
  if (r) return r > 0 ? -1000 - r : r;
  // output maps: a box of 32 rows x 32 columns per epilogue warp (64 bytes a row, fp32 128)
  CUtensorMap tc, tx;
  memset(&tc, 0, sizeof(tc));
  memset(&tx, 0, sizeof(tx));
  const int esz = out_fp32 ? 4 : 2;
  p.tma_store = 0; p.tma_aux = 0;
  if (!(reinterpret_cast<uintptr_t>(C) & 15) && ((ldc * esz) % 16 == 0) && ((c_bs[0] * esz) % 16 == 0) && ((c_bs[1] * esz) % 16 == 0) &&
      (!aux || (!(reinterpret_cast<uintptr_t>(aux) & 15) && (ld_aux * 2) % 16 == 0))) {
    const bool slabs = atomic_out == 2;
    r = encode_2d(&tc, C, (uint64_t)N, (uint64_t)M, (uint64_t)ldc * esz, 32, 32, nb1, slabs ? (uint64_t)splits : nb2,
                  c_bs[0] * esz, slabs ? (uint64_t)M * ldc * esz : c_bs[1] * esz, out_fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                  out_fp32 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B);
    if (r == 0) p.tma_store = 1;
    if (r == 0 && aux) {
      r = encode_2d(&tx, aux, (uint64_t)N, (uint64_t)M, (uint64_t)ld_aux * 2, 32, 32, 1, 1, 0, 0, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                    CU_TENSOR_MAP_SWIZZLE_64B);
      if (r == 0) p.tma_aux = 1; else p.tma_store = 0;
    }
  }
  if (atomic_out == 2 && (!p.tma_store || batch1 != 1 || batch2 != 1)) return -DL4J_ERR_BAD_ARG;
  // bias on the tensor core: needs the bias in the operand format, 16-byte aligned, and alpha = 1 (the accumulator then
  // already holds A.B + bias); the epilogue's per-element broadcast of the bias competes with the MMA operand fetch for
  // the shared-memory path and costs a quarter of a short-K tile
  CUtensorMap tones, tbias;
  memset(&tones, 0, sizeof(tones));
  memset(&tbias, 0, sizeof(tbias));
  p.bias_mma = 0;
  if (bias && !bias_fp32 && alpha == 1.0f && splits == 1 && batch1 == 1 && batch2 == 1 && !(reinterpret_cast<uintptr_t>(bias) & 15)) {
    void* ones = nullptr;
    cudaError_t ce = fmt == 1 ? cudaGetSymbolAddress(&ones, g_ones_bf16) : cudaGetSymbolAddress(&ones, g_ones_f16);
    if (ce == cudaSuccess && encode_2d(&tones, ones, 128, 1, 256, 64, UMMA_K) == 0 &&
        encode_2d(&tbias, bias, (uint64_t)N, 1, (uint64_t)((N + 7) / 8 * 8) * 2, 64, UMMA_K) == 0)
      p.bias_mma = 1;
  }
  {
    const int tn = (N + block_n - 1) / block_n;
    p.raster_gn = tn < 16 ? tn : 16;
  }
  const int tile_m = pair ? 2 * BLOCK_M : BLOCK_M;
  const long tiles_l = (long)((M + tile_m - 1) / tile_m) * ((N + block_n - 1) / block_n) * splits * batch1 * batch2;
  if (tiles_l > 0x7fffffffL) return -DL4J_ERR_BAD_ARG;
  const int tiles = (int)tiles_l;
  if (num_sms <= 0) num_sms = 148;
  const bool full = p.aux || p.act > 1 || p.res_act;
  if (pair) {
    const int pairs = num_sms / 2 > 0 ? num_sms / 2 : 1, grid2 = 2 * (tiles < pairs ? tiles : pairs);
#define DL4J_GEMM_PAIR(AM, BM)                                                                                                   \
    if (a_mn == AM && b_mn == BM)                                                                                                \
      return full ? launch_gemm<256, AM != 0, BM != 0, true, true>(ta, tb, tc, tx, tones, tbias, p, grid2, dev, stream)    \
                  : launch_gemm<256, AM != 0, BM != 0, false, true>(ta, tb, tc, tx, tones, tbias, p, grid2, dev, stream);
    DL4J_GEMM_PAIR(0, 0) DL4J_GEMM_PAIR(0, 1) DL4J_GEMM_PAIR(1, 0) DL4J_GEMM_PAIR(1, 1)
#undef DL4J_GEMM_PAIR
    return -DL4J_ERR_BAD_ARG;
  }
  const int grid = tiles < num_sms ? tiles : num_sms;
#define DL4J_GEMM_CASE(BN, AM, BM)                                                                                              \
  if (block_n == BN && a_mn == AM && b_mn == BM)                                                                               \
    return full ? launch_gemm<BN, AM != 0, BM != 0, true>(ta, tb, tc, tx, tones, tbias, p, grid, dev, stream)                       \
                : launch_gemm<BN, AM != 0, BM != 0, false>(ta, tb, tc, tx, tones, tbias, p, grid, dev, stream);
  DL4J_GEMM_CASE(256, 0, 0) DL4J_GEMM_CASE(256, 0, 1) DL4J_GEMM_CASE(256, 1, 0) DL4J_GEMM_CASE(256, 1, 1)
  DL4J_GEMM_CASE(128, 0, 0) DL4J_GEMM_CASE(128, 0, 1) DL4J_GEMM_CASE(128, 1, 0) DL4J_GEMM_CASE(128, 1, 1)
#undef DL4J_GEMM_CASE
  return -DL4J_ERR_BAD_ARG;
}

// C[M,N] = act(alpha * A·B + bias) (+ residual)
//   a_mn = 0: A stored [M, K] (row stride lda);  a_mn = 1: A stored [K, M] (row stride lda)
//   b_mn = 0: B stored [N, K] (row stride ldb);  b_mn = 1: B stored [K, N] (row stride ldb)
// Alignment contract (checked): base pointers 16-byte aligned, lda/ldb multiples of 8 elements.
DL4J_API int dl4j_gemm(const void* A, const void* B, void* C, void* aux, const void* bias, const void* residual, int M,
                       int N, int K, long lda, long ldb, long ldc, long ld_aux, long ld_res, int a_mn, int b_mn, int fmt,
                       int bias_fp32, int out_fp32, int act, int atomic_out, int splits, float alpha, int block_n,
                       int num_sms, void* stream_) {
  const long z[2] = {0, 0};
  return gemm_impl(A, B, C, aux, bias, residual, M, N, K, lda, ldb, ldc, ld_aux, ld_res, a_mn, b_mn, fmt, bias_fp32, out_fp32,
                   act, atomic_out, splits, alpha, block_n, num_sms, stream_, 1, 1, z, z, z);
}

// out[m, n] = sum over s of part[s][m][n] in order, rounded once.  Memory-bound, and what it reads has just been written: 7 slabs of
// 2456 x 768 are 53 MB in L2.
template <typename T>
static __global__ void __launch_bounds__(256)
split_sum_kernel(const float* __restrict__ part, T* __restrict__ out, int M, int N, long ldo, int splits) {
  const long n4 = N / 4, total = (long)M * n4, slab = (long)M * N;
  for (long g = blockIdx.x * 256L + threadIdx.x; g < total; g += (long)gridDim.x * 256) {
    const long m = g / n4, n = (g - m * n4) * 4;
    const float* s = part + m * N + n;
    float4 a = __ldcs(reinterpret_cast<const float4*>(s));
#pragma unroll 8
    for (int i = 1; i < splits; ++i) {
      const float4 b = __ldcs(reinterpret_cast<const float4*>(s + i * slab));
      a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
    }
    T* o = out + m * ldo + n;
    o[0] = T(a.x); o[1] = T(a.y); o[2] = T(a.z); o[3] = T(a.w);
  }
}

// C[M, N] (16-bit, row pitch ldc) = A B with the reduction split: each split stores its fp32 partial result, one kernel adds them in
// order, so that the result does not depend on timing.  partial: [splits, M, N] fp32, 16-byte aligned, N a multiple of 4.
DL4J_API int dl4j_gemm_split(const void* A, const void* B, float* partial, void* C, int M, int N, int K, long lda, long ldb, long ldc,
                             int a_mn, int b_mn, int fmt, int splits, int num_sms, void* stream_) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (splits < 2 || N % 4 || (fmt != 0 && fmt != 1)) return -DL4J_ERR_BAD_ARG;
  const long z[2] = {0, 0};
  // pairs from 36 steps of K per CTA on, unless their rows are mostly padding, as everywhere
  const long pairs = num_sms > 1 ? num_sms / 2 : 74, tiles = (long)((M + 255) / 256) * ((N + 255) / 256) * splits;
  const long steps = (tiles + pairs - 1) / pairs * (((K + 63) / 64 + splits - 1) / splits);
  const int rc = gemm_impl(A, B, partial, nullptr, nullptr, nullptr, M, N, K, lda, ldb, N, 0, 0, a_mn, b_mn, fmt, 0, 1, 0, 2, splits, 1.0f,
                           steps >= 36 && (M + 255) / 256 * 8 <= (M + 127) / 128 * 5 ? GEMM_PAIR_TILE : 256, num_sms, stream_, 1, 1, z, z, z);
  if (rc) return rc;
  const long blocks = ((long)M * (N / 4) + 255) / 256;
  const int grid = (int)(blocks < 148 * 16 ? blocks : 148 * 16);
  cudaStream_t st = (cudaStream_t)stream_;
  if (fmt == 1) split_sum_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(partial, (__nv_bfloat16*)C, M, N, ldc, splits);
  else split_sum_kernel<__half><<<grid, 256, 0, st>>>(partial, (__half*)C, M, N, ldc, splits);
  return (int)cudaGetLastError();
}

// Batched form: batch index (b1, b2) with per-operand element strides {stride_b1, stride_b2} (multiples of 8 for A and B).
// Used for attention (batch = [heads, examples] over strided views of the fused QKV buffer) and batched_gemm.
DL4J_API int dl4j_gemm_batched(const void* A, const void* B, void* C, int M, int N, int K, long lda, long ldb, long ldc,
                               int a_mn, int b_mn, int fmt, int out_fp32, float alpha, int block_n, int num_sms,
                               int batch1, int batch2, const long* a_bs, const long* b_bs, const long* c_bs, void* stream_) {
  if (batch1 < 1 || batch2 < 1) return 0;
  return gemm_impl(A, B, C, nullptr, nullptr, nullptr, M, N, K, lda, ldb, ldc, 0, 0, a_mn, b_mn, fmt, 0, out_fp32, 0, 0, 1,
                   alpha, block_n, num_sms, stream_, batch1, batch2, a_bs, b_bs, c_bs);
}
