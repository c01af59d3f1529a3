// Persistent LSTM sequence kernels for batches that can be split over the chip: the batch rows fall into groups of R <= 48, and every
// group has its own n / 16 CTAs, so that 16 units' recurrent weights stay in shared memory as in lstm_seq.cu while a CTA takes in only
// its group's rows of h (dz) per step.
//
// What bounds a step is the hand-over of h (dz) between the CTAs, a chain of L2 round trips.  Three things shorten it here:
//  * The values carry their own "written" mark.  The buffer is filled with 0xFFFFFFFF words before the launch, a word that no pair of
//    converted bf16 values can be (a NaN converts to 0x7FFF), and a reader repeats its loads until no mark is left.  No release, no
//    counter, no acquire: one store and one load are on the path instead of store, release (0.7 us), arrival and poll (1.1 us), load.
//    Writers store 32-bit elements with st.relaxed.gpu, readers load them with ld.relaxed.gpu; every element validates itself, so
//    nothing depends on the order in which the elements of a vector, or two vectors, become visible.
//  * The weights are the M operand (64 rows) and the batch rows the N operand (R columns).  An instruction's time is its operand bytes
//    out of shared memory: 64 x 32 B + R x 32 B instead of 128 x 32 B (half of them padding) + 64 x 32 B.
//  * R rows instead of the whole batch: half the L2 -> SM stream at n = 1024, batch 64 (two groups of 64 CTAs), an eighth at n = 256.
//
// Warps 0-3: epilogue; 4-6: MMA issue (one accumulator each, k-blocks me, me + 3, ...); 7-22: loaders, half a 64-column k-block each at a
// time.  They start to ask when their own CTA has published: the others do so at the same time, and a round of answers that are not
// there yet costs as much of the L2 -> SM stream as the values (asking at once: 4.22 / 6.65 us).
// Per step, 50 steps, forward / backward with the weight gradient's product, us, ring kernels of lstm_seq.cu -> here:
//   batch 64 n 1024  5.92 / 8.67 -> 4.00 / 5.88      batch 64 n 512  4.69 / 6.94 -> 2.56 / 3.83      batch 64 n 256  4.12 / 6.30 -> 2.01 / 3.24
//   batch 50 n  768  5.27 / 7.50 -> 2.97 / 4.55      batch 16 n 128  3.35 / 4.46 -> 2.01 / 2.68
// A forward step of n 1024 after its own publication: 2.1 - 2.3 until the others' values are in shared memory, 2.8 products done, 3.0 sums
// out of tensor memory, 3.3 published.
#include "lstm_common.cuh"

namespace dl4j {

constexpr int SP_M = 64;                       // MMA M: weight rows
constexpr int SP_ISS = 3;                      // one thread issues per ~64 clocks, an instruction takes 24 (one issuer: 5.3 us a step)
constexpr int SP_LOADERS = 16;
constexpr int SP_LOAD0 = 4 + SP_ISS;
constexpr int SP_THREADS = 32 * (SP_LOAD0 + SP_LOADERS);
constexpr int SP_MAX_ROWS = 48;
constexpr int SP_MAX_KB = 19;                  // n <= 1216
constexpr int SP_W_KB = SP_M * LS_BK * 2;      // 8 KB of resident weights per k-block
constexpr int SP_XP = SP_M + 4;                // pitch of the forward transposition buffer [R][68]: 4 x (2 pitch) = 8 banks apart
constexpr int SP_TMEM = 256;                   // three accumulators, 64 columns apart

struct LstmSplitFwd {
  const __nv_bfloat16* zx;   // [T, mb, 4n]
  const __nv_bfloat16* rw;   // [4n, n]
  __nv_bfloat16* h_all;      // [T + 1, mb, n]; slot 0 holds h_0, the others are filled with marks
  const float* c0;           // [mb, n]
  float* cs;                 // [T, mb, n]
  __nv_bfloat16* gates;      // [T, mb, 4n]
  int T, mb, n, reverse, rows;
  int* status;
  long long* trace;
};
struct LstmSplitBwd {
  const __nv_bfloat16* dout;   // [T, mb, n]
  const __nv_bfloat16* gates;  // [T, mb, 4n]
  const float* cs;             // [T, mb, n]
  const float* c0;             // [mb, n]
  const __nv_bfloat16* rwt;    // [n, 4n]
  const float* dc_last;        // [mb, n] or null
  __nv_bfloat16* dzx;          // [T, mb, 4n], filled with marks
  __nv_bfloat16* dh0;          // [mb, n] or null
  float* dc0;                  // [mb, n] or null
  int T, mb, n, reverse, rows;
  int* status;
  long long* trace;
};

__device__ __forceinline__ uint4 ld_relaxed_v4(const void* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_v2(void* p, uint32_t a, uint32_t b) {
  asm volatile("st.relaxed.gpu.global.v2.b32 [%0], {%1, %2};" ::"l"(p), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ bool has_mark(const uint4& v) { return max(max(v.x, v.y), max(v.z, v.w)) == 0xffffffffu; }
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float2 unpack2(uint32_t u) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u)); }
__device__ __forceinline__ void unpack4(const uint2& u, float (&o)[4]) {
  const float2 a = unpack2(u.x), b = unpack2(u.y);
  o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
}

// 16 lanes x 32 columns of an M = 64 accumulator: lane l receives rows l / 4 (r[4 j], r[4 j + 1]) and l / 4 + 8 (r[4 j + 2], r[4 j + 3]),
// columns 8 j + 2 (l % 4) and the next
__device__ __forceinline__ void tmem_ld_16x32(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ void sp_stamp(long long* trace, int s, int slot) {
  if (trace != nullptr && blockIdx.x == gridDim.x / 2 && blockIdx.y == 0) trace[s * 32 + slot] = clock64();
}

// The loaders' share of one step.  A unit is half a k-block: R / 2 rows x 128 bytes, L 16-byte loads per lane at most; warp w takes units w
// and w + 16 (and 32 further on), so that the first half of the k-blocks is complete first and the tensor core starts under the rest of
// the stream.  All loads of both units are issued at once; each unit is handed on with one proxy fence (0.15 us).  No index is divided
// here: the addresses were most of a step's instructions with units numbered by rows.  With `poll`, words that still carry the mark are
// read again until they are there; false when that exceeds the bound.
template <int L>
__device__ __forceinline__ bool sp_load(const __nv_bfloat16* src, long stride, int rows_valid, int R, int kblocks, uint8_t* a_smem, uint64_t* full,
                                        int w, bool poll, int* status) {
  const int lane = threadIdx.x & 31, chunk = lane & 7, r0 = lane >> 3, half = R >> 1;
  bool ok = true;
  for (int u = w; u < 2 * kblocks && ok; u += 2 * SP_LOADERS) {
    uint4 v[2][L];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int kb = (u + k * SP_LOADERS) >> 1, row = (u & 1) * half + r0;      // SP_LOADERS is even: both units are the same half
      const char* p = reinterpret_cast<const char*>(src + (long)row * stride + kb * LS_BK) + chunk * 16;
#pragma unroll
      for (int i = 0; i < L; ++i) {
        v[k][i] = make_uint4(0u, 0u, 0u, 0u);
        if (kb < kblocks && r0 + 4 * i < half && row + 4 * i < rows_valid) v[k][i] = ld_relaxed_v4(p + (long)(4 * i) * stride * 2);
      }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int kb = (u + k * SP_LOADERS) >> 1, row = (u & 1) * half + r0;
      if (kb < kblocks && ok) {                        // uniform over the warp
        if (poll) {
          const char* p = reinterpret_cast<const char*>(src + (long)row * stride + kb * LS_BK) + chunk * 16;
          uint32_t spins = 0;
          long long t0 = 0;
          while (true) {
            bool wait = false;
#pragma unroll
            for (int i = 0; i < L; ++i)
              if (has_mark(v[k][i])) { v[k][i] = ld_relaxed_v4(p + (long)(4 * i) * stride * 2); wait = true; }
            if (!wait) break;
            if ((++spins & 0xff) == 0) {
              if (t0 == 0) t0 = clock64();
              if (clock64() - t0 > 4000000000LL || *((volatile int*)status) != 0) {
                atomicCAS(status, 0, DL4J_ERR_TIMEOUT_PEER);
                ok = false;
                break;
              }
            }
          }
        }
        uint8_t* dst = a_smem + kb * R * 128 + row * 128;
#pragma unroll
        for (int i = 0; i < L; ++i)
          if (r0 + 4 * i < half && row + 4 * i < rows_valid) *reinterpret_cast<uint4*>(dst + i * 512 + ((chunk ^ ((row + 4 * i) & 7)) << 4)) = v[k][i];
        fence_proxy_async_smem();
        ok = __all_sync(0xffffffffu, ok);
        if (ok && lane == 0) mbar_arrive(&full[kb]);
      }
    }
  }
  return ok;
}

// Barriers and tensor memory of one CTA, behind the operand tiles.
struct SpBars {
  uint64_t full[SP_MAX_KB];
  uint64_t acc_full, acc_empty, pub;
  uint64_t x_full[2];
  uint32_t tmem;
};

__device__ __forceinline__ void sp_init(SpBars* b, int kblocks, int warp) {
  if (threadIdx.x == 0) {
    for (int i = 0; i < kblocks; ++i) mbar_init(&b->full[i], 2);                      // one arrival per half
    mbar_init(&b->acc_full, (uint32_t)min(SP_ISS, kblocks));      // one commit per issuer that has k-blocks
    mbar_init(&b->acc_empty, 4);
    mbar_init(&b->pub, 128);
    mbar_init(&b->x_full[0], 1);
    mbar_init(&b->x_full[1], 1);
    mbar_fence_init();
  }
  if (warp == 4) {
    tmem_alloc(&b->tmem, SP_TMEM);
    tmem_relinquish();
  }
}

// All rounds of one MMA-issuing thread.
__device__ __forceinline__ void sp_issue(SpBars* bars, uint32_t tmem_base, int me, int rounds, int kblocks, int rows, const uint8_t* w_smem,
                                         const uint8_t* a_smem, int* status) {
  const uint32_t idesc = make_idesc(1, 0, 0, SP_M, rows);
  const uint32_t acc = tmem_base + (uint32_t)(me * 64);
  bool ok = me < kblocks;
  for (int s = 0; s < rounds && ok; ++s) {
    if (!mbar_wait_bounded(&bars->acc_empty, (uint32_t)((s & 1) ^ 1), status, DL4J_ERR_TIMEOUT_MMA)) break;
    tc_fence_after();
    for (int kb = me; kb < kblocks; kb += SP_ISS) {
      if (!mbar_wait_bounded(&bars->full[kb], (uint32_t)(s & 1), status, DL4J_ERR_TIMEOUT_MMA)) { ok = false; break; }
      tc_fence_after();
      const uint64_t da = make_smem_desc_sw128(smem_u32(w_smem + kb * SP_W_KB), 16, 1024);
      const uint64_t db = make_smem_desc_sw128(smem_u32(a_smem + kb * rows * 128), 16, 1024);
#pragma unroll
      for (int k = 0; k < LS_BK / 16; ++k)
        umma_f16(acc, da + ((uint64_t)(k * 32) >> 4), db + ((uint64_t)(k * 32) >> 4), idesc, (kb > me || k > 0) ? 1u : 0u);
    }
    if (ok) umma_commit(&bars->acc_full);
  }
}

// The issuers' partial accumulators, 32 columns from `col` on, summed.
__device__ __forceinline__ void sp_read_acc(uint32_t tmem_base, int q, int col, int naccs, float (&v)[16]) {
  const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + col;
#pragma unroll
  for (int j = 0; j < SP_ISS; ++j)
    if (j < naccs) {
      uint32_t r[16];
      tmem_ld_16x32(taddr + j * 64, r);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = j ? v[i] + __uint_as_float(r[i]) : __uint_as_float(r[i]);
    }
}

// ITEMS: (row, four units) pairs per epilogue thread: 1 up to 32 rows, 2 up to 48
template <int ITEMS>
__global__ void __launch_bounds__(SP_THREADS, 1) lstm_split_fwd_kernel(const LstmSplitFwd p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int kblocks = p.n / LS_BK, R = p.rows;
  uint8_t* w_smem = smem;
  uint8_t* a_smem = w_smem + kblocks * SP_W_KB;
  float* xbuf = reinterpret_cast<float*>(a_smem + kblocks * R * 128);        // [R][SP_XP] accumulators, one batch row after another
  SpBars* bars = reinterpret_cast<SpBars*>(xbuf + R * SP_XP);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int unit0 = blockIdx.x * LS_UNITS, b0 = blockIdx.y * R;
  const int rows_valid = min(R, p.mb - b0);
  const long n4 = 4L * p.n;

  sp_init(bars, kblocks, warp);
  // resident weights: row 16 g + u of the tile is gate g of unit u
  const int cpr = p.n / 8;
  for (int i = threadIdx.x; i < SP_M * cpr; i += SP_THREADS) {
    const int row = i / cpr, col = i % cpr;
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(p.rw + ((long)(row >> 4) * p.n + unit0 + (row & 15)) * p.n) + col);
    *reinterpret_cast<uint4*>(w_smem + (col >> 3) * SP_W_KB + row * 128 + (((col & 7) ^ (row & 7)) << 4)) = v;
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem;

  if (warp >= SP_LOAD0) {
    bool ok = true;
    for (int s = 0; s < p.T && ok; ++s) {
      if (s > 0) {
        // the previous step's MMAs have read the tiles, and this CTA has published
        if (!mbar_wait_bounded(&bars->acc_full, (uint32_t)((s - 1) & 1), p.status, DL4J_ERR_TIMEOUT_PRODUCER)) ok = false;
        if (ok && !mbar_wait_bounded(&bars->pub, (uint32_t)((s - 1) & 1), p.status, DL4J_ERR_TIMEOUT_PRODUCER)) ok = false;
        ok = __all_sync(0xffffffffu, ok);
      }
      if (ok)
        ok = sp_load<ITEMS == 1 ? 4 : 6>(p.h_all + ((long)s * p.mb + b0) * p.n, p.n, rows_valid, R, kblocks, a_smem, bars->full, warp - SP_LOAD0, s > 0,
                                         p.status);
      if (lane == 0) sp_stamp(p.trace, s, 2 + warp - SP_LOAD0);
    }
  } else if (warp >= 4) {
    if (elect_one()) sp_issue(bars, tmem_base, warp - 4, p.T, kblocks, R, w_smem, a_smem, p.status);
  } else {
    const int naccs = min(SP_ISS, kblocks);
    int row[ITEMS];
    float c[ITEMS][4];
    const int u = unit0 + (threadIdx.x & 3) * 4;               // first of this thread's four units
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      row[i] = (int)(threadIdx.x >> 2) + 32 * i;
      if (row[i] < rows_valid) {
        const float4 v = *reinterpret_cast<const float4*>(p.c0 + (long)(b0 + row[i]) * p.n + u);
        c[i][0] = v.x; c[i][1] = v.y; c[i][2] = v.z; c[i][3] = v.w;
      }
    }
    bool ok = true;
    for (int s = 0; s < p.T; ++s) {                            // a failed wait skips the work, never the barriers
      const int t = p.reverse ? p.T - 1 - s : s;
      uint2 zraw[ITEMS][4];                                    // input contribution, fetched before the accumulators are ready
#pragma unroll
      for (int i = 0; i < ITEMS; ++i)
        if (row[i] < rows_valid) {
          const __nv_bfloat16* z = p.zx + ((long)t * p.mb + b0 + row[i]) * n4 + u;
#pragma unroll
          for (int g = 0; g < 4; ++g) zraw[i][g] = __ldg(reinterpret_cast<const uint2*>(z + (long)g * p.n));
        }
      if (ok && !mbar_wait_bounded(&bars->acc_full, (uint32_t)(s & 1), p.status, DL4J_ERR_TIMEOUT_EPILOGUE)) ok = false;
      ok = __all_sync(0xffffffffu, ok);
      if (threadIdx.x == 0) sp_stamp(p.trace, s, 19);
      tc_fence_after();
#pragma unroll
      for (int h = 0; h < ITEMS; ++h) {
        if (!ok) break;                                        // uniform over the warp
        float v[16];
        sp_read_acc(tmem_base, warp, 32 * h, naccs, v);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int b = 32 * h + 8 * j + 2 * (lane & 3);
          if (32 * h + 8 * j < R) {
            float* x = xbuf + b * SP_XP + warp * 16 + (lane >> 2);
            x[0] = v[4 * j]; x[SP_XP] = v[4 * j + 1]; x[8] = v[4 * j + 2]; x[SP_XP + 8] = v[4 * j + 3];
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->acc_empty);            // accumulators drained: the next step's MMAs may overwrite them
      epilogue_bar_sync();
      if (threadIdx.x == 0) sp_stamp(p.trace, s, 20);
      float a[ITEMS][4], f[ITEMS][4], o[ITEMS][4], g[ITEMS][4];
#pragma unroll
      for (int i = 0; i < ITEMS; ++i)
        if (ok && row[i] < rows_valid) {
          const float4* x = reinterpret_cast<const float4*>(xbuf + row[i] * SP_XP) + (threadIdx.x & 3);
          const float4 xa = x[0], xf = x[4], xo = x[8], xg = x[12];
          unpack4(zraw[i][0], a[i]); unpack4(zraw[i][1], f[i]); unpack4(zraw[i][2], o[i]); unpack4(zraw[i][3], g[i]);
          const float ra[4] = {xa.x, xa.y, xa.z, xa.w}, rf[4] = {xf.x, xf.y, xf.z, xf.w}, ro[4] = {xo.x, xo.y, xo.z, xo.w},
                      rg[4] = {xg.x, xg.y, xg.z, xg.w};
          float h[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            a[i][k] = tanh_fast(a[i][k] + ra[k]);
            f[i][k] = sigm_fast(f[i][k] + rf[k]);
            o[i][k] = sigm_fast(o[i][k] + ro[k]);
            g[i][k] = sigm_fast(g[i][k] + rg[k]);
            c[i][k] = fmaf(f[i][k], c[i][k], g[i][k] * a[i][k]);
            h[k] = o[i][k] * tanh_fast(c[i][k]);
          }
          // h_t is what the other CTAs wait for: publish it first, then write what only the backward pass reads
          st_relaxed_v2(p.h_all + ((long)(s + 1) * p.mb + b0 + row[i]) * p.n + u, pack2(h[0], h[1]), pack2(h[2], h[3]));
        }
      mbar_arrive(&bars->pub);
      if (threadIdx.x == 0) sp_stamp(p.trace, s, 21);
#pragma unroll
      for (int i = 0; i < ITEMS; ++i)
        if (ok && row[i] < rows_valid) {
          __nv_bfloat16* gd = p.gates + ((long)t * p.mb + b0 + row[i]) * n4 + u;
          *reinterpret_cast<uint2*>(gd) = make_uint2(pack2(a[i][0], a[i][1]), pack2(a[i][2], a[i][3]));
          *reinterpret_cast<uint2*>(gd + p.n) = make_uint2(pack2(f[i][0], f[i][1]), pack2(f[i][2], f[i][3]));
          *reinterpret_cast<uint2*>(gd + 2L * p.n) = make_uint2(pack2(o[i][0], o[i][1]), pack2(o[i][2], o[i][3]));
          *reinterpret_cast<uint2*>(gd + 3L * p.n) = make_uint2(pack2(g[i][0], g[i][1]), pack2(g[i][2], g[i][3]));
          *reinterpret_cast<float4*>(p.cs + ((long)t * p.mb + b0 + row[i]) * p.n + u) = make_float4(c[i][0], c[i][1], c[i][2], c[i][3]);
        }
      epilogue_bar_sync();                                     // xbuf has been read
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 4) {
    tc_fence_after();
    tmem_dealloc(tmem_base, SP_TMEM);
  }
}

// ----------------------------------------------------------------------------- backward
__device__ __forceinline__ void st_async_v4(uint32_t dst_cluster, float a, float b, float c, float d, uint32_t bar_cluster) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst_cluster), "f"(a), "f"(b),
               "f"(c), "f"(d), "r"(bar_cluster)
               : "memory");
}

// Four CTAs of a cluster own 64 units together.  CTA `rank` keeps RW[those 64 units, gate `rank`'s n columns], takes in that gate's
// dz of its rows and forms the partial sums of dh for all 64 units; quadrant q of the accumulator holds the 16 units that CTA q
// finishes and is sent there, 16 bytes a lane as tcgen05.ld hands them out (st.async, counted on the receiver's mbarrier; with 8 bytes
// in row order the exchange took 0.98 us instead of 0.61).  Walks the steps in reverse; one more round after step 0 yields the gradient
// of the initial hidden state.
// The receive buffer has two halves: a CTA sends round r only after it has read every dz of round r - 1, which the receiver stored
// after it had read its sums of round r - 1.
template <int ITEMS>
__global__ void __launch_bounds__(SP_THREADS, 1) lstm_split_bwd_kernel(const LstmSplitBwd p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int kblocks = p.n / LS_BK, R = p.rows;
  uint8_t* w_smem = smem;
  uint8_t* a_smem = w_smem + kblocks * SP_W_KB;
  float* xbuf = reinterpret_cast<float*>(a_smem + kblocks * R * 128);        // [2][4 senders][R / 8][32 lanes][4], as tcgen05.ld hands them out
  SpBars* bars = reinterpret_cast<SpBars*>(xbuf + 2 * 4 * 16 * R);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();
  const int unit0 = blockIdx.x * LS_UNITS, grp_unit0 = (int)(blockIdx.x / 4) * SP_M, b0 = blockIdx.y * R;
  const int rows_valid = min(R, p.mb - b0);
  const long n4 = 4L * p.n;
  const int rounds = p.T - 1 + (p.dh0 ? 1 : 0);

  sp_init(bars, kblocks, warp);
  const int cpr = p.n / 8;
  for (int i = threadIdx.x; i < SP_M * cpr; i += SP_THREADS) {
    const int row = i / cpr, col = i % cpr;
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(p.rwt + (long)(grp_unit0 + row) * n4 + (long)rank * p.n) + col);
    *reinterpret_cast<uint4*>(w_smem + (col >> 3) * SP_W_KB + row * 128 + (((col & 7) ^ (row & 7)) << 4)) = v;
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                          // the peers' barriers exist before anything is sent to them
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem;

  if (warp >= SP_LOAD0) {
    bool ok = true;
    for (int r = 0; r < rounds && ok; ++r) {
      const int s_src = p.T - 1 - r;                           // step whose dz feeds this round
      const int t_src = p.reverse ? p.T - 1 - s_src : s_src;
      if (r > 0 && !mbar_wait_bounded(&bars->acc_full, (uint32_t)((r - 1) & 1), p.status, DL4J_ERR_TIMEOUT_PRODUCER)) ok = false;
      if (ok && !mbar_wait_bounded(&bars->pub, (uint32_t)(r & 1), p.status, DL4J_ERR_TIMEOUT_PRODUCER)) ok = false;
      ok = __all_sync(0xffffffffu, ok);
      if (ok)
        ok = sp_load<ITEMS == 1 ? 4 : 6>(p.dzx + ((long)t_src * p.mb + b0) * n4 + (long)rank * p.n, n4, rows_valid, R, kblocks, a_smem, bars->full,
                                         warp - SP_LOAD0, true, p.status);
      if (lane == 0) sp_stamp(p.trace, r, 2 + warp - SP_LOAD0);
    }
  } else if (warp >= 4) {
    if (elect_one()) sp_issue(bars, tmem_base, warp - 4, rounds, kblocks, R, w_smem, a_smem, p.status);
  } else {
    const int naccs = min(SP_ISS, kblocks);
    int row[ITEMS];
    float dc[ITEMS][4];
    const int uq = threadIdx.x & 3, u = unit0 + uq * 4;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      row[i] = (int)(threadIdx.x >> 2) + 32 * i;
#pragma unroll
      for (int k = 0; k < 4; ++k) dc[i][k] = 0.f;
      if (row[i] < rows_valid && p.dc_last) {
        const float4 v = *reinterpret_cast<const float4*>(p.dc_last + (long)(b0 + row[i]) * p.n + u);
        dc[i][0] = v.x; dc[i][1] = v.y; dc[i][2] = v.z; dc[i][3] = v.w;
      }
    }
    bool ok = true;
    for (int s = p.T - 1; s >= (p.dh0 ? -1 : 0) && ok; --s) {
      const int r = p.T - 2 - s;                               // MMA round that produced this step's recurrent gradient (none for T - 1)
      const int t = p.reverse ? p.T - 1 - s : s;
      uint2 graw[ITEMS][4], draw[ITEMS];
      float4 ct[ITEMS], cp[ITEMS];
      if (s >= 0) {
        const int tp = p.reverse ? t + 1 : t - 1;
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
          if (row[i] < rows_valid) {
            const long b = b0 + row[i];
            const __nv_bfloat16* gr = p.gates + ((long)t * p.mb + b) * n4 + u;
#pragma unroll
            for (int g = 0; g < 4; ++g) graw[i][g] = __ldg(reinterpret_cast<const uint2*>(gr + (long)g * p.n));
            draw[i] = __ldg(reinterpret_cast<const uint2*>(p.dout + ((long)t * p.mb + b) * p.n + u));
            ct[i] = __ldg(reinterpret_cast<const float4*>(p.cs + ((long)t * p.mb + b) * p.n + u));
            cp[i] = __ldg(reinterpret_cast<const float4*>((s > 0 ? p.cs + ((long)tp * p.mb + b) * p.n : p.c0 + b * p.n) + u));
          }
      }
      float dhr[ITEMS][4];
#pragma unroll
      for (int i = 0; i < ITEMS; ++i)
#pragma unroll
        for (int k = 0; k < 4; ++k) dhr[i][k] = 0.f;
      if (r >= 0) {
        const int par = r & 1;
        if (threadIdx.x == 0) mbar_expect_tx(&bars->x_full[par], (uint32_t)(4 * 16 * 4 * R));
        if (!mbar_wait_bounded(&bars->acc_full, (uint32_t)(r & 1), p.status, DL4J_ERR_TIMEOUT_EPILOGUE)) ok = false;
        ok = __all_sync(0xffffffffu, ok);
        if (threadIdx.x == 0) sp_stamp(p.trace, r, 19);
        tc_fence_after();
        const uint32_t dst0 = mapa_cluster(smem_u32(xbuf + (par * 4 + rank) * 16 * R + lane * 4), (uint32_t)warp);
        const uint32_t bar = mapa_cluster(smem_u32(&bars->x_full[par]), (uint32_t)warp);
#pragma unroll
        for (int h = 0; h < ITEMS; ++h) {
          float v[16];
          sp_read_acc(tmem_base, warp, 32 * h, naccs, v);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (32 * h + 8 * j < R && ok) st_async_v4(dst0 + (uint32_t)(4 * h + j) * 512u, v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3], bar);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->acc_empty);
        if (threadIdx.x == 0) sp_stamp(p.trace, r, 20);
        if (ok && !mbar_wait_bounded_cluster(&bars->x_full[par], (uint32_t)((r >> 1) & 1), p.status, DL4J_ERR_TIMEOUT_PEER)) ok = false;
        if (threadIdx.x == 0) sp_stamp(p.trace, r, 22);
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
          if (row[i] < rows_valid) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              // row b of unit m sits with lane 4 (m % 8) + b % 8 / 2, in element 2 (m / 8) + b % 2
              const float* x = xbuf + (par * 4 + q) * 16 * R + (row[i] >> 3) * 128 + ((uq & 1) * 16 + ((row[i] & 7) >> 1)) * 4 + (uq & 2) + (row[i] & 1);
#pragma unroll
              for (int k = 0; k < 4; ++k) dhr[i][k] += x[k * 16];
            }
          }
      }
      ok = __all_sync(0xffffffffu, ok);
      if (s < 0) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
          if (ok && row[i] < rows_valid)
            *reinterpret_cast<uint2*>(p.dh0 + (long)(b0 + row[i]) * p.n + u) = make_uint2(pack2(dhr[i][0], dhr[i][1]), pack2(dhr[i][2], dhr[i][3]));
        break;
      }
#pragma unroll
      for (int i = 0; i < ITEMS; ++i)
        if (ok && row[i] < rows_valid) {
          float ga[4], gf[4], go[4], gg[4], dh[4];
          unpack4(graw[i][0], ga); unpack4(graw[i][1], gf); unpack4(graw[i][2], go); unpack4(graw[i][3], gg); unpack4(draw[i], dh);
          const float c_[4] = {ct[i].x, ct[i].y, ct[i].z, ct[i].w}, cp_[4] = {cp[i].x, cp[i].y, cp[i].z, cp[i].w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float a = ga[k], f = gf[k], o = go[k], g = gg[k];
            const float dhv = dh[k] + dhr[i][k];
            const float tc = tanh_fast(c_[k]);
            const float dcv = dc[i][k] + dhv * o * (1.f - tc * tc);
            ga[k] = dcv * g * (1.f - a * a);
            gf[k] = dcv * cp_[k] * f * (1.f - f);
            go[k] = dhv * tc * o * (1.f - o);
            gg[k] = dcv * a * g * (1.f - g);
            dc[i][k] = dcv * f;
          }
          __nv_bfloat16* d = p.dzx + ((long)t * p.mb + b0 + row[i]) * n4 + u;
          st_relaxed_v2(d, pack2(ga[0], ga[1]), pack2(ga[2], ga[3]));
          st_relaxed_v2(d + p.n, pack2(gf[0], gf[1]), pack2(gf[2], gf[3]));
          st_relaxed_v2(d + 2L * p.n, pack2(go[0], go[1]), pack2(go[2], go[3]));
          st_relaxed_v2(d + 3L * p.n, pack2(gg[0], gg[1]), pack2(gg[2], gg[3]));
        }
      mbar_arrive(&bars->pub);
      if (threadIdx.x == 0 && r >= 0) sp_stamp(p.trace, r, 21);
    }
    if (p.dc0) {
#pragma unroll
      for (int i = 0; i < ITEMS; ++i)
        if (row[i] < rows_valid)
          *reinterpret_cast<float4*>(p.dc0 + (long)(b0 + row[i]) * p.n + u) = make_float4(dc[i][0], dc[i][1], dc[i][2], dc[i][3]);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 4) {
    tc_fence_after();
    tmem_dealloc(tmem_base, SP_TMEM);
  }
  cluster_sync_all();                                          // no CTA leaves while another may still write into it
}

}  // namespace dl4j

using namespace dl4j;

// Rows per group: the fewest (a multiple of 8, the MMA's N) with which all groups' CTAs are on the chip at once; 0: not covered.
static int sp_rows(int mb, int n, int max_ctas) {
  const int groups = max_ctas / (n / LS_UNITS);
  if (groups < 1) return 0;
  const int rows = ((mb + groups - 1) / groups + 7) / 8 * 8;
  return rows <= SP_MAX_ROWS ? rows : 0;
}
static size_t sp_smem(int n, int rows, bool bwd) {
  const size_t s = 1024 + (size_t)(n / LS_BK) * (SP_W_KB + rows * 128) + (bwd ? (size_t)2 * 4 * 16 * rows : (size_t)rows * SP_XP) * 4 + sizeof(SpBars);
  return s <= 227 * 1024 ? s : 0;
}
static bool sp_aligned(const void* p) { return ((uintptr_t)p & 15) == 0; }

// 1: not covered here; otherwise a CUDA error code (0: launched).  Arguments as dl4j_lstm_seq_fwd.
int dl4j_lstm_split_fwd(const void* zx, const void* rw, void* h_all, const float* c0, float* cs, void* gates, int T, int mb, int n, int reverse,
                        int sms, int* status, long long* trace, cudaStream_t stream) {
  const int rows = sp_rows(mb, n, sms);
  const size_t smem = rows ? sp_smem(n, rows, false) : 0;
  if (!smem || n / LS_BK > SP_MAX_KB || !(sp_aligned(zx) && sp_aligned(rw) && sp_aligned(h_all) && sp_aligned(c0) && sp_aligned(cs) && sp_aligned(gates)))
    return 1;
  LstmSplitFwd p;
  p.zx = reinterpret_cast<const __nv_bfloat16*>(zx);
  p.rw = reinterpret_cast<const __nv_bfloat16*>(rw);
  p.h_all = reinterpret_cast<__nv_bfloat16*>(h_all);
  p.c0 = c0; p.cs = cs;
  p.gates = reinterpret_cast<__nv_bfloat16*>(gates);
  p.T = T; p.mb = mb; p.n = n; p.reverse = reverse; p.rows = rows;
  p.status = status; p.trace = trace;
  void* kern = rows <= 32 ? (void*)lstm_split_fwd_kernel<1> : (void*)lstm_split_fwd_kernel<2>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  e = cudaMemsetAsync(p.h_all + (size_t)mb * n, 0xff, (size_t)T * mb * n * 2, stream);
  if (e != cudaSuccess) return (int)e;
  void* args[] = {(void*)&p};
  return (int)cudaLaunchCooperativeKernel(kern, dim3(n / LS_UNITS, (mb + rows - 1) / rows), dim3(SP_THREADS), args, smem, stream);
}

int dl4j_lstm_split_bwd(const void* dout, const void* gates, const float* cs, const float* c0, const void* rwt, void* dzx, const float* dc_last,
                        void* dh0, float* dc0, int T, int mb, int n, int reverse, int sms, int* status, long long* trace, cudaStream_t stream) {
  if (n / LS_BK > SP_MAX_KB || !(sp_aligned(dout) && sp_aligned(gates) && sp_aligned(cs) && sp_aligned(c0) && sp_aligned(rwt) && sp_aligned(dzx) &&
                                 sp_aligned(dc_last) && sp_aligned(dh0) && sp_aligned(dc0)))
    return 1;
  LstmSplitBwd p;
  p.dout = reinterpret_cast<const __nv_bfloat16*>(dout);
  p.gates = reinterpret_cast<const __nv_bfloat16*>(gates);
  p.cs = cs; p.c0 = c0;
  p.rwt = reinterpret_cast<const __nv_bfloat16*>(rwt);
  p.dc_last = dc_last;
  p.dzx = reinterpret_cast<__nv_bfloat16*>(dzx);
  p.dh0 = reinterpret_cast<__nv_bfloat16*>(dh0);
  p.dc0 = dc0;
  p.T = T; p.mb = mb; p.n = n; p.reverse = reverse;
  p.status = status; p.trace = trace;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = 4; attrs[0].val.clusterDim.y = 1; attrs[0].val.clusterDim.z = 1;
  attrs[1].id = cudaLaunchAttributeCooperative;
  attrs[1].val.cooperative = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(SP_THREADS); cfg.stream = stream; cfg.attrs = attrs; cfg.numAttrs = 2;
  // clusters of four do not tile every GPC: ask how many fit, and take fewer groups until they do
  int ctas = sms;
  for (int tries = 0; tries < 4; ++tries) {
    const int rows = sp_rows(mb, n, ctas);
    const size_t smem = rows ? sp_smem(n, rows, true) : 0;
    if (!smem) return 1;
    void* kern = rows <= 32 ? (void*)lstm_split_bwd_kernel<1> : (void*)lstm_split_bwd_kernel<2>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    const int groups = (mb + rows - 1) / rows;
    cfg.gridDim = dim3(n / LS_UNITS, groups);
    cfg.dynamicSmemBytes = smem;
    int clusters = 0;
    e = cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg);
    if (e != cudaSuccess) return (int)e;
    if (clusters * 4 < groups * (n / LS_UNITS)) { ctas = min(ctas - 1, clusters * 4); continue; }
    p.rows = rows;
    e = cudaMemsetAsync(dzx, 0xff, (size_t)T * mb * 4 * n * 2, stream);
    if (e != cudaSuccess) return (int)e;
    void* args[] = {(void*)&p};
    return (int)cudaLaunchKernelExC(&cfg, kern, args);
  }
  return 1;
}
