// Layer-norm gradient in one sweep: dx, dgain and dbias from a single read of x and dy.
//
//     xhat = (x - mean) * rstd,  dx = rstd * (dy*g - mean(dy*g) - xhat * mean(dy*g*xhat)),  dgain = sum dy*xhat,  dbias = sum dy
//
// x and dy in, dx out: 75 MB at 16384 x 768 bf16, 11.6 us at the copy rate.  A row belongs to WPR warps (8 or 16 columns per thread, 24 for
// up to 768 columns, where one warp per row needs no barrier); the column sums stay in registers over all rows of a warp.  What bounds it
// above the copy rate is instruction issue and the chain of a row's reductions at 16 warps per SM: a copy ring alone changed nothing
// (23.1 -> 23.9 us).  So a 16-bit row is passed over twice instead of three times, with one round of reductions, and two columns share an
// instruction (fma.rn.f32x2); the ring then keeps the loads off that chain: 23.1 -> 18.8 us.  The row statistics are computed here unless
// the caller has them.  Column sums leave the kernel as one partial per block and a second kernel adds them in block order (4.8 -> 4.3 us): no
// atomics, the result does not depend on timing.
#include "vec8.cuh"

namespace dl4j {

constexpr int LG_THREADS = 256;
constexpr int LG_WARPS = LG_THREADS / 32;

constexpr int LG_STAGES = 3;           // ring slots per row group, 2 where only they fit

// Two fp32 values in one 64-bit register: the packed instructions of sm_100 do two operations per issue slot.
__device__ __forceinline__ uint64_t f2_pack(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 f2_unpack(uint64_t v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float f2_sum(uint64_t v) { const float2 f = f2_unpack(v); return f.x + f.y; }

template <typename T> __device__ __forceinline__ void lg_pairs(const Raw8<T>& q, uint64_t (&v)[4]) {
  float f[8];
  unpack8(q, f);
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] = f2_pack(f[2 * j], f[2 * j + 1]);
}

// One row of x or dy into shared memory by the copy engine; bytes and both addresses are multiples of 16.
__device__ __forceinline__ void lg_bulk_load(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(smem_dst)), "l"(gsrc), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// Rows of whole 16-byte vectors.  BULK: rows come through a ring of `stages` slots per row group, one elected thread's bulk copies one or
// two rows ahead, so that a warp's next rows are on their way while it works on the present one, which it reads from its slot in every
// pass.  Otherwise the row stays packed in registers and is unpacked at each of its uses.
template <typename T, int NV, int WPR, bool STATS, bool BULK>
__global__ void __launch_bounds__(LG_THREADS, 2)
layer_norm_grad_kernel(const T* __restrict__ dy, const T* __restrict__ x, const float* __restrict__ gain,
                       const float* __restrict__ mean_in, const float* __restrict__ rstd_in, T* __restrict__ dx,
                       float* __restrict__ out_g, float* __restrict__ out_b, long long out_stride, int accumulate, long long rows,
                       int C, float eps, int stages, int* __restrict__ status) {
  constexpr bool GREG = NV <= 2 || (NV == 3 && sizeof(T) == 2 && BULK);      // a thread's gain columns stay in registers
  // 16-bit rows take their statistics from one pass over x - the mean of its first eight values: sums of a sample-shifted row lose at
  // most a few bits of 24 where the result keeps 8 or 11.  fp32 rows take the mean first.
  constexpr bool ONE_PASS = !STATS && sizeof(T) == 2;
  constexpr int RPB = LG_WARPS / WPR;                 // rows in flight per block
  constexpr int TPR = 32 * WPR;                       // threads per row
  extern __shared__ __align__(128) unsigned char lg_ring[];
  __shared__ uint64_t bars[BULK ? RPB * LG_STAGES : 1];
  __shared__ float4 xch[2][2][LG_WARPS];              // cross-warp exchange: round, row parity, warp
  __shared__ float fold[RPB > 1 ? 2 * NV * 8 * TPR : 1];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int grp = wid / WPR;
  const int tr = threadIdx.x - grp * TPR;             // thread within its row
  const int nvec = C / 8;
  uint64_t ag[NV][4], ab[NV][4];
#pragma unroll
  for (int i = 0; i < NV; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) ag[i][j] = ab[i][j] = 0ull;
  const long long stride = (long long)gridDim.x * RPB;
  long long row = (long long)blockIdx.x * RPB + grp;
  const float inv_c = 1.f / C;
  const uint32_t row_bytes = (uint32_t)C * sizeof(T);
  unsigned char* ring = lg_ring + (size_t)grp * stages * 2 * row_bytes;
  uint64_t* bar = bars + (BULK ? grp * LG_STAGES : 0);
  auto issue = [&](int slot, long long r) {            // the row group's first thread only
    mbar_expect_tx(&bar[slot], 2 * row_bytes);
    lg_bulk_load(ring + (size_t)slot * 2 * row_bytes, dy + r * C, row_bytes, &bar[slot]);
    lg_bulk_load(ring + ((size_t)slot * 2 + 1) * row_bytes, x + r * C, row_bytes, &bar[slot]);
  };
  if constexpr (BULK) {
    if (tr == 0) {
#pragma unroll
      for (int i = 0; i < LG_STAGES; ++i) mbar_init(&bar[i], 1);
      mbar_fence_init();
#pragma unroll
      for (int i = 0; i < LG_STAGES; ++i)
        if (i < stages && row + i * stride < rows) issue(i, row + i * stride);
    }
    __syncthreads();
  }
  auto load_gain = [&](int vi, uint64_t (&g)[4]) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(gain) + vi * 2), c = __ldg(reinterpret_cast<const float4*>(gain) + vi * 2 + 1);
    g[0] = f2_pack(a.x, a.y); g[1] = f2_pack(a.z, a.w); g[2] = f2_pack(c.x, c.y); g[3] = f2_pack(c.z, c.w);
  };
  uint64_t greg[GREG ? NV : 1][4];
  if constexpr (GREG) {
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (tr + i * TPR < nvec) load_gain(tr + i * TPR, greg[i]);
  }
  auto gains = [&](int i, int vi, uint64_t (&g)[4]) {
    if constexpr (GREG) {
#pragma unroll
      for (int j = 0; j < 4; ++j) g[j] = greg[i][j];
    } else {
      load_gain(vi, g);
    }
  };
  int it = 0;
  auto row_sum = [&](float4 v, int round) {            // z and w are used with ONE_PASS only
    v.x = warp_sum(v.x);
    v.y = warp_sum(v.y);
    if (ONE_PASS) { v.z = warp_sum(v.z); v.w = warp_sum(v.w); }
    if constexpr (WPR > 1) {
      if (lane == 0) xch[round][it & 1][wid] = v;
      asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "r"(TPR) : "memory");
      v = xch[round][it & 1][grp * WPR];
#pragma unroll
      for (int w = 1; w < WPR; ++w) {
        const float4 o = xch[round][it & 1][grp * WPR + w];
        v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
      }
    }
    return v;
  };
  int slot = 0;
  uint32_t phase = 0;
  for (; row < rows; row += stride, ++it) {
    if constexpr (BULK) {
      if (!mbar_wait_bounded(&bar[slot], phase, status, DL4J_ERR_TIMEOUT_PRODUCER)) break;
    }
    Raw8<T> qd[BULK ? 1 : NV], qx[BULK ? 1 : NV];
    const T* sd = reinterpret_cast<const T*>(ring + (size_t)slot * 2 * row_bytes);
    if constexpr (!BULK) {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int vi = tr + i * TPR;
        if (vi < nvec && DL4J_IN_BOUNDS(row * C + vi * 8 + 7, rows * C)) {
          qd[i] = ld_raw8(dy + row * C + vi * 8);
          qx[i] = ld_raw8(x + row * C + vi * 8);
        } else {
          qd[i] = qx[i] = Raw8<T>();
        }
      }
    }
    auto get = [&](int i, int vi, uint64_t (&xv)[4], uint64_t (&d)[4]) {
      if constexpr (BULK) {
        lg_pairs<T>(*reinterpret_cast<const Raw8<T>*>(sd + C + vi * 8), xv);
        lg_pairs<T>(*reinterpret_cast<const Raw8<T>*>(sd + vi * 8), d);
      } else {
        lg_pairs<T>(qx[i], xv);
        lg_pairs<T>(qd[i], d);
      }
    };
    float mean = STATS ? mean_in[row] : 0.f, rstd = STATS ? rstd_in[row] : 0.f, s1, s2;
    float shift = 0.f;
    if constexpr (ONE_PASS) {
      uint64_t h[4];
      lg_pairs<T>(BULK ? *reinterpret_cast<const Raw8<T>*>(sd + C) : ld_raw8(x + row * C), h);
      shift = f2_sum(f2_add(f2_add(h[0], h[1]), f2_add(h[2], h[3]))) * 0.125f;
    }
    if constexpr (ONE_PASS || STATS) {                 // sums of dy*g, dy*g*xs, xs, xs^2 with xs = x - shift (given statistics: x - mean, the first two)
      const float ref = STATS ? mean : shift;
      const uint64_t neg = f2_pack(-ref, -ref);
      uint64_t a0 = 0ull, a1 = 0ull, a2 = 0ull, a3 = 0ull;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int vi = tr + i * TPR;
        if (vi < nvec) {
          uint64_t xv[4], d[4], g[4];
          get(i, vi, xv, d);
          gains(i, vi, g);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint64_t xs = f2_add(xv[j], neg), dg = f2_mul(d[j], g[j]);
            a0 = f2_add(a0, dg);
            a1 = f2_fma(dg, xs, a1);
            if (!STATS) { a2 = f2_add(a2, xs); a3 = f2_fma(xs, xs, a3); }
          }
        }
      }
      const float4 s = row_sum(make_float4(f2_sum(a0), f2_sum(a1), STATS ? 0.f : f2_sum(a2), STATS ? 0.f : f2_sum(a3)), 0);
      s1 = s.x * inv_c;
      if (STATS) {
        s2 = s.y * rstd * inv_c;
      } else {
        const float off = s.z * inv_c;                 // mean - shift
        mean = shift + off;
        float var = fmaf(-off, off, s.w * inv_c);
        if (var < 0.f) var = 0.f;                      // NaN stays
        rstd = rsqrtf(var + eps);
        s2 = fmaf(-off, s.x, s.y) * rstd * inv_c;
      }
    } else {
      uint64_t a0 = 0ull, a1 = 0ull;                   // sums of dy*g and x, then of (x - mean)^2 and dy*g*(x - mean)
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int vi = tr + i * TPR;
        if (vi < nvec) {
          uint64_t xv[4], d[4], g[4];
          get(i, vi, xv, d);
          gains(i, vi, g);
#pragma unroll
          for (int j = 0; j < 4; ++j) { a0 = f2_fma(d[j], g[j], a0); a1 = f2_add(a1, xv[j]); }
        }
      }
      const float4 s = row_sum(make_float4(f2_sum(a0), f2_sum(a1), 0.f, 0.f), 0);
      mean = s.y * inv_c;
      const uint64_t neg = f2_pack(-mean, -mean);
      a0 = a1 = 0ull;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int vi = tr + i * TPR;
        if (vi < nvec) {
          uint64_t xv[4], d[4], g[4];
          get(i, vi, xv, d);
          gains(i, vi, g);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint64_t xc = f2_add(xv[j], neg);
            a0 = f2_fma(xc, xc, a0);
            a1 = f2_fma(f2_mul(d[j], g[j]), xc, a1);
          }
        }
      }
      const float4 t = row_sum(make_float4(f2_sum(a0), f2_sum(a1), 0.f, 0.f), 1);
      rstd = rsqrtf(t.x * inv_c + eps);
      s1 = s.x * inv_c;
      s2 = t.y * rstd * inv_c;
    }
    const uint64_t neg = f2_pack(-mean, -mean), r2 = f2_pack(rstd, rstd), m1 = f2_pack(-s1, -s1), m2 = f2_pack(-s2, -s2);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int vi = tr + i * TPR;
      if (vi < nvec) {
        uint64_t xv[4], d[4], g[4];
        float o[8];
        get(i, vi, xv, d);
        gains(i, vi, g);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint64_t xh = f2_mul(f2_add(xv[j], neg), r2);
          ag[i][j] = f2_fma(d[j], xh, ag[i][j]);
          ab[i][j] = f2_add(ab[i][j], d[j]);
          const float2 v = f2_unpack(f2_mul(r2, f2_fma(xh, m2, f2_fma(d[j], g[j], m1))));
          o[2 * j] = v.x; o[2 * j + 1] = v.y;
        }
        Vec8<T>::store(dx + row * C + vi * 8, o);
      }
    }
    if constexpr (BULK) {                              // the row group has done with the slot: refill it
      if constexpr (WPR == 1) __syncwarp();
      else asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "r"(TPR) : "memory");
      if (tr == 0 && row + stages * stride < rows) issue(slot, row + stages * stride);
      if (++slot == stages) { slot = 0; phase ^= 1; }
    }
  }
  float sg[NV][8], sb[NV][8];
#pragma unroll
  for (int i = 0; i < NV; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 g = f2_unpack(ag[i][j]), c = f2_unpack(ab[i][j]);
      sg[i][2 * j] = g.x; sg[i][2 * j + 1] = g.y; sb[i][2 * j] = c.x; sb[i][2 * j + 1] = c.y;
    }
  if constexpr (RPB > 1) {
    // the block's row groups add up in shared memory, one after the other; slot (i, j) of thread tr sits at ((i * 8 + j) * TPR + tr)
    for (int w = 0; w < RPB; ++w) {
      if (grp == w) {
#pragma unroll
        for (int i = 0; i < NV; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int k = (i * 8 + j) * TPR + tr;
            if (w == 0) { fold[k] = sg[i][j]; fold[NV * 8 * TPR + k] = sb[i][j]; }
            else { fold[k] += sg[i][j]; fold[NV * 8 * TPR + k] += sb[i][j]; }
          }
      }
      __syncthreads();
    }
    if (grp != 0) return;
#pragma unroll
    for (int i = 0; i < NV; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int k = (i * 8 + j) * TPR + tr;
        sg[i][j] = fold[k];
        sb[i][j] = fold[NV * 8 * TPR + k];
      }
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int vi = tr + i * TPR;
    if (vi < nvec) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const long long o = blockIdx.x * out_stride + vi * 8 + j;
        if (out_g) out_g[o] = accumulate ? out_g[o] + sg[i][j] : sg[i][j];
        if (out_b) out_b[o] = accumulate ? out_b[o] + sb[i][j] : sb[i][j];
      }
    }
  }
}

// Any width and alignment: one element per thread and access, rows straight from global memory.
template <typename T, int NV, int WPR, bool STATS>
__global__ void __launch_bounds__(LG_THREADS, 2)
layer_norm_grad_scalar_kernel(const T* __restrict__ dy, const T* __restrict__ x, const float* __restrict__ gain,
                              const float* __restrict__ mean_in, const float* __restrict__ rstd_in, T* __restrict__ dx,
                              float* __restrict__ out_g, float* __restrict__ out_b, long long out_stride, int accumulate, long long rows,
                              int C, float eps) {
  constexpr int RPB = LG_WARPS / WPR;                 // rows in flight per block
  constexpr int TPR = 32 * WPR;                       // threads per row
  __shared__ float2 xch[2][2][LG_WARPS];              // cross-warp exchange: round, row parity, warp
  __shared__ float fold[RPB > 1 ? 2 * NV * TPR : 1];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int grp = wid / WPR;
  const int tr = threadIdx.x - grp * TPR;             // thread within its row
  float ag[NV], ab[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) ag[i] = ab[i] = 0.f;
  const long long stride = (long long)gridDim.x * RPB;
  long long row = (long long)blockIdx.x * RPB + grp;
  const float inv_c = 1.f / C;
  int parity = 0;
  auto row_sum = [&](float2 v, int round) {
    v.x = warp_sum(v.x);
    v.y = warp_sum(v.y);
    if constexpr (WPR > 1) {
      if (lane == 0) xch[round][parity][wid] = v;
      asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "r"(TPR) : "memory");
      v = xch[round][parity][grp * WPR];
#pragma unroll
      for (int w = 1; w < WPR; ++w) { const float2 o = xch[round][parity][grp * WPR + w]; v.x += o.x; v.y += o.y; }
    }
    return v;
  };
  for (; row < rows; row += stride) {
    T qd[NV], qx[NV];
    float2 s = make_float2(0.f, 0.f);                  // sum of x, sum of dy*g
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = tr + i * TPR;
      qd[i] = qx[i] = T(0.f);
      if (c < C && DL4J_IN_BOUNDS(row * C + c, rows * C)) { qd[i] = dy[row * C + c]; qx[i] = x[row * C + c]; }
    }
    float mean = STATS ? mean_in[row] : 0.f, rstd = STATS ? rstd_in[row] : 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = tr + i * TPR;
      if (c < C) {
        if (!STATS) s.x += ldf(&qx[i]);
        s.y = fmaf(ldf(&qd[i]), gain[c], s.y);
      }
    }
    if (!STATS) {
      s = row_sum(s, 0);
      mean = s.x * inv_c;
    }
    float2 t = make_float2(0.f, 0.f);                  // sum of (x - mean)^2 (given statistics: of dy*g), sum of dy*g*(x - mean)
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = tr + i * TPR;
      if (c < C) {
        const float xc = ldf(&qx[i]) - mean;
        if (!STATS) t.x = fmaf(xc, xc, t.x);
        t.y = fmaf(ldf(&qd[i]) * gain[c], xc, t.y);
      }
    }
    if (STATS) t.x = s.y;
    t = row_sum(t, 1);
    if (!STATS) rstd = rsqrtf(t.x * inv_c + eps);
    const float s1 = (STATS ? t.x : s.y) * inv_c, s2 = t.y * rstd * inv_c;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = tr + i * TPR;
      if (c < C) {
        const float d = ldf(&qd[i]), xh = (ldf(&qx[i]) - mean) * rstd;
        ag[i] = fmaf(d, xh, ag[i]);
        ab[i] += d;
        stf(dx + row * C + c, rstd * (fmaf(d, gain[c], -s1) - xh * s2));
      }
    }
    parity ^= 1;
  }
  if constexpr (RPB > 1) {
    // the block's row groups add up in shared memory, one after the other
    for (int w = 0; w < RPB; ++w) {
      if (grp == w) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          const int k = i * TPR + tr;
          if (w == 0) { fold[k] = ag[i]; fold[NV * TPR + k] = ab[i]; }
          else { fold[k] += ag[i]; fold[NV * TPR + k] += ab[i]; }
        }
      }
      __syncthreads();
    }
    if (grp != 0) return;
#pragma unroll
    for (int i = 0; i < NV; ++i) { ag[i] = fold[i * TPR + tr]; ab[i] = fold[NV * TPR + i * TPR + tr]; }
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = tr + i * TPR;
    if (c < C) {
      const long long o = blockIdx.x * out_stride + c;
      if (out_g) out_g[o] = accumulate ? out_g[o] + ag[i] : ag[i];
      if (out_b) out_b[o] = accumulate ? out_b[o] + ab[i] : ab[i];
    }
  }
}

// partial[blocks][2][C] -> dgain, dbias.  32 columns x 32 row lanes per block, all of a thread's (up to ten) rows in flight at once; each
// thread adds its rows in order.
constexpr int LG_COL_LANES = 32;
__global__ void __launch_bounds__(32 * LG_COL_LANES)
layer_norm_grad_cols_kernel(const float* __restrict__ partial, int blocks, int C, float* __restrict__ dgain, float* __restrict__ dbias,
                            int accumulate) {
  __shared__ float red[LG_COL_LANES][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + tx;
  float s = 0.f;
  if (c < 2 * C) {
#pragma unroll 10
    for (int b = ty; b < blocks; b += LG_COL_LANES) s += __ldcs(partial + (long long)b * 2 * C + c);
  }
  red[ty][tx] = s;
  __syncthreads();
  const float t = warp_sum(red[tx][ty]);               // warp ty: column ty, its lanes' sums pairwise
  const int col = blockIdx.x * 32 + ty;
  if (tx == 0 && col < 2 * C) {
    float* dst = col < C ? (dgain ? dgain + col : nullptr) : (dbias ? dbias + (col - C) : nullptr);
    if (dst) *dst = accumulate ? *dst + t : t;
  }
}

}  // namespace dl4j

using namespace dl4j;

namespace {

struct LgArgs {
  const void *dy, *x;
  const float *gain, *mean, *rstd;
  void* dx;
  float *dgain, *dbias, *partial;
  long long rows;
  int C;
  float eps;
  int accumulate, sms;
  cudaStream_t stream;
};

constexpr size_t LG_RING_MAX = 100 * 1024;      // of a block: two share the SM's 227 KB with the fold buffers (up to 12 KB each)

template <typename T, int NV, int WPR, bool STATS, bool BULK>
int lg_launch(const LgArgs& a, int grid, int stages, size_t smem, float* og, float* ob, long long os, int acc) {
  auto kern = layer_norm_grad_kernel<T, NV, WPR, STATS, BULK>;
  int dev = 0;
  cudaGetDevice(&dev);
  static SmemLimit limit;
  if (smem) {
    const cudaError_t e = raise_smem_limit((const void*)kern, dev, (int)smem, limit);
    if (e != cudaSuccess) return (int)e;
  }
  kern<<<grid, LG_THREADS, smem, a.stream>>>((const T*)a.dy, (const T*)a.x, a.gain, a.mean, a.rstd, (T*)a.dx, og, ob, os, acc, a.rows, a.C, a.eps, stages,
                                             dl4j_status_word(dev));
  return (int)cudaGetLastError();
}

template <typename T, bool VEC, int NV, int WPR>
int lg_run(const LgArgs& a) {
  constexpr int RPB = LG_WARPS / WPR;
  const long long need = (a.rows + RPB - 1) / RPB;
  const long long cap = (long long)a.sms * 2;
  const int grid = (int)(need < cap ? need : cap);
  // one block writes the sums itself; otherwise they go through the partials
  const bool direct = grid == 1;
  float* og = direct ? a.dgain : a.partial;
  float* ob = direct ? a.dbias : a.partial + a.C;
  const long long os = direct ? 0 : 2LL * a.C;
  const int acc = direct ? a.accumulate : 0;
  int rc = 0;
  if constexpr (VEC) {
    // the ring is worth its set-up from the second row of a group on, and two blocks must fit an SM with it
    const size_t slots = (size_t)RPB * 2 * a.C * sizeof(T);
    const int stages = LG_STAGES * slots <= LG_RING_MAX ? LG_STAGES : 2;
    const size_t ring = stages * slots;
    const bool bulk = need > cap && ring <= LG_RING_MAX;
    if (a.mean) rc = bulk ? lg_launch<T, NV, WPR, true, true>(a, grid, stages, ring, og, ob, os, acc) : lg_launch<T, NV, WPR, true, false>(a, grid, 0, 0, og, ob, os, acc);
    else rc = bulk ? lg_launch<T, NV, WPR, false, true>(a, grid, stages, ring, og, ob, os, acc) : lg_launch<T, NV, WPR, false, false>(a, grid, 0, 0, og, ob, os, acc);
  } else {
    auto kern = a.mean ? layer_norm_grad_scalar_kernel<T, NV, WPR, true> : layer_norm_grad_scalar_kernel<T, NV, WPR, false>;
    kern<<<grid, LG_THREADS, 0, a.stream>>>((const T*)a.dy, (const T*)a.x, a.gain, a.mean, a.rstd, (T*)a.dx, og, ob, os, acc, a.rows, a.C, a.eps);
    rc = (int)cudaGetLastError();
  }
  if (rc) return rc;
  if (!direct && (a.dgain || a.dbias))
    layer_norm_grad_cols_kernel<<<(2 * a.C + 31) / 32, 32 * LG_COL_LANES, 0, a.stream>>>(a.partial, grid, a.C, a.dgain, a.dbias, a.accumulate);
  return (int)cudaGetLastError();
}

template <typename T>
int lg_dispatch(const LgArgs& a) {
  const bool vec = a.C % 8 == 0 && (((uintptr_t)a.dy | (uintptr_t)a.x | (uintptr_t)a.dx | (uintptr_t)a.gain) & 15) == 0;
  const int C = a.C;
  if (vec) {
    if (C <= 256) return lg_run<T, true, 1, 1>(a);
    if (C <= 512) return lg_run<T, true, 2, 1>(a);
    if (C <= 768) return lg_run<T, true, 3, 1>(a);
    if (C <= 1024) return lg_run<T, true, 2, 2>(a);
    if (C <= 2048) return lg_run<T, true, 2, 4>(a);
    if (C <= 4096) return lg_run<T, true, 2, 8>(a);
    return lg_run<T, true, 4, 8>(a);
  }
  if (C <= 256) return lg_run<T, false, 8, 1>(a);
  if (C <= 512) return lg_run<T, false, 16, 1>(a);
  if (C <= 1024) return lg_run<T, false, 16, 2>(a);
  if (C <= 2048) return lg_run<T, false, 16, 4>(a);
  if (C <= 4096) return lg_run<T, false, 16, 8>(a);
  return lg_run<T, false, 32, 8>(a);
}

}  // namespace

// mean / rstd: the forward's row statistics, or null (both) to compute them here with `eps`.  dgain / dbias may be null; they are
// overwritten, or added to with `accumulate`.  partial: room for 2 * num_sms * 2 * C floats.  Limits: 1 <= C <= 8192.
DL4J_API int dl4j_layer_norm_grad(const void* dy, const void* x, const float* gain, const float* mean, const float* rstd, void* dx,
                                  float* dgain, float* dbias, float* partial, long long rows, int C, float eps, int dtype,
                                  int accumulate, int num_sms, void* stream) {
  if (rows < 1 || C < 1 || C > 8192 || num_sms < 1 || !dy || !x || !gain || !dx || !partial || (!mean) != (!rstd)) return -DL4J_ERR_BAD_ARG;
  const LgArgs a{dy, x, gain, mean, rstd, dx, dgain, dbias, partial, rows, C, eps, accumulate, num_sms, (cudaStream_t)stream};
  if (dtype == 1) return lg_dispatch<__nv_bfloat16>(a);
  if (dtype == 0) return lg_dispatch<__half>(a);
  if (dtype == 2) return lg_dispatch<float>(a);
  return -DL4J_ERR_BAD_ARG;
}
