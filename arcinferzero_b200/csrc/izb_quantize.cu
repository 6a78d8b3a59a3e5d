// Activation quantiser: f32 rows -> int8 per 32-block + f32 scale (+ int16 sums per 16), HBM-bound.
// Arithmetic of quantize_act_cpu (src/quants.h:626-643) = quant_store16 (zero/kernels/ops.cl:38-72), bit for bit:
//   amax = max|x|;  inv = amax > 0 ? 127.0f / amax : 0;  q = rint(x * inv);  scale = amax / 127.0f
// The divisions and the product are written with the round-to-nearest intrinsics so no contraction or reciprocal
// approximation can change a bit.
//
// (Many rows.)  One CTA covers 32 token rows x 256 columns: every lane owns 8 consecutive values (two 128-bit loads), four lanes make
// a 32-block.  The int8 row stores are 256 contiguous bytes per warp; the scales, whose layout is block-major
// ([K/32][Mp]), go through shared memory so that each block's 32 token scales leave as one 128-byte line.
#include "izb_common.cuh"

namespace {

// kMode 0: quantise x.  1 (SwiGLU): x holds gate | up at column offset F, quantise h = silu(gate) * up; hout: optional
// f32 copy of h.
template <int kMode>
__global__ void __launch_bounds__(256) quantize_act_kernel(const float* __restrict__ x, int ldx, int M, int Mp, int K,
                                                           int8_t* __restrict__ aq, float* __restrict__ asc,
                                                           int16_t* __restrict__ absum, float* __restrict__ hout,
                                                           int F /* mode 1: up projection at column offset F */) {
  constexpr bool kSwiglu = kMode == 1;
  __shared__ float s_sc[8][33];
  __shared__ int16_t s_sum[16][34];
  const int sb = blockIdx.x, m0 = blockIdx.y * 32, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = sb * 256 + lane * 8;
  pdl_launch_next();
  pdl_wait();
  float v[4][8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + warp + 8 * i;
    if (m < M) {
      const float4* p = reinterpret_cast<const float4*>(x + (size_t)m * ldx + col);
      const float4 a = __ldcs(p), b = __ldcs(p + 1);
      v[i][0] = a.x; v[i][1] = a.y; v[i][2] = a.z; v[i][3] = a.w;
      v[i][4] = b.x; v[i][5] = b.y; v[i][6] = b.z; v[i][7] = b.w;
      if (kSwiglu) {  // v holds the gate g: h = g / (1 + exp(-g)) * u   (zero/kernels/ops.cl:272-315)
        const float4* pu = reinterpret_cast<const float4*>(x + (size_t)m * ldx + F + col);
        const float4 c = __ldcs(pu), d = __ldcs(pu + 1);
        const float u[8] = {c.x, c.y, c.z, c.w, d.x, d.y, d.z, d.w};
#pragma unroll
        for (int k = 0; k < 8; ++k) v[i][k] = __fmul_rn(__fdiv_rn(v[i][k], __fadd_rn(1.0f, expf(-v[i][k]))), u[k]);
        if (hout) {
          float4* ph = reinterpret_cast<float4*>(hout + (size_t)m * F + col);
          ph[0] = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
          ph[1] = make_float4(v[i][4], v[i][5], v[i][6], v[i][7]);
        }
      }
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) v[i][k] = 0.0f;
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = warp + 8 * i, m = m0 + r;
    float amax = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) amax = fmaxf(amax, fabsf(v[i][k]));
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
    const float inv = amax > 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
    int q[8], s8 = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      // lrintf's x86 result for products outside the int range or NaN (only when amax is so small that 127 / amax
      // overflows): INT_MIN, whose low byte is 0
      const float p = __fmul_rn(v[i][k], inv);
      q[k] = fabsf(p) <= 2147483520.0f ? __float2int_rn(p) : 0;
      s8 += q[k];
    }
    const int s16 = s8 + __shfl_xor_sync(0xFFFFFFFFu, s8, 1);
    if (m < Mp) {
      uint2 pk;
      pk.x = (q[0] & 0xFF) | ((q[1] & 0xFF) << 8) | ((q[2] & 0xFF) << 16) | ((uint32_t)(q[3] & 0xFF) << 24);
      pk.y = (q[4] & 0xFF) | ((q[5] & 0xFF) << 8) | ((q[6] & 0xFF) << 16) | ((uint32_t)(q[7] & 0xFF) << 24);
      *reinterpret_cast<uint2*>(aq + (size_t)m * K + col) = pk;
    }
    if ((lane & 3) == 0) s_sc[lane >> 2][r] = __fdiv_rn(amax, 127.0f);
    if ((lane & 1) == 0) s_sum[lane >> 1][r] = (int16_t)s16;
  }
  __syncthreads();
  {
    const int b = threadIdx.x >> 5, r = threadIdx.x & 31;
    if (m0 + r < Mp) {
      asc[(size_t)(sb * 8 + b) * Mp + m0 + r] = s_sc[b][r];
      if (absum) {
        absum[(size_t)(sb * 16 + b) * Mp + m0 + r] = s_sum[b][r];
        absum[(size_t)(sb * 16 + 8 + b) * Mp + m0 + r] = s_sum[8 + b][r];
      }
    }
  }
}

// One value per thread, a warp per 32-block: the block's scale and sums from the warp.  kNan: a block that is all NaN has the scale NaN, as the residual
// addition's rows have it, else 0, as the quantisers' and the other norm's have it.
template <bool kNan>
__device__ __forceinline__ void quantize_value(float v, int row, int col, int Mp, int K, int8_t* __restrict__ aq, float* __restrict__ asc, int16_t* __restrict__ absum) {
  const int lane = threadIdx.x & 31;
  float amax = kNan ? fabsf(v) : fmaxf(0.0f, fabsf(v));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
  const float inv = amax > 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
  const float p = __fmul_rn(v, inv);
  const int q = fabsf(p) <= 2147483520.0f ? __float2int_rn(p) : 0;  // (see quantize_act_kernel)
  aq[(size_t)row * K + col] = (int8_t)q;
  if (lane == 0) asc[(size_t)(col >> 5) * Mp + row] = __fdiv_rn(amax, 127.0f);
  if (absum) {
    int s16 = q;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) s16 += __shfl_xor_sync(0xFFFFFFFFu, s16, o);
    if ((lane & 15) == 0) absum[(size_t)(col >> 4) * Mp + row] = (int16_t)s16;
  }
}

// The same for few rows: one thread per value, a warp per 32-block, a CTA per row and 256 columns (one CTA more for the padding rows).  What bounds
// a decode step's quantiser is the latency of one thread's values: eight of them, each with an exponential and two divisions (SwiGLU).
template <int kMode>
__global__ void __launch_bounds__(256) quantize_few_kernel(const float* __restrict__ x, int ldx, int M, int Mp, int K, int8_t* __restrict__ aq, float* __restrict__ asc,
                                                           int16_t* __restrict__ absum, float* __restrict__ hout, int F) {
  const int sb = blockIdx.x, row = blockIdx.y, col = sb * 256 + threadIdx.x;
  pdl_launch_next();
  pdl_wait();
  if (row == M) {
    for (int i = threadIdx.x; i < (Mp - M) * 16; i += 256) {
      const int m = M + (i >> 4), c = i & 15;
      *reinterpret_cast<uint4*>(aq + (size_t)m * K + sb * 256 + 16 * c) = make_uint4(0, 0, 0, 0);
      if (c < 8) asc[(size_t)(sb * 8 + c) * Mp + m] = 0.0f;
      if (absum) absum[(size_t)(sb * 16 + c) * Mp + m] = 0;
    }
    return;
  }
  float v = x[(size_t)row * ldx + col];
  if (kMode == 1) {
    const float u = x[(size_t)row * ldx + F + col];
    v = __fmul_rn(__fdiv_rn(v, __fadd_rn(1.0f, expf(-v))), u);
    if (hout) hout[(size_t)row * F + col] = v;
  }
  quantize_value<false>(v, row, col, Mp, K, aq, asc, absum);
}

// Sum over the CTA's 256 threads in the defined order: xor butterfly 16, 8, 4, 2, 1 inside every warp, then the eight
// warp sums added in warp order; every thread returns the same value.  s_w: 8 floats of shared memory.
__device__ __forceinline__ float cta_sum_ordered(float v, float* s_w) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
  __syncthreads();  // (s_w may still be read from a call before)
  if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = s_w[0];
#pragma unroll
  for (int w = 1; w < 8; ++w) t = __fadd_rn(t, s_w[w]);
  return t;
}

// rows M..Mp-1 of a quantised activation buffer: zeros with scale 0 (one CTA per row, or columns c0 .. c1 - 1 of a row)
__device__ __forceinline__ void zero_pad_cols(int m, int c0, int c1, int Mp, int K, int8_t* __restrict__ aq, float* __restrict__ asc, int16_t* __restrict__ absum) {
  int8_t* row = aq + (size_t)m * K;
  const bool wide = (reinterpret_cast<uintptr_t>(row) & 15) == 0;  // (add_norm_quant takes any alignment)
  for (int i = c0 / 16 + threadIdx.x; i < c1 / 16; i += blockDim.x) {
    if (wide) reinterpret_cast<uint4*>(row)[i] = make_uint4(0, 0, 0, 0);
    else
      for (int j = 0; j < 16; ++j) row[16 * i + j] = 0;
    if (!(i & 1)) asc[(size_t)(i >> 1) * Mp + m] = 0.0f;
    if (absum) absum[(size_t)i * Mp + m] = 0;
  }
}
__device__ __forceinline__ void zero_pad_row(int m, int Mp, int K, int8_t* __restrict__ aq, float* __restrict__ asc, int16_t* __restrict__ absum) {
  zero_pad_cols(m, 0, K, Mp, K, aq, asc, absum);
}

// add_norm_quant (zero/kernels/ops_attn_g.cl:617-680), one CTA of 256 threads per row, K <= 256 * kAnqMax:
//   x = (x + (t * r) * w) * s with r = 1/sqrt(sum(t^2)/K + eps);  y = w2 ? (x * r2) * w2 : x with r2 from the new x;
//   y quantised per 32-block.  Thread j owns elements j, j + 256, ...: a warp owns one 32-block per step, so the
// block maximum is a warp reduction; the new x stays in registers between the two steps.  Both sums of squares are
// taken in the defined order of cta_sum_ordered over per-thread fused-multiply-add chains.
// A few decode rows are bound by latency: NK (elements per thread, rounded up) is a compile-time number so that all of a
// thread's loads are in flight before the first reduction and the chains unroll.  (With a run-time bound over 64 elements
// the loads were issued one step at a time: 5 rows of 4096 took 35 us.)  Up to 20 elements (K = 5120) the norm weights are
// requested with the rows; above that they would not fit the registers and come from L2 behind the first reduction.
// kHold: t stays in registers from the first sum to the update.  Not for long rows (K > 8192) when there are more of them than SMs: with
// both rows held one block fills an SM's registers, and the next row waits (16384, 200 rows: 72 us held, 38 read twice; 4096 rows: 1033 and 609).
constexpr int kAnqMax = 64;
template <int NK, bool kHold>
__global__ void __launch_bounds__(256) add_norm_quant_kernel(float* __restrict__ x, const float* __restrict__ t,
                                                             const float* __restrict__ w, int K, float eps, float s,
                                                             const float* __restrict__ w2, int M, int Mp, int8_t* __restrict__ aq,
                                                             float* __restrict__ asc, int16_t* __restrict__ absum) {
  __shared__ float s_w[8];
  constexpr bool kAhead = NK <= 20;
  const int m = blockIdx.x, lane = threadIdx.x & 31;
  pdl_launch_next();
  pdl_wait();
  if (m >= M) {
    zero_pad_row(m, Mp, K, aq, asc, absum);
    return;
  }
  float* xr = x + (size_t)m * K;
  const float* tr = t + (size_t)m * K;
  const int nk = K / 256;
  float tv[kHold ? NK : 1], xv[NK], wv[kAhead ? NK : 1], w2v[kAhead ? NK : 1];
  if (kHold) {
#pragma unroll
    for (int k = 0; k < NK; ++k)
      if (k < nk) tv[k] = tr[threadIdx.x + 256 * k];
#pragma unroll
    for (int k = 0; k < NK; ++k)
      if (k < nk) xv[k] = xr[threadIdx.x + 256 * k];
  }
  if (kAhead) {
#pragma unroll
    for (int k = 0; k < NK; ++k)
      if (k < nk) {
        wv[k] = w[threadIdx.x + 256 * k];
        if (w2) w2v[k] = w2[threadIdx.x + 256 * k];
      }
  }
  float ss = 0.0f;
  if (kHold) {
#pragma unroll
    for (int k = 0; k < NK; ++k)
      if (k < nk) ss = __fmaf_rn(tv[k], tv[k], ss);
  } else {
    for (int k = 0; k < nk; ++k) {
      const float v = tr[threadIdx.x + 256 * k];
      ss = __fmaf_rn(v, v, ss);
    }
  }
  ss = cta_sum_ordered(ss, s_w);
  const float r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)K), eps)));
  float s2 = 0.0f;
#pragma unroll
  for (int k = 0; k < NK; ++k) {
    if (k < nk) {
      const int i = threadIdx.x + 256 * k;
      const float v = __fmul_rn(__fadd_rn(kHold ? xv[k] : xr[i], __fmul_rn(__fmul_rn(kHold ? tv[k] : tr[i], r), kAhead ? wv[k] : w[i])), s);
      xv[k] = v;
      xr[i] = v;
      s2 = __fmaf_rn(v, v, s2);
    }
  }
  float r2 = 1.0f;
  if (w2) {
    s2 = cta_sum_ordered(s2, s_w);
    r2 = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(s2, (float)K), eps)));
  }
#pragma unroll
  for (int k = 0; k < NK; ++k) {
    if (k < nk) {
      const int i = threadIdx.x + 256 * k;
      const float y = w2 ? __fmul_rn(__fmul_rn(xv[k], r2), kAhead ? w2v[k] : w2[i]) : xv[k];
      float amax = fabsf(y);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
      const float inv = amax > 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
      const float p = __fmul_rn(y, inv);
      const int q = fabsf(p) <= 2147483520.0f ? __float2int_rn(p) : 0;  // (see quantize_act_kernel)
      aq[(size_t)m * K + i] = (int8_t)q;
      const int b = i >> 5;
      if (lane == 0) asc[(size_t)b * Mp + m] = __fdiv_rn(amax, 127.0f);
      if (absum) {
        int s16 = q;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) s16 += __shfl_xor_sync(0xFFFFFFFFu, s16, o);
        if ((lane & 15) == 0) absum[(size_t)(2 * b + (lane >> 4)) * Mp + m] = (int16_t)s16;
      }
    }
  }
}

// The same for few rows of 1280 to 5120: a cluster of up to eight CTAs per row.  Every CTA takes both sums over the whole row, in the same order, and then
// updates and quantises its share of it (up to three steps of 256): one SM's issue slots, not its loads, are what a row took its time for.
// The new x goes over the old one that the other CTAs read: they store behind the cluster's barrier.
constexpr int kFewSteps = 3;
template <int NK>
__global__ void __launch_bounds__(256) add_norm_few_kernel(float* __restrict__ x, const float* __restrict__ t, const float* __restrict__ w, int K, float eps, float s,
                                                           const float* __restrict__ w2, int M, int Mp, int8_t* __restrict__ aq, float* __restrict__ asc,
                                                           int16_t* __restrict__ absum, int steps) {
  __shared__ float s_w[8];
  const int m = blockIdx.y, first = blockIdx.x * steps, nk = K / 256;
  pdl_launch_next();
  pdl_wait();
  if (m >= M) {
    zero_pad_cols(m, 256 * first, min(256 * (first + steps), K), Mp, K, aq, asc, absum);
    return;
  }
  float* xr = x + (size_t)m * K;
  const float* tr = t + (size_t)m * K;
  float tv[NK], xv[NK], wv[NK], to[kFewSteps], xo[kFewSteps], wo[kFewSteps], w2o[kFewSteps];
#pragma unroll
  for (int k = 0; k < NK; ++k)
    if (k < nk) tv[k] = tr[threadIdx.x + 256 * k];
  if (w2) {
#pragma unroll
    for (int k = 0; k < NK; ++k)
      if (k < nk) {
        xv[k] = xr[threadIdx.x + 256 * k];
        wv[k] = w[threadIdx.x + 256 * k];
      }
  }
#pragma unroll
  for (int k = 0; k < kFewSteps; ++k)
    if (k < steps && first + k < nk) {
      const int i = threadIdx.x + 256 * (first + k);
      to[k] = tr[i];
      xo[k] = xr[i];
      wo[k] = w[i];
      if (w2) w2o[k] = w2[i];
    }
  float ss = 0.0f;
#pragma unroll
  for (int k = 0; k < NK; ++k)
    if (k < nk) ss = __fmaf_rn(tv[k], tv[k], ss);
  ss = cta_sum_ordered(ss, s_w);
  const float r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)K), eps)));
  auto updated = [&](float xe, float te, float we) { return __fmul_rn(__fadd_rn(xe, __fmul_rn(__fmul_rn(te, r), we)), s); };
  float s2 = 0.0f;
  if (w2) {
#pragma unroll
    for (int k = 0; k < NK; ++k)
      if (k < nk) {
        const float v = updated(xv[k], tv[k], wv[k]);
        s2 = __fmaf_rn(v, v, s2);
      }
  }
#pragma unroll
  for (int k = 0; k < kFewSteps; ++k)
    if (k < steps && first + k < nk) xo[k] = updated(xo[k], to[k], wo[k]);
  asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");  // this CTA has read the row
  float r2 = 1.0f;
  if (w2) {
    s2 = cta_sum_ordered(s2, s_w);
    r2 = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(s2, (float)K), eps)));
  }
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
#pragma unroll
  for (int k = 0; k < kFewSteps; ++k)
    if (k < steps && first + k < nk) {
      const int i = threadIdx.x + 256 * (first + k);
      xr[i] = xo[k];
      quantize_value<true>(w2 ? __fmul_rn(__fmul_rn(xo[k], r2), w2o[k]) : xo[k], m, i, Mp, K, aq, asc, absum);
    }
}

// rmsnorm_quant (zero/kernels/ops.cl:104-141), one CTA of 256 threads per row, in the quantiser's lane layout: thread j owns
// the groups of 8 consecutive values j, j + 256, ... .  Step 1: the sum of squares, a chain of fused multiply-adds over the
// thread's values in index order, then cta_sum_ordered (this order is part of the definition: the oracle repeats it).
// Step 2: y = (x * r) * w, optional f32 copy, and per 32-block (four adjacent threads) int8 + scale + sums of 16.
// G = groups per thread rounded up: row and norm weights are requested together before the reduction and stay in
// registers (one pass over the row, one latency instead of two; a row read twice through L1 / L2 measured 56 us at 8192 x
// 5120 and 5.8 us for one row of 5120).  G = 0: rows too long for that (K > 16384), or many long ones, read twice.
template <int G>
__global__ void __launch_bounds__(256) rmsnorm_quant_row_kernel(const float* __restrict__ x, int ldx, const float* __restrict__ w,
                                                                int K, float eps, int M, int Mp, float* __restrict__ hout,
                                                                int8_t* __restrict__ aq, float* __restrict__ asc,
                                                                int16_t* __restrict__ absum) {
  __shared__ float s_w[8];
  constexpr int GR = G > 0 ? G : 1;
  const int m = blockIdx.x, ng = K / 8;
  pdl_launch_next();
  pdl_wait();
  if (m >= M) {
    zero_pad_row(m, Mp, K, aq, asc, absum);
    return;
  }
  const float* xr = x + (size_t)m * ldx;
  float4 xa[GR], xb[GR], wa[GR], wb[GR];
  float ss = 0.0f;
  auto square = [&](const float4& a, const float4& b) {
    ss = __fmaf_rn(a.x, a.x, ss); ss = __fmaf_rn(a.y, a.y, ss); ss = __fmaf_rn(a.z, a.z, ss); ss = __fmaf_rn(a.w, a.w, ss);
    ss = __fmaf_rn(b.x, b.x, ss); ss = __fmaf_rn(b.y, b.y, ss); ss = __fmaf_rn(b.z, b.z, ss); ss = __fmaf_rn(b.w, b.w, ss);
  };
  if (G > 0) {
#pragma unroll
    for (int k = 0; k < G; ++k) {
      const int g = threadIdx.x + 256 * k;
      if (g < ng) {
        xa[k] = reinterpret_cast<const float4*>(xr)[2 * g];
        xb[k] = reinterpret_cast<const float4*>(xr)[2 * g + 1];
      }
    }
#pragma unroll
    for (int k = 0; k < G; ++k) {
      const int g = threadIdx.x + 256 * k;
      if (g < ng) {
        wa[k] = reinterpret_cast<const float4*>(w)[2 * g];
        wb[k] = reinterpret_cast<const float4*>(w)[2 * g + 1];
      }
    }
#pragma unroll
    for (int k = 0; k < G; ++k)
      if (threadIdx.x + 256 * k < ng) square(xa[k], xb[k]);
  } else {
    for (int g = threadIdx.x; g < ng; g += 256) square(reinterpret_cast<const float4*>(xr)[2 * g], reinterpret_cast<const float4*>(xr)[2 * g + 1]);
  }
  ss = cta_sum_ordered(ss, s_w);
  const float r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)K), eps)));
  auto group = [&](int g, const float4& a, const float4& b, const float4& c, const float4& d) {  // (K / 8 is a multiple of 32: whole warps take part in the shuffles)
    const int col = 8 * g;
    float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    const float wv[8] = {c.x, c.y, c.z, c.w, d.x, d.y, d.z, d.w};
    float amax = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      v[k] = __fmul_rn(__fmul_rn(v[k], r), wv[k]);
      amax = fmaxf(amax, fabsf(v[k]));
    }
    if (hout) {
      float4* ph = reinterpret_cast<float4*>(hout + (size_t)m * K + col);
      ph[0] = make_float4(v[0], v[1], v[2], v[3]);
      ph[1] = make_float4(v[4], v[5], v[6], v[7]);
    }
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
    const float inv = amax > 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
    int q[8], s8 = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float p = __fmul_rn(v[k], inv);
      q[k] = fabsf(p) <= 2147483520.0f ? __float2int_rn(p) : 0;  // (see quantize_act_kernel)
      s8 += q[k];
    }
    uint2 pk;
    pk.x = (q[0] & 0xFF) | ((q[1] & 0xFF) << 8) | ((q[2] & 0xFF) << 16) | ((uint32_t)(q[3] & 0xFF) << 24);
    pk.y = (q[4] & 0xFF) | ((q[5] & 0xFF) << 8) | ((q[6] & 0xFF) << 16) | ((uint32_t)(q[7] & 0xFF) << 24);
    *reinterpret_cast<uint2*>(aq + (size_t)m * K + col) = pk;
    if ((g & 3) == 0) asc[(size_t)(g >> 2) * Mp + m] = __fdiv_rn(amax, 127.0f);
    if (absum) {
      const int s16 = s8 + __shfl_xor_sync(0xFFFFFFFFu, s8, 1);
      if ((g & 1) == 0) absum[(size_t)(g >> 1) * Mp + m] = (int16_t)s16;
    }
  };
  if (G > 0) {
#pragma unroll
    for (int k = 0; k < G; ++k)
      if (threadIdx.x + 256 * k < ng) group(threadIdx.x + 256 * k, xa[k], xb[k], wa[k], wb[k]);
  } else {
    for (int g = threadIdx.x; g < ng; g += 256)
      group(g, reinterpret_cast<const float4*>(xr)[2 * g], reinterpret_cast<const float4*>(xr)[2 * g + 1], reinterpret_cast<const float4*>(w)[2 * g],
            reinterpret_cast<const float4*>(w)[2 * g + 1]);
  }
}

// The same for few rows: several CTAs per row, each with the whole row's sum in the same order and two steps of 256 values to quantise (see
// add_norm_few_kernel; nothing is written over what another CTA reads).
template <int G>
__global__ void __launch_bounds__(256) rmsnorm_few_kernel(const float* __restrict__ x, int ldx, const float* __restrict__ w, int K, float eps, int M, int Mp, float* __restrict__ hout,
                                                          int8_t* __restrict__ aq, float* __restrict__ asc, int16_t* __restrict__ absum) {
  __shared__ float s_w[8];
  const int m = blockIdx.y, ng = K / 8, i0 = blockIdx.x * 512 + threadIdx.x, i1 = i0 + 256;
  pdl_launch_next();
  pdl_wait();
  if (m >= M) {
    zero_pad_cols(m, blockIdx.x * 512, min(blockIdx.x * 512 + 512, K), Mp, K, aq, asc, absum);
    return;
  }
  const float* xr = x + (size_t)m * ldx;
  float4 xa[G], xb[G];
#pragma unroll
  for (int k = 0; k < G; ++k) {
    const int g = threadIdx.x + 256 * k;
    if (g < ng) {
      xa[k] = reinterpret_cast<const float4*>(xr)[2 * g];
      xb[k] = reinterpret_cast<const float4*>(xr)[2 * g + 1];
    }
  }
  const bool two = i1 < K;  // (uniform over the CTA, as K is a multiple of 256)
  const float x0 = xr[i0], w0 = w[i0], x1 = two ? xr[i1] : 0.0f, w1 = two ? w[i1] : 0.0f;
  float ss = 0.0f;
#pragma unroll
  for (int k = 0; k < G; ++k)
    if (threadIdx.x + 256 * k < ng) {
      ss = __fmaf_rn(xa[k].x, xa[k].x, ss); ss = __fmaf_rn(xa[k].y, xa[k].y, ss); ss = __fmaf_rn(xa[k].z, xa[k].z, ss); ss = __fmaf_rn(xa[k].w, xa[k].w, ss);
      ss = __fmaf_rn(xb[k].x, xb[k].x, ss); ss = __fmaf_rn(xb[k].y, xb[k].y, ss); ss = __fmaf_rn(xb[k].z, xb[k].z, ss); ss = __fmaf_rn(xb[k].w, xb[k].w, ss);
    }
  ss = cta_sum_ordered(ss, s_w);
  const float r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)K), eps)));
  const float v0 = __fmul_rn(__fmul_rn(x0, r), w0), v1 = __fmul_rn(__fmul_rn(x1, r), w1);
  if (hout) hout[(size_t)m * K + i0] = v0;
  quantize_value<false>(v0, m, i0, Mp, K, aq, asc, absum);
  if (two) {
    if (hout) hout[(size_t)m * K + i1] = v1;
    quantize_value<false>(v1, m, i1, Mp, K, aq, asc, absum);
  }
}

int check_quant_args(const float* x, int ldx, int M, int Mp, int K, const int8_t* aq, const float* asc, int width_needed) {
  if (!x || !aq || !asc) IZB_FAIL(IZB_ERR_ARG, "quantize: null pointer");
  if (K <= 0 || K % 256) IZB_FAIL(IZB_ERR_SHAPE, "quantize: K = %d is not a positive multiple of 256", K);
  if (Mp <= 0 || Mp % 16 || M < 0 || M > Mp) IZB_FAIL(IZB_ERR_SHAPE, "quantize: rows %d of Mp = %d (Mp must be a multiple of 16)", M, Mp);
  if (ldx < width_needed) IZB_FAIL(IZB_ERR_SHAPE, "quantize: row stride %d shorter than the row (%d)", ldx, width_needed);
  if (ldx % 4 || !izb_aligned(x, 16)) IZB_FAIL(IZB_ERR_ALIGN, "quantize: input rows must be 16-byte aligned (ldx %% 4 == 0)");
  if (!izb_aligned(aq, 16) || !izb_aligned(asc, 4)) IZB_FAIL(IZB_ERR_ALIGN, "quantize: outputs not aligned");
  return IZB_OK;
}

}  // namespace

// two byte ranges share memory
static bool overlap(const void* a, size_t na, const void* b, size_t nb) {
  const uintptr_t x = (uintptr_t)a, y = (uintptr_t)b;
  return x < y + nb && y < x + na;
}

// Few rows -- blocks of one row that fit the device at once, four times as many with the SwiGLU product -- take a thread per value.  (us, a thread
// per eight values / per value: quantise 1 x 5120 2.2 / 1.2, 32 x 768 2.1 / 1.2, 128 x 2048 2.1 / 2.0, 64 x 5120 2.2 / 2.3, 256 x 5120 3.7 / 5.9; SwiGLU 1 x
// 17408 2.9 / 1.4, 32 x 5120 4.7 / 2.0, 64 x 17408 7.5 / 5.8, 100 x 17408 7.8 / 8.3, 512 x 5120 8.5 / 11.9.)
template <int kMode>
static int launch_quantize(const char* what, const float* x, int ldx, int M, int Mp, int K, int8_t* aq, float* asc, int16_t* absum, float* hout, cudaStream_t st) {
  const dim3 few(K / 256, M + (Mp > M ? 1 : 0));
  if (izb_one_wave(dim3(few.x, kMode == 1 ? (few.y + 3) / 4 : few.y), 256) && Mp - M <= 256) {
    IZB_LAUNCH(what, st, izb_launch_pdl(quantize_few_kernel<kMode>, few, 256, 0, st, x, ldx, M, Mp, K, aq, asc, absum, hout, K));
  } else {
    dim3 grid(K / 256, (Mp + 31) / 32);
    IZB_LAUNCH(what, st, izb_launch_pdl(quantize_act_kernel<kMode>, grid, 256, 0, st, x, ldx, M, Mp, K, aq, asc, absum, hout, K));
  }
  return IZB_OK;
}

extern "C" int izb_quantize_act(const float* d_x, int ldx, int M_valid, int Mp, int K, int8_t* d_aq, float* d_asc,
                                int16_t* d_absum, void* stream) {
  if (int rc = check_quant_args(d_x, ldx, M_valid, Mp, K, d_aq, d_asc, K)) return rc;
  return launch_quantize<0>("quantize_act", d_x, ldx, M_valid, Mp, K, d_aq, d_asc, d_absum, nullptr, (cudaStream_t)stream);
}

extern "C" int izb_swiglu_quant(const float* d_gu, int ldgu, int split, int M_valid, int Mp, int F, float* d_h, int8_t* d_aq,
                                float* d_asc, int16_t* d_absum, void* stream) {
  if (int rc = check_quant_args(d_gu, ldgu, M_valid, Mp, F, d_aq, d_asc, split ? 2 * F : F)) return rc;
  if (d_h && !izb_aligned(d_h, 16)) IZB_FAIL(IZB_ERR_ALIGN, "swiglu_quant: h not 16-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  return split ? launch_quantize<1>("swiglu_quant", d_gu, ldgu, M_valid, Mp, F, d_aq, d_asc, d_absum, d_h, st)
               : launch_quantize<0>("quantize_act", d_gu, ldgu, M_valid, Mp, F, d_aq, d_asc, d_absum, nullptr, st);
}

extern "C" int izb_rmsnorm_quant(const float* d_x, int ldx, const float* d_w, float eps, int M_valid, int Mp, int K, float* d_h,
                                 int8_t* d_aq, float* d_asc, int16_t* d_absum, void* stream) {
  if (int rc = check_quant_args(d_x, ldx, M_valid, Mp, K, d_aq, d_asc, K)) return rc;
  if (!d_w) IZB_FAIL(IZB_ERR_ARG, "rmsnorm_quant: null weight");
  if (!izb_aligned(d_w, 16) || (d_h && !izb_aligned(d_h, 16))) IZB_FAIL(IZB_ERR_ALIGN, "rmsnorm_quant: w and h must be 16-byte aligned");
  if (!(eps >= 0.0f)) IZB_FAIL(IZB_ERR_ARG, "rmsnorm_quant: eps = %g", (double)eps);
  cudaStream_t st = (cudaStream_t)stream;
  const int groups = (K / 8 + 255) / 256;  // of 8 values per thread
  // decode steps over long rows (us, a CTA per row / several: 4096, one row 2.0/1.8, eight 2.1/2.1; 5120, one 2.3/1.9, eight 2.4/2.2, sixteen 2.4/3.0; 12288, one
  // 3.6/2.7, eight 3.6/3.4; 2048, one 1.5/1.6)
  // (not over its own input, which other blocks still read)
  const size_t xb = M_valid > 0 ? ((size_t)(M_valid - 1) * ldx + K) * 4 : 0;
  const bool apart = !(d_h && overlap(d_x, xb, d_h, (size_t)M_valid * K * 4)) && !overlap(d_x, xb, d_aq, (size_t)Mp * K) && !overlap(d_x, xb, d_asc, (size_t)Mp * (K / 8)) &&
                     !(d_absum && overlap(d_x, xb, d_absum, (size_t)Mp * (K / 8)));
  if (M_valid <= 8 && K >= 4096 && groups <= 8 && Mp <= 65535 && apart) {
    auto kernel = groups <= 2 ? rmsnorm_few_kernel<2> : groups <= 3 ? rmsnorm_few_kernel<3> : groups <= 4 ? rmsnorm_few_kernel<4> : rmsnorm_few_kernel<8>;
    IZB_LAUNCH("rmsnorm_quant", st, izb_launch_pdl(kernel, dim3((K + 511) / 512, Mp), 256, 0, st, d_x, ldx, d_w, K, eps, M_valid, Mp, d_h, d_aq, d_asc, d_absum));
    return IZB_OK;
  }
  // Rows held in registers cost blocks per SM: many long rows are faster read twice (us, held / read twice: 16384, 296 rows 13.5/12.9, 450 rows
  // 17.6/15.2, 4096 rows 126/83; 8448, 1000 rows 14.6/16.1, 4096 rows 54/46; 12288, 2000 rows 35/39, 4096 rows 66/63)
  int dev = 0;
  if (groups > 4) IZB_CUDA(cudaGetDevice(&dev));
  const bool hold = groups <= 4 || M_valid <= izb_sm_count(dev) * (groups <= 6 ? 14 : 2);
  auto kernel = !hold ? rmsnorm_quant_row_kernel<0> : groups <= 1 ? rmsnorm_quant_row_kernel<1> : groups <= 2 ? rmsnorm_quant_row_kernel<2> : groups <= 3 ? rmsnorm_quant_row_kernel<3>
              : groups <= 4 ? rmsnorm_quant_row_kernel<4> : groups <= 6 ? rmsnorm_quant_row_kernel<6> : groups <= 8 ? rmsnorm_quant_row_kernel<8>
                                                                                                                 : rmsnorm_quant_row_kernel<0>;
  IZB_LAUNCH("rmsnorm_quant", st, izb_launch_pdl(kernel, Mp, 256, 0, st, d_x, ldx, d_w, K, eps, M_valid, Mp, d_h, d_aq, d_asc, d_absum));
  return IZB_OK;
}

extern "C" int izb_add_norm_quant(float* d_x, const float* d_t, const float* d_w, float eps, float s, const float* d_w2, int M_valid,
                                  int Mp, int K, int8_t* d_aq, float* d_asc, int16_t* d_absum, void* stream) {
  if (!d_x || !d_t || !d_w || !d_aq || !d_asc) IZB_FAIL(IZB_ERR_ARG, "add_norm_quant: null pointer");
  if (K <= 0 || K % 256 || K > 256 * kAnqMax) IZB_FAIL(IZB_ERR_SHAPE, "add_norm_quant: K = %d (a multiple of 256 up to %d)", K, 256 * kAnqMax);
  if (Mp <= 0 || Mp % 16 || M_valid < 0 || M_valid > Mp) IZB_FAIL(IZB_ERR_SHAPE, "add_norm_quant: rows %d of Mp = %d (Mp must be a multiple of 16)", M_valid, Mp);
  if (!(eps >= 0.0f)) IZB_FAIL(IZB_ERR_ARG, "add_norm_quant: eps = %g", (double)eps);
  cudaStream_t st = (cudaStream_t)stream;
  const int nk = K / 256;  // elements per thread
  int dev = 0;
  IZB_CUDA(cudaGetDevice(&dev));
  // A cluster per row while there are up to three CTAs per SM (us, a CTA per row / a cluster: 2048, one row 4.0/2.6, 100 rows 5.3/4.3; 4096, one 6.6/3.0,
  // 32 6.9/4.2, 64 7.4/7.3, 100 7.6/9.6; 5120, one 8.2/3.5, 100 9.4/11; 1024, one 2.7/2.5, 100 3.0/3.1).  It ends at 5120 because every CTA holds the whole of three
  // rows in registers, 60 per thread there; it is not written for longer rows, of which a CTA takes 18 us for eight of 8192
  const int cl = nk <= 16 ? (nk + 1) / 2 : 7, steps = (nk + cl - 1) / cl;
  if (nk > 4 && nk <= 20 && (long long)cl * Mp <= 3 * izb_sm_count(dev)) {
    auto kernel = nk <= 8 ? add_norm_few_kernel<8> : nk <= 16 ? add_norm_few_kernel<16> : add_norm_few_kernel<20>;
    IZB_LAUNCH("add_norm_quant", st, izb_launch_pdl_cluster(kernel, cl, dim3(cl, Mp), 256, 0, st, d_x, d_t, d_w, K, eps, s, d_w2, M_valid, Mp, d_aq, d_asc, d_absum, steps));
    return IZB_OK;
  }
  auto kernel = nk <= 4 ? add_norm_quant_kernel<4, true> : nk <= 8 ? add_norm_quant_kernel<8, true> : nk <= 16 ? add_norm_quant_kernel<16, true>
              : nk <= 20 ? add_norm_quant_kernel<20, true> : nk <= 32 ? add_norm_quant_kernel<32, true>
              : M_valid <= izb_sm_count(dev) ? add_norm_quant_kernel<kAnqMax, true> : add_norm_quant_kernel<kAnqMax, false>;
  IZB_LAUNCH("add_norm_quant", st, izb_launch_pdl(kernel, Mp, 256, 0, st, d_x, d_t, d_w, K, eps, s, d_w2, M_valid, Mp, d_aq, d_asc, d_absum));
  return IZB_OK;
}

// ---------------------------------------------------------------------------------------------- logit soft-cap
// softcap_rows (zero/kernels/ops_attn_g.cl:724) and the output head's HEAD_OUT (zero/kernels/decode.cl:882-887):
// v = cap * tanh(v * (1 / cap)) on columns off .. off+N-1 of `rows` rows.  One float4 per thread where the row start is
// 16-byte aligned, scalars otherwise.
namespace {
template <bool kAhead>  // launched ahead of the kernel before
__global__ void __launch_bounds__(256) softcap_rows_kernel(float* __restrict__ C, int ld, int off, int N, float cap, float rcap, int vec) {
  float* p = C + (size_t)blockIdx.y * ld + off;
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (kAhead) {
    pdl_launch_next();
    pdl_wait();
  }
  if (vec) {
    if (4 * i + 3 < N) {
      float4 v = *reinterpret_cast<float4*>(p + 4 * i);
      v.x = __fmul_rn(cap, tanhf(__fmul_rn(v.x, rcap)));
      v.y = __fmul_rn(cap, tanhf(__fmul_rn(v.y, rcap)));
      v.z = __fmul_rn(cap, tanhf(__fmul_rn(v.z, rcap)));
      v.w = __fmul_rn(cap, tanhf(__fmul_rn(v.w, rcap)));
      *reinterpret_cast<float4*>(p + 4 * i) = v;
    } else {
      for (int n = 4 * i; n < N; ++n) p[n] = __fmul_rn(cap, tanhf(__fmul_rn(p[n], rcap)));
    }
  } else if (i < N) {
    p[i] = __fmul_rn(cap, tanhf(__fmul_rn(p[i], rcap)));
  }
}
}  // namespace

extern "C" int izb_softcap_rows(float* d_C, int rows, int ld, int off, int N, float cap, void* stream) {
  if (!d_C) IZB_FAIL(IZB_ERR_ARG, "softcap_rows: null pointer");
  if (rows < 0 || N < 0 || off < 0 || (rows > 1 && ld < off + N)) IZB_FAIL(IZB_ERR_SHAPE, "softcap_rows: rows=%d ld=%d off=%d N=%d", rows, ld, off, N);
  if (!(cap > 0.0f)) IZB_FAIL(IZB_ERR_ARG, "softcap_rows: cap = %g (must be positive)", (double)cap);
  if (rows == 0 || N == 0) return IZB_OK;
  if (rows > 65535) IZB_FAIL(IZB_ERR_LIMIT, "softcap_rows: %d rows (at most 65535 per call)", rows);
  cudaStream_t st = (cudaStream_t)stream;
  const int vec = izb_aligned(d_C, 16) && ld % 4 == 0 && off % 4 == 0;
  const int per_row = vec ? (N + 3) / 4 : N;
  dim3 grid((per_row + 255) / 256, rows);
  // (us with / without dependent launch: 8192 logits x 1000 rows 10.1/9.2, x 8 rows 1.8/2.3)
  if (izb_one_wave(grid, 256))
    IZB_LAUNCH("softcap_rows", st, izb_launch_pdl(softcap_rows_kernel<true>, grid, 256, 0, st, d_C, ld, off, N, cap, 1.0f / cap, vec));
  else
    IZB_LAUNCH("softcap_rows", st, softcap_rows_kernel<false><<<grid, 256, 0, st>>>(d_C, ld, off, N, cap, 1.0f / cap, vec));
  return IZB_OK;
}

// ---------------------------------------------------------------------------------------------- SwiGLU of interleaved columns
// gu [M][ldgu]: the outputs of a gate | up weight whose rows alternate in groups of 32 (izb_weight_create_gateup): columns
// 64 j .. 64 j + 31 are gate outputs, 64 j + 32 .. 64 j + 63 the up outputs of the same FFN rows.
// C[m][c_off + 32 j + i] = up * silu(gate) (zero/kernels/gemm.cl:562-565).  Used where the tensor-core GEMM, which forms
// this product in its epilogue, does not take the call.
namespace {
__global__ void __launch_bounds__(256) swiglu_pairs_kernel(const float* __restrict__ gu, int ldgu, int F, float* __restrict__ C, int ldc, int c_off) {
  const int f = blockIdx.x * 256 + threadIdx.x;
  if (f >= F) return;
  const float* row = gu + (size_t)blockIdx.y * ldgu + 64 * (f >> 5) + (f & 31);
  const float g = row[0], u = row[32];
  C[(size_t)blockIdx.y * ldc + c_off + f] = __fmul_rn(u, __fdiv_rn(g, __fadd_rn(1.0f, expf(-g))));
}
}  // namespace

int izb_swiglu_pairs_launch(const float* gu, int ldgu, int M, int F, float* C, int ldc, int c_off, cudaStream_t st) {
  dim3 grid((F + 255) / 256, M);
  IZB_LAUNCH("swiglu_pairs", st, swiglu_pairs_kernel<<<grid, 256, 0, st>>>(gu, ldgu, F, C, ldc, c_off));
  return IZB_OK;
}
