// One to eight activation rows against a weight matrix on the warp-level integer matrix instruction (mma.sync, K = 16: int8 x
// int8 -> int32): decode batches and the per-tile mixture-of-experts products (the latter by dp4a while a tile has one or two slots).
//
// Such a call is bound by the weights' bytes, but the dot-product kernels (csrc/izb_gemv_stream.cu, csrc/izb_types.cu) spend
// instructions per weight AND token: at five rows the unpacked nibbles are multiplied five times by dp4a.  One matrix
// instruction multiplies 16 weight rows x 16 elements with eight tokens at once, so eight tokens cost what one does.  (The
// tcgen05 kernel wants 128 tokens per tile; at eight it is all latency.)
//
// The sums are those of gemv_stream_kernel, gemv_q6p_kernel and the per-tile expert kernels bit for bit, so that a row's result does not
// depend on which of these its call's size selects (a decode step requantises it, and one value that crosses a rounding boundary changes
// every layer after it).  Not those of the Q4_K kernels for one to four rows of K % 1024 == 0, N >= 1024 (gemv_q4k_*), which add in an order of
// their own: there four and five rows differ in last bits.  Per
// output the same 32 partial sums -- superblock index modulo kSubs x piece of a superblock -- each added up in superblock order
// with the same roundings, then the same pairwise tree.  A piece is 16 elements of a block pair (Q4_K), 16 elements (Q8_0) or a
// 32-block (Q6_K), hence K = 16.  (One sum per output with the min term on a bf16 matrix instruction is a third of the f32
// work and took 24 us for 34816 x 5120 at five rows, but moved int8 values of the next projection's input.)  Products of the
// small integers and fp16 scales that those kernels multiply one after the other are exact in f32, so they may be formed once per
// row and block: P = fma(d * sc, dot, -(dmin * mn) * asum).
//
// Lane mapping (g = lane / 4, t = lane % 4): the weight rows are the instruction's M side, the tokens its N side.  A lane supplies
// bytes 4t .. 4t+3 of a 16-element half of rows g, g + 8 and of token g, and receives rows g, g + 8 against tokens 2t, 2t + 1:
// register pairs, so all f32 work runs on packed pairs.  Dots reach f32 by starting the accumulator at the bits of 1.5 * 2^23 and
// subtracting that number (|dot| < 2^22): exact and cheaper than a conversion.  High nibbles are multiplied in place as 16 q.
//
// Both operands come from shared memory: each warp has a ring of 16-row x one-superblock chunks filled by TMA (row pitches of 4 mod
// 8 words: 32-bit reads of eight rows x four words touch every bank once), the activations are staged once per CTA, and what
// a row's header holds is expanded once per chunk (per row and block) for the whole quad.  kSubs warps share
// a tile, so that neighbouring superblocks of the same rows are in flight together: rings of scattered tiles ran at half the
// DRAM rate.  The ring's first fill is issued before pdl_wait() (no kernel writes weights).
//
// Up to four tokens would leave half of the instruction's columns empty, and with them half of every lane's f32 work.  There one instruction
// takes 32 elements, two pieces: columns 0-3 are the tokens with zeros for the second piece, columns 4-7 the same tokens with zeros for
// the first, so that each lane has half of the pieces and all of its work counts (mul4; the K = 32 instruction takes the tensor pipe's 8 clk like
// the K = 16 one).  The sums are the same and in the same order; half as many accumulators also halve what the warps of a tile exchange.
// (us before / now: Q6_K 151936 x 5120 three rows 149 / 118, 32000 x 4096 three 30 / 24; Q4_K 16384 x 5376 three 20.8 / 16.5, 5120 x 13824 four 27 /
// 19; Q8_0 4096 x 14336 one 17.2 / 15.1, 8192 x 4096 four 8.8 / 7.8.)
//
// Measured (us, dot-product kernels / this one; the time at the copy's bandwidth): Q4_K 34816 x 5120 five rows 52.3 / 34.4 (15.3), eight
// 75.7 / 35.1; 128000 x 4096 eight 218 / 89 (45); Q8_0 151936 x 2048 eight 136 / 57 (51); Q6_K 32000 x 4096 three 44 / 24 (17).  The
// Q4_K case is bound by instruction issue (56 % of the cycles) and shared-memory latency: about 450 warp instructions per chunk, of
// which 128 are the 32 partial sums' f32 work that the other kernels' order asks for.
#include <cuda.h>
#include <string.h>

#include "izb_common.cuh"

namespace {

constexpr uint32_t kMagic = 0x4B400000u;  // 1.5 * 2^23

// d = c + rows g (d[0], d[1]) and g + 8 (d[2], d[3]) . tokens 2t, 2t + 1, over 16 elements
__device__ __forceinline__ void dot16_u8(int (&d)[4], uint32_t w0, uint32_t w1, uint32_t x, uint32_t c0 = kMagic, uint32_t c1 = kMagic) {
  asm("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%8,%7,%8};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(w0), "r"(w1), "r"(x), "r"(c0), "r"(c1));
}
__device__ __forceinline__ void dot16_s8(int (&d)[4], uint32_t w0, uint32_t w1, uint32_t x) {
  asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(w0), "r"(w1), "r"(x), "r"(kMagic));
}

// The same with up to four tokens: 32 elements, of which columns 0-3 meet the first 16 (their words of the other 16 are zero) and
// columns 4-7, the same tokens again, the last 16.
__device__ __forceinline__ void dot32_u8(int (&d)[4], uint32_t w0, uint32_t w1, uint32_t v0, uint32_t v1, uint32_t x, uint32_t y, uint32_t c0 = kMagic, uint32_t c1 = kMagic) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%10,%11};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(w0), "r"(w1), "r"(v0), "r"(v1), "r"(x), "r"(y), "r"(c0), "r"(c1));
}
__device__ __forceinline__ void dot32_s8(int (&d)[4], uint32_t w0, uint32_t w1, uint32_t v0, uint32_t v1, uint32_t x, uint32_t y) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(w0), "r"(w1), "r"(v0), "r"(v1), "r"(x), "r"(y), "r"(kMagic));
}

// f32 pairs (tokens 2t, 2t + 1): two IEEE operations per instruction
typedef unsigned long long f2;
__device__ __forceinline__ f2 f2_of(float x, float y) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ float f2_get(f2 a, int i) { return __uint_as_float((uint32_t)(i ? a >> 32 : a)); }
// the integer instruction's accumulators of row g + 8 r as f32: minus the number they started from
__device__ __forceinline__ f2 unmagic(const int (&d)[4], int r) {
  return f2_add(f2_of(__int_as_float(d[2 * r]), __int_as_float(d[2 * r + 1])), 0xCB400000CB400000ull);
}
// c + the unsigned bytes of w . the signed bytes of x
__device__ __forceinline__ int dot_u8(uint32_t w, uint32_t x, int c) {
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(w), "r"(x), "r"(c));
  return d;
}
// unsigned byte k of a word as f32: 0x4B000000 | byte is 2^23 + byte
__device__ __forceinline__ float byte_f(uint32_t w, int k) { return __fsub_rn(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440 + k)), 8388608.0f); }

// What the weights are multiplied with, in shared memory (offsets of this lane):
//   q   token g: words of the first and second 16 elements of a block, `qs` bytes per block
//   sc  scales of tokens 2t, 2t + 1, four pairs per block
//   ex  per block and half, four pairs: Q4_K the sum of the 16 values as f32; Q6_K the accumulator's start, kMagic - 32 * that sum
// For mul4 token g % 4, tokens 2 (t % 2), + 1, and of two pieces the one that the column meets.
struct Acts {
  const unsigned char* q;
  const f2* sc;
  const f2* ex;
  int qs;
  f2 neg_zero;  // (-0, -0), from a number that only the launch knows
  uint32_t first, last;  // mul4: masks, all ones in lanes whose column g meets the first / the last 16 elements
};

// ---- weight forms.  prep() expands the headers of a chunk into `hd` ([block][row]); mul() multiplies a chunk into
// the piece sums acc[piece][r]: rows g, g + 8 against tokens 2t, 2t + 1.  mul4(), for up to four tokens: rows g, g + 8 against tokens
// 2 (t % 2), + 1, and the half of the pieces whose number has t / 2 at bit kLaneBit.
struct RQ4K {
  static constexpr int SBB = 144, kPitch = 144, kSubs = 4, kPieces = 8, kDotWarps = 16;
  static constexpr bool kEx = true, kPrep = true;
  // (d * sc, -dmin * mn) of a row's blocks 4 up .. + 3; the sub-block scales and mins as bytes (get_scale_min_k4,
  // src/quants.h:61-69).  Odd blocks meet 16 q: their d * sc is divided by 16.
  static __device__ __forceinline__ void header(const unsigned char* chunk, int row, int up, float2 (&o)[4]) {
    const uint4 h = *reinterpret_cast<const uint4*>(chunk + row * kPitch);
    const float2 d = __half22float2(*reinterpret_cast<const __half2*>(&h.x));
    const uint32_t sc = up ? (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u) : h.y & 0x3F3F3F3Fu;
    const uint32_t mn = up ? ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u) : h.z & 0x3F3F3F3Fu;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      o[k] = make_float2(__fmul_rn((k & 1) ? d.x * 0.0625f : d.x, byte_f(sc, k)), __fmul_rn(-d.y, byte_f(mn, k)));
    }
  }
  static __device__ __forceinline__ void prep(const unsigned char* chunk, float2* hd, int lane) {
    const int row = lane >> 1, up = lane & 1;
    float2 h[4];
    header(chunk, row, up, h);
#pragma unroll
    for (int k = 0; k < 4; ++k) hd[(4 * up + k) * 16 + row] = h[k];
  }
  // The same products by dp4a: lane <-> row lane % 16 and pieces 4 up .. + 3 of the superblock (up = lane / 16), TT tokens of the T staged
  template <int TT>
  static __device__ __forceinline__ void dot(const unsigned char* chunk, const unsigned char* act, int nb, int T, int sb, int lane, float (&acc)[TT][kPieces / 2]) {
    const int row = lane & 15, up = lane >> 4, b0 = 8 * sb + 4 * up;
    float2 hd[4];
    header(chunk, row, up, hd);
    const float* sc = reinterpret_cast<const float*>(act + (size_t)nb * 32 * T) + b0 * 8;
    const float* ex = reinterpret_cast<const float*>(act + (size_t)nb * 32 * T) + nb * 8 + b0 * 16;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const uint4* w = reinterpret_cast<const uint4*>(chunk + row * kPitch + 16 + 64 * up + 32 * c);
      const uint4 w0 = w[0], w1 = w[1];
#pragma unroll
      for (int j = 0; j < TT; ++j) {
        if (j >= T) break;
        const uint4 *l = reinterpret_cast<const uint4*>(act + (size_t)((b0 + 2 * c) * T + j) * 32), *h = l + 2 * T;
        const uint4 l0 = l[0], l1 = l[1], h0 = h[0], h1 = h[1];  // (words of the two halves alternate)
        const float* e = ex + 32 * c + j;
        const float sl = sc[16 * c + j], sh = sc[16 * c + 8 + j];
        int dl0 = 0, dl1 = 0, dh0 = 0, dh1 = 0;
        dl0 = dot_u8(w0.x & 0x0F0F0F0Fu, l0.x, dl0); dl0 = dot_u8(w0.y & 0x0F0F0F0Fu, l0.z, dl0); dl0 = dot_u8(w0.z & 0x0F0F0F0Fu, l1.x, dl0); dl0 = dot_u8(w0.w & 0x0F0F0F0Fu, l1.z, dl0);
        dl1 = dot_u8(w1.x & 0x0F0F0F0Fu, l0.y, dl1); dl1 = dot_u8(w1.y & 0x0F0F0F0Fu, l0.w, dl1); dl1 = dot_u8(w1.z & 0x0F0F0F0Fu, l1.y, dl1); dl1 = dot_u8(w1.w & 0x0F0F0F0Fu, l1.w, dl1);
        dh0 = dot_u8(w0.x & 0xF0F0F0F0u, h0.x, dh0); dh0 = dot_u8(w0.y & 0xF0F0F0F0u, h0.z, dh0); dh0 = dot_u8(w0.z & 0xF0F0F0F0u, h1.x, dh0); dh0 = dot_u8(w0.w & 0xF0F0F0F0u, h1.z, dh0);
        dh1 = dot_u8(w1.x & 0xF0F0F0F0u, h0.y, dh1); dh1 = dot_u8(w1.y & 0xF0F0F0F0u, h0.w, dh1); dh1 = dot_u8(w1.z & 0xF0F0F0F0u, h1.y, dh1); dh1 = dot_u8(w1.w & 0xF0F0F0F0u, h1.w, dh1);
        const float2 a = hd[2 * c], b = hd[2 * c + 1];
        const float p0 = __fmaf_rn(a.x, (float)dl0, __fmul_rn(a.y, e[0])), q0 = __fmaf_rn(b.x, (float)dh0, __fmul_rn(b.y, e[16]));
        const float p1 = __fmaf_rn(a.x, (float)dl1, __fmul_rn(a.y, e[8])), q1 = __fmaf_rn(b.x, (float)dh1, __fmul_rn(b.y, e[24]));
        acc[j][2 * c] = __fadd_rn(acc[j][2 * c], __fmaf_rn(sl, p0, __fmul_rn(sh, q0)));
        acc[j][2 * c + 1] = __fadd_rn(acc[j][2 * c + 1], __fmaf_rn(sl, p1, __fmul_rn(sh, q1)));
      }
    }
  }
  static __device__ __forceinline__ void mul(const unsigned char* chunk, const float2* hd, const Acts& a, int sb, int g, int t, f2 (&acc)[kPieces][2]) {
    const unsigned char* p = chunk + g * kPitch + 16 + 4 * t;
    const unsigned char* xq = a.q + 8 * sb * a.qs;
    const f2 *xs = a.sc + 32 * sb, *xe = a.ex + 64 * sb;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const uint2 xl = *reinterpret_cast<const uint2*>(xq + 2 * c * a.qs), xh = *reinterpret_cast<const uint2*>(xq + (2 * c + 1) * a.qs);
      const f2 sl = xs[8 * c], sh = xs[8 * c + 4];
      f2 hl[2][2], hh[2][2];  // (d * sc, -dmin * mn) of rows g, g + 8: low-nibble and high-nibble block
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float2 u = hd[2 * c * 16 + g + 8 * r], v = hd[(2 * c + 1) * 16 + g + 8 * r];
        hl[r][0] = f2_of(u.x, u.x); hl[r][1] = f2_of(u.y, u.y);
        hh[r][0] = f2_of(v.x, v.x); hh[r][1] = f2_of(v.y, v.y);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t w0 = *reinterpret_cast<const uint32_t*>(p + 32 * c + 16 * h), w1 = *reinterpret_cast<const uint32_t*>(p + 8 * kPitch + 32 * c + 16 * h);
        const f2 el = xe[16 * c + 4 * h], eh = xe[16 * c + 8 + 4 * h];
        int dl[4], dh[4];
        dot16_u8(dl, w0 & 0x0F0F0F0Fu, w1 & 0x0F0F0F0Fu, h ? xl.y : xl.x);
        dot16_u8(dh, w0 & 0xF0F0F0F0u, w1 & 0xF0F0F0F0u, h ? xh.y : xh.x);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const f2 P = f2_fma(hl[r][0], unmagic(dl, r), f2_mul(hl[r][1], el)), Q = f2_fma(hh[r][0], unmagic(dh, r), f2_mul(hh[r][1], eh));
          acc[2 * c + h][r] = f2_add(acc[2 * c + h][r], f2_fma(sl, P, f2_mul(sh, Q)));
        }
      }
    }
  }
  // lane's pieces: 2c + t / 2
  static constexpr int kLaneBit = 0;
  static __device__ __forceinline__ void mul4(const unsigned char* chunk, const float2* hd, const Acts& a, int sb, int g, int t, f2 (&acc)[kPieces / 2][2]) {
    const unsigned char* p = chunk + g * kPitch + 16 + 4 * t;
    const unsigned char* xq = a.q + 8 * sb * a.qs;
    const f2 *xs = a.sc + 32 * sb, *xe = a.ex + 64 * sb;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const uint32_t xl = *reinterpret_cast<const uint32_t*>(xq + 2 * c * a.qs), xh = *reinterpret_cast<const uint32_t*>(xq + (2 * c + 1) * a.qs);
      const f2 sl = xs[8 * c], sh = xs[8 * c + 4], el = xe[16 * c], eh = xe[16 * c + 8];
      const uint32_t w0 = *reinterpret_cast<const uint32_t*>(p + 32 * c), w1 = *reinterpret_cast<const uint32_t*>(p + 8 * kPitch + 32 * c);
      const uint32_t v0 = *reinterpret_cast<const uint32_t*>(p + 32 * c + 16), v1 = *reinterpret_cast<const uint32_t*>(p + 8 * kPitch + 32 * c + 16);
      int dl[4], dh[4];
      dot32_u8(dl, w0 & 0x0F0F0F0Fu, w1 & 0x0F0F0F0Fu, v0 & 0x0F0F0F0Fu, v1 & 0x0F0F0F0Fu, xl & a.first, xl & a.last);
      dot32_u8(dh, w0 & 0xF0F0F0F0u, w1 & 0xF0F0F0F0u, v0 & 0xF0F0F0F0u, v1 & 0xF0F0F0F0u, xh & a.first, xh & a.last);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float2 u = hd[2 * c * 16 + g + 8 * r], v = hd[(2 * c + 1) * 16 + g + 8 * r];
        const f2 P = f2_fma(f2_of(u.x, u.x), unmagic(dl, r), f2_mul(f2_of(u.y, u.y), el)), Q = f2_fma(f2_of(v.x, v.x), unmagic(dh, r), f2_mul(f2_of(v.y, v.y), eh));
        acc[c][r] = f2_add(acc[c][r], f2_fma(sl, P, f2_mul(sh, Q)));
      }
    }
  }
};

struct RQ80 {
  static constexpr int SBB = 272, kPitch = 272, kSubs = 2, kPieces = 16, kDotWarps = 16;
  static constexpr bool kEx = false, kPrep = false;
  static __device__ __forceinline__ void prep(const unsigned char*, float2*, int) {}
  template <int TT>
  static __device__ __forceinline__ void dot(const unsigned char* chunk, const unsigned char* act, int nb, int T, int sb, int lane, float (&acc)[TT][kPieces / 2]) {
    const int row = lane & 15, up = lane >> 4, b0 = 8 * sb + 4 * up;
    const uint2 hd = *reinterpret_cast<const uint2*>(chunk + row * kPitch + 8 * up);
    const float* sc = reinterpret_cast<const float*>(act + (size_t)nb * 32 * T) + b0 * 8;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const uint4* w = reinterpret_cast<const uint4*>(chunk + row * kPitch + 16 + 128 * up + 32 * b);
      const uint4 w0 = w[0], w1 = w[1];
      const uint32_t hw = b < 2 ? hd.x : hd.y;
      const float d = half_bits_to_float((b & 1) ? hw >> 16 : hw & 0xFFFFu);
#pragma unroll
      for (int j = 0; j < TT; ++j) {
        if (j >= T) break;
        const uint4* x = reinterpret_cast<const uint4*>(act + (size_t)((b0 + b) * T + j) * 32);
        const uint4 x0 = x[0], x1 = x[1];  // (words of the two halves alternate)
        int d0 = 0, d1 = 0;
        d0 = __dp4a((int)w0.x, (int)x0.x, d0); d0 = __dp4a((int)w0.y, (int)x0.z, d0); d0 = __dp4a((int)w0.z, (int)x1.x, d0); d0 = __dp4a((int)w0.w, (int)x1.z, d0);
        d1 = __dp4a((int)w1.x, (int)x0.y, d1); d1 = __dp4a((int)w1.y, (int)x0.w, d1); d1 = __dp4a((int)w1.z, (int)x1.y, d1); d1 = __dp4a((int)w1.w, (int)x1.w, d1);
        const float sd = __fmul_rn(sc[8 * b + j], d);
        acc[j][2 * b] = __fmaf_rn(sd, (float)d0, acc[j][2 * b]);
        acc[j][2 * b + 1] = __fmaf_rn(sd, (float)d1, acc[j][2 * b + 1]);
      }
    }
  }
  static __device__ __forceinline__ void mul(const unsigned char* chunk, const float2*, const Acts& a, int sb, int g, int t, f2 (&acc)[kPieces][2]) {
    const unsigned char* p = chunk + g * kPitch;
    const uint4 hd[2] = {*reinterpret_cast<const uint4*>(p), *reinterpret_cast<const uint4*>(p + 8 * kPitch)};
    p += 16 + 4 * t;
    const unsigned char* xq = a.q + 8 * sb * a.qs;
    const f2* xs = a.sc + 32 * sb;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const uint2 x = *reinterpret_cast<const uint2*>(xq + b * a.qs);
      f2 sd[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const uint32_t w = (b >> 1) == 0 ? hd[r].x : (b >> 1) == 1 ? hd[r].y : (b >> 1) == 2 ? hd[r].z : hd[r].w;
        const float d = half_bits_to_float((b & 1) ? w >> 16 : w & 0xFFFFu);
        sd[r] = f2_mul(xs[4 * b], f2_of(d, d));
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        int d[4];
        dot16_s8(d, *reinterpret_cast<const uint32_t*>(p + 32 * b + 16 * h), *reinterpret_cast<const uint32_t*>(p + 8 * kPitch + 32 * b + 16 * h), h ? x.y : x.x);
#pragma unroll
        for (int r = 0; r < 2; ++r) acc[2 * b + h][r] = f2_fma(sd[r], unmagic(d, r), acc[2 * b + h][r]);
      }
    }
  }
  // lane's pieces: 2b + t / 2
  static constexpr int kLaneBit = 0;
  static __device__ __forceinline__ void mul4(const unsigned char* chunk, const float2*, const Acts& a, int sb, int g, int t, f2 (&acc)[kPieces / 2][2]) {
    const unsigned char* p = chunk + g * kPitch;
    const uint4 hd[2] = {*reinterpret_cast<const uint4*>(p), *reinterpret_cast<const uint4*>(p + 8 * kPitch)};
    p += 16 + 4 * t;
    const unsigned char* xq = a.q + 8 * sb * a.qs;
    const f2* xs = a.sc + 32 * sb;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const uint32_t x = *reinterpret_cast<const uint32_t*>(xq + b * a.qs);
      int d[4];
      dot32_s8(d, *reinterpret_cast<const uint32_t*>(p + 32 * b), *reinterpret_cast<const uint32_t*>(p + 8 * kPitch + 32 * b), *reinterpret_cast<const uint32_t*>(p + 32 * b + 16),
               *reinterpret_cast<const uint32_t*>(p + 8 * kPitch + 32 * b + 16), x & a.first, x & a.last);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const uint32_t w = (b >> 1) == 0 ? hd[r].x : (b >> 1) == 1 ? hd[r].y : (b >> 1) == 2 ? hd[r].z : hd[r].w;
        const float s = half_bits_to_float((b & 1) ? w >> 16 : w & 0xFFFFu);
        acc[b][r] = f2_fma(f2_mul(xs[4 * b], f2_of(s, s)), unmagic(d, r), acc[b][r]);
      }
    }
  }
};

// Q6_K packed: ql[128] | qh[64] | int8 scale[16] | fp16 d (csrc/izb_types.cu: q6p_word).  The quants' offset of 32 is taken off by the
// accumulators' start.
struct RQ6K {
  static constexpr int SBB = kQ6pSbBytes, kPitch = 240, kSubs = 4, kPieces = 8, kDotWarps = 8;
  static constexpr bool kEx = true, kPrep = true;
  static __device__ __forceinline__ void prep(const unsigned char* chunk, float2* hd, int lane) {
    // lane <-> row lane / 2, blocks 4 (lane & 1) .. + 3: (scale of the first half, of the second half)
    const int row = lane >> 1, up = lane & 1;
    const uint2 s = *reinterpret_cast<const uint2*>(chunk + row * kPitch + 192 + 8 * up);
    const uint32_t w[2] = {s.x ^ 0x80808080u, s.y ^ 0x80808080u};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float a = __fsub_rn(byte_f(w[k >> 1], 2 * (k & 1)), 128.0f), b = __fsub_rn(byte_f(w[k >> 1], 2 * (k & 1) + 1), 128.0f);
      hd[(4 * up + k) * 16 + row] = make_float2(a, b);
    }
  }
  static __device__ __forceinline__ uint32_t word(uint32_t ql, uint32_t qh, int sub) {  // 0 .. 63 per byte
    const uint32_t hi = sub == 0 ? qh << 4 : sub == 1 ? qh << 2 : sub == 2 ? qh : qh >> 2;
    return (((sub & 2) ? ql >> 4 : ql) & 0x0F0F0F0Fu) | (hi & 0x30303030u);
  }
  static __device__ __forceinline__ void mul(const unsigned char* chunk, const float2* hd, const Acts& a, int sb, int g, int t, f2 (&acc)[kPieces][2]) {
    const unsigned char* p = chunk + g * kPitch;
    const float d0 = half_bits_to_float(*reinterpret_cast<const unsigned short*>(p + 208)), d1 = half_bits_to_float(*reinterpret_cast<const unsigned short*>(p + 8 * kPitch + 208));
    const f2 wd[2] = {f2_of(d0, d0), f2_of(d1, d1)};
    p += 4 * t;
    const unsigned char* xq = a.q + 8 * sb * a.qs;
    const f2 *xs = a.sc + 32 * sb, *xe = a.ex + 64 * sb;
#pragma unroll
    for (int nh = 0; nh < 2; ++nh) {
      uint32_t hq[2][2];
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int i = 0; i < 2; ++i) hq[r][i] = *reinterpret_cast<const uint32_t*>(p + 8 * r * kPitch + 128 + 32 * nh + 16 * i);
#pragma unroll
      for (int lo = 0; lo < 2; ++lo) {  // sub-blocks lo and lo + 2 share their low-nibble bytes
        uint32_t l[2][2];
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int i = 0; i < 2; ++i) l[r][i] = *reinterpret_cast<const uint32_t*>(p + 8 * r * kPitch + 64 * nh + 32 * lo + 16 * i);
#pragma unroll
        for (int up = 0; up < 2; ++up) {
          const int sub = lo + 2 * up, b = 4 * nh + sub;
          const uint2 x = *reinterpret_cast<const uint2*>(xq + b * a.qs), c0 = *reinterpret_cast<const uint2*>(xe + 8 * b), c1 = *reinterpret_cast<const uint2*>(xe + 8 * b + 4);
          int d[4], e[4];
          dot16_u8(d, word(l[0][0], hq[0][0], sub), word(l[1][0], hq[1][0], sub), x.x, c0.x, c0.y);
          dot16_u8(e, word(l[0][1], hq[0][1], sub), word(l[1][1], hq[1][1], sub), x.y, c1.x, c1.y);
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const float2 s = hd[b * 16 + g + 8 * r];
            // (both products and their sum are integers below 2^24: exact)
            const f2 v = f2_fma(f2_of(s.x, s.x), unmagic(d, r), f2_mul(f2_of(s.y, s.y), unmagic(e, r)));
            // the product is rounded before it is added: fma(x, y, -0) with a -0 that the compiler does not know (a packed product and a packed addition
            // came out as of one rounding, also as a fma with the constant; single values take a seventh more instructions)
            acc[b][r] = f2_add(acc[b][r], f2_fma(f2_mul(xs[4 * b], wd[r]), v, a.neg_zero));
          }
        }
      }
    }
  }
  // lane's pieces, the blocks of a superblock: 4 nh + lo + 2 (t / 2)
  static constexpr int kLaneBit = 1;
  static __device__ __forceinline__ void mul4(const unsigned char* chunk, const float2* hd, const Acts& a, int sb, int g, int t, f2 (&acc)[kPieces / 2][2]) {
    const unsigned char* p = chunk + g * kPitch;
    const float d0 = half_bits_to_float(*reinterpret_cast<const unsigned short*>(p + 208)), d1 = half_bits_to_float(*reinterpret_cast<const unsigned short*>(p + 8 * kPitch + 208));
    const f2 wd[2] = {f2_of(d0, d0), f2_of(d1, d1)};
    p += 4 * t;
    const unsigned char* xq = a.q + 8 * sb * a.qs;
    const f2 *xs = a.sc + 32 * sb, *xe = a.ex + 64 * sb;
    hd += (t >> 1) * 32 + g;
#pragma unroll
    for (int nh = 0; nh < 2; ++nh) {
      uint32_t hq[2][2];
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int i = 0; i < 2; ++i) hq[r][i] = *reinterpret_cast<const uint32_t*>(p + 8 * r * kPitch + 128 + 32 * nh + 16 * i);
#pragma unroll
      for (int lo = 0; lo < 2; ++lo) {  // sub-blocks lo and lo + 2 share their low-nibble bytes
        const int b = 4 * nh + lo;
        const uint2 x = *reinterpret_cast<const uint2*>(xq + b * a.qs), c0 = *reinterpret_cast<const uint2*>(xe + 8 * b), c1 = *reinterpret_cast<const uint2*>(xe + 8 * b + 4);
        int d[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          uint32_t l[2];
#pragma unroll
          for (int r = 0; r < 2; ++r) l[r] = *reinterpret_cast<const uint32_t*>(p + 8 * r * kPitch + 64 * nh + 32 * lo + 16 * i);
          const uint32_t v = i ? x.y : x.x;
          dot32_u8(d[i], word(l[0], hq[0][i], lo), word(l[1], hq[1][i], lo), word(l[0], hq[0][i], lo + 2), word(l[1], hq[1][i], lo + 2), v & a.first, v & a.last, i ? c1.x : c0.x, i ? c1.y : c0.y);
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float2 s = hd[b * 16 + 8 * r];
          const f2 v = f2_fma(f2_of(s.x, s.x), unmagic(d[0], r), f2_mul(f2_of(s.y, s.y), unmagic(d[1], r)));
          acc[2 * nh + lo][r] = f2_add(acc[2 * nh + lo][r], f2_fma(f2_mul(xs[4 * b], wd[r]), v, a.neg_zero));  // (see mul)
        }
      }
    }
  }
};

// ---- a warp's ring of chunks (16 rows x one superblock each), filled by TMA
__device__ __forceinline__ uint32_t r_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
template <class F>
struct Ring {
  static constexpr int kSlot = (16 * F::kPitch + 127) & ~127;
  static constexpr uint32_t kSpin = 1u << 24;
  unsigned char* base;
  uint64_t* bars;
  int slots, put = 0, get = 0;
  uint32_t parity = 0;
  __device__ __forceinline__ void init(int lane) {
    if (lane == 0) {
      for (int s = 0; s < slots; ++s) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(r_u32(&bars[s])) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
  }
  // (every lane keeps the position, lane 0 issues)
  __device__ __forceinline__ void fill(const void* tmap, int sb, int row, int lane) {
    if (lane == 0) {
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(r_u32(&bars[put])), "r"(16 * F::kPitch) : "memory");
      asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(r_u32(base + put * kSlot)),
                   "l"(tmap), "r"(sb * (F::SBB / 4)), "r"(row), "r"(r_u32(&bars[put]))
                   : "memory");
    }
    if (++put == slots) put = 0;
  }
  // The next chunk in order; null when the bounded wait ran out.  Every lane gets the same answer: a lane that left alone would wait at the
  // tile's barrier for lanes that wait for it at the next __syncwarp.
  __device__ __forceinline__ const unsigned char* wait() const {
    for (uint32_t it = 0; it < kSpin; ++it) {
      uint32_t ok;
      asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                   : "=r"(ok) : "r"(r_u32(&bars[get])), "r"(parity) : "memory");
      if (__all_sync(0xFFFFFFFFu, ok)) return base + get * kSlot;
    }
    return nullptr;
  }
  __device__ __forceinline__ void next() {
    if (++get == slots) { get = 0; parity ^= 1; }
  }
  // after a wait that ran out: the other requests in flight, with the same limit (their slots must outlive them)
  __device__ __forceinline__ void drain() {
    for (int s = 1; s < slots; ++s) {
      next();
      wait();
    }
  }
};

// ---- shared memory: activations | rings | 4 KB per warp, 2 KB with half the sums (expanded headers, exchanged sums) | barriers
template <class F>
__host__ __device__ __forceinline__ size_t act_bytes(int K, int T) { return ((size_t)(K / 32) * (32 * T + 32 + (F::kEx ? 64 : 0)) + 127) & ~(size_t)127; }
template <bool kFour>
constexpr int kXch = kFour ? 2048 : 4096;
template <class F, bool kFour>
__host__ __device__ __forceinline__ size_t rows_smem(int K, int T, int nw, int slots) {
  return act_bytes<F>(K, T) + (size_t)nw * (slots * (Ring<F>::kSlot + 8) + kXch<kFour>);
}

// Activations of T tokens (rows `src(j)` of aq, columns of asc), as Acts describes them.  Four items per thread and pass, so that their
// loads are in flight together.
template <class F, bool kFour, class Src>
__device__ __forceinline__ Acts stage_acts(unsigned char* smem, int K, int T, const int8_t* __restrict__ aq, const float* __restrict__ asc, int Mp, int g, int t, Src src) {
  const int nb = K / 32, items = nb * T;
  float* s_sc = reinterpret_cast<float*>(smem + (size_t)nb * 32 * T);
  float* s_ex = s_sc + nb * 8;
  constexpr int kBatch = 4;
  for (int i0 = threadIdx.x; i0 < items; i0 += kBatch * blockDim.x) {
    uint4 x[kBatch], y[kBatch];
    float s[kBatch];
    int bb[kBatch], jj[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int i = i0 + u * blockDim.x;
      bb[u] = i / T;
      jj[u] = i - bb[u] * T;
      if (i < items) {
        const int row = src(jj[u]);
        const uint4* p = reinterpret_cast<const uint4*>(aq + (size_t)row * K) + 2 * bb[u];
        x[u] = p[0];
        y[u] = p[1];
        s[u] = asc[(size_t)bb[u] * Mp + row];
      }
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int b = bb[u], j = jj[u];
      if (i0 + u * (int)blockDim.x >= items) continue;
      uint4* o = reinterpret_cast<uint4*>(smem + (size_t)(b * T + j) * 32);
      o[0] = make_uint4(x[u].x, y[u].x, x[u].y, y[u].y);
      o[1] = make_uint4(x[u].z, y[u].z, x[u].w, y[u].w);
      s_sc[b * 8 + j] = s[u];
      if (F::kEx) {
        const uint32_t w[8] = {x[u].x, x[u].y, x[u].z, x[u].w, y[u].x, y[u].y, y[u].z, y[u].w};
        int s0 = 0, s1 = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          s0 = __dp4a((int)w[k], 0x01010101, s0);
          s1 = __dp4a((int)w[4 + k], 0x01010101, s1);
        }
        const bool q4 = F::SBB == 144;
        s_ex[b * 16 + j] = q4 ? (float)s0 : __int_as_float((int)kMagic - 32 * s0);
        s_ex[b * 16 + 8 + j] = q4 ? (float)s1 : __int_as_float((int)kMagic - 32 * s1);
      }
    }
  }
  Acts a;
  a.qs = 32 * T;
  a.first = g < 4 ? 0xFFFFFFFFu : 0u;
  a.last = ~a.first;
  a.q = smem + min(kFour ? g & 3 : g, T - 1) * 32 + 8 * t;  // (lanes past the last token repeat it; their results are not stored)
  a.sc = reinterpret_cast<const f2*>(s_sc) + (kFour ? t & 1 : t);
  a.ex = reinterpret_cast<const f2*>(s_ex) + (kFour ? t & 1 : t);
  if (kFour && F::kLaneBit == 0) {  // columns 4-7: the second half of a block
    a.q += 4 * (g >> 2);
    a.ex += 4 * (t >> 1);
  } else if (kFour) {  // ... the block after the next
    a.q += 2 * a.qs * (g >> 2);
    a.sc += 8 * (t >> 1);
    a.ex += 16 * (t >> 1);
  }
  const uint32_t nz = 0x80000000u | (uint32_t)(K >> 31);  // (K > 0)
  a.neg_zero = (f2)nz << 32 | nz;
  return a;
}

// One chunk after the other of this warp's share of a tile (superblocks part, part + kSubs, ...) into acc.  false: a wait ran out.
template <class F, bool kFour>
constexpr int kLanePieces = kFour ? F::kPieces / 2 : F::kPieces;
template <class F, bool kFour, class Request>
__device__ __forceinline__ bool accumulate(Ring<F>& ring, float2* hd, const Acts& acts, int part, int nsb, int lane, f2 (&acc)[kLanePieces<F, kFour>][2], Request request) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int p = 0; p < kLanePieces<F, kFour>; ++p) acc[p][0] = acc[p][1] = 0ull;
  for (int s = part; s < nsb; s += F::kSubs) {
    const unsigned char* chunk = ring.wait();
    if (!chunk) {
      ring.drain();
      return false;
    }
    if (F::kPrep) {
      F::prep(chunk, hd, lane);
      __syncwarp();
    }
    if constexpr (kFour) F::mul4(chunk, hd, acts, s, g, t, acc);
    else F::mul(chunk, hd, acts, s, g, t, acc);
    __syncwarp();  // every lane has read the chunk: its slot takes the next request
    ring.next();
    request();
  }
  return true;
}

// the pieces of a lane into acc[0], pairs `H` apart and then nearer ones (mul4: the step over the bit kLaneBit is between lanes)
template <class F, bool kFour, int H>
__device__ __forceinline__ void fold_pieces(f2 (&acc)[kLanePieces<F, kFour>][2]) {
  constexpr bool kLanes = kFour && H == 1 << F::kLaneBit;
  constexpr int kHave = kFour && H >= 1 << F::kLaneBit ? H : 2 * H, kLeft = kLanes ? kHave : kHave / 2;  // the lane's pieces before and after
#pragma unroll
  for (int p = 0; p < kLeft; ++p)
#pragma unroll
    for (int r = 0; r < 2; ++r) acc[p][r] = f2_add(acc[p][r], kLanes ? __shfl_xor_sync(0xFFFFFFFFu, acc[p][r], 2) : acc[p + kLeft][r]);
  if constexpr (H > 1) fold_pieces<F, kFour, H / 2>(acc);
}

// The tree over a tile's 32 partial sums per output: superblock parts p, p ^ 2, then p ^ 1 (through shared memory: parts 2 and 3
// hand theirs to 0 and 1, part 1 to 0), then the pieces halves first.  All warps of a tile call it (a named barrier per tile: the
// tiles of a CTA need not keep step); the result is valid in part 0.  `xch`: this CTA's exchange areas, one per warp.
template <class F>
__device__ __forceinline__ void tile_sync(int mine) { asm volatile("bar.sync %0, %1;" ::"r"(1 + mine), "n"(F::kSubs * 32) : "memory"); }
// (mul4: lanes t and t + 2 both have the result.)
template <class F, bool kFour>
__device__ __forceinline__ void reduce_tile(f2 (&acc)[kLanePieces<F, kFour>][2], unsigned char* xch, int warp, int lane) {
  constexpr int kMine = kLanePieces<F, kFour>;
  static_assert(F::kSubs == 4 ? F::kPieces == 8 : F::kSubs == 2 && F::kPieces == 16, "exchange areas: 4 KB per warp");
  const int part = warp % F::kSubs, mine = warp / F::kSubs;
  auto area = [&](int w) { return reinterpret_cast<ulonglong2*>(xch + (size_t)w * kXch<kFour>) + lane; };  // [piece][lane] of 16 bytes
  auto give = [&](int w) {
#pragma unroll
    for (int p = 0; p < kMine; ++p) area(w)[32 * p] = make_ulonglong2(acc[p][0], acc[p][1]);
  };
  auto take = [&](int w) {
#pragma unroll
    for (int p = 0; p < kMine; ++p) {
      const ulonglong2 v = area(w)[32 * p];
      acc[p][0] = f2_add(acc[p][0], v.x);
      acc[p][1] = f2_add(acc[p][1], v.y);
    }
  };
  if (F::kSubs == 4) {
    if (part >= 2) give(warp);  // (a warp's own area: only its own headers were there)
    tile_sync<F>(mine);
    if (part < 2) take(warp + 2);
    if (part == 1) give(warp);
    tile_sync<F>(mine);
    if (part == 0) take(warp + 1);
    tile_sync<F>(mine);  // the areas take headers again
  } else {
    if (part == 1) give(warp - 1);  // (sixteen pieces: the areas of both warps)
    tile_sync<F>(mine);
    if (part == 0) take(warp);
    tile_sync<F>(mine);
  }
  fold_pieces<F, kFour, F::kPieces / 2>(acc);
}

// C[token][c_off + row] (= or +=) for T tokens.  The grid walks groups of (warps / kSubs) row tiles.
template <class F, bool kFour>
__global__ void __launch_bounds__(512, 1) rows_kernel(const __grid_constant__ CUtensorMap tm, int wrow0, int N, int K, const int8_t* __restrict__ aq,
                                                      const float* __restrict__ asc, int T, int Mp, float* __restrict__ C, int ldc, int c_off, int acc_mode, int slots,
                                                      uint32_t* err) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int NW = blockDim.x >> 5, kPer = NW / F::kSubs;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int part = warp % F::kSubs, mine = warp / F::kSubs, nsb = K >> 8, groups = ((N + 15) / 16 + kPer - 1) / kPer;
  unsigned char* rings = smem + act_bytes<F>(K, T);
  unsigned char* xch = rings + (size_t)NW * slots * Ring<F>::kSlot;
  Ring<F> ring;
  ring.slots = slots;
  ring.base = rings + (size_t)warp * slots * Ring<F>::kSlot;
  ring.bars = reinterpret_cast<uint64_t*>(xch + NW * kXch<kFour>) + warp * slots;
  __shared__ int s_gave_up;
  volatile int* gave_up = &s_gave_up;
  if (threadIdx.x == 0) s_gave_up = 0;
  ring.init(lane);
  // chunks still to request: superblock `ps` of the tile in group `pg`
  int pg = blockIdx.x, ps = part;
  auto request = [&]() {
    if (pg >= groups || part >= nsb) return;
    ring.fill(&tm, ps, wrow0 + (pg * kPer + mine) * 16, lane);
    if ((ps += F::kSubs) >= nsb) { ps = part; pg += gridDim.x; }
  };
  for (int s = 0; s < slots; ++s) request();
  pdl_launch_next();
  pdl_wait();
  const Acts acts = stage_acts<F, kFour>(smem, K, T, aq, asc, Mp, g, t, [](int j) { return j; });
  __syncthreads();
  bool ok = true;
  for (int gr = blockIdx.x; gr < groups; gr += gridDim.x) {
    f2 acc[kLanePieces<F, kFour>][2];
    if (ok) ok = accumulate<F, kFour>(ring, reinterpret_cast<float2*>(xch + (size_t)warp * kXch<kFour>), acts, part, nsb, lane, acc, request);
    if (!ok) {  // (bounded wait gave up: nothing of this CTA is stored any more)
      if (lane == 0) atomicOr(err, 64u);
      *gave_up = 1;
    }
    reduce_tile<F, kFour>(acc, xch, warp, lane);
    if (part == 0 && !*gave_up) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = (gr * kPer + mine) * 16 + g + 8 * (i >> 1), tok = 2 * (kFour ? t & 1 : t) + (i & 1);
        if (kFour && (t >> 1) != i >> 1) continue;  // (both pairs of lanes have the sums: one stores rows g, the other g + 8)
        if (row < N && tok < T) {
          float* c = C + (size_t)tok * ldc + c_off + row;
          const float v = f2_get(acc[0][i >> 1], i & 1);
          *c = acc_mode ? __fadd_rn(*c, v) : v;
        }
      }
    }
  }
}

// A warp's whole 16-row tile for TT tokens by dp4a, its chunks in superblock order; the same 32 partial sums per output and the same tree.
// out[j]: row lane % 16 (both half-warps) against token j.  false: a wait ran out.
template <class F, int TT, class Request>
__device__ __forceinline__ bool dot_tile(Ring<F>& ring, const unsigned char* act, int nsb, int T, int lane, float (&out)[2], Request request) {
  constexpr int kLocal = F::kPieces / 2;
  float acc[F::kSubs][TT][kLocal];
#pragma unroll
  for (int s = 0; s < F::kSubs; ++s)
#pragma unroll
    for (int j = 0; j < TT; ++j)
#pragma unroll
      for (int p = 0; p < kLocal; ++p) acc[s][j][p] = 0.0f;
  // (acc[0] is always the next superblock's: the sums move up by one per chunk, which costs less than the loop body four times over
  // in the instruction cache; past the last superblock they move on until number 0 is in place)
  auto turn = [&]() {
#pragma unroll
    for (int j = 0; j < TT; ++j)
#pragma unroll
      for (int p = 0; p < kLocal; ++p) {
        const float a = acc[0][j][p];
#pragma unroll
        for (int s = 0; s + 1 < F::kSubs; ++s) acc[s][j][p] = acc[s + 1][j][p];
        acc[F::kSubs - 1][j][p] = a;
      }
  };
#pragma unroll 1
  for (int sb = 0; sb < nsb; ++sb) {
    const unsigned char* chunk = ring.wait();
    if (!chunk) {
      ring.drain();
      return false;
    }
    F::template dot<TT>(chunk, act, nsb * 8, T, sb, lane, acc[0]);
    __syncwarp();  // every lane has read the chunk: its slot takes the next request
    ring.next();
    request();
    turn();
  }
#pragma unroll 1
  for (int sb = nsb; sb % F::kSubs; ++sb) turn();
#pragma unroll
  for (int j = 0; j < TT; ++j) {
    float v[kLocal];
#pragma unroll
    for (int p = 0; p < kLocal; ++p) {
      v[p] = F::kSubs == 4 ? __fadd_rn(__fadd_rn(acc[0][j][p], acc[F::kSubs - 2][j][p]), __fadd_rn(acc[1][j][p], acc[F::kSubs - 1][j][p])) : __fadd_rn(acc[0][j][p], acc[1][j][p]);
      v[p] = __fadd_rn(v[p], __shfl_xor_sync(0xFFFFFFFFu, v[p], 16));
    }
#pragma unroll
    for (int h = kLocal / 2; h > 0; h >>= 1)
#pragma unroll
      for (int p = 0; p < h; ++p) v[p] = __fadd_rn(v[p], v[p + h]);
    out[j] = v[0];
  }
  return true;
}
// Mixture of experts: an item is a tile (up to 8 slots of one expert) x as many row tiles as the CTA has warps; how many tiles there are
// is known on the device only.  A CTA takes a run of consecutive items, which mostly share their tile: the activations are staged once
// per tile, and the rings run on from item to item.  (One CTA per possible item left at once for most of them: 2048 x 768 of 128
// experts, 32 slots: 8448 CTAs for some 1800 items; a 4-token step took 120 us, walked like this 97.)
// A tile of up to kFewSlots slots -- most, while a step has few tokens -- goes by dp4a, each warp a row tile of its own: a third of the
// matrix instruction's instructions at one slot and no exchange between warps (the step: 69 -> 50 us; at three slots the two ways
// are equal).  What bounds it is the latency of a chunk, about 1 us with the three warps per SMSP that fit: contiguous runs of
// whole rows instead of 16-row chunks wanted four times the header work per weight (94 us).
// gate/up (pair): h[slot][N] = silu(x Wg^T) * (x Wu^T), token rows through stok; down: y[slot][N] = swt * (hq Wd^T).
constexpr int kFewSlots = 2;
// (small CTAs: items are divided among them as they come, and a tile's activations hold up four warps only; three per SM leave the two
// ways 168 registers, which do not hold everything either: 100 bytes a thread are spilt for Q4_K, 176 for Q8_0)
constexpr int kMoeWarps = 4, kMoeCtas = 3;
// Where the items are fewer than the blocks that fit, a block takes kPer row tiles of one tile instead of kMoeWarps, its kSubs warps per row
// tile sharing the superblocks also for few slots: gate / up 1024 x 512 of 8 experts Q4_K, four slots, 10.8 -> 6.0 us, sixteen 16.1 -> 6.9; 4096 x
// 1536 of 16, two slots, 21.0 -> 11.6.  At most two items per SM: with a third the walk below is faster.  `slots`: the ring's, set up by
// the caller.  (Out of line: beside the walk in one body it cost that one registers.)
template <class F>
__device__ __noinline__ void moe_fine(const CUtensorMap& tg, const CUtensorMap& tu, int pair, int N, int K, const int8_t* aq, const float* asc, int Mp, const int32_t* tiles,
                                      const int32_t* stok, const float* swt, float* out, int slots, volatile int* gave_up, uint32_t* err) {
  extern __shared__ __align__(1024) unsigned char smem[];
  constexpr int NW = kMoeWarps, kPer = NW / F::kSubs;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int part = warp % F::kSubs, mine = warp / F::kSubs, nsb = K >> 8, groups = ((N + 15) / 16 + kPer - 1) / kPer;
  const int ti = blockIdx.x / groups, row_tile = (blockIdx.x - ti * groups) * kPer + mine;
  if (ti >= tiles[0]) return;
  unsigned char* rings = smem + act_bytes<F>(K, 8);
  unsigned char* xch = rings + (size_t)NW * slots * Ring<F>::kSlot;
  Ring<F> ring;
  ring.slots = slots;
  ring.base = rings + (size_t)warp * slots * Ring<F>::kSlot;
  ring.bars = reinterpret_cast<uint64_t*>(xch + NW * kXch<false>) + warp * slots;
  const int row = tiles[1 + 3 * ti] * N + row_tile * 16, s0 = tiles[2 + 3 * ti], T = tiles[3 + 3 * ti];
  int pm = 0, ps = part;
  auto request = [&]() {
    if (pm > pair || part >= nsb) return;
    ring.fill(pm ? &tu : &tg, ps, row, lane);
    if ((ps += F::kSubs) >= nsb) { ps = part; ++pm; }
  };
  for (int s = 0; s < slots; ++s) request();
  const Acts acts = stage_acts<F, false>(smem, K, T, aq, asc, Mp, g, t, [&](int j) { return stok ? stok[s0 + j] : s0 + j; });
  __syncthreads();
  bool ok = true;
  float first[4];
  for (int m = 0; m <= pair; ++m) {
    f2 acc[F::kPieces][2];
    if (ok) ok = accumulate<F, false>(ring, reinterpret_cast<float2*>(xch + (size_t)warp * kXch<false>), acts, part, nsb, lane, acc, request);
    if (!ok) {
      if (lane == 0) atomicOr(err, 64u);
      *gave_up = 1;
    }
    reduce_tile<F, false>(acc, xch, warp, lane);
    if (part != 0 || *gave_up) continue;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int n = row_tile * 16 + g + 8 * (i >> 1), slot = 2 * t + (i & 1);
      const float v = f2_get(acc[0][i >> 1], i & 1);
      if (m < pair) first[i] = v;
      else if (n < N && slot < T) out[(size_t)(s0 + slot) * N + n] = pair ? __fmul_rn(__fdiv_rn(first[i], __fadd_rn(1.0f, expf(-first[i]))), v) : __fmul_rn(swt[s0 + slot], v);
    }
  }
}
template <class F>
__global__ void __launch_bounds__(kMoeWarps * 32, kMoeCtas) moe_rows_kernel(const __grid_constant__ CUtensorMap tg, const __grid_constant__ CUtensorMap tu, int pair, int N, int K,
                                                          const int8_t* __restrict__ aq, const float* __restrict__ asc, int Mp, const int32_t* __restrict__ tiles,
                                                          const int32_t* __restrict__ stok, const float* __restrict__ swt, float* __restrict__ out, int slots, int fine_items, uint32_t* err) {
  extern __shared__ __align__(1024) unsigned char smem[];
  constexpr int NW = kMoeWarps, kPer = NW / F::kSubs;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int part = warp % F::kSubs, mine = warp / F::kSubs, nsb = K >> 8, groups = ((N + 15) / 16 + NW - 1) / NW;
  unsigned char* rings = smem + act_bytes<F>(K, 8);
  unsigned char* xch = rings + (size_t)NW * slots * Ring<F>::kSlot;
  Ring<F> ring;
  ring.slots = slots;
  ring.base = rings + (size_t)warp * slots * Ring<F>::kSlot;
  ring.bars = reinterpret_cast<uint64_t*>(xch + NW * kXch<false>) + warp * slots;
  __shared__ int s_gave_up;
  volatile int* gave_up = &s_gave_up;
  if (threadIdx.x == 0) s_gave_up = 0;
  ring.init(lane);
  pdl_launch_next();
  pdl_wait();
  {  // (fine_items 0 for the down product; not for short K and few slots: dp4a without the exchange between warps is as fast there)
    const int n_tiles = tiles[0], saved = 2 * (nsb - (nsb + F::kSubs - 1) / F::kSubs);
    if ((long long)n_tiles * (((N + 15) / 16 + kPer - 1) / kPer) <= fine_items &&
        (saved > 1 || __any_sync(0xFFFFFFFFu, lane < n_tiles && tiles[3 + 3 * lane] > kFewSlots))) {  // (a look at the first 32 tiles)
      moe_fine<F>(tg, tu, pair, N, K, aq, asc, Mp, tiles, stok, swt, out, slots, gave_up, err);
      return;
    }
  }
  const long long items = (long long)tiles[0] * groups;
  const int lo = (int)(items * blockIdx.x / gridDim.x), hi = (int)(items * (blockIdx.x + 1) / gridDim.x);
  // Chunks still to request: superblock `ps` of matrix `pm` (gate, up) of this warp's row tile in round `pr` of item `pi`.  Few slots:
  // one round, every superblock; else kSubs rounds of kPer row tiles, every kSubs-th superblock.
  // (no divisions: a warp asks once per chunk.)
  int left = hi - lo, pt = lo / groups, pg = lo - pt * groups, row = 0, rounds = 1, pr = 0, pm = 0, ps = 0, by = 1, from = 0;
  auto enter = [&]() {  // tile pt
    const bool few = tiles[3 + 3 * pt] <= kFewSlots;
    row = tiles[1 + 3 * pt] * N + (pg * NW + (few ? warp : mine)) * 16;
    rounds = few ? 1 : F::kSubs;
    by = few ? 1 : F::kSubs;
    ps = from = few ? 0 : part;
  };
  auto request = [&]() {
    while (left > 0) {
      const bool any = ps < nsb;
      if (any) {
        ring.fill(pm ? &tu : &tg, ps, row + pr * kPer * 16, lane);
        if ((ps += by) < nsb) return;
      }
      ps = from;
      if (pm++ >= pair) {
        pm = 0;
        if (++pr >= rounds) {
          pr = 0;
          row += NW * 16;
          if (--left > 0 && ++pg == groups) {
            pg = 0;
            ++pt;
            enter();
          }
        }
      }
      if (any) return;
    }
  };
  if (left > 0) enter();
  for (int s = 0; s < slots; ++s) request();
  Acts acts;
  int s0 = 0, T = 0;
  bool ok = true;
  auto store = [&](int n, int slot, float gate, float v) {
    if (n < N && slot < T) out[(size_t)(s0 + slot) * N + n] = pair ? __fmul_rn(__fdiv_rn(gate, __fadd_rn(1.0f, expf(-gate))), v) : __fmul_rn(swt[s0 + slot], v);
  };
  auto note = [&]() {  // (bounded wait gave up: nothing of this CTA is stored any more)
    if (lane == 0) atomicOr(err, 64u);
    *gave_up = 1;
  };
  int ti = lo / groups, gi = lo - ti * groups;
  for (int it = lo; it < hi; ++it, ++gi) {
    if (it == lo || gi == groups) {
      if (it != lo) {
        __syncthreads();  // the last tile's activations have been read
        gi = 0;
        ++ti;
      }
      s0 = tiles[2 + 3 * ti];
      T = tiles[3 + 3 * ti];
      acts = stage_acts<F, false>(smem, K, T, aq, asc, Mp, g, t, [&](int j) { return stok ? stok[s0 + j] : s0 + j; });
      __syncthreads();
    }
    const int tile0 = gi * NW;
    if (T <= kFewSlots) {
      float first[2] = {0.0f, 0.0f}, v[2] = {0.0f, 0.0f};
#pragma unroll 1
      for (int m = 0; m <= pair; ++m) {
#pragma unroll
        for (int j = 0; j < 2; ++j) first[j] = v[j];
        if (ok) ok = T == 1 ? dot_tile<F, 1>(ring, smem, nsb, T, lane, v, request) : dot_tile<F, 2>(ring, smem, nsb, T, lane, v, request);
      }
      if (!ok) note();
      if (!*gave_up && lane < 16) {
#pragma unroll
        for (int j = 0; j < kFewSlots; ++j) store((tile0 + warp) * 16 + lane, j, first[j], v[j]);
      }
      continue;
    }
    for (int r = 0; r < F::kSubs; ++r) {
      float first[4];
      for (int m = 0; m <= pair; ++m) {
        f2 acc[F::kPieces][2];
        if (ok) ok = accumulate<F, false>(ring, reinterpret_cast<float2*>(xch + (size_t)warp * kXch<false>), acts, part, nsb, lane, acc, request);
        if (!ok) note();
        reduce_tile<F, false>(acc, xch, warp, lane);
        if (m < pair) {
#pragma unroll
          for (int i = 0; i < 4; ++i) first[i] = f2_get(acc[0][i >> 1], i & 1);
        } else if (part == 0 && !*gave_up) {
#pragma unroll
          for (int i = 0; i < 4; ++i) store((tile0 + r * kPer + mine) * 16 + g + 8 * (i >> 1), 2 * t + (i & 1), first[i], f2_get(acc[0][i >> 1], i & 1));
        }
      }
    }
  }
}

// Warps per CTA, CTAs per SM and ring slots (2 to 4) for `tiles` row tiles.  The fewest rounds of the grid, weighted by what a round of
// fewer slots takes longer (three for two 1.15; four for three 1.04, up to eight warps per SM: with twelve three are enough); of equals
// the smaller CTA, which spreads the tiles of a single round over more SMs.  (us, 16 warps / 12: Q4_K 5120 x 13824, one row, 17.5 / 14.9,
// 6144 x 4096, five, 9.3 / 8.6; Q6_K 5120 x 17408, three, 27.8 / 20.5 with eight in two rounds.  One CTA of twelve / three of four: Q6_K 5120 x 5120, one row,
// 7.9 / 7.0; of sixteen / two of eight: Q4_K 16384 x 5376, three, 17.0 / 15.4.  Two of four, three slots / one of eight, four: Q8_0 8192 x 4096, eight,
// 10.9 / 9.7.)
constexpr size_t kSmemPerSm = 226 * 1024;
struct Split {
  int warps, ctas, slots;  // slots 0: the activations leave no room
};
template <class F, bool kFour>
Split pick_split(int K, int T, int tiles, int sms) {
  constexpr double kDepth[5] = {0, 0, 1.0, 1.15, 1.2};
  Split best = {0, 0, 0};
  double least = 0;
  for (int nw = 4; nw <= 16; nw += 4) {
    const int groups = (tiles + nw / F::kSubs - 1) / (nw / F::kSubs);
    for (int c = 1; c * nw <= 16 && (c - 1) * sms < groups; ++c) {
      const size_t room = kSmemPerSm / c - (c > 1 ? 1024 : 0);
      int slots = 4;
      while (slots >= 2 && rows_smem<F, kFour>(K, T, nw, slots) > room) --slots;
      if (slots < 2) break;
      const int rounds = (groups + c * sms - 1) / (c * sms);
      const double time = rounds / kDepth[slots == 4 && c * nw >= 12 ? 3 : slots];
      if (best.slots == 0 || time < least * 0.999) {
        least = time;
        best = {nw, c, slots};
      }
    }
  }
  return best;
}

template <class F, bool kFour>
int rows_of(const izb_weight* w, int mat, const int8_t* aq, const float* asc, int T, int Mp, float* C, int ldc, int c_off, int acc, cudaStream_t st) {
  const int sms = izb_sm_count(w->device), tiles = (w->N + 15) / 16;
  const Split sp = pick_split<F, kFour>(w->K, T, tiles, sms);
  // Half the tokens at a time, the second pass finding part of the weights in L2; not where the dot-product kernel's warps (kDotWarps per SM)
  // take every row in one round (us, halves / dot products, eight rows of 17408 Q6_K: 1024 rows 34/28, 1280 rows 34/42; of 18944 Q4_K:
  // 2304 rows 35/33, 2560 rows 45/60).
  if (!sp.slots) {
    if (T < 2 || w->N <= F::kDotWarps * sms) return 1;
    const int h = (T + 1) / 2;
    if (const int rc = rows_of<F, true>(w, mat, aq, asc, h, Mp, C, ldc, c_off, acc, st)) return rc;
    return rows_of<F, true>(w, mat, aq + (size_t)h * w->K, asc + h, T - h, Mp, C + (size_t)h * ldc, ldc, c_off, acc, st);
  }
  IZB_SMEM_OPTIN((rows_kernel<F, kFour>), kSmemPerSm, w->device);
  const int groups = (tiles + sp.warps / F::kSubs - 1) / (sp.warps / F::kSubs), grid = groups < sms * sp.ctas ? groups : sms * sp.ctas;
  uint32_t* err = izb_device_error_word(w->device);
  if (!err) IZB_FAIL(IZB_ERR_NOMEM, "gemv: no device error word");
  CUtensorMap tm;
  memcpy(&tm, w->tmap16_raw, sizeof tm);
  IZB_LAUNCH("gemv_rows", st, izb_launch_pdl(rows_kernel<F, kFour>, grid, sp.warps * 32, rows_smem<F, kFour>(w->K, T, sp.warps, sp.slots), st, tm, mat * w->N, w->N, w->K, aq, asc, T, Mp, C, ldc,
                                             c_off, acc, sp.slots, err));
  return IZB_OK;
}
template <class F>
int moe_rows_of(const izb_weight* wg, const izb_weight* wu, const int8_t* aq, const float* asc, int Mp, const int32_t* tiles, int max_tiles, const int32_t* stok, const float* swt,
                float* out, cudaStream_t st) {
  const int sms = izb_sm_count(wg->device);
  if ((long long)max_tiles * ((wg->N + 15) / 16) > (1ll << 30)) return 1;
  int ctas = kMoeCtas, slots = 0;
  for (; ctas > 0; --ctas) {
    const size_t room = kSmemPerSm / ctas - (ctas > 1 ? 1024 : 0);
    for (slots = 4; slots >= 2 && rows_smem<F, false>(wg->K, 8, kMoeWarps, slots) > room;) --slots;
    if (slots >= 2) break;
  }
  if (ctas == 0) return 1;
  uint32_t* err = izb_device_error_word(wg->device);
  if (!err) IZB_FAIL(IZB_ERR_NOMEM, "moe: no device error word");
  CUtensorMap tg, tu;
  memcpy(&tg, wg->tmap16_raw, sizeof tg);
  memcpy(&tu, (wu ? wu : wg)->tmap16_raw, sizeof tu);
  // (one kernel for both products: as two, the second finds its code out of the instruction cache, 1 us of a 4-token step)
  IZB_SMEM_OPTIN((moe_rows_kernel<F>), kSmemPerSm, wg->device);
  IZB_LAUNCH(wu ? "moe_gateup" : "moe_down", st, izb_launch_pdl(moe_rows_kernel<F>, sms * ctas, kMoeWarps * 32, rows_smem<F, false>(wg->K, 8, kMoeWarps, slots), st, tg, tu, wu ? 1 : 0,
                                                               wg->N, wg->K, aq, asc, Mp, tiles, stok, swt, out, slots, wu ? sms * (ctas < 2 ? ctas : 2) : 0, err));
  return IZB_OK;
}

}  // namespace

// up to 8 rows; +1: not taken (another weight form, no tensor map, or activations that do not fit in shared memory)
int izb_rows_launch(const izb_weight* w, int mat, const int8_t* aq, const float* asc, int T, int Mp, float* C, int ldc, int c_off, int acc, cudaStream_t st) {
  if (!w->has_tmap16 || T > 8) return 1;
  auto of = w->type == IZB_Q4_K ? (T <= 4 ? rows_of<RQ4K, true> : rows_of<RQ4K, false>) : w->type == IZB_Q8_0 ? (T <= 4 ? rows_of<RQ80, true> : rows_of<RQ80, false>)
          : T <= 4 ? rows_of<RQ6K, true> : rows_of<RQ6K, false>;
  return of(w, mat, aq, asc, T, Mp, C, ldc, c_off, acc, st);
}

// gate / up (wu given) or down (wu = null, swt given) over tiles of up to 8 slots; +1: not taken
int izb_moe_rows_launch(const izb_weight* wg, const izb_weight* wu, const int8_t* aq, const float* asc, int Mp, const int32_t* tiles, int max_tiles, const int32_t* stok,
                        const float* swt, float* out, cudaStream_t st) {
  if (!wg->has_tmap16 || (wu && !wu->has_tmap16)) return 1;
  return wg->type == IZB_Q4_K ? moe_rows_of<RQ4K>(wg, wu, aq, asc, Mp, tiles, max_tiles, stok, swt, out, st)
                              : moe_rows_of<RQ80>(wg, wu, aq, asc, Mp, tiles, max_tiles, stok, swt, out, st);
}
