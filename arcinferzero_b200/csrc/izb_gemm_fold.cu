// Prefill GEMM on the 5th-generation tensor cores (tcgen05, TMEM operands and accumulators) for plain stores of Q4_K and Q5_K products: the
// block scales travel in the operands.  (csrc/izb_gemm_tc.cu: the kernel with plain integers in its operands, for every other call.)
//
// Problem: C[m][n] = sum over 32-blocks b of asc[m][b] * wscale[n][b] * dot_b[m][n]  (- the min term of Q4_K and Q5_K), where dot_b
// is an exact integer.  Both operands carry a scale per block.  Left out of the operands, the scales force every block's 128 x 128 dot products
// through TMEM reads and an fma on the CUDA cores before the next block may be added: that, not the MMA, bounds such a kernel (550 clk per
// 128 x 128 x 32 block).  Here they are folded into the operands and the accumulators leave TMEM once per superblock (256 of K):
//   * activations: asc[m][b] * a as TWO fp16 terms.  Per row and superblock asc[m][b] = r[m][b] * s[m], s a 128th of the largest |asc|, so
//     |r * a| <= 2^14; r * a = hi + lo, hi a multiple of 4 or 8, lo = fp16(r * a - hi): 23 to 24 bits of the largest value.
//     s is applied in f32.
//   * weights: sub-scale * quant <= 1953, exact in one fp16 term.
//   * so a block costs two MMAs (a_lo, a_hi), 256 clk of a 128 x 128 x 32 block, and the CUDA cores per superblock and element:
//     res += s[m] * (d[n] * D - dmin[n] * D2).
//   * D2[m][n] = sum_b (r * asum)[m][b] * mn[n][b]: one more MMA of K = 16 per superblock, the eight blocks' hi and lo terms.
// Where a row's scales lie more than 4 : 1 apart inside a superblock, 24 bits of the largest block's values are too few of the smallest's: the large block's
// weights may be zeros.  Such rows have a third term, on 16 more MMAs into an accumulator of its own; beyond 4096 : 1, and where a scale is no finite
// number, the blocks are multiplied one by one (split_scale).  A tile whose rows are all plain in its part of K runs the loops of plain rows, and a
// row's sums do not depend on what the others are.  (Two terms alone: 1.4e-6 of the result at 40 : 1, 2e-4 at 2^13 : 1.)
// The tensor core adds in f32 but rounds towards zero, which would shrink every sum a little with every MMA (6e-7 of the result over a
// superblock's 32).  Hence the order of a superblock's MMAs: first all with a_lo, on sums some 2^12 times smaller; then a_hi, whose products
// and sums are multiples of 4 or 8, mostly of less than 24 bits, and lose nothing but, once, the fraction that they found.
//
// What bounds it: in long calls power.  The MMAs take 256 clk of a block and the whole 390, but at 1000 W the SM clock falls to some 1.45 GHz
// (the kernel with one MMA per block keeps 1.94).  Measured, us with the quantiser, before and now: 8192 x 17408 x 5120 3079 / 2740,
// 3401 x 4528 x 3584 275 / 242, 1108 x 4560 x 2048 76 / 56, 37 x 5120 x 5120 30.5 / 17.9, Q5_K 14 x 3920 x 16896 57 / 30.  Two-term weights
// (Q8_0, Q6_K) would need four MMAs per block and end up where the other kernel is (512 x 4096 x 4096 Q8_0 65 us at 1.75 GHz against 67 at 1.96).
// With one block of every superblock 40 (2^15) times the others, all rows, us against the other kernel now: 8192 x 17408 x 5120 4126 (12207) / 2920, 1108 x
// 4560 x 2048 87 (238) / 74, 300 x 5120 x 5120 69 (217) / 55, 37 x 5120 x 5120 26.8 (61) / 26.4, Q5_K 14 x 3920 x 16896 51 (116) / 51.
//
// Plain stores of long K under IZB_GEMM_AUTO only, as with the cut of K: what the other store modes write is mostly quantised to int8 next, where a last
// bit can become a whole step, and they keep the sums that they had.
//
// The weight rows are the MMA's M (TMEM lanes), the token rows its N (TMEM columns): a dequantiser thread owns a weight row and writes its
// operand straight from registers to its TMEM lane (no shared-memory round trip, no swizzle), a short token tile costs a short MMA, and a
// store of a warp fills whole 32-byte sectors.
//
// CTA = one output tile of 128 weight rows x up to 128 token rows, 20 warps:
//   warps 0-7    dequantisers, two groups of four: one thread per weight row; raw superblock -> fp16 operand in TMEM (four slots
//                of 64 K-elements; group g fills slots g and g + 2), scales and mins to shared memory;
//   warps 8-15   combine: once per superblock tcgen05.ld and the f32 arithmetic above; final store;
//   warp 16      activation producer: cp.async.bulk of pre-swizzled operand images (made by the pre-pass) into a ring; finds out what rows are not plain;
//   warp 17      producer of the row scales s and the min-term images;
//   warp 18      weight producer: TMA (cp.async.bulk.tensor.2d) of the raw GGUF superblocks of 128 rows into a ring;
//   warp 19      issues tcgen05.mma (one elected thread).
// All waits are bounded: a wait that gives up sets a CTA-wide abort flag and a device error word, the CTA drains and
// returns without storing (izb_device_status reports it).
#include <cuda.h>
#include <string.h>

#include <type_traits>

#include "izb_fold.cuh"

namespace {

// error-word codes (which wait gave up)
enum : uint32_t { E_APROD = 1, E_WPROD = 2, E_DEQ = 4, E_MMA = 16, E_EPI = 32 };

// ---------------------------------------------------------------------------------------------- PTX wrappers
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_if(uint32_t bar, bool pred) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(bar), "r"((uint32_t)pred) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// non-blocking look at a barrier's phase
__device__ __forceinline__ uint32_t mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok)
               : "r"(bar), "r"(parity)
               : "memory");
  return ok;
}
// Bounded wait of a whole warp: every lane gets the same answer, so no lane leaves for the CTA's last barrier while the others go
// on to an instruction that needs all 32 (elect.sync under the MMA and the commit, the TMEM reads, __syncwarp).  (A lane that has seen its
// phase complete sees it again: the phase after it needs this warp.)  The vote costs nothing that shows: 8192 x 17408 x 5120 Q4_K 3.05 ms
// with and without.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag, uint32_t* err,
                                               uint32_t limit, uint32_t code) {
  constexpr uint32_t kAll = 0xFFFFFFFFu;
  if (__all_sync(kAll, mbar_test(bar, parity))) return true;
  for (uint32_t it = 0; it < limit; ++it) {
    if (__all_sync(kAll, mbar_try_wait(bar, parity))) return true;
    if ((it & 255u) == 255u && __any_sync(kAll, *abort_flag)) return false;
  }
  *abort_flag = 1;
  atomicOr(err, code);
  return false;
}
// several barriers at once: the looks overlap
struct Wait { uint32_t bar, parity; };
__device__ __forceinline__ bool mbar_wait_warp(const Wait (&w)[4], volatile uint32_t* abort_flag, uint32_t* err, uint32_t limit, uint32_t code) {
  uint32_t ok = 1;
#pragma unroll
  for (int i = 0; i < 4; ++i) ok &= mbar_test(w[i].bar, w[i].parity);
  if (__all_sync(0xFFFFFFFFu, ok)) return true;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (!mbar_wait_warp(w[i].bar, w[i].parity, abort_flag, err, limit, code)) return false;
  return true;
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
               "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void tma_2d(uint32_t dst, const void* tmap, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
               "l"(tmap), "r"(x), "r"(y), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// MMA and commit are issued by one lane, elected once.  What they need is the same for the whole warp and known to be (see the kernel's
// `warp`), so it stays in uniform registers; moved there one by one for every instruction an MMA took some 70 clk to issue.
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\tselp.u32 %0, 1, 0, e;\n\t}" : "=r"(e));
  return e != 0;
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// A from TMEM (lane = row, 32-bit column = two K-elements), B from shared memory
__device__ __forceinline__ void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc),
               "r"(idesc), "r"(accumulate)
               : "memory");
}
__device__ __forceinline__ void tc_mma_ss(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem), "l"(adesc), "l"(bdesc),
               "r"(idesc), "r"(accumulate)
               : "memory");
}
// sixteen registers to sixteen columns of the thread's TMEM lane
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// TMEM loads + wait, delivered as register pairs (two neighbouring columns) for the f32x2 arithmetic.  The loads, the wait and the moves are one
// asm block: nothing that uses the values can be scheduled before the wait.
// 16 TMEM lanes x 32 columns as matrix fragments: register pair 2g + r holds lane 8 r + threadlane / 4, columns 8 g + 2 (threadlane % 4) and
// the one after.  A thread then meets few columns and few rows: factors that belong to a column cost a fourth of the shared-memory reads
// that one lane x 32 columns per thread does (a 16-byte read of one address by the whole warp takes four passes).  Two such loads at once:
__device__ __forceinline__ void tc_ld_frag2(uint32_t ta, uint32_t tb, unsigned long long (&r)[8], unsigned long long (&q)[8]) {
  asm volatile(
      "{\n\t.reg .b32 t<16>, u<16>;\n\t"
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {t0,t1,t2,t3,t4,t5,t6,t7,t8,t9,t10,t11,t12,t13,t14,t15}, [%16];\n\t"
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {u0,u1,u2,u3,u4,u5,u6,u7,u8,u9,u10,u11,u12,u13,u14,u15}, [%17];\n\t"
      "tcgen05.wait::ld.sync.aligned;\n\t"
      "mov.b64 %0, {t0,t1};\n\t"
      "mov.b64 %1, {t2,t3};\n\t"
      "mov.b64 %2, {t4,t5};\n\t"
      "mov.b64 %3, {t6,t7};\n\t"
      "mov.b64 %4, {t8,t9};\n\t"
      "mov.b64 %5, {t10,t11};\n\t"
      "mov.b64 %6, {t12,t13};\n\t"
      "mov.b64 %7, {t14,t15};\n\t"
      "mov.b64 %8, {u0,u1};\n\t"
      "mov.b64 %9, {u2,u3};\n\t"
      "mov.b64 %10, {u4,u5};\n\t"
      "mov.b64 %11, {u6,u7};\n\t"
      "mov.b64 %12, {u8,u9};\n\t"
      "mov.b64 %13, {u10,u11};\n\t"
      "mov.b64 %14, {u12,u13};\n\t"
      "mov.b64 %15, {u14,u15};\n\t"
      "}"
      : "=l"(r[0]), "=l"(r[1]), "=l"(r[2]), "=l"(r[3]), "=l"(r[4]), "=l"(r[5]), "=l"(r[6]), "=l"(r[7]), "=l"(q[0]), "=l"(q[1]), "=l"(q[2]), "=l"(q[3]), "=l"(q[4]), "=l"(q[5]), "=l"(q[6]), "=l"(q[7])
      : "r"(ta), "r"(tb)
      : "memory");
}
// packed f32x2 arithmetic (two IEEE round-to-nearest operations per instruction)
__device__ __forceinline__ void ffma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long fmul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long pack2(float x) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ unsigned long long pair(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float lo_f(unsigned long long a) { return __uint_as_float((uint32_t)a); }
__device__ __forceinline__ float hi_f(unsigned long long a) { return __uint_as_float((uint32_t)(a >> 32)); }

// Shared-memory operands, K-major.  tcgen05 descriptor: start address >> 4, stride byte offset (8-row groups) >> 4 at bit 32, version 1 at
// bit 46, swizzle mode at bit 61; the leading byte offset is not used when the MMA's K extent lies inside one swizzled row.
// 128-byte rows, 128-byte swizzle (mode 2: the 16-byte chunk's number ^= row & 7):
__device__ __forceinline__ uint64_t umma_desc128(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// 32-byte rows, 32-byte swizzle (mode 6: chunk ^= (row >> 2) & 1):
__device__ __forceinline__ uint64_t umma_desc32(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(256 >> 4) << 32) | (1ull << 46) | (6ull << 61);
}
// instruction descriptor, kind::f16: D = f32 (bit 4), A and B fp16 (0 at bits 7 / 10), both K-major, N >> 3 at bit 17, M = 128 (M >> 4) at bit 24
__device__ __forceinline__ uint32_t umma_idesc(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24); }

__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
__device__ __forceinline__ __half2 bits_h2(uint32_t u) { return *reinterpret_cast<const __half2*>(&u); }
__device__ __forceinline__ __half2 h2_const(unsigned short b) { return __half2half2(__ushort_as_half(b)); }

// four int8 (offset by 128 into unsigned bytes) of `x` -> two half2, element order kept
__device__ __forceinline__ __half2 q8_pair(uint32_t x_biased, uint32_t sel) {
  return __hsub2(bits_h2(__byte_perm(x_biased, 0x64646464u, sel)), h2_const(0x6480));  // (1024 + q + 128) - 1152
}

constexpr int BN = 128;                       // weight rows of a tile: TMEM lanes
constexpr int BT = 128;                       // token rows of a tile at most: TMEM columns of an accumulator
constexpr int UNIT_BYTES = 2 * BT * 128;      // a unit of the activation ring: 2 x 64 K-elements of the token rows

constexpr int kThreads = 640;
// registers per thread of the roles (setmaxnreg): together no more than the CTA was launched with (640 x 96), or an increase waits for ever
constexpr int kRegsDeq = 72, kRegsComb = 144, kRegsOther = 48;
constexpr int kRoleRegs = (8 * kRegsDeq + 8 * kRegsComb + 4 * kRegsOther) * 32;

// ---- what differs between the weight forms
struct FQ4K { static constexpr int SBB = 144, NA = 5, NR = 2, NM = 3; };
struct FQ5K { static constexpr int SBB = kK16SbBytes, NA = 4, NR = 2, NM = 2; };

// TMEM columns: two accumulators and the min term's, the weight operand's four slots
constexpr int TM_D = 0, TM_D2 = 2 * BT, TM_W = 3 * BT;

// shared memory map (bytes from a 1024-aligned base)
template <class F>
struct Map {
  static constexpr int NA = F::NA, NR = F::NR, NM = F::NM, RAW = BN * F::SBB;
  static constexpr int OFF_A = 0;                                  // NA activation units
  static constexpr int OFF_RAW = OFF_A + NA * UNIT_BYTES;          // NR raw weight tiles
  static constexpr int OFF_W2 = OFF_RAW + NR * RAW;                // 2 x [128 rows][16] fp16, the weights' side of the min term
  static constexpr int OFF_MIN = OFF_W2 + 2 * 4096;                // NM x [tokens][16] fp16, the activations' side
  static constexpr int OFF_S = OFF_MIN + NM * 4096;                // NM x [tokens] f32 row scales s
  static constexpr int OFF_SCL = OFF_S + NM * 512;                 // 4 x 128 weight rows: f32 d, then f32 -16 dmin
  static constexpr int SCL = 1024;
  static constexpr int OFF_BAR = OFF_SCL + 4 * SCL;
  static constexpr int SMEM_BYTES = OFF_BAR + 512 + 1024;          // barriers + alignment slack
  // 8-byte mbarriers
  static constexpr int A_FULL = 0, A_EMPTY = A_FULL + NA, W_FULL = A_EMPTY + NA, W_EMPTY = W_FULL + 4, RAW_FULL = W_EMPTY + 4,
                       RAW_EMPTY = RAW_FULL + NR, S_FULL = RAW_EMPTY + NR, S_EMPTY = S_FULL + NM, W2_FULL = S_EMPTY + NM, W2_EMPTY = W2_FULL + 2,
                       D_FULL = W2_EMPTY + 2, D_EMPTY = D_FULL + 2, D2_EMPTY = D_EMPTY + 2, NUM_BARS = D2_EMPTY + 1;
  static_assert(SMEM_BYTES <= 232448, "shared memory per CTA");
  static_assert(NUM_BARS * 8 + 56 + 4 * NM <= 512, "barrier area");
  static_assert(OFF_RAW % 1024 == 0 && RAW % 1024 == 0 && OFF_W2 % 1024 == 0, "alignment of the operand and TMA areas");
};

// bytes per token row and superblock of the operand images, of the third term's, and of what goes beside them (min-term factors, s; kind)
constexpr int kImgRow = 1024, kFineRow = 512, kTailCopy = 36, kTailRow = kTailCopy + 1;

// position p (0..7) inside a 16-byte chunk of the Q4_K operand row holds element perm8[p] of that group of eight:
// the order in which the dequantiser's two-nibbles-per-word extraction delivers them
__device__ __forceinline__ int q4k_perm8(int p) { return (p & 4) | ((p & 1) << 1) | ((p >> 1) & 1); }

// ---------------------------------------------------------------------------------------------- activation pre-pass
// Per token tile and superblock: the operand images (above) and what goes beside them.  One CTA = 32 rows x one superblock, a warp per row,
// a lane per eight values (= one 16-byte chunk of an image); the images go out in whole 128-byte lines, what belongs to a row or block only
// once is collected in shared memory first.
struct PrepRows {
  float sc[8][33], v[8][33];  // [block of the superblock][row]: activation scale, r * (sum of the quants) / 16
  float s[32];
  unsigned char kind[32];
};
// asc = r * s for the eight blocks of a row's superblock; the whole warp calls it, lane l with block l / 4.  s is a 128th of the largest
// |asc| (down at 2^-118 that itself, which would lose bits).  `kind`, for scales that differ more and more:
//   kPlain   all r that are not 0 at least 32: hi + lo keep 21 to 22 bits of the smallest block's largest value
//   kSpread  at least 2^-5: a third term, all three on grids that the blocks share.  (Finer grids for smaller blocks would do with two terms, but
//            sums that larger blocks make long then lose those bits MMA by MMA and always towards zero: 5e-7 of the result for 256 : 1.)  s is negative.
//   kWide    all else, also scales that are no finite numbers: r = 1 and s = 0, and the GEMM takes the blocks one by one
enum : uint32_t { kPlain = 0, kSpread = 1, kWide = 2 };
struct RowScale {
  float r, s;
  uint32_t kind;
};
__device__ __forceinline__ RowScale split_scale(float asc) {
  constexpr uint32_t kAll = 0xFFFFFFFFu;
  const uint32_t mag = __float_as_uint(asc) & 0x7FFFFFFFu;
  uint32_t mx = max(mag, __shfl_xor_sync(kAll, mag, 4));
  mx = max(mx, __shfl_xor_sync(kAll, mx, 8));
  mx = max(mx, __shfl_xor_sync(kAll, mx, 16));
  const float m = __uint_as_float(mx);
  const bool tiny = m < 0x1p-118f;
  RowScale o = {mag == 0 ? 0.0f : __fmul_rn(tiny ? 1.0f : 128.0f, __fdiv_rn(asc, m)), tiny ? m : 0.0078125f * m, kPlain};
  if (__any_sync(kAll, mag != 0 && !(fabsf(o.r) >= 32.0f))) {
    if (__any_sync(kAll, mx >= 0x7F800000u || (mag != 0 && !(fabsf(o.r) >= 0x1p-5f)))) o = {1.0f, 0.0f, kWide};
    else o.s = -o.s, o.kind = kSpread;
  }
  return o;
}
// where a row's chunks go: the images of its tile and superblock, and the third term's
struct RowImg {
  unsigned char *img, *fine;
  int tt, row;
};
__device__ __forceinline__ RowImg row_img(unsigned char* img, unsigned char* fine, size_t sb, int tt, int row) {
  return {img + sb * kImgRow * tt, fine + sb * kFineRow * tt, tt, row};
}
// the chunk of eight values r * q, chunk `c` (0 .. 31) of a superblock: hi a multiple of 4, of 8 from 2^13 on; a spread row's lo a multiple of 2^-9; a wide row's
// hi all of q.  Q5_K, whose weights have a bit more, hi a multiple of 8 (plain rows' of 4 while r is below 64): of two errors that grow in opposite
// directions, the bits that the tensor core's sums lose and lo's own, the smaller sum (K = 2048 and 5120: 1.2e-7, multiples of 4 1.5e-7; Q4_K 1.1e-7).
template <bool kQ4K>
__device__ __forceinline__ void put_chunk(const RowImg& o, int c, const RowScale& rs, const int (&q)[8]) {
  uint32_t hi[4], lo[4], fine[4];
  // x + round - round: x as a multiple of round / (1.5 * 2^23)
  const float round = rs.kind == kWide ? 0x1.8p23f : kQ4K || (rs.kind == kPlain && fabsf(rs.r) < 64.0f) ? 0x1.8p25f : 0x1.8p26f;
  constexpr float kRoundLo = 0x1.8p14f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float x = (float)q[kQ4K ? q4k_perm8(2 * j) : 2 * j], y = (float)q[kQ4K ? q4k_perm8(2 * j + 1) : 2 * j + 1];
    const __half2 h = __floats2half2_rn(__fsub_rn(__fmaf_rn(rs.r, x, round), round), __fsub_rn(__fmaf_rn(rs.r, y, round), round));
    const float2 hf = __half22float2(h);
    float2 rest = make_float2(__fmaf_rn(rs.r, x, -hf.x), __fmaf_rn(rs.r, y, -hf.y));
    hi[j] = h2_bits(h);
    if (rs.kind == kSpread) {
      const float2 l = make_float2(__fsub_rn(__fadd_rn(rest.x, kRoundLo), kRoundLo), __fsub_rn(__fadd_rn(rest.y, kRoundLo), kRoundLo));
      fine[j] = h2_bits(__floats2half2_rn(__fsub_rn(rest.x, l.x), __fsub_rn(rest.y, l.y)));
      rest = l;
    }
    lo[j] = h2_bits(__floats2half2_rn(rest.x, rest.y));
  }
  const size_t at = (size_t)(c >> 3) * 128 * o.tt + o.row * 128 + (((c & 7) ^ (o.row & 7)) << 4);
  *reinterpret_cast<uint4*>(o.img + at) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  *reinterpret_cast<uint4*>(o.img + at + 512 * o.tt) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
  if (rs.kind == kSpread) *reinterpret_cast<uint4*>(o.fine + at) = make_uint4(fine[0], fine[1], fine[2], fine[3]);
}
// (after a barrier, the whole CTA) what goes beside the images, for the lane's row: row r of a tile
__device__ __forceinline__ void put_tail(const PrepRows& p, unsigned char* sb_tail, int tt, int r, int warp, int lane) {
  if (warp > 2) return;
  if (warp == 2) {
    reinterpret_cast<float*>(sb_tail + 32 * tt)[r] = p.s[lane];
    sb_tail[36 * tt + r] = p.kind[lane];
    return;
  }
  uint32_t o[4];  // warp 0: the eight hi terms, warp 1: the eight lo terms
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float x = p.v[2 * j][lane], y = p.v[2 * j + 1][lane];
    __half2 h = __floats2half2_rn(x, y);
    if (warp) {
      const float2 b = __half22float2(h);
      h = __floats2half2_rn(__fsub_rn(x, b.x), __fsub_rn(y, b.y));
    }
    o[j] = h2_bits(h);
  }
  *reinterpret_cast<uint4*>(sb_tail + r * 32 + ((warp ^ ((r >> 2) & 1)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
}
// one row's images from its int8 values and their block's scale (this lane's eight and its block's)
template <bool kPerm>
__device__ __forceinline__ void put_row(PrepRows& p, const RowImg& o, int row, int lane, float asc, const int (&q)[8]) {
  const RowScale rs = split_scale(asc);
  put_chunk<kPerm>(o, lane, rs, q);
  int sum = q[0] + q[1] + q[2] + q[3] + q[4] + q[5] + q[6] + q[7];
  sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
  sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 2);  // the four chunks of a 32-block
  if ((lane & 3) == 0) p.v[lane >> 2][row] = __fmul_rn(rs.r, 0.0625f * (float)sum);  // (at most 2^15)
  if (lane == 0) p.s[row] = rs.s, p.kind[row] = (unsigned char)rs.kind;
}

template <bool kPerm>
__global__ void __launch_bounds__(256) fold_prepare_kernel(const int8_t* __restrict__ aq, const float* __restrict__ asc, int lda, int K, int rows_total,
                                                           unsigned char* __restrict__ img, unsigned char* __restrict__ fine, unsigned char* __restrict__ tail, int tt, int n_rows,
                                                           uint32_t* __restrict__ part_bad) {
  __shared__ PrepRows s;
  const int sb = blockIdx.y, nsb = K >> 8, m0 = blockIdx.x * 32, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_launch_next();
  pdl_wait();
  if (part_bad && sb == 0 && blockIdx.x == 0 && threadIdx.x == 0) *part_bad = 0;
  s.sc[warp][lane] = m0 + lane < rows_total ? asc[(size_t)(sb * 8 + warp) * lda + m0 + lane] : 0.0f;
  uint2 x[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + warp + 8 * i;
    x[i] = m < rows_total ? *reinterpret_cast<const uint2*>(aq + (size_t)m * K + sb * 256 + lane * 8) : make_uint2(0, 0);
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int rr = warp + 8 * i, m = m0 + rr, tile = m / tt;
    if (m >= n_rows) break;
    int a[8];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      a[k] = (int)(int8_t)(x[i].x >> (8 * k));
      a[4 + k] = (int)(int8_t)(x[i].y >> (8 * k));
    }
    put_row<kPerm>(s, row_img(img, fine, (size_t)tile * nsb + sb, tt, m - tile * tt), rr, lane, s.sc[lane >> 2][rr], a);
  }
  __syncthreads();
  const int m = m0 + lane, tile = m / tt;
  if (m < n_rows) put_tail(s, tail + ((size_t)tile * nsb + sb) * kTailRow * tt, tt, m - tile * tt, warp, lane);
}

// ---------------------------------------------------------------------------------------------- quantiser + pre-pass in one
// izb_quantize_act (csrc/izb_quantize.cu, the arithmetic of quantize_act_cpu, src/quants.h:626-643, bit for bit) and
// fold_prepare_kernel above in one pass over the f32 rows: a lane owns 8 consecutive values (= one 16-byte operand chunk),
// four lanes a 32-block.  Writes aq / asc exactly as the quantiser does (the caller's buffers stay valid for every other
// kernel) and, from the same registers, the operand images and what goes beside them: the int8 rows are not read back and the
// second launch is gone.  One CTA = 8 kR rows x one superblock: four rows a warp, or one where that leaves SMs without work.
template <bool kPerm, int kR>
__global__ void __launch_bounds__(256) fold_quant_prepare_kernel(const float* __restrict__ x, int ldx, int M, int Mp, int K,
                                                            int8_t* __restrict__ aq, float* __restrict__ asc,
                                                            unsigned char* __restrict__ img, unsigned char* __restrict__ fine, unsigned char* __restrict__ tail, int tt, int n_tiles,
                                                            uint32_t* __restrict__ part_bad) {
  __shared__ PrepRows s;
  const int sb = blockIdx.x, nsb = K >> 8, m0 = blockIdx.y * (8 * kR), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = sb * 256 + lane * 8;
  pdl_launch_next();
  pdl_wait();
  if (part_bad && sb == 0 && blockIdx.y == 0 && threadIdx.x == 0) *part_bad = 0;
  float v[kR][8];
#pragma unroll
  for (int i = 0; i < kR; ++i) {
    const int m = m0 + warp + 8 * i;
    if (m < M) {
      const float4* p = reinterpret_cast<const float4*>(x + (size_t)m * ldx + col);
      const float4 a = __ldcs(p), b = __ldcs(p + 1);
      v[i][0] = a.x; v[i][1] = a.y; v[i][2] = a.z; v[i][3] = a.w;
      v[i][4] = b.x; v[i][5] = b.y; v[i][6] = b.z; v[i][7] = b.w;
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) v[i][k] = 0.0f;
    }
  }
#pragma unroll
  for (int i = 0; i < kR; ++i) {
    const int rr = warp + 8 * i, m = m0 + rr;
    float amax = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) amax = fmaxf(amax, fabsf(v[i][k]));
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
    const float inv = amax > 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
    int q[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float pr = __fmul_rn(v[i][k], inv);
      q[k] = fabsf(pr) <= 2147483520.0f ? __float2int_rn(pr) : 0;  // (see quantize_act_kernel: the overflow case)
      q[k] = (int)(int8_t)q[k];  // the stored byte is what the GEMM multiplies
    }
    const float sc = __fdiv_rn(amax, 127.0f);
    if (m < Mp) {
      uint2 pk;
      pk.x = (q[0] & 0xFF) | ((q[1] & 0xFF) << 8) | ((q[2] & 0xFF) << 16) | ((uint32_t)(q[3] & 0xFF) << 24);
      pk.y = (q[4] & 0xFF) | ((q[5] & 0xFF) << 8) | ((q[6] & 0xFF) << 16) | ((uint32_t)(q[7] & 0xFF) << 24);
      *reinterpret_cast<uint2*>(aq + (size_t)m * K + col) = pk;
    }
    if ((lane & 3) == 0) s.sc[lane >> 2][rr] = sc;
    const int tile = m / tt;
    if (tile < n_tiles)  // (padding rows past the last tile the GEMM reads: aq / asc only)
      put_row<kPerm>(s, row_img(img, fine, (size_t)tile * nsb + sb, tt, m - tile * tt), rr, lane, sc, q);
  }
  __syncthreads();
  if (lane >= 8 * kR) return;
  if (m0 + lane < Mp) asc[(size_t)(sb * 8 + warp) * Mp + m0 + lane] = s.sc[warp][lane];
  const int tile = (m0 + lane) / tt;
  if (tile < n_tiles) put_tail(s, tail + ((size_t)tile * nsb + sb) * kTailRow * tt, tt, m0 + lane - tile * tt, warp, lane);
}

// ---------------------------------------------------------------------------------------------- weight forms
// What a weight row's superblock becomes.  Every form offers
//   load(row)              the superblock's header into registers
//   load_stage(c, row)     the quants of blocks 2c, 2c + 1 into registers
//   half<kH>(c, o)         the 32 elements of block 2c + kH as fp16 pairs, K order
//   put_scales(scl, t)     what the combine warps need of row t
//   mins(u)                the eight blocks' mn as fp16
struct DeqQ4K {
  uint4 hdr, q0, q1;
  // (scale, min) bytes of sub-blocks 2c and 2c + 1 (get_scale_min_k4, src/quants.h:61-69), without a branch on c
  __device__ __forceinline__ void pair(int c, uint32_t& sc2, uint32_t& mn2) const {
    const int sh = 16 * (c & 1);
    const uint32_t a = hdr.y >> sh, b = hdr.z >> sh, d = hdr.w >> sh;
    sc2 = c >= 2 ? ((d & 0x0F0Fu) | ((a >> 2) & 0x3030u)) : (a & 0x3F3Fu);
    mn2 = c >= 2 ? (((d >> 4) & 0x0F0Fu) | ((b >> 2) & 0x3030u)) : (b & 0x3F3Fu);
  }
  __device__ __forceinline__ void load(const unsigned char* row) { hdr = *reinterpret_cast<const uint4*>(row); }
  __device__ __forceinline__ void load_stage(int c, const unsigned char* row) {
    q0 = *reinterpret_cast<const uint4*>(row + 16 + 32 * c);
    q1 = *reinterpret_cast<const uint4*>(row + 32 + 32 * c);
  }
  __device__ __forceinline__ void put_scales(unsigned char* scl, int t) const {
    reinterpret_cast<float*>(scl)[t] = half_bits_to_float(hdr.x & 0xFFFFu);
    reinterpret_cast<float*>(scl)[128 + t] = -16.0f * half_bits_to_float(hdr.x >> 16);
  }
  template <int kH>
  __device__ __forceinline__ void half(int c, uint32_t (&o)[16]) const {
    const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
    // the block's 6-bit sub-block scale as (sc, sc) and (-1024 sc, -1024 sc): 0x6400 | sc is the fp16 number 1024 + sc
    uint32_t sc2, mn_unused;
    pair(c, sc2, mn_unused);
    __half2 sc = __hsub2(bits_h2(__byte_perm(sc2, 0x64646464u, kH ? 0x4141 : 0x4040)), h2_const(0x6400));
    __half2 neg = __hmul2(sc, h2_const(0xE400));
    // High nibbles stay where they are: (word & 0x00F000F0) | 0x6400 is the fp16 number 1024 + 16 q, and
    // (1024 + 16 q) * (sc / 16) - 64 sc = sc * q exactly (one rounding, of an integer below 2^11).  One shift per
    // word (for its upper bytes) instead of three.
    if (kH) { sc = __hmul2(sc, h2_const(0x2C00)); neg = __hmul2(neg, h2_const(0x2C00)); }
    constexpr uint32_t mask = kH ? 0x00F000F0u : 0x000F000Fu;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      o[2 * j] = h2_bits(__hfma2(bits_h2((w[j] & mask) | 0x64006400u), sc, neg));
      o[2 * j + 1] = h2_bits(__hfma2(bits_h2(((w[j] >> 8) & mask) | 0x64006400u), sc, neg));
    }
  }
  __device__ __forceinline__ void mins(uint32_t (&u)[4]) const {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t sc_unused, mn2;
      pair(c, sc_unused, mn2);
      u[c] = h2_bits(__hsub2(bits_h2(__byte_perm(mn2, 0x64646464u, 0x4140)), h2_const(0x6400)));
    }
  }
};

// Q5_K in the generic form: f32 d | f32 dmin | int8 scale[16] | uint8 min[16] | pad | int8 quant[256]
struct DeqQ5K {
  uint4 h0, h1, h2, qs[4];
  __device__ __forceinline__ void load(const unsigned char* row) {
    h0 = *reinterpret_cast<const uint4*>(row);
    h1 = *reinterpret_cast<const uint4*>(row + 16);
    h2 = *reinterpret_cast<const uint4*>(row + 32);
  }
  __device__ __forceinline__ void put_scales(unsigned char* scl, int t) const {
    reinterpret_cast<float*>(scl)[t] = __uint_as_float(h0.x);
    reinterpret_cast<float*>(scl)[128 + t] = -16.0f * __uint_as_float(h0.y);
  }
  __device__ __forceinline__ void load_stage(int c, const unsigned char* row) {
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) qs[jj] = *reinterpret_cast<const uint4*>(row + 48 + 64 * c + 16 * jj);
  }
  template <int kH>
  __device__ __forceinline__ void half(int c, uint32_t (&o)[16]) const {
    const uint32_t scw = c == 0 ? h0.z : c == 1 ? h0.w : c == 2 ? h1.x : h1.y;  // the four halves' scales
#pragma unroll
    for (int jj = 0; jj < 2; ++jj) {
      const uint4 q = qs[2 * kH + jj];
      const uint32_t x[4] = {q.x, q.y, q.z, q.w};
      const __half2 f = __half2half2(__int2half_rn((int)(int8_t)(scw >> (8 * (2 * kH + jj)))));
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        o[8 * jj + 2 * k] = h2_bits(__hmul2(q8_pair(x[k] ^ 0x80808080u, 0x4140), f));
        o[8 * jj + 2 * k + 1] = h2_bits(__hmul2(q8_pair(x[k] ^ 0x80808080u, 0x4342), f));
      }
    }
  }
  __device__ __forceinline__ void mins(uint32_t (&u)[4]) const {
    const uint32_t m[4] = {h1.z, h1.w, h2.x, h2.y};  // (both halves of a block share it)
#pragma unroll
    for (int k = 0; k < 4; ++k) u[k] = h2_bits(__hsub2(bits_h2(__byte_perm(m[k], 0x64646464u, 0x4240)), h2_const(0x6400)));
  }
};

template <class F> struct DeqOf;
template <> struct DeqOf<FQ4K> { using type = DeqQ4K; };
template <> struct DeqOf<FQ5K> { using type = DeqQ5K; };

// ---------------------------------------------------------------------------------------------- the GEMM kernel
template <class F>
__global__ void __launch_bounds__(kThreads, 1) gemm_fold_kernel(const __grid_constant__ CUtensorMap tmW, const FoldParams p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  using MP = Map<F>;
  constexpr int NA = MP::NA, NR = MP::NR, NM = MP::NM, RAW = MP::RAW, SBB = F::SBB;
  constexpr int ND = 2;                 // accumulators: superblocks take them in turn
  constexpr int UNITS = 4;              // units of the activation ring per superblock
  constexpr int NCH = 2;                // groups of 32 columns of a combine warp
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + MP::OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + MP::OFF_BAR + MP::NUM_BARS * 8);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + MP::OFF_BAR + MP::NUM_BARS * 8 + 4);
  uint32_t* unit_kinds = reinterpret_cast<uint32_t*>(smem + MP::OFF_BAR + MP::NUM_BARS * 8 + 8);  // [4], items with rows that are not plain: superblocks in turn
  uint32_t* s_kinds = unit_kinds + 4;                                                                // [NM], with the ring of scales
  uint32_t *unit_item = s_kinds + NM, *s_item = unit_item + 4;                                       // [4] each, items in turn
  const uint32_t bar0 = smem_u32(bars);
  auto bar = [&](int i) -> uint32_t { return bar0 + 8u * (uint32_t)i; };
  // (through a shuffle: the compiler then knows that the role branches and what follows from them are the same for the whole warp, and keeps
  // the MMAs' operands in uniform registers)
  const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    // Shared memory is released by an arrival of every thread, accumulators by one of every warp, what the tensor core reads by a tcgen05.commit.
    for (int i = 0; i < NA; ++i) { mbar_init(bar(MP::A_FULL + i), 1); mbar_init(bar(MP::A_EMPTY + i), 1); }
    for (int i = 0; i < 4; ++i) { mbar_init(bar(MP::W_FULL + i), 128); mbar_init(bar(MP::W_EMPTY + i), 1); }
    for (int i = 0; i < NR; ++i) { mbar_init(bar(MP::RAW_FULL + i), 1); mbar_init(bar(MP::RAW_EMPTY + i), 256); }
    for (int i = 0; i < NM; ++i) { mbar_init(bar(MP::S_FULL + i), 1); mbar_init(bar(MP::S_EMPTY + i), 256 + 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(bar(MP::W2_FULL + i), 128); mbar_init(bar(MP::W2_EMPTY + i), 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(bar(MP::D_FULL + i), 1); mbar_init(bar(MP::D_EMPTY + i), 8); }
    mbar_init(bar(MP::D2_EMPTY), 8);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 16) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xFFFFFFFFu, *tmem_slot, 0);

  // ---- the CTA's work: items blockIdx.x, blockIdx.x + gridDim.x, ... of (token tiles) x (weight tiles) x (K parts), K part
  // fastest, then weight tile.  Every role walks the same list; its ring positions and barrier parities run on from item to
  // item, so the producers, the dequantisers and the issuer are already inside the next one while the combine warps store.
  const int n_ntiles = (p.N + BN - 1) / BN, nsb = p.K >> 8;
  const int n_work = p.n_mtiles * n_ntiles * p.n_split;
  struct Item { int tile, nt, ks, s0, s1, r0, nr, n; };  // r0, nr: the tile's token rows; n: columns of its MMAs
  auto item = [&](int w) -> Item {
    Item it;
    it.ks = 0;
    int q = w;
    if (p.n_split > 1) { q = w / p.n_split; it.ks = w - q * p.n_split; }
    it.tile = q / n_ntiles;
    it.nt = q - it.tile * n_ntiles;
    it.s0 = it.ks * nsb / p.n_split;
    it.s1 = (it.ks + 1) * nsb / p.n_split;
    it.r0 = it.tile * p.tt;
    it.nr = min(p.tt, p.M - it.r0);
    it.n = (it.nr + 15) & ~15;
    return it;
  };

  // Kinds of a tile's rows.  Both producers of the token side look them up, the issuer and the combine warps find them in shared memory: for an item, whose
  // loops then are those for plain rows alone or the longer ones, and in the latter for a superblock (`sb` of all tiles').
  auto load_kinds = [&](size_t sb, int n) -> uint32_t {
    return 4 * lane < n ? *reinterpret_cast<const uint32_t*>(p.tail + sb * kTailRow * p.tt + kTailCopy * p.tt + 4 * lane) : 0u;
  };
  auto all_kinds = [&](uint32_t k) -> uint32_t {
    k = __reduce_or_sync(0xFFFFFFFFu, k);
    k |= k >> 16;
    return (k | k >> 8) & 3u;
  };
  auto item_kinds = [&](const Item& it) -> uint32_t {  // a lane 16 rows: four superblocks a load, kAhead loads in flight
    constexpr int kAhead = 8;
    const unsigned char* k = p.tail + (size_t)it.tile * nsb * kTailRow * p.tt + kTailCopy * p.tt + 16 * (lane & 7);
    uint32_t any = 0;
    for (int s = it.s0 + (lane >> 3); 16 * (lane & 7) < it.n && s < it.s1; s += 4 * kAhead) {
      uint4 v[kAhead];
#pragma unroll
      for (int i = 0; i < kAhead; ++i) v[i] = *reinterpret_cast<const uint4*>(k + (size_t)min(s + 4 * i, it.s1 - 1) * kTailRow * p.tt);
#pragma unroll
      for (int i = 0; i < kAhead; ++i) any |= v[i].x | v[i].y | v[i].z | v[i].w;
    }
    __syncwarp();
    return all_kinds(any);
  };

  if (warp >= 16) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOther));
    // Every role loop below is executed by its whole warp (uniform waits, an elected lane issues), so no lane of a role warp
    // sits at the final CTA barrier while another lane of the same warp is still working.
    if (warp == 16) {
      // ================= activation producer: the tile's stage images lie back to back in global memory
      pdl_wait();  // (the pre-pass; the weights depend on no kernel and are on their way by then)
      int sa = 0, pa = 1, sbc = 0, n_item = 0;
      bool ok = true;
      for (int w = blockIdx.x; w < n_work && ok; w += gridDim.x, ++n_item) {
        const Item it = item(w);
        const uint32_t half = (uint32_t)it.n * 128;  // bytes of a stage; a unit of the ring is two of them
        const int step = 256 * p.tt;
        auto copy = [&](const unsigned char* src) {
          const uint32_t dst = smem_u32(smem + MP::OFF_A + sa * UNIT_BYTES);
          if (it.n == p.tt) {
            bulk_g2s(dst, src, 2 * half, bar(MP::A_FULL + sa));
          } else {
            bulk_g2s(dst, src, half, bar(MP::A_FULL + sa));
            bulk_g2s(dst + half, src + 128 * p.tt, half, bar(MP::A_FULL + sa));
          }
        };
        auto next = [&]() { if (++sa == NA) { sa = 0; pa ^= 1; } };
        auto unit = [&](const unsigned char* src, bool skip) -> bool {
          if (!mbar_wait_warp(bar(MP::A_EMPTY + sa), pa, abort_flag, p.err, p.spin_limit, E_APROD)) return false;
          if (lane == 0 && !skip) {
            mbar_expect_tx(bar(MP::A_FULL + sa), 2 * half);
            copy(src);
          }
          __syncwarp();
          next();
          return true;
        };
        const size_t sb0 = (size_t)it.tile * nsb;
        const unsigned char* src = p.img + sb0 * kImgRow * p.tt;
        // the item's first unit: its bytes are on their way while the kinds are looked up, and count as arrived with this thread's arrival
        if (!mbar_wait_warp(bar(MP::A_EMPTY + sa), pa, abort_flag, p.err, p.spin_limit, E_APROD)) break;
        const bool skip = it.s0 * UNITS == p.skip_stage;  // (skip_stage: diagnostics only, makes the waits of this unit run out)
        if (lane == 0 && !skip) copy(src + (size_t)(it.s0 * UNITS) * step);
        __syncwarp();
        const uint32_t any = item_kinds(it);
        uint32_t more = any ? all_kinds(load_kinds(sb0 + it.s0, it.n)) : 0u;
        if (lane == 0) {
          unit_item[n_item & 3] = any;
          unit_kinds[sbc & 3] = more;
          if (!skip) mbar_expect_tx(bar(MP::A_FULL + sa), 2 * half);
        }
        __syncwarp();
        next();
        if (!any) {
          for (int g = it.s0 * UNITS + 1; g < it.s1 * UNITS && ok; ++g) ok = unit(src + (size_t)g * step, g == p.skip_stage);
          sbc += it.s1 - it.s0;
          continue;
        }
        for (int s = it.s0; s < it.s1 && ok; ++s, ++sbc) {
          const uint32_t ahead = s + 1 < it.s1 ? load_kinds(sb0 + s + 1, it.n) : 0u;
          const unsigned char *u = src + (size_t)(s * UNITS) * step, *fine = p.fine + (sb0 + s) * kFineRow * p.tt;
          if (s > it.s0) {
            if (lane == 0) unit_kinds[sbc & 3] = more;  // (before this thread's arrival for the unit)
            ok = unit(u, s * UNITS == p.skip_stage);
          }
          if (ok && (more & kSpread)) ok = unit(fine, false) && unit(fine + step, false);
          for (int i = 1; i < UNITS && ok; ++i) ok = unit(u + i * step, s * UNITS + i == p.skip_stage);
          more = all_kinds(ahead);
        }
      }
    } else if (warp == 17) {
      // ================= per superblock: row scales and the min term's activation side
      pdl_wait();
      int sq = 0, pq = 1, n_item = 0;
      bool ok = true;
      for (int w = blockIdx.x; w < n_work && ok; w += gridDim.x, ++n_item) {
        const Item it = item(w);
        const size_t sb_bytes = (size_t)kTailRow * p.tt;
        const unsigned char* src = p.tail + ((size_t)it.tile * nsb + it.s0) * sb_bytes;
        const uint32_t any = item_kinds(it);
        for (int s = it.s0; s < it.s1; ++s, src += sb_bytes) {
          uint32_t more = 0;
          if (any) more = all_kinds(load_kinds((size_t)it.tile * nsb + s, it.n));
          if (!mbar_wait_warp(bar(MP::S_EMPTY + sq), pq, abort_flag, p.err, p.spin_limit, E_WPROD)) { ok = false; break; }
          const uint32_t dst = smem_u32(smem + MP::OFF_S + sq * 512), full = bar(MP::S_FULL + sq);
          if (lane == 0) {
            if (s == it.s0) s_item[n_item & 3] = any;  // (before this thread's arrival)
            s_kinds[sq] = more;
            mbar_expect_tx(full, it.n * kTailCopy);
            bulk_g2s(smem_u32(smem + MP::OFF_MIN + sq * 4096), src, it.n * 32, full);
            bulk_g2s(dst, src + 32 * p.tt, it.n * 4, full);
          }
          __syncwarp();
          if (++sq == NM) { sq = 0; pq ^= 1; }
        }
      }
    } else if (warp == 18) {
      // ================= weight producer: TMA of the raw superblocks of the tile's 128 weight rows
      int rb = 0, pr = 1;
      bool ok = true;
      for (int w = blockIdx.x; w < n_work && ok; w += gridDim.x) {
        const Item it = item(w);
        const int wrow = p.mat * p.N + it.nt * BN;
        for (int s = it.s0; s < it.s1; ++s) {
          if (!mbar_wait_warp(bar(MP::RAW_EMPTY + rb), pr, abort_flag, p.err, p.spin_limit, E_WPROD)) { ok = false; break; }
          if (lane == 0) {
            mbar_expect_tx(bar(MP::RAW_FULL + rb), RAW);
            tma_2d(smem_u32(smem + MP::OFF_RAW + rb * RAW), &tmW, s * (SBB / 4), wrow, bar(MP::RAW_FULL + rb));
          }
          __syncwarp();
          if (++rb == NR) { rb = 0; pr ^= 1; }
        }
      }
    } else {
      // ================= MMA issuer
      bool ok = true;
      const bool leader = elect_one();
      int sa = 0, pa = 0, sq = 0, pq = 0, d = 0, pd = 1, sbc = 0, n_item = 0;  // ring positions and wait parities, superblocks and items done: they run on across items
      for (int w = blockIdx.x; w < n_work && ok; w += gridDim.x, ++n_item) {
        const Item it = item(w);
        const uint32_t idesc = umma_idesc(it.n), half = (uint32_t)it.n * 128;
        // K = 16 step k of stage c's weights x an activation stage
        auto mma = [&](uint32_t dt, int c, int k, uint32_t a_addr, uint32_t accumulate) {
          tc_mma_ts(dt, tmem_base + (uint32_t)(TM_W + c * 32 + 8 * k), umma_desc128(a_addr + 32 * k), idesc, accumulate);
        };
        auto a_base = [&](int u) -> uint32_t { return smem_u32(smem + MP::OFF_A + u * UNIT_BYTES); };
        auto next = [&]() { if (++sa == NA) { sa = 0; pa ^= 1; } };
        // (the item's first unit tells which of the two loops)
        if (!mbar_wait_warp(bar(MP::A_FULL + sa), pa, abort_flag, p.err, p.spin_limit, E_MMA)) break;
        if (__shfl_sync(0xFFFFFFFFu, unit_item[n_item & 3], 0)) {  // (a shuffle: see `warp`)
          // with rows that are not plain
          auto wait = [&](int b, int parity) -> bool { return mbar_wait_warp(bar(b), (uint32_t)parity, abort_flag, p.err, p.spin_limit, E_MMA); };
          auto next_d = [&]() { if (++d == ND) { d = 0; pd ^= 1; } };
          struct Place { int u, parity; };  // in the ring of units, `ahead` places on
          auto place = [&](int ahead) -> Place {
            Place o = {sa, pa};
            for (int i = 0; i < ahead; ++i)
              if (++o.u == NA) { o.u = 0; o.parity ^= 1; }
            return o;
          };
          auto unit = [&](Place at) -> Wait { return {bar(MP::A_FULL + at.u), (uint32_t)at.parity}; };
          // (the leader) eight K steps, half h of the superblock
          auto issue = [&](int u, uint32_t dt, int h, bool fresh, bool last) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              mma(dt, 2 * h + (e >> 2), e & 3, a_base(u) + (e >> 2) * half, fresh && e == 0 ? 0u : 1u);
              if ((e & 3) == 3 && last) tc_commit(bar(MP::W_EMPTY + 2 * h + (e >> 2)));
            }
          };
          // one superblock.  Compiled for each of the common combinations of kinds: tests of them between its MMAs cost these their uniform registers
          // (1108 x 4560 x 2048: 66 us with all rows plain in this loop, 51 in the one below)
          auto superblock = [&](auto spread_known, auto wide_known) -> bool {
            const bool spread = decltype(spread_known)::value, wide = decltype(wide_known)::value;
            const int b = sbc & 1;
            const uint32_t pw = b;
            const Place lo0 = place(0);
            const Wait w2{bar(MP::W_FULL + 2), pw}, w3{bar(MP::W_FULL + 3), pw};
            const int at = spread ? 3 : 1;
            if (spread) {
              // the third term, into an accumulator of its own.  Before the others, although the first of those lies before it in the ring: the combine
              // warps take it while these run, and the next superblock's while they take these
              const Place f0 = place(1), f1 = place(2);
              const Wait need[4] = {unit(f0), unit(f1), w2, w3};
              if (!mbar_wait_warp(need, abort_flag, p.err, p.spin_limit, E_MMA)) return false;
              tc_fence_after();
              if (leader) {
                const uint32_t dt = tmem_base + (uint32_t)(TM_D + d * BT);
                issue(f0.u, dt, 0, true, false);
                tc_commit(bar(MP::A_EMPTY + f0.u));
                issue(f1.u, dt, 1, false, false);
                tc_commit(bar(MP::A_EMPTY + f1.u));
                tc_commit(bar(MP::D_FULL + d));
              }
              __syncwarp();
              next_d();
            }
            const Place lo1 = place(at), hi0 = place(at + 1), hi1 = place(at + 2);
            const uint32_t dt = tmem_base + (uint32_t)(TM_D + d * BT);
            const Wait need[4] = {{bar(MP::D_EMPTY + d), (uint32_t)pd}, unit(lo1), w2, w3};
            if (!mbar_wait_warp(need, abort_flag, p.err, p.spin_limit, E_MMA)) return false;
            tc_fence_after();
            if (leader) {
              issue(lo0.u, dt, 0, true, false);
              tc_commit(bar(MP::A_EMPTY + lo0.u));
              issue(lo1.u, dt, 1, false, false);
              tc_commit(bar(MP::A_EMPTY + lo1.u));
            }
            __syncwarp();
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
              const Place hi = h ? hi1 : hi0;
              if (!wait(MP::A_FULL + hi.u, hi.parity)) return false;
              tc_fence_after();
              if (leader) {
                issue(hi.u, dt, h, false, !wide);
                if (!wide) tc_commit(bar(MP::A_EMPTY + hi.u));
              }
              __syncwarp();
            }
            const Wait w2_full{bar(MP::W2_FULL + b), (uint32_t)(sbc >> 1) & 1u}, s_full{bar(MP::S_FULL + sq), (uint32_t)pq};
            const Wait min_term[4] = {w2_full, s_full, {bar(MP::D2_EMPTY), pw ^ 1u}, s_full};
            if (!mbar_wait_warp(min_term, abort_flag, p.err, p.spin_limit, E_MMA)) return false;
            tc_fence_after();
            if (leader) {
              tc_mma_ss(tmem_base + TM_D2, umma_desc32(smem_u32(smem + MP::OFF_W2 + b * 4096)), umma_desc32(smem_u32(smem + MP::OFF_MIN + sq * 4096)), idesc, 0);
              if (!wide) tc_commit(bar(MP::W2_EMPTY + b));
              tc_commit(bar(MP::S_EMPTY + sq));
              tc_commit(bar(MP::D_FULL + d));
            }
            __syncwarp();
            if (++sq == NM) { sq = 0; pq ^= 1; }
            next_d();
            if (wide) {
              // the hi images once more, whose wide rows are whole numbers (their lo images are zeros): block by block, each into an accumulator of its own
#pragma unroll 1
              for (int blk = 0; blk < 8; ++blk) {
                if (!wait(MP::D_EMPTY + d, pd)) return false;
                tc_fence_after();
                if (leader) {
                  const uint32_t a = a_base(blk < 4 ? hi0.u : hi1.u) + (blk >> 1 & 1) * half, to = tmem_base + (uint32_t)(TM_D + d * BT);
                  mma(to, blk >> 1, 2 * (blk & 1), a, 0u);
                  mma(to, blk >> 1, 2 * (blk & 1) + 1, a, 1u);
                  tc_commit(bar(MP::D_FULL + d));
                }
                __syncwarp();
                next_d();
              }
              if (leader) {
#pragma unroll
                for (int c = 0; c < 4; ++c) tc_commit(bar(MP::W_EMPTY + c));
                tc_commit(bar(MP::A_EMPTY + hi0.u));
                tc_commit(bar(MP::A_EMPTY + hi1.u));
              }
              __syncwarp();
              // (the combine warps read the weights' side of the min term: it is free when they are done with the last block's accumulator)
              const int e = d + 1 < ND ? d + 1 : 0;
              if (!wait(MP::D_EMPTY + e, e ? pd : pd ^ 1)) return false;
              mbar_arrive_if(bar(MP::W2_EMPTY + b), lane == 0);
            }
            for (int i = 0; i < at + 3; ++i) next();
            return true;
          };
          using Yes = std::true_type;
          using No = std::false_type;
          for (int s = it.s0; s < it.s1 && ok; ++s, ++sbc) {
            const Wait first[4] = {unit(place(0)), {bar(MP::W_FULL), (uint32_t)(sbc & 1)}, {bar(MP::W_FULL + 1), (uint32_t)(sbc & 1)}, {bar(MP::D_EMPTY + d), (uint32_t)pd}};
            ok = mbar_wait_warp(first, abort_flag, p.err, p.spin_limit, E_MMA);
            if (!ok) break;
            const uint32_t more = __shfl_sync(0xFFFFFFFFu, unit_kinds[sbc & 3], 0);
            ok = more == 0 ? superblock(No{}, No{}) : more == kSpread ? superblock(Yes{}, No{}) : more == kWide ? superblock(No{}, Yes{}) : superblock(Yes{}, Yes{});
          }
          continue;
        }
        for (int s = it.s0; s < it.s1 && ok; ++s, ++sbc) {
          const uint32_t pw = sbc & 1;
          // a superblock: the lo images (two units of two stages), then the hi images, all into one accumulator; the min term into its own
          const uint32_t dt = tmem_base + (uint32_t)(TM_D + d * BT);
#pragma unroll 1
          for (int h = 0; h < 2; ++h) {
            const Wait need[4] = {{bar(MP::A_FULL + sa), (uint32_t)pa}, {bar(MP::W_FULL + 2 * h), pw}, {bar(MP::W_FULL + 2 * h + 1), pw}, {bar(MP::D_EMPTY + d), (uint32_t)pd}};
            if (!mbar_wait_warp(need, abort_flag, p.err, p.spin_limit, E_MMA)) { ok = false; break; }
            tc_fence_after();
            if (leader) {
#pragma unroll
              for (int e = 0; e < 8; ++e) mma(dt, 2 * h + (e >> 2), e & 3, a_base(sa) + (e >> 2) * half, h + e ? 1u : 0u);
              tc_commit(bar(MP::A_EMPTY + sa));
            }
            __syncwarp();
            next();
          }
          if (!ok) break;
#pragma unroll 1
          for (int h = 0; h < 2; ++h) {
            if (!mbar_wait_warp(bar(MP::A_FULL + sa), pa, abort_flag, p.err, p.spin_limit, E_MMA)) { ok = false; break; }
            tc_fence_after();
            if (leader) {
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                mma(dt, 2 * h + (e >> 2), e & 3, a_base(sa) + (e >> 2) * half, 1u);
                if ((e & 3) == 3) tc_commit(bar(MP::W_EMPTY + 2 * h + (e >> 2)));
              }
              tc_commit(bar(MP::A_EMPTY + sa));
            }
            __syncwarp();
            next();
          }
          if (!ok) break;
          const int b = sbc & 1;
          const Wait s_full{bar(MP::S_FULL + sq), (uint32_t)pq};
          const Wait need[4] = {{bar(MP::W2_FULL + b), (uint32_t)(sbc >> 1) & 1u}, s_full, {bar(MP::D2_EMPTY), pw ^ 1u}, s_full};
          if (!mbar_wait_warp(need, abort_flag, p.err, p.spin_limit, E_MMA)) { ok = false; break; }
          tc_fence_after();
          if (leader) {
            tc_mma_ss(tmem_base + TM_D2, umma_desc32(smem_u32(smem + MP::OFF_W2 + b * 4096)), umma_desc32(smem_u32(smem + MP::OFF_MIN + sq * 4096)), idesc, 0);
            tc_commit(bar(MP::W2_EMPTY + b));
            tc_commit(bar(MP::S_EMPTY + sq));
            tc_commit(bar(MP::D_FULL + d));
          }
          __syncwarp();
          if (++sq == NM) { sq = 0; pq ^= 1; }
          if (++d == ND) { d = 0; pd ^= 1; }
        }
      }
    }
  } else if (warp < 8) {
    // ================= dequantisers: TMEM lane t <-> weight row n0 + t
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsDeq));
    const int grp = warp >> 2, t = threadIdx.x & 127;
    const uint32_t t_lane = tmem_base + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)TM_W;
    bool ok = true;
    int rb = 0, pr = 0, sbc = 0;
    for (int w = blockIdx.x; w < n_work && ok; w += gridDim.x) {
      const Item it = item(w);
      for (int s = it.s0; s < it.s1; ++s, ++sbc) {
        if (!mbar_wait_warp(bar(MP::RAW_FULL + rb), pr, abort_flag, p.err, p.spin_limit, E_DEQ)) { ok = false; break; }
        const unsigned char* rrow = smem + MP::OFF_RAW + rb * RAW + t * SBB;
        typename DeqOf<F>::type dq;
        dq.load(rrow);
        if (grp == 0) dq.put_scales(smem + MP::OFF_SCL + (sbc & 3) * MP::SCL, t);
#pragma unroll 1  // (rolled on purpose: with the role loops resident at once, code size costs more than the loop)
        for (int c = grp; c < 4; c += 2) {
          dq.load_stage(c, rrow);
          uint32_t o[16];
          dq.template half<0>(c, o);
          if (!mbar_wait_warp(bar(MP::W_EMPTY + c), (sbc & 1) ^ 1, abort_flag, p.err, p.spin_limit, E_DEQ)) { ok = false; break; }
          tc_fence_after();
          tc_st16(t_lane + (uint32_t)(c * 32), o);
          dq.template half<1>(c, o);
          tc_st16(t_lane + (uint32_t)(c * 32 + 16), o);
          tc_wait_st();
          tc_fence_before();
          mbar_arrive(bar(MP::W_FULL + c));  // (every thread after its own stores)
        }
        if (!ok) break;
        if (grp == 1) {  // the weights' side of the min term: mn of the eight blocks, against the hi and against the lo factors
          uint32_t u[4];
          dq.mins(u);
          if (!mbar_wait_warp(bar(MP::W2_EMPTY + (sbc & 1)), ((sbc >> 1) & 1) ^ 1, abort_flag, p.err, p.spin_limit, E_DEQ)) { ok = false; break; }
          uint4* o = reinterpret_cast<uint4*>(smem + MP::OFF_W2 + (sbc & 1) * 4096 + t * 32);
          o[0] = o[1] = make_uint4(u[0], u[1], u[2], u[3]);  // (both chunks alike: the swizzle moves nothing)
          fence_proxy_async();
          mbar_arrive(bar(MP::W2_FULL + (sbc & 1)));
        }
        mbar_arrive(bar(MP::RAW_EMPTY + rb));
        if (++rb == NR) { rb = 0; pr ^= 1; }
      }
    }
  } else {
    // ================= combine: a warp holds 32 weight rows (TMEM lanes 32 * (warp % 4) ..) x one or two groups of 32 tokens as fragments (tc_ld_frag2).
    // All f32 arithmetic is done on register pairs (fma.rn.f32x2): half the instructions for the same IEEE results.
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsComb));
    pdl_wait();  // (C belongs to kernels before this one until they are done)
    const int q = warp & 3, grp = (warp - 8) >> 2;
    const int row0 = 32 * q + (lane >> 2), cl = 2 * (lane & 3);  // this thread's rows row0 + 8 k, k < 4; tokens column(i) + 8 g + cl, + 1
    const uint32_t t_lane = tmem_base + ((uint32_t)(32 * q) << 16);
    auto column = [&](int i) -> int { return 32 * (grp + 2 * i); };
    bool ok = true;
    int d = 0, pd = 0, sq = 0, pq = 0, sbc = 0, n_item = 0;
    for (int w = blockIdx.x; w < n_work && ok; w += gridDim.x, ++n_item) {
      __syncwarp();
      const Item it = item(w);
      unsigned long long res[NCH][2][8];  // [group][rows 16 hr ..][2 g + r]: row 16 hr + 8 r, token pair 8 g
#pragma unroll
      for (int i = 0; i < NCH; ++i)
#pragma unroll
        for (int j = 0; j < 16; ++j) res[i][j >> 3][j & 7] = 0ull;
      if (!mbar_wait_warp(bar(MP::S_FULL + sq), pq, abort_flag, p.err, p.spin_limit, E_EPI)) break;
      int s = it.s0;
      if (__shfl_sync(0xFFFFFFFFu, s_item[n_item & 3], 0)) {
        // with rows that are not plain
        auto wait = [&](int b, int parity) -> bool { return mbar_wait_warp(bar(b), (uint32_t)parity, abort_flag, p.err, p.spin_limit, E_EPI); };
        auto done = [&]() {  // with an accumulator
          tc_fence_before();
          __syncwarp();
          mbar_arrive_if(bar(MP::D_EMPTY + d), lane == 0);
          if (++d == ND) { d = 0; pd ^= 1; }
        };
        for (; s < it.s1 && ok; ++s, ++sbc) {
          ok = false;  // (until the superblock is through)
          if (!wait(MP::S_FULL + sq, pq)) break;
          const uint32_t more = __shfl_sync(0xFFFFFFFFu, s_kinds[sq], 0);
          const unsigned char* scl = smem + MP::OFF_SCL + (sbc & 3) * MP::SCL;
          const float* sv = reinterpret_cast<const float*>(smem + MP::OFF_S + sq * 512) + cl;
          if (!wait(MP::D_FULL + d, pd)) break;
          tc_fence_after();
          unsigned long long d2[4], nd2[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            d2[k] = pack2(reinterpret_cast<const float*>(scl)[row0 + 8 * k]);
            nd2[k] = pack2(reinterpret_cast<const float*>(scl)[128 + row0 + 8 * k]);
          }
          if (more & kSpread) {  // the third term; what comes of rows without one may be anything (their image is what was there) and is not taken
#pragma unroll
            for (int i = 0; i < NCH; ++i) {
              const int col = column(i);
              if (col >= it.n) break;
              unsigned long long v[8], x[8];
              const uint32_t at = t_lane + (uint32_t)(col + TM_D + d * BT);
              tc_ld_frag2(at, at + (16u << 16), v, x);
#pragma unroll
              for (int g = 0; g < 4; ++g) {
                const unsigned long long ss = *reinterpret_cast<const unsigned long long*>(sv + col + 8 * g);
                const unsigned long long t2 = ss ^ 0x8000000080000000ull;
                const float s0 = lo_f(ss), s1 = hi_f(ss);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                  const unsigned long long y = (k >> 1 ? x : v)[2 * g + (k & 1)];
                  ffma2(res[i][k >> 1][2 * g + (k & 1)], t2, fmul2(d2[k], pair(s0 < 0.0f ? lo_f(y) : 0.0f, s1 < 0.0f ? hi_f(y) : 0.0f)));
                }
              }
            }
            done();
            if (!wait(MP::D_FULL + d, pd)) break;
            tc_fence_after();
          }
#pragma unroll
          for (int i = 0; i < NCH; ++i) {  // the first two terms, as for plain rows (s of wide ones is 0)
            const int col = column(i);
            if (col >= it.n) break;
            unsigned long long ss[4];
#pragma unroll
            for (int g = 0; g < 4; ++g) ss[g] = *reinterpret_cast<const unsigned long long*>(sv + col + 8 * g) & 0x7FFFFFFF7FFFFFFFull;
#pragma unroll
            for (int hr = 0; hr < 2; ++hr) {
              unsigned long long v[8], x[8];
              const uint32_t at = t_lane + ((uint32_t)(16 * hr) << 16) + (uint32_t)col;
              tc_ld_frag2(at + (uint32_t)(TM_D + d * BT), at + (uint32_t)TM_D2, v, x);
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                unsigned long long a = fmul2(d2[2 * hr + (j & 1)], v[j]);
                ffma2(a, nd2[2 * hr + (j & 1)], x[j]);
                ffma2(res[i][hr][j], ss[j >> 1], a);
              }
            }
          }
          done();
          mbar_arrive_if(bar(MP::D2_EMPTY), lane == 0);
          if (more & kWide) {
            // Wide rows, block by block: the sums are whole numbers, the scales come from memory, the min term is taken on the CUDA cores.  A lane holds the
            // factors of one row per group, and every lane takes those of its tokens from there.
            if (!wait(MP::W2_FULL + (sbc & 1), sbc >> 1 & 1)) break;
            const unsigned char* mnp = smem + MP::OFF_W2 + (sbc & 1) * 4096 + row0 * 32;
            const unsigned char* kp = p.tail + ((size_t)it.tile * nsb + s) * kTailRow * p.tt + kTailCopy * p.tt;
            bool mine[NCH], any[NCH];
            float tr[NCH], ar[NCH];
#pragma unroll
            for (int i = 0; i < NCH; ++i) {
              const int row = column(i) + lane;
              mine[i] = row < it.n && __ldcg(kp + row) == kWide;
              any[i] = __any_sync(0xFFFFFFFFu, mine[i]);
            }
            auto fetch = [&](int b) {
#pragma unroll
              for (int i = 0; i < NCH; ++i) {
                const int row = column(i) + lane;
                tr[i] = ar[i] = 0.0f;
                if (mine[i]) {
                  tr[i] = __ldcg(p.asc + (size_t)(8 * s + b) * p.lda + it.r0 + row);
                  const unsigned char* vr = smem + MP::OFF_MIN + sq * 4096 + row * 32 + 2 * b;
                  const int sw = (row >> 2 & 1) << 4;
                  ar[i] = __fadd_rn(__half2float(*reinterpret_cast<const __half*>(vr + sw)), __half2float(*reinterpret_cast<const __half*>(vr + (sw ^ 16))));
                }
              }
            };
            fetch(0);
            int b = 0;
#pragma unroll 1
            for (; b < 8; ++b) {
              const float t_now[NCH] = {tr[0], tr[1]}, a_now[NCH] = {ar[0], ar[1]};
              if (b < 7) fetch(b + 1);
              if (!wait(MP::D_FULL + d, pd)) break;
              tc_fence_after();
              unsigned long long mn[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) mn[k] = fmul2(nd2[k], pack2(__half2float(*reinterpret_cast<const __half*>(mnp + 256 * k + 2 * b))));
#pragma unroll
              for (int i = 0; i < NCH; ++i) {
                if (!any[i]) continue;
                unsigned long long v[8], x[8];
                const uint32_t at = t_lane + (uint32_t)(column(i) + TM_D + d * BT);
                tc_ld_frag2(at, at + (16u << 16), v, x);
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                  const int row = 8 * g + cl;
                  const unsigned long long t2 = pair(__shfl_sync(0xFFFFFFFFu, t_now[i], row), __shfl_sync(0xFFFFFFFFu, t_now[i], row + 1));
                  const unsigned long long a2 = pair(__shfl_sync(0xFFFFFFFFu, a_now[i], row), __shfl_sync(0xFFFFFFFFu, a_now[i], row + 1));
#pragma unroll
                  for (int k = 0; k < 4; ++k) {
                    unsigned long long y = fmul2(d2[k], (k >> 1 ? x : v)[2 * g + (k & 1)]);
                    ffma2(y, mn[k], a2);
                    ffma2(res[i][k >> 1][2 * g + (k & 1)], t2, y);
                  }
                }
              }
              done();
            }
            if (b < 8) break;
          }
          mbar_arrive(bar(MP::S_EMPTY + sq));
          if (++sq == NM) { sq = 0; pq ^= 1; }
          ok = true;
        }
      }
      for (; s < it.s1 && ok; ++s, ++sbc) {
        if (!mbar_wait_warp(bar(MP::S_FULL + sq), pq, abort_flag, p.err, p.spin_limit, E_EPI)) { ok = false; break; }
        const unsigned char* scl = smem + MP::OFF_SCL + (sbc & 3) * MP::SCL;
        const float* sv = reinterpret_cast<const float*>(smem + MP::OFF_S + sq * 512) + cl;
        if (!mbar_wait_warp(bar(MP::D_FULL + d), pd, abort_flag, p.err, p.spin_limit, E_EPI)) { ok = false; break; }
        tc_fence_after();
        unsigned long long d2[4], nd2[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          d2[k] = pack2(reinterpret_cast<const float*>(scl)[row0 + 8 * k]);
          nd2[k] = pack2(reinterpret_cast<const float*>(scl)[128 + row0 + 8 * k]);
        }
#pragma unroll
        for (int i = 0; i < NCH; ++i) {
          const int col = column(i);
          if (col >= it.n) break;
          unsigned long long ss[4];
#pragma unroll
          for (int g = 0; g < 4; ++g) ss[g] = *reinterpret_cast<const unsigned long long*>(sv + col + 8 * g);
#pragma unroll
          for (int hr = 0; hr < 2; ++hr) {
            unsigned long long v[8], x[8];
            const uint32_t at = t_lane + ((uint32_t)(16 * hr) << 16) + (uint32_t)col;
            tc_ld_frag2(at + (uint32_t)(TM_D + d * BT), at + (uint32_t)TM_D2, v, x);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              unsigned long long a = fmul2(d2[2 * hr + (j & 1)], v[j]);
              ffma2(a, nd2[2 * hr + (j & 1)], x[j]);
              ffma2(res[i][hr][j], ss[j >> 1], a);
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        mbar_arrive_if(bar(MP::D_EMPTY + d), lane == 0);  // the accumulators may be overwritten
        mbar_arrive_if(bar(MP::D2_EMPTY), lane == 0);
        if (++d == ND) { d = 0; pd ^= 1; }
        mbar_arrive(bar(MP::S_EMPTY + sq));
        if (++sq == NM) { sq = 0; pq ^= 1; }
      }
      if (!ok || *abort_flag) continue;
      // ---- the item's outputs: a store of the warp is eight neighbouring columns of C (a 32-byte sector) for four tokens
      const int n0 = it.nt * BN + row0;
      float* cp = p.n_split > 1 ? p.part + ((size_t)it.ks * p.M + it.r0 + cl) * p.N + n0 : p.C + (size_t)(it.r0 + cl) * p.ldc + p.c_off + n0;
      const size_t ld = p.n_split > 1 ? (size_t)p.N : (size_t)p.ldc;
#pragma unroll
      for (int i = 0; i < NCH; ++i)
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int c = column(i) + 8 * ((j >> 1) & 3), n = 16 * (j >> 3) + 8 * (j & 1);  // (then + cl, + n0)
          float* o = cp + (size_t)c * ld + n;
          if (n0 + n < p.N && c + cl < it.nr) o[0] = lo_f(res[i][j >> 3][j & 7]);
          if (n0 + n < p.N && c + cl + 1 < it.nr) o[ld] = hi_f(res[i][j >> 3][j & 7]);
        }
    }
  }
  // ---- teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // a wait gave up: let copies and MMAs still in flight land before shared memory and TMEM are released
    pdl_wait();  // (the pre-pass clears the flag)
    if (p.n_split > 1 && threadIdx.x == 0) atomicOr(p.part_bad, 1u);
    for (int i = 0; i < 64; ++i) __nanosleep(20000);
    __syncthreads();
  }
  if (warp == 16) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
  }
}

template <class F>
int launch(const izb_weight* w, const FoldParams& p, int grid, cudaStream_t st) {
  constexpr int SMEM_BYTES = Map<F>::SMEM_BYTES;
  static izb_device_once once;
  if (int rc = once.run(w->device, [&]() -> int {
        cudaFuncAttributes fa;
        IZB_CUDA(cudaFuncGetAttributes(&fa, gemm_fold_kernel<F>));
        if (fa.numRegs * kThreads < kRoleRegs) IZB_FAIL(IZB_ERR_SELFCHECK, "gemm: built with %d registers for each of %d threads, the roles share %d", fa.numRegs, kThreads, kRoleRegs);
        IZB_CUDA(cudaFuncSetAttribute(gemm_fold_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        return IZB_OK;
      }))
    return rc;
  CUtensorMap tm;
  memcpy(&tm, w->tmap_raw, sizeof tm);
  if (p.pdl)
    IZB_LAUNCH("gemm_fold", st, izb_launch_pdl(gemm_fold_kernel<F>, dim3(grid), dim3(kThreads), SMEM_BYTES, st, tm, p));
  else
    IZB_LAUNCH("gemm_fold", st, gemm_fold_kernel<F><<<grid, kThreads, SMEM_BYTES, st>>>(tm, p));
  return IZB_OK;
}

}  // namespace

// The cut of M whose rounds of tiles over the SMs cost least.  A tile's time follows its rows while its MMAs set the pace, and stops following
// them below 64 rows, where the dequantisers do; every tile has a fill and a drain.  (The rows' results do not depend on it while K is not cut; the number of
// tiles has a part in how it is.)
int izb_fold_tile_rows(int device, int M, int N) {
  const int sms = izb_sm_count(device), n_ntiles = (N + BN - 1) / BN;
  int best = BT;
  long long best_cost = -1;
  for (int n_tt = (M + BT - 1) / BT, i = 0; i < 8; ++i, ++n_tt) {
    const int tt = ((M + n_tt - 1) / n_tt + 15) & ~15;
    const long long rounds = ((long long)((M + tt - 1) / tt) * n_ntiles + sms - 1) / sms;
    const long long cost = rounds * ((tt < 64 ? 64 : tt) + 4);
    if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = tt; }
    if (tt == 16) break;
  }
  return best;
}

size_t izb_fold_img_bytes(int rows, int K) { return (size_t)rows * (K / 256) * kImgRow; }
size_t izb_fold_fine_bytes(int rows, int K) { return (size_t)rows * (K / 256) * kFineRow; }
size_t izb_fold_tail_bytes(int rows, int K) { return ((size_t)rows * (K / 256) * kTailRow + 255) & ~(size_t)255; }

int izb_fold_prepare(const izb_weight* w, const int8_t* aq, const float* asc, int lda, int rows, const FoldParams& p, cudaStream_t st) {
  const int n_rows = p.n_mtiles * p.tt;
  dim3 grid((n_rows + 31) / 32, w->K / 256);
  auto kernel = w->type == IZB_Q4_K ? fold_prepare_kernel<true> : fold_prepare_kernel<false>;
  IZB_LAUNCH("act_prepare", st, izb_launch_pdl(kernel, grid, 256, 0, st, aq, asc, lda, w->K, rows, p.img, p.fine, p.tail, p.tt, n_rows, p.part_bad));
  return IZB_OK;
}

int izb_fold_quant_prepare(const izb_weight* w, const float* x, int ldx, int M, int Mp, int8_t* aq, float* asc, const FoldParams& p, cudaStream_t st) {
  const int rows = p.n_mtiles * p.tt;  // (every row of every tile is written, rows past M as zeros)
  const int all = rows > Mp ? rows : Mp;
  const bool one = izb_one_row_per_warp(all, w->K);
  dim3 grid(w->K / 256, one ? (all + 7) / 8 : (all + 31) / 32);
  auto kernel = w->type == IZB_Q4_K ? (one ? fold_quant_prepare_kernel<true, 1> : fold_quant_prepare_kernel<true, 4>)
                                    : one ? fold_quant_prepare_kernel<false, 1> : fold_quant_prepare_kernel<false, 4>;
  IZB_LAUNCH("quant_prepare", st, izb_launch_pdl(kernel, grid, 256, 0, st, x, ldx, M, Mp, w->K, aq, asc, p.img, p.fine, p.tail, p.tt, p.n_mtiles, p.part_bad));
  return IZB_OK;
}

int izb_fold_gemm(const izb_weight* w, const FoldParams& p, int grid, cudaStream_t st) {
  return w->type == IZB_Q4_K ? launch<FQ4K>(w, p, grid, st) : launch<FQ5K>(w, p, grid, st);
}
