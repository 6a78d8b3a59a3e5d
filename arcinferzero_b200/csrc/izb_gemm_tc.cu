// Prefill GEMM on the 5th-generation tensor cores (tcgen05, TMEM accumulators), exact per-32-block semantics; the host side of this kernel and of
// the folded one (csrc/izb_gemm_fold.cu), which takes plain stores of Q4_K and Q5_K products of long K under IZB_GEMM_AUTO.
//
// Problem: C[m][n] = sum over 32-blocks b of asc[m][b] * wscale[n][b] * dot_b[m][n]  (- the Q4_K min term), where dot_b
// is an exact integer.  Both operands carry a scale per block, so a block's dot product must leave the tensor core
// before the next one is added: the f32 combine on the CUDA cores (M*N*K/32 fused multiply-adds), not the MMA, bounds
// the kernel.  The design therefore minimises CUDA-core work per (m, n, block) to ONE fma:
//   * operands are fed as fp16 holding exact integers: activations a in [-127,127]; Q4_K weights as sc*q in [0,945]
//     (the 6-bit sub-block scale folded in, exactly representable), Q8_0 weights q in [-128,127].  tcgen05.mma
//     kind::f16 then leaves (float)(sc*dot) in TMEM: every product and every partial sum is an integer below 2^24,
//     so the f32 accumulator holds it exactly (the verification mode reads these accumulators back and the tests
//     compare them bit for bit with the CPU's int32 dots).  A kind::i8 accumulator would need an int->float
//     conversion and a second multiply per element, which costs more than the slower fp16 MMA rate saves.
//   * Q4_K:  tq += asc[m][b] * D_b   per block;   res = fma(d[n], tq, res)   per superblock.
//     The min term  - sum_b (asc*asum)[m][b] * (dmin*mn)[n][b]  never touches the CUDA cores: it is one more GEMM on the
//     tensor cores, accumulated over the whole of K in a fourth TMEM accumulator and read once per tile.  Both factors
//     are f32 numbers, fed as bf16 triples (v = v1+v2+v3, u = u1+u2+u3, the six products that matter: v1u1, v1u2, v2u1,
//     v1u3, v2u2, v3u1; u = -dmin*mn has 17 significant bits, so its split is exact, v is exact to 2^-24).  Those 48
//     K-entries per superblock travel as a fifth "stage" through the same operand ring as the four fp16 stages.
//   * Q8_0:  res += (asc[m][b] * d[n][b]) * D_b.
//
// CTA = one 128 (tokens, TMEM lanes) x 128 (weight rows, TMEM columns) output tile, 16 warps:
//   warp 0      activation producer: cp.async.bulk of pre-swizzled operand tiles (made by act_prepare_kernel) into the
//               operand ring;
//   warp 3      weight producer: TMA (cp.async.bulk.tensor.2d) of the raw GGUF superblocks of 128 rows into a ring, and
//               the tile's activation scales;
//   warps 4-7   dequantisers: one thread per weight row, nibbles -> fp16 sc*q written in the 128-byte-swizzled K-major
//               operand layout, the min-term operand, block scales to shared memory;
//   warps 1-2   issue tcgen05.mma (one thread each, alternating stages) into a ring of three 128-column accumulators +
//               the min-term accumulator (always warp 2, so that one thread orders all updates of it);
//   warps 8-15  combine: tcgen05.ld of 16 rows x 64 columns at a time, one fma per element, final store with the reference's
//               store modes.
// The combine warps read accumulators as fragments: a thread meets 4 token rows x 8 column pairs, not 1 x 64 columns.  With a lane per row the
// column scales (Q8_0: 64 per block) were 16-byte reads of one address by the whole warp, four passes each: the shared-memory pipe stood at 86 %
// of its peak for Q8_0.  Together with role branches the compiler knows to be warp-uniform, and SwiGLU products two at a time (us, before and
// now): 300 x 5120 x 17408 Q6_K 235 / 216, 512 x 4096 x 4096 Q8_0 67.6 / 64.9, feed-forward block of 1000 x 5120 x 17408 Q4_K 1387 / 1297, of
// 94 x 2048 x 7168 123 / 111, 4096 tokens x 8 of 128 experts 1163 / 1148.  Tried: sixteen combine warps of 16 rows x 64 columns and two groups of
// dequantisers (28 warps, 72 registers at launch): Q8_0 62, but the feed-forward block 1482 and the experts 1200.
// All waits are bounded: a wait that gives up sets a CTA-wide abort flag and a device error word, the CTA drains and
// returns without storing (izb_device_status reports it).
#include <cuda.h>
#include <cuda_bf16.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <exception>
#include <mutex>
#include <vector>

#include "izb_fold.cuh"

void izb_set_tc_ok(int device, int ok);
void izb_note_noalloc_status(int device, uint32_t* status);
int izb_get_tc_ok(int device);
int izb_gemm_core_launch(const izb_weight* w, const uint8_t* raw, const int8_t* aq, const float* asc, int M, int Mp, float* C,
                         int ldc, int c_off, int acc, int32_t* dots, cudaStream_t st);

namespace {

constexpr int BM = 128, BN = 128, KS = 64;
constexpr int ND1 = 3;                    // accumulators of a 32-block in the ring
constexpr int STAGE_BYTES = BM * KS * 2;  // 16 KB: 128 rows x 128 B
constexpr int kThreads = 512;
constexpr uint32_t kSpinLimit = 1u << 24;
constexpr int NASC = 3;

// ---- what differs between the weight forms
//   kMin    superblock mins (Q4_K, Q5_K): a fifth operand stage per superblock carries the min term
//   kTerms  fp16 terms of scale * quant: one where the product fits 11 bits (Q4_K 63 * 15, Q5_K 63 * 31, Q8_0's plain quant);
//           two where it reaches 4096 (Q6_K, IQ4_XS): scale * quant = hi + lo with hi even and lo in {0, 1}, both exact
//   kColScale  a scale per block and weight row applied in the combine (Q8_0) instead of one per superblock
struct FQ4K { static constexpr int SBB = 144, kTerms = 1, NA = 6, NB = 4, NR = 2; static constexpr bool kMin = true, kColScale = false; };
struct FQ80 { static constexpr int SBB = 272, kTerms = 1, NA = 4, NB = 4, NR = 2; static constexpr bool kMin = false, kColScale = true; };
struct FQ5K { static constexpr int SBB = kK16SbBytes, kTerms = 1, NA = 4, NB = 4, NR = 2; static constexpr bool kMin = true, kColScale = false; };
struct FQ6K { static constexpr int SBB = kQ6pSbBytes, kTerms = 2, NA = 3, NB = 3, NR = 2; static constexpr bool kMin = false, kColScale = false; };
struct FIQ4 { static constexpr int SBB = kK16SbBytes, kTerms = 2, NA = 3, NB = 3, NR = 1; static constexpr bool kMin = false, kColScale = false; };

// shared memory map (bytes from a 1024-aligned base).  The two operands of a stage travel through rings of their own: an
// activation image is a bulk copy from L2 whose latency (not its bandwidth) is what has to be covered, so its ring is as
// deep as shared memory allows; a weight tile is written by the dequantiser warps from a raw tile already in shared memory.
template <class F>
struct Map {
  static constexpr int NA = F::NA, NB = F::NB, NR = F::NR, RAW = BN * F::SBB;
  static constexpr int BSTAGE = STAGE_BYTES * F::kTerms;
  static constexpr int OFF_A = 0;
  static constexpr int OFF_B = OFF_A + NA * STAGE_BYTES;
  static constexpr int OFF_RAW = OFF_B + NB * BSTAGE;
  static constexpr int OFF_SCL = OFF_RAW + NR * RAW;                          // 4 x [128] f32 superblock scales d; Q8_0: 4 x [8][128] f32 block scales
  static constexpr int OFF_ASC = OFF_SCL + (F::kColScale ? 4 * 4096 : 4 * 512);  // NASC x [8 blocks][128 rows] f32 activation scales
  static constexpr int OFF_BAR = OFF_ASC + NASC * 4096;
  static constexpr int SMEM_BYTES = OFF_BAR + 1024 + 1024;                    // barriers + alignment slack
  // 8-byte mbarriers
  static constexpr int A_FULL = 0, A_EMPTY = A_FULL + NA, B_FULL = A_EMPTY + NA, B_EMPTY = B_FULL + NB, RAW_FULL = B_EMPTY + NB,
                       RAW_EMPTY = RAW_FULL + NR, D1_FULL = RAW_EMPTY + NR, D1_EMPTY = D1_FULL + ND1, D2_FULL = D1_EMPTY + ND1,
                       D2_EMPTY = D2_FULL + 1, ASC_FULL = D2_EMPTY + 1, ASC_EMPTY = ASC_FULL + NASC, NUM_BARS = ASC_EMPTY + NASC;
  static_assert(SMEM_BYTES <= 232448, "shared memory per CTA");
  static_assert(NUM_BARS * 8 + 16 <= 1024, "barrier area");
  static_assert(OFF_RAW % 1024 == 0 && OFF_SCL % 16 == 0 && RAW % 128 == 0, "alignment of the TMA destinations");
};

// error-word codes (which wait gave up)
enum : uint32_t { E_APROD = 1, E_WPROD = 2, E_DEQ = 4, E_MMA = 16, E_EPI = 32 };

struct TcParams {
  const uint16_t* aimg;   // [tiles][stages][128][64] 16-bit operand tiles, rows 128-byte swizzled; stages = K/64, and
                          // for weights with mins one bf16 min-term tile after every four (5 per superblock)
  const float* ascimg;    // [tiles][K/32][128] f32: the tile rows' activation scales, gathered
  const int32_t* tiles;   // grouped: [1 + 3*max_tiles]; dense: null
  const float* rowscale;  // per output row factor or null
  int M;                  // dense: rows to store
  int n_mtiles;           // dense: row tiles (grouped: tiles[0], read on the device)
  int N, K;               // per matrix
  int mat;                // dense: matrix of the stack
  int n_split;            // parts the K range of every tile is cut into (dense only)
  float* part;            // n_split > 1: [n_split][M][N] partial sums, stored instead of C
  uint32_t* part_bad;     // n_split > 1: set when a wait gave up (split_reduce_kernel then stores nothing)
  float* C;
  int ldc, c_off, acc;
  int32_t* dots;          // verification mode output or null
  uint32_t* err;
  uint32_t spin_limit;    // polls after which a wait gives up
  int skip_stage;         // diagnostics: the operand stage the activation producer leaves out (-1: none)
  int pdl;                // programmatic dependent launch (tc_pdl)
};

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
// Bounded wait of one thread.  false = gave up (or another thread did): the caller leaves its loop.  The lanes of a warp may get different
// answers when the limit runs out: for roles whose threads work by themselves.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag, uint32_t* err,
                                          uint32_t limit, uint32_t code) {
  // (a satisfied wait is the common case: one non-blocking look costs less than the blocking form)
  if (mbar_test(bar, parity)) return true;
  for (uint32_t it = 0; it < limit; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 255u) == 255u && *abort_flag) return false;
  }
  *abort_flag = 1;
  atomicOr(err, code);
  return false;
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
// MMA and commit are issued by a whole converged warp with one elected lane's predicate inside the statement: the operands
// then stay in uniform registers.  Behind a lane test they are moved there one by one for every instruction, which
// measured 98 clk per MMA and per commit; in this form four MMAs and three commits take 168.
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_mma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\telect.sync _|e, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// tcgen05.ld of 16 TMEM lanes x 64 columns + wait as matrix fragments: register pair 2g + r holds lane 8 r + threadlane / 4, columns
// 8 g + 2 (threadlane % 4) and the one after
__device__ __forceinline__ void tc_ld_frag64(uint32_t taddr, unsigned long long (&r)[16]) {
  asm volatile(
      "{\n\t.reg .b32 t<32>;\n\t"
      "tcgen05.ld.sync.aligned.16x256b.x8.b32 {t0,t1,t2,t3,t4,t5,t6,t7,t8,t9,t10,t11,t12,t13,t14,t15,t16,t17,t18,t19,t20,t21,t22,t23,t24,t25,t26,t27,t28,t29,t30,t31}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;\n\t"
      "mov.b64 %0, {t0,t1};\n\t"
      "mov.b64 %1, {t2,t3};\n\t"
      "mov.b64 %2, {t4,t5};\n\t"
      "mov.b64 %3, {t6,t7};\n\t"
      "mov.b64 %4, {t8,t9};\n\t"
      "mov.b64 %5, {t10,t11};\n\t"
      "mov.b64 %6, {t12,t13};\n\t"
      "mov.b64 %7, {t14,t15};\n\t"
      "mov.b64 %8, {t16,t17};\n\t"
      "mov.b64 %9, {t18,t19};\n\t"
      "mov.b64 %10, {t20,t21};\n\t"
      "mov.b64 %11, {t22,t23};\n\t"
      "mov.b64 %12, {t24,t25};\n\t"
      "mov.b64 %13, {t26,t27};\n\t"
      "mov.b64 %14, {t28,t29};\n\t"
      "mov.b64 %15, {t30,t31};\n\t"
      "}"
      : "=l"(r[0]), "=l"(r[1]), "=l"(r[2]), "=l"(r[3]), "=l"(r[4]), "=l"(r[5]), "=l"(r[6]), "=l"(r[7]), "=l"(r[8]), "=l"(r[9]), "=l"(r[10]), "=l"(r[11]), "=l"(r[12]), "=l"(r[13]), "=l"(r[14]), "=l"(r[15])
      : "r"(taddr)
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
// up * silu(gate) (zero/kernels/gemm.cl:562-565).  Two at a time, for their latency; out of line on purpose:
// the epilogues call it 32 and 16 times per thread, and the role loops of the kernel compete for the instruction cache.
__device__ __noinline__ float2 swiglu_mul2(float2 g, float2 u) {
  return make_float2(__fmul_rn(u.x, __fdiv_rn(g.x, __fadd_rn(1.0f, expf(-g.x)))), __fmul_rn(u.y, __fdiv_rn(g.y, __fadd_rn(1.0f, expf(-g.y)))));
}
__device__ __forceinline__ float lo_f(unsigned long long a) { return __uint_as_float((uint32_t)a); }
__device__ __forceinline__ float hi_f(unsigned long long a) { return __uint_as_float((uint32_t)(a >> 32)); }

// K-major operand tile of 128-byte rows, 128-byte swizzle: 8-row groups 1024 bytes apart (tcgen05 shared-memory
// descriptor: start address >> 4, stride byte offset >> 4 at bit 32, descriptor version 1 at bit 46, swizzle mode 2
// (128 B) at bit 61; the leading byte offset is not used when the MMA's K extent lies inside one swizzled row).
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// instruction descriptor, kind::f16: D = f32 (bit 4), A/B format at bits 7 / 10 (0 fp16, 1 bf16), both K-major,
// N >> 3 at bit 17, M >> 4 at bit 24
constexpr uint32_t kIdescF16 = (1u << 4) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
constexpr uint32_t kIdescBF16 = kIdescF16 | (1u << 7) | (1u << 10);

// position p (0..7) inside a 16-byte chunk of the Q4_K operand row holds element perm8[p] of that group of eight:
// the order in which the dequantiser's two-nibbles-per-word extraction delivers them
__device__ __forceinline__ int q4k_perm8(int p) { return (p & 4) | ((p & 1) << 1) | ((p >> 1) & 1); }

// ---------------------------------------------------------------------------------------------- activation pre-pass
// Per 128-row tile: fp16 operand images (one 16 KB swizzled stage per 64 elements of K), the tile's activation scales
// and, with sps == 5 (the Q4_K GEMM), after every four stages one more 16 KB image: the min-term factor
// v = asc * (float)asum of the superblock's eight blocks as three bf16 terms, laid out as the six 16-byte K-chunks
// (v1, v1, v2, v1, v2, v3) x eight blocks that meet the weight side's (u1, u2, u1, u3, u2, u1).
// Bound by its writes, so one CTA = 32 rows x one superblock: the image goes out in whole 128-byte lines, and scales and min terms, whose
// neighbours in memory belong to other rows, are collected in shared memory first.  (One thread per chunk, rows one after the other, wrote
// them as 4- and 2-byte pieces: 32768 gathered rows of K = 2048 took 94 us, now 42.)
struct PrepRows {
  float sc[8][33], v[8][33];  // [block of the superblock][row]: scale, scale * sum
};
// (after a barrier) the scales and, sps == 5, the min-term chunks of the kN rows from row r0 of the tile on
template <int kN>
__device__ __forceinline__ void put_scales(const PrepRows& p, float* __restrict__ ascimg, uint8_t* tile_img, int tile, int K, int sb, int r0, int sps) {
  {
    const int b = threadIdx.x >> 5, r = threadIdx.x & 31;
    if (r < kN) ascimg[((size_t)tile * (K / 32) + sb * 8 + b) * BM + r0 + r] = p.sc[b][r];
  }
  if (sps != 5) return;
  const int r = threadIdx.x >> 3, k = threadIdx.x & 7;
  if (k >= 6 || r >= kN) return;
  const int term = k == 2 || k == 4 ? 1 : k == 5 ? 2 : 0;
  uint32_t o[4];
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const float v = p.v[b][r];
    const __nv_bfloat16 h1 = __float2bfloat16_rn(v);
    const float r1 = __fsub_rn(v, __bfloat162float(h1));
    const __nv_bfloat16 h2 = __float2bfloat16_rn(r1);
    const __nv_bfloat16 h3 = __float2bfloat16_rn(__fsub_rn(r1, __bfloat162float(h2)));
    const uint32_t h = __bfloat16_as_ushort(term == 0 ? h1 : term == 1 ? h2 : h3);
    o[b >> 1] = (b & 1) ? o[b >> 1] | (h << 16) : h;
  }
  *reinterpret_cast<uint4*>(tile_img + ((size_t)sb * 5 + 4) * STAGE_BYTES + (r0 + r) * 128 + ((k ^ (r & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
}
// the operand chunk of eight int8 values: row r of the tile, chunk `c` (0 .. 31) of superblock sb
template <bool kPerm>
__device__ __forceinline__ void put_chunk(uint8_t* tile_img, int sb, int sps, int r, int c, const int (&q)[8]) {
  uint32_t o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int e0 = kPerm ? q4k_perm8(2 * j) : 2 * j, e1 = kPerm ? q4k_perm8(2 * j + 1) : 2 * j + 1;
    const __half2 h = __floats2half2_rn((float)q[e0], (float)q[e1]);
    o[j] = *reinterpret_cast<const uint32_t*>(&h);
  }
  *reinterpret_cast<uint4*>(tile_img + ((size_t)sb * sps + (c >> 3)) * STAGE_BYTES + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
}

template <bool kPerm>
__global__ void __launch_bounds__(256) act_prepare_kernel(const int8_t* __restrict__ aq, const float* __restrict__ asc, int lda,
                                                          int K, int rows_total, const int32_t* __restrict__ tiles,
                                                          const int32_t* __restrict__ rowmap, uint16_t* __restrict__ aimg,
                                                          float* __restrict__ ascimg, int sps,
                                                          uint32_t* __restrict__ part_bad) {
  __shared__ PrepRows s;
  const int sb = blockIdx.y, tile = blockIdx.x >> 2, m0 = (blockIdx.x & 3) * 32, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int r0, nr;
  pdl_launch_next();
  pdl_wait();
  if (part_bad && sb == 0 && blockIdx.x == 0 && threadIdx.x == 0) *part_bad = 0;
  if (tiles) {
    if (tile >= tiles[0]) return;
    r0 = tiles[2 + 3 * tile];
    nr = tiles[3 + 3 * tile];
    if (m0 >= nr) return;  // (rows past the tile's slots reach no result: every accumulator row belongs to one operand row)
  } else {
    r0 = tile * BM;
    nr = min(BM, rows_total - r0);
  }
  // this lane's row of the 32, for the scales; the rows a warp copies come from it by shuffle
  const int src = m0 + lane < nr ? (rowmap ? rowmap[r0 + m0 + lane] : r0 + m0 + lane) : -1;
  if (asc) s.sc[warp][lane] = src >= 0 ? asc[(size_t)(sb * 8 + warp) * lda + src] : 0.0f;  // (null in the block-dot verification mode)
  uint2 x[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int from = __shfl_sync(0xFFFFFFFFu, src, warp + 8 * i);
    x[i] = from >= 0 ? *reinterpret_cast<const uint2*>(aq + (size_t)from * K + sb * 256 + lane * 8) : make_uint2(0, 0);
  }
  __syncthreads();
  uint8_t* tile_img = reinterpret_cast<uint8_t*>(aimg) + (size_t)tile * (K / 256) * sps * STAGE_BYTES;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int rr = warp + 8 * i;
    int a[8];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      a[k] = (int)(int8_t)(x[i].x >> (8 * k));
      a[4 + k] = (int)(int8_t)(x[i].y >> (8 * k));
    }
    put_chunk<kPerm>(tile_img, sb, sps, m0 + rr, lane, a);
    int sum = a[0] + a[1] + a[2] + a[3] + a[4] + a[5] + a[6] + a[7];
    sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
    sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 2);  // the four chunks of a 32-block
    if ((lane & 3) == 0) s.v[lane >> 2][rr] = __fmul_rn(s.sc[lane >> 2][rr], (float)sum);
  }
  if (!asc) return;
  __syncthreads();
  put_scales<32>(s, ascimg, tile_img, tile, K, sb, m0, sps);
}

// ---------------------------------------------------------------------------------------------- quantiser + pre-pass in one
// izb_quantize_act (csrc/izb_quantize.cu, the arithmetic of quantize_act_cpu, src/quants.h:626-643, bit for bit) and
// act_prepare_kernel above in one pass over the f32 rows: a lane owns 8 consecutive values (= one 16-byte operand chunk),
// four lanes a 32-block.  Writes aq / asc exactly as the quantiser does (the caller's buffers stay valid for every other
// kernel) and, from the same registers, the operand images, the gathered scales and the min-term factors of the dense
// tensor-core GEMM: the int8 rows are not read back and the second launch is gone.  One CTA = 8 kR rows x one superblock: four rows a
// warp, or one where that leaves SMs without work.
template <bool kPerm, int kR>
__global__ void __launch_bounds__(256) quant_prepare_kernel(const float* __restrict__ x, int ldx, int M, int Mp, int K,
                                                            int8_t* __restrict__ aq, float* __restrict__ asc,
                                                            uint16_t* __restrict__ aimg, float* __restrict__ ascimg, int sps, int n_tiles,
                                                            uint32_t* __restrict__ part_bad) {
  __shared__ PrepRows s_rows;
  const int sb = blockIdx.x, m0 = blockIdx.y * (8 * kR), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = sb * 256 + lane * 8;
  const int tile = m0 >> 7;  // (the rows lie in one tile)
  uint8_t* tile_img = reinterpret_cast<uint8_t*>(aimg) + (size_t)tile * (K / 256) * sps * STAGE_BYTES;
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
    int q[8], s = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float pr = __fmul_rn(v[i][k], inv);
      q[k] = fabsf(pr) <= 2147483520.0f ? __float2int_rn(pr) : 0;  // (see quantize_act_kernel: the overflow case)
      q[k] = (int)(int8_t)q[k];  // the stored byte is what the GEMM multiplies
      s += q[k];
    }
    s += __shfl_xor_sync(0xFFFFFFFFu, s, 1);
    s += __shfl_xor_sync(0xFFFFFFFFu, s, 2);
    const float sc = __fdiv_rn(amax, 127.0f);
    if (m < Mp) {
      uint2 pk;
      pk.x = (q[0] & 0xFF) | ((q[1] & 0xFF) << 8) | ((q[2] & 0xFF) << 16) | ((uint32_t)(q[3] & 0xFF) << 24);
      pk.y = (q[4] & 0xFF) | ((q[5] & 0xFF) << 8) | ((q[6] & 0xFF) << 16) | ((uint32_t)(q[7] & 0xFF) << 24);
      *reinterpret_cast<uint2*>(aq + (size_t)m * K + col) = pk;
    }
    if ((lane & 3) == 0) {
      s_rows.sc[lane >> 2][rr] = sc;
      s_rows.v[lane >> 2][rr] = __fmul_rn(sc, (float)s);
    }
    if (tile < n_tiles) put_chunk<kPerm>(tile_img, sb, sps, m & 127, lane, q);  // (padding rows past the last tile the GEMM reads: aq / asc only)
  }
  __syncthreads();
  {
    const int b = threadIdx.x >> 5, r = threadIdx.x & 31;
    if (r < 8 * kR && m0 + r < Mp) asc[(size_t)(sb * 8 + b) * Mp + m0 + r] = s_rows.sc[b][r];
  }
  if (tile < n_tiles) put_scales<8 * kR>(s_rows, ascimg, tile_img, tile, K, sb, m0 & 127, sps);
}

// ---------------------------------------------------------------------------------------------- the GEMM kernel
// What one superblock of a weight row becomes in shared memory.  Every form offers
//   load(row)                    the row's superblock header into registers
//   store_scales(smem, slot, t)  the scales the combine warps apply
//   load_stage(c, row)           the quants of blocks 2c, 2c + 1 into registers
//   stage(c, out, t)             those 64 elements as fp16 operand rows, 128-byte swizzled (hi at out, lo 16 KB on)
//   mins(u)                      -dmin * mn of the eight blocks
__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
__device__ __forceinline__ __half2 bits_h2(uint32_t u) { return *reinterpret_cast<const __half2*>(&u); }
__device__ __forceinline__ __half2 h2_const(unsigned short b) { return __half2half2(__ushort_as_half(b)); }
__device__ __forceinline__ void put16(unsigned char* orow, int chunk, int t, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  *reinterpret_cast<uint4*>(orow + ((chunk ^ (t & 7)) << 4)) = make_uint4(a, b, c, d);
}

template <bool kDots>
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
  __device__ __forceinline__ void store_scales(unsigned char* scl, int slot, int t) const {
    reinterpret_cast<float*>(scl + slot * 512)[t] = half_bits_to_float(hdr.x & 0xFFFFu);
  }
  __device__ __forceinline__ void stage(int c, unsigned char* orow, int t) const {
    const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
    // the chunk's two 6-bit sub-block scales as half2 pairs (sc, sc) and (-1024 sc, -1024 sc): 0x6400 | sc is the
    // fp16 number 1024 + sc
    uint32_t sc2 = 0x0101u, mn_unused;
    if (!kDots) pair(c, sc2, mn_unused);
    const __half2 k1024 = h2_const(0x6400), kneg = h2_const(0xE400), k16th = h2_const(0x2C00);
    const __half2 slo = __hsub2(bits_h2(__byte_perm(sc2, 0x64646464u, 0x4040)), k1024), shi = __hsub2(bits_h2(__byte_perm(sc2, 0x64646464u, 0x4141)), k1024);
    const __half2 nlo = __hmul2(slo, kneg), nhi16 = __hmul2(__hmul2(shi, kneg), k16th), shi16 = __hmul2(shi, k16th);
    // High nibbles stay where they are: (word & 0x00F000F0) | 0x6400 is the fp16 number 1024 + 16 q, and
    // (1024 + 16 q) * (sc / 16) - 64 sc = sc * q exactly (one rounding, of an integer below 2^11).  One shift per
    // word (for its upper bytes) instead of three.
    auto cv = [](uint32_t word, uint32_t mask, __half2 scale, __half2 neg) -> uint32_t { return h2_bits(__hfma2(bits_h2((word & mask) | 0x64006400u), scale, neg)); };
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
      const uint32_t w0 = w[2 * jj], w1 = w[2 * jj + 1], x0 = w0 >> 8, x1 = w1 >> 8;
      put16(orow, jj, t, cv(w0, 0x000F000Fu, slo, nlo), cv(x0, 0x000F000Fu, slo, nlo), cv(w1, 0x000F000Fu, slo, nlo), cv(x1, 0x000F000Fu, slo, nlo));
      put16(orow, 4 + jj, t, cv(w0, 0x00F000F0u, shi16, nhi16), cv(x0, 0x00F000F0u, shi16, nhi16), cv(w1, 0x00F000F0u, shi16, nhi16), cv(x1, 0x00F000F0u, shi16, nhi16));
    }
  }
  __device__ __forceinline__ void mins(float (&u)[8]) const {
    const float ndmin = -half_bits_to_float(hdr.x >> 16);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t sc_unused, mn2;
      pair(c, sc_unused, mn2);
      u[2 * c] = __fmul_rn(ndmin, (float)(mn2 & 0xFFu));
      u[2 * c + 1] = __fmul_rn(ndmin, (float)(mn2 >> 8));
    }
  }
};

// four int8 (offset by 128 into unsigned bytes) of `x` -> two half2, element order kept
__device__ __forceinline__ __half2 q8_pair(uint32_t x_biased, uint32_t sel) {
  return __hsub2(bits_h2(__byte_perm(x_biased, 0x64646464u, sel)), h2_const(0x6480));  // (1024 + q + 128) - 1152
}

struct DeqQ80 {
  uint4 hdr, qs[4];
  __device__ __forceinline__ void load(const unsigned char* row) { hdr = *reinterpret_cast<const uint4*>(row); }
  __device__ __forceinline__ void store_scales(unsigned char* scl, int slot, int t) const {
    float* d8 = reinterpret_cast<float*>(scl + slot * 4096);
    const uint32_t hw[4] = {hdr.x, hdr.y, hdr.z, hdr.w};
#pragma unroll
    for (int b = 0; b < 8; ++b) d8[b * 128 + t] = half_bits_to_float((b & 1) ? hw[b >> 1] >> 16 : hw[b >> 1] & 0xFFFFu);
  }
  __device__ __forceinline__ void load_stage(int c, const unsigned char* row) {
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) qs[jj] = *reinterpret_cast<const uint4*>(row + 16 + 64 * c + 16 * jj);
  }
  __device__ __forceinline__ void stage(int, unsigned char* orow, int t) const {
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
      const uint4 q = qs[jj];
      const uint32_t x0 = q.x ^ 0x80808080u, x1 = q.y ^ 0x80808080u, x2 = q.z ^ 0x80808080u, x3 = q.w ^ 0x80808080u;
      put16(orow, 2 * jj, t, h2_bits(q8_pair(x0, 0x4140)), h2_bits(q8_pair(x0, 0x4342)), h2_bits(q8_pair(x1, 0x4140)), h2_bits(q8_pair(x1, 0x4342)));
      put16(orow, 2 * jj + 1, t, h2_bits(q8_pair(x2, 0x4140)), h2_bits(q8_pair(x2, 0x4342)), h2_bits(q8_pair(x3, 0x4140)), h2_bits(q8_pair(x3, 0x4342)));
    }
  }
  __device__ __forceinline__ void mins(float (&)[8]) const {}
};

// an integer -128 .. 127 as (s, s)
__device__ __forceinline__ __half2 small_h2(int s) { return __half2half2(__int2half_rn(s)); }
// sixteen quants of one 16-element half with its scale: words of four quants q + 128 (biased) -> chunk pair `ch`, `ch` + 1
template <int kTerms>
__device__ __forceinline__ void put_half(unsigned char* orow, int ch, int t, const uint32_t (&xb)[4], int sc) {
  uint32_t hi[8], lo[8];
  const __half2 s_hi = small_h2(kTerms == 2 ? sc & ~1 : sc), s_lo = small_h2(sc & 1);  // sc = (sc & ~1) + (sc & 1), also below zero
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const __half2 a = q8_pair(xb[k], 0x4140), b = q8_pair(xb[k], 0x4342);
    hi[2 * k] = h2_bits(__hmul2(a, s_hi));
    hi[2 * k + 1] = h2_bits(__hmul2(b, s_hi));
    if (kTerms == 2) {
      lo[2 * k] = h2_bits(__hmul2(a, s_lo));
      lo[2 * k + 1] = h2_bits(__hmul2(b, s_lo));
    }
  }
  put16(orow, ch, t, hi[0], hi[1], hi[2], hi[3]);
  put16(orow, ch + 1, t, hi[4], hi[5], hi[6], hi[7]);
  if (kTerms == 2) {
    put16(orow + STAGE_BYTES, ch, t, lo[0], lo[1], lo[2], lo[3]);
    put16(orow + STAGE_BYTES, ch + 1, t, lo[4], lo[5], lo[6], lo[7]);
  }
}

// Q5_K and IQ4_XS in the generic form: f32 d | f32 dmin | int8 scale[16] | uint8 min[16] | pad | int8 quant[256]
template <int kTerms>
struct DeqK16 {
  uint4 h0, h1, h2, qs[4];
  __device__ __forceinline__ void load(const unsigned char* row) {
    h0 = *reinterpret_cast<const uint4*>(row);
    h1 = *reinterpret_cast<const uint4*>(row + 16);
    h2 = *reinterpret_cast<const uint4*>(row + 32);
  }
  __device__ __forceinline__ void store_scales(unsigned char* scl, int slot, int t) const { reinterpret_cast<uint32_t*>(scl + slot * 512)[t] = h0.x; }
  __device__ __forceinline__ void load_stage(int c, const unsigned char* row) {
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) qs[jj] = *reinterpret_cast<const uint4*>(row + 48 + 64 * c + 16 * jj);
  }
  __device__ __forceinline__ void stage(int c, unsigned char* orow, int t) const {
    const uint32_t scw = c == 0 ? h0.z : c == 1 ? h0.w : c == 2 ? h1.x : h1.y;  // the four halves' scales
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
      const uint4 q = qs[jj];
      const uint32_t xb[4] = {q.x ^ 0x80808080u, q.y ^ 0x80808080u, q.z ^ 0x80808080u, q.w ^ 0x80808080u};
      put_half<kTerms>(orow, 2 * jj, t, xb, (int)(int8_t)(scw >> (8 * jj)));
    }
  }
  __device__ __forceinline__ void mins(float (&u)[8]) const {
    const float ndmin = -__uint_as_float(h0.y);
    const uint32_t m[4] = {h1.z, h1.w, h2.x, h2.y};
#pragma unroll
    for (int b = 0; b < 8; ++b) u[b] = __fmul_rn(ndmin, (float)((m[b >> 1] >> (16 * (b & 1))) & 0xFFu));  // (both halves of a block share it)
  }
};

// Q6_K packed: ql[128] | qh[64] | int8 scale[16] | fp16 d (csrc/izb_types.cu: q6p_word)
struct DeqQ6K {
  uint4 sc, h[2], l[4];
  uint32_t d;
  __device__ __forceinline__ void load(const unsigned char* row) {
    sc = *reinterpret_cast<const uint4*>(row + 192);
    d = *reinterpret_cast<const unsigned short*>(row + 208);
  }
  __device__ __forceinline__ void store_scales(unsigned char* scl, int slot, int t) const { reinterpret_cast<float*>(scl + slot * 512)[t] = half_bits_to_float(d); }
  __device__ __forceinline__ void load_stage(int c, const unsigned char* row) {
    const unsigned char* pl = row + 64 * (c >> 1);
    const unsigned char* ph = row + 128 + 32 * (c >> 1);
#pragma unroll
    for (int i = 0; i < 4; ++i) l[i] = *reinterpret_cast<const uint4*>(pl + 16 * i);
#pragma unroll
    for (int i = 0; i < 2; ++i) h[i] = *reinterpret_cast<const uint4*>(ph + 16 * i);
  }
  __device__ __forceinline__ void stage(int c, unsigned char* orow, int t) const {
    const int up = c & 1;  // blocks 2c, 2c + 1: sub-blocks 2 up, 2 up + 1 of half c / 2
    const uint32_t scw = c == 0 ? sc.x : c == 1 ? sc.y : c == 2 ? sc.z : sc.w;
#pragma unroll
    for (int hl = 0; hl < 2; ++hl) {
      const uint32_t hw[4] = {h[hl].x, h[hl].y, h[hl].z, h[hl].w};
#pragma unroll
      for (int o = 0; o < 2; ++o) {  // sub-block 2 up + o
        const uint4 lq = l[2 * o + hl];
        const uint32_t lw[4] = {lq.x, lq.y, lq.z, lq.w};
        uint32_t xb[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t qu = ((lw[k] >> (4 * up)) & 0x0F0F0F0Fu) | (((hw[k] >> (4 * up + 2 * o)) & 0x03030303u) << 4);
          xb[k] = qu + 0x60606060u;  // 0..63 -> q + 128 (96..159 per byte, no carry)
        }
        put_half<2>(orow, 4 * o + 2 * hl, t, xb, (int)(int8_t)(scw >> (8 * (2 * o + hl))));
      }
    }
  }
  __device__ __forceinline__ void mins(float (&)[8]) const {}
};

template <class F, bool kDots> struct DeqOf;
template <bool kDots> struct DeqOf<FQ4K, kDots> { using type = DeqQ4K<kDots>; };
template <bool kDots> struct DeqOf<FQ80, kDots> { using type = DeqQ80; };
template <bool kDots> struct DeqOf<FQ5K, kDots> { using type = DeqK16<1>; };
template <bool kDots> struct DeqOf<FIQ4, kDots> { using type = DeqK16<2>; };
template <bool kDots> struct DeqOf<FQ6K, kDots> { using type = DeqQ6K; };

// What a hand-over costs (measured on one SM): a satisfied mbarrier test has 54 clk of latency, an arrival is seen by a waiting
// warp of the same CTA 135 clk later, a tcgen05.commit 182 clk after the last MMA; with three accumulators in the ring
// that alone allows no block in under 175 clk.  An MMA or commit behind a lane test takes 98 clk to issue, with the elected
// predicate inside the statement about 25 (6 % of the kernel).  The rest of a block's time is the combine warps' own
// chain: test, two TMEM reads and the packed FMAs; in calls of a millisecond the board is at its 1000 W as well.
template <class F, bool kDots>
__global__ void __launch_bounds__(kThreads, 1) gemm_tc_kernel(const __grid_constant__ CUtensorMap tmW, const TcParams p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  using MP = Map<F>;
  constexpr int NA = MP::NA, NB = MP::NB, NR = MP::NR, RAW = MP::RAW, SBB = F::SBB;
  constexpr bool kMins = F::kMin && !kDots;
  constexpr int SPS = kMins ? 5 : 4;  // operand stages per superblock: four of 64 K-elements (+ the min-term stage)
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + MP::OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + MP::OFF_BAR + MP::NUM_BARS * 8);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + MP::OFF_BAR + MP::NUM_BARS * 8 + 4);
  const uint32_t bar0 = smem_u32(bars);
  auto bar = [&](int i) -> uint32_t { return bar0 + 8u * (uint32_t)i; };
  // (through a shuffle: the compiler then knows it to be the same for the whole warp and keeps what follows from it in uniform registers)
  const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    // Consumers release a buffer with one arrival per THREAD (128 dequantisers, 256 combine threads): one elected arrival per
    // warp, predicated without a branch, measured 5 % slower (8192 x 17408 x 5120: 3.25 against 3.10 ms).  A_EMPTY / B_EMPTY: one
    // tcgen05.commit each
    for (int i = 0; i < NA; ++i) { mbar_init(bar(MP::A_FULL + i), 1); mbar_init(bar(MP::A_EMPTY + i), 1); }
    for (int i = 0; i < NB; ++i) { mbar_init(bar(MP::B_FULL + i), 128); mbar_init(bar(MP::B_EMPTY + i), 1); }
    for (int i = 0; i < NR; ++i) { mbar_init(bar(MP::RAW_FULL + i), 1); mbar_init(bar(MP::RAW_EMPTY + i), 128); }
    for (int i = 0; i < ND1; ++i) { mbar_init(bar(MP::D1_FULL + i), 1); mbar_init(bar(MP::D1_EMPTY + i), 8); }
    mbar_init(bar(MP::D2_FULL), 1);
    mbar_init(bar(MP::D2_EMPTY), 8);
    for (int i = 0; i < NASC; ++i) { mbar_init(bar(MP::ASC_FULL + i), 1); mbar_init(bar(MP::ASC_EMPTY + i), 256); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xFFFFFFFFu, *tmem_slot, 0);

  // ---- the CTA's work: items blockIdx.x, blockIdx.x + gridDim.x, ... of (row tiles) x (column tiles) x (K parts), K part
  // fastest, then column tile.  Every role walks the same list; its ring positions and barrier parities run on from item to
  // item, so the producers, the dequantisers and the issuers are already inside the next one while the combine warps store.
  const int n_ntiles = (p.N + BN - 1) / BN, nsb = p.K >> 8, nb = p.K >> 5;
  const int n_work = (p.tiles ? p.tiles[0] : p.n_mtiles) * n_ntiles * p.n_split;
  struct Item { int tile, nt, ks, s0, s1; };
  auto item = [&](int w) -> Item {
    Item it;
    it.ks = 0;
    int q = w;
    if (p.n_split > 1) { q = w / p.n_split; it.ks = w - q * p.n_split; }
    it.tile = q / n_ntiles;
    it.nt = q - it.tile * n_ntiles;
    it.s0 = it.ks * nsb / p.n_split;
    it.s1 = (it.ks + 1) * nsb / p.n_split;
    return it;
  };

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    // Every role loop below is executed by its whole warp (uniform waits, an elected lane issues), so no lane of a role warp
    // sits at the final CTA barrier while another lane of the same warp is still working.
    if (warp == 0) {
      // ================= activation producer: the tile's stage images lie back to back in global memory
      pdl_wait();  // (the pre-pass; the weights depend on no kernel and are on their way by then)
      int sa = 0, pa = 1;
      bool ok = true;
      for (int w = blockIdx.x; w < n_work && ok; w += gridDim.x) {
        const Item it = item(w);
        const unsigned char* src = reinterpret_cast<const unsigned char*>(p.aimg) + (size_t)it.tile * nsb * SPS * STAGE_BYTES;
        for (int g = it.s0 * SPS; g < it.s1 * SPS; ++g) {
          if (!mbar_wait_warp(bar(MP::A_EMPTY + sa), pa, abort_flag, p.err, p.spin_limit, E_APROD)) { ok = false; break; }
          if (lane == 0 && g != p.skip_stage) {  // (skip_stage: diagnostics only, makes the waits of this stage run out)
            mbar_expect_tx(bar(MP::A_FULL + sa), STAGE_BYTES);
            bulk_g2s(smem_u32(smem + MP::OFF_A + sa * STAGE_BYTES), src + (size_t)g * STAGE_BYTES, STAGE_BYTES, bar(MP::A_FULL + sa));
          }
          __syncwarp();
          if (++sa == NA) { sa = 0; pa ^= 1; }
        }
      }
    } else if (warp == 3) {
      // ================= weight producer: TMA of the raw superblocks of the tile's 128 weight rows, and per superblock the
      // 8 x 128 activation scales the combine warps need
      int rb = 0, pr = 1, sq = 0, pq = 1;
      bool ok = true;
      for (int w = blockIdx.x; w < n_work && ok; w += gridDim.x) {
        const Item it = item(w);
        const int wrow = (p.tiles ? p.tiles[1 + 3 * it.tile] : p.mat) * p.N + it.nt * BN;
        for (int s = it.s0; s < it.s1; ++s) {
          if (!mbar_wait_warp(bar(MP::RAW_EMPTY + rb), pr, abort_flag, p.err, p.spin_limit, E_WPROD)) { ok = false; break; }
          if (lane == 0) {
            mbar_expect_tx(bar(MP::RAW_FULL + rb), RAW);
            tma_2d(smem_u32(smem + MP::OFF_RAW + rb * RAW), &tmW, s * (SBB / 4), wrow, bar(MP::RAW_FULL + rb));
          }
          if (++rb == NR) { rb = 0; pr ^= 1; }
          if (!kDots) {
            if (!mbar_wait_warp(bar(MP::ASC_EMPTY + sq), pq, abort_flag, p.err, p.spin_limit, E_WPROD)) { ok = false; break; }
            pdl_wait();  // (the scales are the pre-pass's; the first weights are on their way; later calls return at once)
            if (lane == 0) {
              mbar_expect_tx(bar(MP::ASC_FULL + sq), 4096);
              bulk_g2s(smem_u32(smem + MP::OFF_ASC + sq * 4096), p.ascimg + ((size_t)it.tile * nb + 8 * s) * BM, 4096, bar(MP::ASC_FULL + sq));
            }
            if (++sq == NASC) { sq = 0; pq ^= 1; }
          }
          __syncwarp();
        }
      }
    } else {
      // ================= MMA issuers.  Of a superblock's stages 0..3 (two 32-blocks each, every block into its own
      // accumulator buffer: two MMAs of K = 16 per term + one commit) warp 1 takes 0 and 2, warp 2 takes 1, 3 and the min-term
      // stage 4 (three bf16 MMAs of K = 16 accumulated into the fourth TMEM buffer over the item's K range).  Two issuers
      // because what a warp pays per block -- barrier tests and commits between MMAs -- is longer than the 128 cycles the two
      // MMAs run; one issuer for the min term so that its accumulator is updated in program order.
      bool ok = true;
      int n_item = 0, gs = 0, jb = 0;  // items, stages and blocks done: they run on across items
      for (int w = blockIdx.x; w < n_work && ok; w += gridDim.x, ++n_item) {
        const Item it = item(w);
        for (int s = it.s0; s < it.s1 && ok; ++s, gs += SPS, jb += 8) {
          for (int t = warp - 1; t < (warp == 1 ? 4 : SPS) && ok; t += (t == 3 ? 1 : 2)) {
            const int g = gs + t, sa = g % NA, sb = g % NB;
            const uint32_t b_ok = mbar_test(bar(MP::B_FULL + sb), (g / NB) & 1), a_ok = mbar_test(bar(MP::A_FULL + sa), (g / NA) & 1);
            if (!__all_sync(0xFFFFFFFFu, b_ok && a_ok)) {
              if (!mbar_wait_warp(bar(MP::B_FULL + sb), (g / NB) & 1, abort_flag, p.err, p.spin_limit, E_MMA)) { ok = false; break; }
              if (!mbar_wait_warp(bar(MP::A_FULL + sa), (g / NA) & 1, abort_flag, p.err, p.spin_limit, E_MMA)) { ok = false; break; }
            }
            tc_fence_after();
            const uint32_t a_addr = smem_u32(smem + MP::OFF_A + sa * STAGE_BYTES), b_addr = smem_u32(smem + MP::OFF_B + sb * MP::BSTAGE);
            if (t < 4) {
#pragma unroll
              for (int blk = 0; blk < 2; ++blk) {
                const int j = jb + 2 * t + blk, d = j % ND1;
                if (!mbar_wait_warp(bar(MP::D1_EMPTY + d), ((j / ND1) & 1) ^ 1, abort_flag, p.err, p.spin_limit, E_MMA)) { ok = false; break; }
                tc_fence_after();
                const uint32_t dt = tmem_base + (uint32_t)(d * BN);
#pragma unroll
                for (int term = 0; term < F::kTerms; ++term)
#pragma unroll
                  for (int k16 = 0; k16 < 2; ++k16)
                    tc_mma_f16(dt, umma_desc(a_addr + blk * 64 + k16 * 32), umma_desc(b_addr + term * STAGE_BYTES + blk * 64 + k16 * 32), kIdescF16, term | k16);
                tc_commit(bar(MP::D1_FULL + d));
              }
              if (!ok) break;
            } else {
              // the min-term accumulator of the item before must have been read before this item's first MMA clears it
              if (s == it.s0 && n_item > 0 && !mbar_wait_warp(bar(MP::D2_EMPTY), (n_item - 1) & 1, abort_flag, p.err, p.spin_limit, E_MMA)) { ok = false; break; }
              tc_fence_after();
#pragma unroll
              for (int k16 = 0; k16 < 3; ++k16)
                tc_mma_f16(tmem_base + ND1 * BN, umma_desc(a_addr + k16 * 32), umma_desc(b_addr + k16 * 32), kIdescBF16, (s > it.s0 || k16) ? 1u : 0u);
            }
            tc_commit(bar(MP::A_EMPTY + sa));
            tc_commit(bar(MP::B_EMPTY + sb));
            if (kMins && t == 4 && s == it.s1 - 1) tc_commit(bar(MP::D2_FULL));
          }
        }
      }
    }
  } else if (warp < 8) {
    // ================= dequantisers: thread t <-> weight row n0 + t
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    const int t = threadIdx.x - 128;
    bool ok = true;
    int sbq = 0, pbq = 1;  // operand ring position and wait parity
    int rb = 0, pr = 0;    // raw ring
    int sbc = 0;           // superblocks done (all items): position in the 4-deep ring of superblock scales
    for (int w = blockIdx.x; w < n_work && ok; w += gridDim.x) {
      const Item it = item(w);
      for (int s = it.s0; s < it.s1 && ok; ++s, ++sbc) {
        if (!mbar_wait(bar(MP::RAW_FULL + rb), pr, abort_flag, p.err, p.spin_limit, E_DEQ)) { ok = false; break; }
        const unsigned char* rrow = smem + MP::OFF_RAW + rb * RAW + t * SBB;
        typename DeqOf<F, kDots>::type dq;
        dq.load(rrow);
        if (!kDots) dq.store_scales(smem + MP::OFF_SCL, sbc & 3, t);
        auto deliver = [&]() {
          fence_proxy_async();
          mbar_arrive(bar(MP::B_FULL + sbq));  // (every thread after its own stores and fence)
          if (++sbq == NB) { sbq = 0; pbq ^= 1; }
        };
#pragma unroll 1  // (rolled on purpose: with the role loops resident at once, code size costs more than the loop)
        for (int c = 0; c < 4; ++c) {
          dq.load_stage(c, rrow);
          if (!mbar_wait(bar(MP::B_EMPTY + sbq), pbq, abort_flag, p.err, p.spin_limit, E_DEQ)) { ok = false; break; }
          dq.stage(c, smem + MP::OFF_B + sbq * MP::BSTAGE + t * 128, t);
          deliver();
        }
        if (!ok) break;
        mbar_arrive(bar(MP::RAW_EMPTY + rb));
        if (++rb == NR) { rb = 0; pr ^= 1; }
        if (kMins) {
          // the min-term stage: u[b] = -dmin * mn[b] (exact in f32: 11 x 6 bits) as three bf16 terms u1 + u2 + u3; the
          // stage's six 16-byte chunks hold (u1, u2, u1, u3, u2, u1) for the eight blocks, against the activation side's
          // (v1, v1, v2, v1, v2, v3)
          float u[8];
          dq.mins(u);
          uint32_t u1[4], u2[4], u3[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const __nv_bfloat162 h1 = __floats2bfloat162_rn(u[2 * k], u[2 * k + 1]);
            const float ra = __fsub_rn(u[2 * k], __low2float(h1)), rb2 = __fsub_rn(u[2 * k + 1], __high2float(h1));
            const __nv_bfloat162 h2 = __floats2bfloat162_rn(ra, rb2);
            const __nv_bfloat162 h3 = __floats2bfloat162_rn(__fsub_rn(ra, __low2float(h2)), __fsub_rn(rb2, __high2float(h2)));
            u1[k] = *reinterpret_cast<const uint32_t*>(&h1);
            u2[k] = *reinterpret_cast<const uint32_t*>(&h2);
            u3[k] = *reinterpret_cast<const uint32_t*>(&h3);
          }
          if (!mbar_wait(bar(MP::B_EMPTY + sbq), pbq, abort_flag, p.err, p.spin_limit, E_DEQ)) { ok = false; break; }
          unsigned char* orow = smem + MP::OFF_B + sbq * MP::BSTAGE + t * 128;
          put16(orow, 0, t, u1[0], u1[1], u1[2], u1[3]);
          put16(orow, 1, t, u2[0], u2[1], u2[2], u2[3]);
          put16(orow, 2, t, u1[0], u1[1], u1[2], u1[3]);
          put16(orow, 3, t, u3[0], u3[1], u3[2], u3[3]);
          put16(orow, 4, t, u2[0], u2[1], u2[2], u2[3]);
          put16(orow, 5, t, u1[0], u1[1], u1[2], u1[3]);
          deliver();
        }
      }
    }
  } else {
    // ================= combine: a warp holds 32 token rows (TMEM lanes 32 * (warp % 4) ..) x 64 of the 128 columns as fragments (tc_ld_frag64).
    // All f32 arithmetic is done on register pairs (fma.rn.f32x2): half the instructions for the same IEEE results.
    asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    pdl_wait();  // (C belongs to kernels before this one until they are done)
    const int q = warp & 3, half = (warp - 8) >> 2;
    const int row0 = 32 * q + (lane >> 2), cl = 64 * half + 2 * (lane & 3);  // this thread's rows row0 + 8 k, k < 4; columns cl + 8 g, + 1, g < 8
    const uint32_t t_lane = tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)(half * 64);
    bool ok = true;
    int d = 0, pd = 0, sq = 0, pq = 0;  // accumulator ring / scale ring positions and wait parities
    int sbc = 0, n_item = 0;            // superblocks and items done
    for (int w = blockIdx.x; w < n_work && ok; w += gridDim.x, ++n_item) {
      __syncwarp();  // (rows that are not stored come here first)
      const Item it = item(w);
      const int n0 = it.nt * BN + cl;
      const int r0 = p.tiles ? p.tiles[2 + 3 * it.tile] : it.tile * BM;
      const int nr = p.tiles ? p.tiles[3 + 3 * it.tile] : min(BM, p.M - r0);
      unsigned long long res2[4][8], tq2[4][8];  // [row][column pair]
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int g = 0; g < 8; ++g) res2[k][g] = tq2[k][g] = 0ull;
      for (int s = it.s0; s < it.s1 && ok; ++s, ++sbc) {
        const float* as = reinterpret_cast<const float*>(smem + MP::OFF_ASC + sq * 4096) + row0;  // the rows' eight block scales
        if (!kDots && !mbar_wait_warp(bar(MP::ASC_FULL + sq), pq, abort_flag, p.err, p.spin_limit, E_EPI)) { ok = false; break; }
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          unsigned long long a2[4];
          if (!kDots) {
#pragma unroll
            for (int k = 0; k < 4; ++k) a2[k] = pack2(as[b * BM + 8 * k]);
          }
          if (!mbar_wait_warp(bar(MP::D1_FULL + d), pd, abort_flag, p.err, p.spin_limit, E_EPI)) { ok = false; break; }
          tc_fence_after();
          unsigned long long dd[8];
          if (F::kColScale && !kDots) {
#pragma unroll
            for (int g = 0; g < 8; ++g) dd[g] = *reinterpret_cast<const unsigned long long*>(smem + MP::OFF_SCL + (sbc & 3) * 4096 + b * 512 + (cl + 8 * g) * 4);
          }
#pragma unroll
          for (int hr = 0; hr < 2; ++hr) {  // 16 rows at a time: the block loop's working set stays inside the register budget
            unsigned long long v[16];
            tc_ld_frag64(t_lane + ((uint32_t)(16 * hr) << 16) + (uint32_t)(d * BN), v);
            if (hr == 1) {
              tc_fence_before();
              mbar_arrive_if(bar(MP::D1_EMPTY + d), lane == 0);  // the accumulator buffer may be overwritten (the loads were the whole warp's)
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const int k = 2 * hr + (j & 1), g = j >> 1;
              if (kDots) {
                const int row = row0 + 8 * k;
                if (row < nr && n0 + 8 * g < p.N) {  // (N is a multiple of 16: pairs are whole)
                  int32_t* o = p.dots + ((size_t)(r0 + row) * p.N + n0 + 8 * g) * nb + 8 * s + b;
                  o[0] = __float2int_rn(lo_f(v[j]));
                  o[nb] = __float2int_rn(hi_f(v[j]));
                }
              } else if (F::kColScale) {
                ffma2(res2[k][g], fmul2(a2[k], dd[g]), v[j]);
              } else if (b == 0) {
                tq2[k][g] = fmul2(a2[k], v[j]);
              } else {
                ffma2(tq2[k][g], a2[k], v[j]);
              }
            }
          }
          if (++d == ND1) { d = 0; pd ^= 1; }
        }
        if (!ok) break;
        if (!kDots) {  // the superblock's scales are read: its ring slot may be refilled
          mbar_arrive(bar(MP::ASC_EMPTY + sq));
          if (++sq == NASC) { sq = 0; pq ^= 1; }
        }
        if (!kDots && !F::kColScale) {  // res += d * tq
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            const unsigned long long dd = *reinterpret_cast<const unsigned long long*>(smem + MP::OFF_SCL + (sbc & 3) * 512 + (cl + 8 * g) * 4);
#pragma unroll
            for (int k = 0; k < 4; ++k) ffma2(res2[k][g], dd, tq2[k][g]);
          }
        }
      }
      if (kMins && ok) {  // the min term of the whole K range (already negative)
        ok = mbar_wait_warp(bar(MP::D2_FULL), n_item & 1, abort_flag, p.err, p.spin_limit, E_EPI);
        if (ok) {
          tc_fence_after();
          const unsigned long long one2 = pack2(1.0f);
#pragma unroll
          for (int hr = 0; hr < 2; ++hr) {
            unsigned long long v[16];
            tc_ld_frag64(t_lane + ((uint32_t)(16 * hr) << 16) + (uint32_t)(ND1 * BN), v);
            if (hr == 1) {
              tc_fence_before();
              mbar_arrive_if(bar(MP::D2_EMPTY), lane == 0);  // the next item's min term may start
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) ffma2(res2[2 * hr + (j & 1)][j >> 1], one2, v[j]);
          }
        }
      }
      if (!ok || kDots || *abort_flag) continue;
      if (p.acc == 3) {
        // Gate and up projections in one weight whose rows alternate in groups of 32 (izb_weight_create_gateup): this
        // thread's columns are gate outputs (g < 4) and the up outputs of the same FFN rows (g + 4), so the SwiGLU product
        // up * silu(gate) (zero/kernels/gemm.cl:562-565) is formed in registers and only the F-wide result is stored.
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (row0 + 8 * k >= nr) break;
          float* cp = p.C + (size_t)(r0 + row0 + 8 * k) * p.ldc + p.c_off + ((it.nt * BN) >> 1) + half * 32 + 2 * (lane & 3);
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            const unsigned long long g2 = res2[k][g], u2 = res2[k][g + 4];
            *reinterpret_cast<float2*>(cp + 8 * g) = swiglu_mul2(make_float2(lo_f(g2), hi_f(g2)), make_float2(lo_f(u2), hi_f(u2)));
          }
        }
        continue;
      }
      const int acc = p.acc;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int out_row = r0 + row0 + 8 * k;
        if (row0 + 8 * k >= nr) break;
        float* cp = p.n_split > 1 ? p.part + ((size_t)it.ks * p.M + out_row) * p.N + n0 : p.C + (size_t)out_row * p.ldc + p.c_off + n0;
        const float rs = p.rowscale ? p.rowscale[out_row] : 1.0f;
        float2 old[8];
        if (acc != 0) {
#pragma unroll
          for (int g = 0; g < 8; ++g) old[g] = n0 + 8 * g < p.N ? *reinterpret_cast<const float2*>(cp + 8 * g) : make_float2(0.0f, 0.0f);
        }
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          if (n0 + 8 * g >= p.N) break;
          float2 y = make_float2(lo_f(res2[k][g]), hi_f(res2[k][g]));
          if (p.rowscale) y = make_float2(__fmul_rn(rs, y.x), __fmul_rn(rs, y.y));
          if (acc == 1) y = make_float2(__fadd_rn(y.x, old[g].x), __fadd_rn(y.y, old[g].y));
          else if (acc == 2) y = swiglu_mul2(old[g], y);  // C holds the gate projection: C = y * silu(C)   (zero/kernels/gemm.cl:562-565)
          *reinterpret_cast<float2*>(cp + 8 * g) = y;
        }
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
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------- partial sums of a cut K range
// C = part 0 + part 1 + ... in order.  One thread per four output columns.
__global__ void __launch_bounds__(256) split_reduce_kernel(const float* __restrict__ part, int n_split, int M, int N, float* __restrict__ C, int ldc, int c_off,
                                                           const uint32_t* __restrict__ part_bad) {
  pdl_launch_next();
  pdl_wait();
  if (*part_bad) return;
  const int c = (blockIdx.x * 256 + threadIdx.x) * 4, m = blockIdx.y;
  if (c >= N) return;
  const float* src = part + (size_t)m * N + c;
  float4 v = *reinterpret_cast<const float4*>(src);
  for (int k = 1; k < n_split; ++k) {
    const float4 o = *reinterpret_cast<const float4*>(src + (size_t)k * M * N);
    v.x = __fadd_rn(v.x, o.x); v.y = __fadd_rn(v.y, o.y); v.z = __fadd_rn(v.z, o.z); v.w = __fadd_rn(v.w, o.w);
  }
  *reinterpret_cast<float4*>(C + (size_t)m * ldc + c_off + c) = v;
}

// ---------------------------------------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn get_encode() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

// Diagnostics hook (izb_debug_wait_test): the spin limit of the bounded waits and the operand stage the activation
// producer leaves out, for the NEXT launch only.
std::atomic<uint32_t> g_test_spin{0};
std::atomic<int> g_test_skip{-1};

template <class F, bool kDots>
int launch_tc(const izb_weight* w, TcParams& p, dim3 grid, cudaStream_t st) {
  constexpr int SMEM_BYTES = Map<F>::SMEM_BYTES;
  IZB_SMEM_OPTIN((gemm_tc_kernel<F, kDots>), SMEM_BYTES, w->device);
  const uint32_t spin = g_test_spin.exchange(0);
  p.spin_limit = spin ? spin : kSpinLimit;
  p.skip_stage = g_test_skip.exchange(-1);
  CUtensorMap tm;
  memcpy(&tm, w->tmap_raw, sizeof tm);
  if (p.pdl)
    IZB_LAUNCH("gemm_tc", st, izb_launch_pdl(gemm_tc_kernel<F, kDots>, grid, dim3(kThreads), SMEM_BYTES, st, tm, p));
  else
    IZB_LAUNCH("gemm_tc", st, gemm_tc_kernel<F, kDots><<<grid, kThreads, SMEM_BYTES, st>>>(tm, p));
  return IZB_OK;
}
int launch_tc_of(const izb_weight* w, TcParams& p, dim3 grid, cudaStream_t st) {
  if (w->type == IZB_Q4_K) return p.dots ? launch_tc<FQ4K, true>(w, p, grid, st) : launch_tc<FQ4K, false>(w, p, grid, st);
  if (w->type == IZB_Q8_0) return p.dots ? launch_tc<FQ80, true>(w, p, grid, st) : launch_tc<FQ80, false>(w, p, grid, st);
  if (p.dots) return 1;
  return w->packed6 ? launch_tc<FQ6K, false>(w, p, grid, st) : w->has_min ? launch_tc<FQ5K, false>(w, p, grid, st) : launch_tc<FIQ4, false>(w, p, grid, st);
}

// operand stages per superblock: weights with mins carry the min term as a fifth one
int tc_sps(const izb_weight* w, bool dots) { return (w->type == IZB_Q4_K || (w->type == IZB_K16 && w->has_min)) && !dots ? 5 : 4; }
// Weights that the CUDA-core kernel takes without an arena, and took alone before this kernel did: a call whose arena cannot be had goes there
bool tc_optional(const izb_weight* w) { return w->type == IZB_K16 || w->N % BN != 0; }
// does the kernel take this weight at all
bool tc_takes(const izb_weight* w) { return w->has_tmap && w->N % 16 == 0 && w->K % 256 == 0; }

// persistent grid: one CTA per SM (shared memory allows no more), fewer when there are fewer items
int tc_grid(int device, int n_work) {
  const int sms = izb_sm_budget(device);
  return n_work < sms ? (n_work > 0 ? n_work : 1) : sms;
}

// Programmatic dependent launch behind the pre-pass, for dense calls of one wave: barriers, TMEM and the first weights are there when it ends (us
// without / with: 37 x 5120 x 5120 Q4_K 22.6/18.9, 18 x 512 x 768 Q6_K 18.6/14.5, 512 x 4096 x 4096 Q8_0 63.6/61.3).  Not for more items: CTAs placed while the
// pre-pass drains land on the SMs in the order in which these fall free, and neighbouring items, which share operands, no longer run on neighbours
// (the down projections of 4096 tokens x 8 experts: 392 us against 345).  The GEMM itself lets no kernel in before its end: what waits beside it
// takes issue slots and power (the first of these calls 21.9, 300 x 5120 x 17408 Q6_K 211 -> 225).
bool tc_pdl(bool grouped, int grid, int n_work) { return !grouped && n_work <= grid; }

// Parts the K range of every output tile is cut into, when the tiles alone would leave more than half the SMs idle: as many as fill
// them once, each at least two superblocks.  The parts' sums are at most one 64 KB tile per SM.  The device's SMs count, not the part of them
// that izb_set_sm_limit leaves: that call caps the grid and changes no result.  Long K and plain stores only.  Short K: a part's pipeline fill
// and the summing launch eat the gain (K = 1024: some 10 us uncut).  Other store modes: sums cut in parts are rounded in other places, and what
// those modes write (the residual, the SwiGLU product) is mostly quantised to int8 next, where a last bit can become a whole step.  (A plain
// store may be quantised next as well; there the cut was taken for its speed.)
int tc_split(int device, int n_items, int nsb) {
  if (nsb < 8) return 1;
  const int s = izb_sm_count(device) / (n_items > 0 ? n_items : 1);
  return s < 2 ? 1 : s < nsb / 2 ? s : nsb / 2;
}
constexpr size_t kSplitBytes = (size_t)BM * BN * 4;  // per SM; the flag of a failed part follows them

size_t split_area(int device) { return kSplitBytes * izb_sm_count(device) + 256; }
uint32_t* split_flag(float* split_ws, int device) { return split_ws ? (uint32_t*)((unsigned char*)split_ws + kSplitBytes * izb_sm_count(device)) : nullptr; }

// scratch of one call: the operand images (sps stage images of 16 KB per superblock and tile) and the gathered scales
void tc_scratch_bytes(int n_tiles, int K, int sps, size_t* img_bytes, size_t* asc_bytes) {
  *img_bytes = (size_t)n_tiles * (K / 256) * sps * STAGE_BYTES;
  *asc_bytes = (size_t)n_tiles * (K / 32) * BM * 4;
}

int launch_split_reduce(const float* part, int n_split, int M, int N, float* C, int ldc, int c_off, const uint32_t* part_bad, cudaStream_t st) {
  dim3 grid((N / 4 + 255) / 256, M);
  IZB_LAUNCH("split_reduce", st, izb_launch_pdl(split_reduce_kernel, grid, 256, 0, st, part, n_split, M, N, C, ldc, c_off, part_bad));
  return IZB_OK;
}

// the activation pre-pass + the GEMM on scratch the caller owns (img_bytes + asc_bytes of tc_scratch_bytes, then, where the
// call may be cut along K, `split_ws`)
int run_tc_on(const izb_weight* w, int mat, const int8_t* aq, const float* asc, int lda, int rows_total, const int32_t* tiles,
              int n_tiles_grid, const int32_t* rowmap, const float* rowscale, int M_store, float* C, int ldc, int c_off, int acc,
              int32_t* dots, void* ws, float* split_ws, uint32_t* err, cudaStream_t st, bool reuse_images) {
  const int K = w->K, sps = tc_sps(w, dots != nullptr);
  size_t img_bytes, asc_bytes;
  tc_scratch_bytes(n_tiles_grid, K, sps, &img_bytes, &asc_bytes);
  uint16_t* aimg = (uint16_t*)ws;
  float* ascimg = (float*)((unsigned char*)ws + img_bytes);
  if (!reuse_images) {
    dim3 pg(n_tiles_grid * 4, K / 256);
    auto kernel = w->type == IZB_Q4_K ? act_prepare_kernel<true> : act_prepare_kernel<false>;
    IZB_LAUNCH("act_prepare", st, izb_launch_pdl(kernel, pg, 256, 0, st, aq, asc, lda, K, rows_total, tiles, rowmap, aimg, ascimg, sps, split_flag(split_ws, w->device)));
  }
  TcParams p;
  p.aimg = aimg;
  p.ascimg = ascimg;
  p.tiles = tiles;
  p.rowscale = rowscale;
  p.M = M_store;
  p.N = w->N;
  p.K = K;
  p.mat = mat;
  p.C = C;
  p.ldc = ldc;
  p.c_off = c_off;
  p.acc = acc;
  p.dots = dots;
  p.err = err;
  p.n_mtiles = n_tiles_grid;
  const int n_items = (w->N + BN - 1) / BN * n_tiles_grid;
  p.n_split = split_ws && acc == 0 && !tiles && !dots ? tc_split(w->device, n_items, K / 256) : 1;
  p.part = split_ws;
  p.part_bad = split_flag(split_ws, w->device);
  const int grid = tc_grid(w->device, n_items * p.n_split);
  p.pdl = tc_pdl(tiles != nullptr, grid, n_items * p.n_split);
  if (int rc = launch_tc_of(w, p, dim3(grid), st)) return rc;
  return p.n_split > 1 ? launch_split_reduce(split_ws, p.n_split, M_store, w->N, C, ldc, c_off, p.part_bad, st) : IZB_OK;
}

// the activation pre-pass + the GEMM for one tile set
int run_tc(const izb_weight* w, int mat, const int8_t* aq, const float* asc, int lda, int rows_total, const int32_t* tiles,
           int n_tiles_grid, const int32_t* rowmap, const float* rowscale, int M_store, float* C, int ldc, int c_off, int acc,
           int32_t* dots, int ws_slot, cudaStream_t st, bool reuse_images = false, bool may_cut = true) {
  // reuse_images: the call before this one, on the same stream and arena, prepared the same activation rows for a weight
  // of the same type and K (the up projection after the gate projection): its operand images are still there
  if (!tc_takes(w)) return 1;
  size_t img_bytes, asc_bytes;
  tc_scratch_bytes(n_tiles_grid, w->K, tc_sps(w, dots != nullptr), &img_bytes, &asc_bytes);
  const size_t split_bytes = tiles || dots || !may_cut ? 0 : split_area(w->device);
  void* ws = nullptr;
  if (int rc = izb_workspace(w->device, ws_slot, img_bytes + asc_bytes + split_bytes, st, &ws, !tiles && !dots && tc_optional(w) ? kWsOrElse : kWsMust)) return rc;
  uint32_t* err = izb_device_error_word(w->device);
  if (!err) IZB_FAIL(IZB_ERR_NOMEM, "gemm: no device error word");
  float* split_ws = split_bytes ? (float*)((unsigned char*)ws + img_bytes + asc_bytes) : nullptr;
  return run_tc_on(w, mat, aq, asc, lda, rows_total, tiles, n_tiles_grid, rowmap, rowscale, M_store, C, ldc, c_off, acc, dots, ws, split_ws, err,
                   st, reuse_images);
}

// A plain store with the scales folded into the operands (csrc/izb_gemm_fold.cu), of long K as with tc_split, and for the same reasons: short K
// gains little (a tile is mostly fill and drain), and keeps the sums of the other store modes; x: the quantiser's input (aq and asc are written), or
// null where aq and asc are there.  +1: not taken, or its arena (2.3 times the other kernel's) cannot be had in a capture or without memory:
// the caller goes on with the other kernel.
int run_fold(const izb_weight* w, int mat, const float* x, int ldx, int T, int8_t* aq, float* asc, int Mp, int M_store, float* C, int ldc, int c_off, cudaStream_t st, bool may_cut = true) {
  if (!tc_takes(w) || !izb_fold_takes(w) || w->K < 2048) return 1;
  FoldParams p;
  p.tt = izb_fold_tile_rows(w->device, M_store, w->N);
  p.n_mtiles = (M_store + p.tt - 1) / p.tt;
  const int rows = p.n_mtiles * p.tt;
  if ((rows + 31) / 32 > 65535) return 1;
  const size_t img_bytes = izb_fold_img_bytes(rows, w->K), fine_bytes = izb_fold_fine_bytes(rows, w->K), tail_bytes = izb_fold_tail_bytes(rows, w->K);
  void* ws = nullptr;
  if (int rc = izb_workspace(w->device, kWsGemm, img_bytes + fine_bytes + tail_bytes + split_area(w->device), st, &ws, kWsOrBlock)) return rc;
  uint32_t* err = izb_device_error_word(w->device);
  if (!err) IZB_FAIL(IZB_ERR_NOMEM, "gemm: no device error word");
  p.img = (unsigned char*)ws;
  p.fine = p.img + img_bytes;
  p.tail = p.fine + fine_bytes;
  p.part = (float*)(p.tail + tail_bytes);
  p.part_bad = split_flag(p.part, w->device);
  p.asc = asc;
  p.lda = Mp;
  p.M = M_store;
  p.N = w->N;
  p.K = w->K;
  p.mat = mat;
  p.C = C;
  p.ldc = ldc;
  p.c_off = c_off;
  p.err = err;
  const uint32_t spin = g_test_spin.exchange(0);
  p.spin_limit = spin ? spin : kSpinLimit;
  p.skip_stage = g_test_skip.exchange(-1);
  const int n_items = (w->N + BN - 1) / BN * p.n_mtiles;
  p.n_split = may_cut ? tc_split(w->device, n_items, w->K / 256) : 1;
  // (rows that are not stored count as zeros: what is in them must not send a tile through the longer loops)
  if (int rc = x ? izb_fold_quant_prepare(w, x, ldx, T, Mp, aq, asc, p, st) : izb_fold_prepare(w, aq, asc, Mp, M_store, p, st)) return rc;
  const int grid = tc_grid(w->device, n_items * p.n_split);
  p.pdl = tc_pdl(false, grid, n_items * p.n_split);
  if (int rc = izb_fold_gemm(w, p, grid, st)) return rc;
  return p.n_split > 1 ? launch_split_reduce(p.part, p.n_split, M_store, w->N, C, ldc, c_off, p.part_bad, st) : IZB_OK;
}

}  // namespace

// scratch bytes of a tensor-core GEMM over `rows` activation rows (izb_reserve sizes the arenas with it); folded: of dense calls, which may run the
// folded kernel
size_t izb_gemm_tc_scratch_bytes(int device, int type, int rows, int K, bool folded) {
  size_t img_bytes, asc_bytes;
  tc_scratch_bytes((rows + BM - 1) / BM, K, type == IZB_Q4_K ? 5 : 4, &img_bytes, &asc_bytes);
  if (!folded) return img_bytes + asc_bytes + split_area(device);
  const size_t fold = izb_fold_img_bytes(rows + BM, K) + izb_fold_fine_bytes(rows + BM, K) + izb_fold_tail_bytes(rows + BM, K);  // (tiles round the rows up by less than one)
  return std::max(img_bytes + asc_bytes, fold) + split_area(device);
}

extern "C" int izb_debug_wait_test(uint32_t spin_limit, int skip_stage) {
  g_test_spin.store(spin_limit);
  g_test_skip.store(skip_stage);
  return IZB_OK;
}

// Tensor map over the raw rows in boxes of `box_rows` rows x `box_bytes` bytes
static int make_map(const izb_weight* w, int box_bytes, int box_rows, unsigned char* out) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return IZB_ERR_CUDA;
  const cuuint64_t rows = (cuuint64_t)w->n_mats * w->N;
  if (rows < 1 || w->row_bytes % 16) return IZB_ERR_ALIGN;
  cuuint64_t dims[2] = {(cuuint64_t)(w->row_bytes / 4), rows};
  cuuint64_t strides[1] = {(cuuint64_t)w->row_bytes};
  cuuint32_t box[2] = {(cuuint32_t)(box_bytes / 4), (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUtensorMap tm;
  const CUresult r = enc(&tm, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, w->raw, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return IZB_ERR_CUDA;
  memcpy(out, &tm, sizeof tm);
  return IZB_OK;
}
int izb_make_raw_tensor_map(izb_weight* w) { return make_map(w, w->sb_bytes, BN, w->tmap_raw); }
// chunks of the few-row kernel: a superblock; Q6_K 16 bytes more, for a row pitch its shared-memory reads want
int izb_make_rows_tensor_map(izb_weight* w) { return make_map(w, w->packed6 ? w->sb_bytes + 16 : w->sb_bytes, 16, w->tmap16_raw); }

// may_cut: the K range may be cut into parts, and scales be folded into the operands (IZB_GEMM_AUTO); IZB_GEMM_TC names this kernel, and gives the
// sums of izb_gemm_noalloc
int izb_gemm_tc_launch(const izb_weight* w, int mat, const int8_t* aq, const float* asc, int M, int Mp, float* C, int ldc, int c_off,
                       int acc, int32_t* dots, cudaStream_t st, bool may_cut) {
  if (may_cut && acc == 0 && !dots) {
    const int rc = run_fold(w, mat, nullptr, 0, 0, const_cast<int8_t*>(aq), const_cast<float*>(asc), Mp, M, C, ldc, c_off, st);
    if (rc <= 0) return rc;
  }
  const int n_tiles = (M + BM - 1) / BM;
  if (n_tiles > 65535) return 1;
  return run_tc(w, mat, aq, asc, Mp, Mp, nullptr, n_tiles, nullptr, nullptr, M, C, ldc, c_off, acc, dots, kWsGemm, st, false, may_cut);
}

// quantise + multiply in one call (dense): the fused pre-pass over the M valid rows (rows up to Mp zeroed), then the GEMM on
// its images.  +1 = shape not taken.
int izb_gemm_tc_quant_launch(const izb_weight* w, int mat, const float* x, int ldx, int M, int Mp, int8_t* aq, float* asc, float* C,
                             int ldc, int c_off, int acc, cudaStream_t st) {
  if (acc == 0) {
    const int rc = run_fold(w, mat, x, ldx, M, aq, asc, Mp, Mp, C, ldc, c_off, st);
    if (rc <= 0) return rc;
  }
  const int n_tiles = (Mp + BM - 1) / BM;  // (the GEMM runs over the padded rows, as izb_matmul's does)
  if (n_tiles > 65535 || !tc_takes(w)) return 1;
  const int K = w->K, sps = tc_sps(w, false);
  size_t img_bytes, asc_bytes;
  tc_scratch_bytes(n_tiles, K, sps, &img_bytes, &asc_bytes);
  void* ws = nullptr;
  if (int rc = izb_workspace(w->device, kWsGemm, img_bytes + asc_bytes + split_area(w->device), st, &ws, tc_optional(w) ? kWsOrElse : kWsMust)) return rc;
  uint32_t* err = izb_device_error_word(w->device);
  if (!err) IZB_FAIL(IZB_ERR_NOMEM, "gemm: no device error word");
  uint16_t* aimg = (uint16_t*)ws;
  float* ascimg = (float*)((unsigned char*)ws + img_bytes);
  float* split_ws = (float*)((unsigned char*)ws + img_bytes + asc_bytes);
  const int rows_img = n_tiles * BM > Mp ? n_tiles * BM : Mp;  // every row of every tile is written (rows past M as zeros)
  const bool one = izb_one_row_per_warp(rows_img, K);
  dim3 grid(K / 256, one ? (rows_img + 7) / 8 : (rows_img + 31) / 32);
  auto kernel = w->type == IZB_Q4_K ? (one ? quant_prepare_kernel<true, 1> : quant_prepare_kernel<true, 4>) : one ? quant_prepare_kernel<false, 1> : quant_prepare_kernel<false, 4>;
  IZB_LAUNCH("quant_prepare", st, izb_launch_pdl(kernel, grid, 256, 0, st, x, ldx, M, Mp, K, aq, asc, aimg, ascimg, sps, n_tiles, split_flag(split_ws, w->device)));
  return run_tc_on(w, mat, aq, asc, Mp, Mp, nullptr, n_tiles, nullptr, nullptr, Mp, C, ldc, c_off, acc, nullptr, ws, split_ws, err, st, true);
}

// Up to one wave of the smaller blocks: in a short call a warp's four rows come one after the other while most SMs are idle (us, quantise + GEMM, four
// rows a warp / one: Q4_K 37 x 5120 x 5120 18.4 / 17.4, 64 x 1024 x 2304 13.0 / 11.3, 256 x 1024 x 2304 14.6 / 13.6, Q6_K 37 x 2048 x 8192 22.5 / 21.9; 512 x 1024 x 1024
// Q8_0 18.9 / 19.4).
bool izb_one_row_per_warp(int rows, int K) { return izb_one_wave(dim3(K / 256, (rows + 7) / 8), 256); }

// MoE on the tensor cores: the slots of each expert are tiles of up to 128 rows (izb_moe_sort with TM = 128); gate then up
// with the fused-SwiGLU store mode (h = up * silu(gate)), down with the routing weight as row scale.
int izb_moe_gateup_tc(const izb_weight* wg, const izb_weight* wu, const int8_t* d_aq, const float* d_asc, int Mp,
                      const int32_t* d_tiles, int max_tiles, const int32_t* d_stok, float* d_h, cudaStream_t st) {
  const int F = wg->N;
  int rc = run_tc(wg, 0, d_aq, d_asc, Mp, 0, d_tiles, max_tiles, d_stok, nullptr, 0, d_h, F, 0, 0, nullptr, kWsMoe, st);
  if (rc != 0) return rc;
  const bool same = wu->type == wg->type && wu->K == wg->K;
  return run_tc(wu, 0, d_aq, d_asc, Mp, 0, d_tiles, max_tiles, d_stok, nullptr, 0, d_h, F, 0, 2, nullptr, kWsMoe, st, same);
}

// gate and up of every expert in one interleaved stack (izb_weight_create_gateup): one grouped GEMM, SwiGLU in its epilogue
int izb_moe_gateup_fused_tc(const izb_weight* wgu, const int8_t* d_aq, const float* d_asc, int Mp, const int32_t* d_tiles,
                            int max_tiles, const int32_t* d_stok, float* d_h, cudaStream_t st) {
  return run_tc(wgu, 0, d_aq, d_asc, Mp, 0, d_tiles, max_tiles, d_stok, nullptr, 0, d_h, wgu->N / 2, 0, 3, nullptr, kWsMoe, st);
}

int izb_moe_down_tc(const izb_weight* wd, const int8_t* d_hq, const float* d_hsc, int Sp, const int32_t* d_tiles, int max_tiles,
                    const float* d_swt, float* d_y, cudaStream_t st) {
  return run_tc(wd, 0, d_hq, d_hsc, Sp, 0, d_tiles, max_tiles, nullptr, d_swt, 0, d_y, wd->N, 0, 0, nullptr, kWsMoe, st);
}

// ---------------------------------------------------------------------------------------------- start-up check
// Seeded data, every weight form, all store modes, a part of a column tile, and the plain store with K cut into parts and not, in this kernel and, of the
// forms it takes, in the folded one (whose rows are of all its kinds):
// tensor-core dots == CUDA-core dots bit for bit (Q4_K, Q8_0: the forms that have this mode), outputs within 1e-5 of max|ref|
// (Engine::xmx_check, zero/engine_setup.h:424-622, does the same for its XMX kernel against DP4a).
int izb_gemm_k16_launch(const izb_weight* w, const uint8_t* raw, const int8_t* aq, const float* asc, int M, int Mp, float* C, int ldc,
                        int c_off, int acc, int32_t* dots, cudaStream_t st);
namespace {
__global__ void fill_quants(int8_t* p, size_t n, uint32_t seed) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t x = (uint32_t)i * 2654435761u + seed;
  x ^= x >> 15; x *= 2246822519u; x ^= x >> 13; x *= 3266489917u; x ^= x >> 16;
  p[i] = (int8_t)((int)(x % 255u) - 127);
}
// (few_small: one of 64 is 2^-15 of that)
__global__ void fill_scales(float* p, size_t n, uint32_t seed, bool few_small) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t x = (uint32_t)i * 2654435761u + seed;
  x ^= x >> 15; x *= 2246822519u; x ^= x >> 13;
  p[i] = (0.005f + (float)(x & 0xFFFF) * (0.03f / 65535.0f)) * (few_small && (x >> 26) == 0 ? 0x1p-15f : 1.0f);
}
// out[0] = count of differing ints, out[1] = max|a-b| bits, out[2] = max|b| bits
__global__ void compare_kernel(const float* a, const float* b, size_t n, int as_int, unsigned int* out) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (as_int) {
    if (reinterpret_cast<const int*>(a)[i] != reinterpret_cast<const int*>(b)[i]) atomicAdd(&out[0], 1u);
  } else {
    const float d = fabsf(a[i] - b[i]);
    if (!(d == d)) atomicAdd(&out[0], 1u);
    atomicMax(&out[1], __float_as_uint(d == d ? d : 0.0f));
    atomicMax(&out[2], __float_as_uint(fabsf(b[i])));
  }
}
// file rows: random bytes, the fp16 factors of each superblock (Q8_0: block) between 0.0002 and 0.005
std::vector<uint8_t> seeded_rows(int type, size_t n_sb) {
  const size_t sb = type == IZB_Q4_K ? 144 : type == IZB_Q5_K ? 176 : type == IZB_Q6_K ? 210 : type == IZB_IQ4_XS ? 136 : 272;
  std::vector<uint8_t> rows(n_sb * sb);
  uint32_t x = 17u + (uint32_t)type;
  auto next = [&]() { x = x * 1664525u + 1013904223u; return x >> 16; };
  for (uint8_t& v : rows) v = (uint8_t)next();
  auto factor = [&](size_t at) {
    const unsigned short h = __half_as_ushort(__float2half(0.0002f + (float)next() * (0.0048f / 65535.0f)));
    rows[at] = (uint8_t)h;
    rows[at + 1] = (uint8_t)(h >> 8);
  };
  for (size_t i = 0; i < n_sb; ++i) {
    if (type == IZB_Q8_0) {
      for (int b = 0; b < 8; ++b) factor(i * sb + 34 * b);
    } else {
      factor(i * sb + (type == IZB_Q6_K ? 208 : 0));
      if (type == IZB_Q4_K || type == IZB_Q5_K) factor(i * sb + 2);
    }
  }
  return rows;
}
struct WeightHolder {
  izb_weight* w = nullptr;
  ~WeightHolder() { if (w) izb_weight_destroy(w); }
};

// one weight form; IZB_ERR_SELFCHECK: the kernels disagree, other errors: the check could not run
int check_form(int device, int type) {
  constexpr int M = 200, Mp = 256, N = 272, K = 2048, nb = K / 32;
  WeightHolder h;
  try {
    const std::vector<uint8_t> rows = seeded_rows(type, (size_t)N * (K / 256));
    if (int rc = izb_weight_create(type, rows.data(), 1, N, K, device, &h.w)) return rc;
  } catch (const std::exception&) {
    IZB_FAIL(IZB_ERR_NOMEM, "selfcheck: host memory for the seeded rows");
  }
  const izb_weight* w = h.w;
  if (!w->has_tmap) IZB_FAIL(IZB_ERR_SELFCHECK, "selfcheck: cannot encode a tensor map");
  const bool k16 = w->type == IZB_K16;
  auto core = [&](const int8_t* aq, const float* asc, int mp, float* C, int acc, int32_t* dots) {
    return k16 ? izb_gemm_k16_launch(w, w->raw, aq, asc, M, mp, C, N, 0, acc, dots, 0) : izb_gemm_core_launch(w, w->raw, aq, asc, M, mp, C, N, 0, acc, dots, 0);
  };
  const size_t n_out = (size_t)Mp * N, n_dots = (size_t)M * N * nb;
  void* ws = nullptr;
  if (int rc = izb_workspace(device, kWsCheck, (size_t)Mp * K + (size_t)nb * Mp * 4 + 2 * n_out * 4 + 2 * n_dots * 4 + 4096, 0, &ws)) return rc;
  int8_t* aq = (int8_t*)ws;
  float* asc = (float*)(aq + (size_t)Mp * K);
  float *c_tc = asc + (size_t)nb * Mp, *c_core = c_tc + n_out;
  int32_t *d_tc = (int32_t*)(c_core + n_out), *d_core = d_tc + n_dots;
  unsigned int* cmp = (unsigned int*)(d_core + n_dots);
  unsigned int out[3];
  auto blocks = [](size_t n) { return (unsigned)((n + 255) / 256); };
  fill_quants<<<blocks((size_t)Mp * K), 256>>>(aq, (size_t)Mp * K, 99u);
  fill_scales<<<blocks((size_t)nb * Mp), 256>>>(asc, (size_t)nb * Mp, 7u, true);
  IZB_CUDA(cudaGetLastError());
  if (!k16) {
    int rc = izb_gemm_tc_launch(w, 0, aq, nullptr, M, M, nullptr, 0, 0, 0, d_tc, 0, false);
    if (rc == 0) rc = core(aq, nullptr, M, nullptr, 0, d_core);
    if (rc != 0) return rc < 0 ? rc : IZB_ERR_SELFCHECK;
    IZB_CUDA(cudaMemset(cmp, 0, 12));
    compare_kernel<<<blocks(n_dots), 256>>>((const float*)d_tc, (const float*)d_core, n_dots, 1, cmp);
    IZB_CUDA(cudaMemcpy(out, cmp, 12, cudaMemcpyDeviceToHost));
    if (out[0]) IZB_FAIL(IZB_ERR_SELFCHECK, "selfcheck: type %d: %u block dots differ between the tensor-core and CUDA-core kernels", type, out[0]);
  }
  constexpr struct {
    const char* what;
    int acc;
    bool folded, cut;
  } modes[] = {{"plain store, K cut", 0, false, true}, {"adding store", 1, false, false}, {"SwiGLU store", 2, false, false}, {"plain store", 0, false, false},
               {"plain store, folded, K cut", 0, true, true}, {"plain store, folded", 0, true, false}};
  for (const auto& mode : modes) {
    if (mode.folded && !izb_fold_takes(w)) continue;
    const int acc = mode.acc;
    fill_scales<<<blocks(n_out), 256>>>(c_tc, n_out, 3u, false);
    fill_scales<<<blocks(n_out), 256>>>(c_core, n_out, 3u, false);
    int rc = mode.folded ? run_fold(w, 0, nullptr, 0, 0, aq, asc, Mp, M, c_tc, N, 0, 0, mode.cut)
                         : run_tc(w, 0, aq, asc, Mp, Mp, nullptr, (M + BM - 1) / BM, nullptr, nullptr, M, c_tc, N, 0, acc, nullptr, kWsGemm, 0, false, mode.cut);
    if (mode.folded && rc > 0) continue;  // (without memory for its arena: its calls go to this kernel)
    if (rc == 0) rc = core(aq, asc, Mp, c_core, acc, nullptr);
    if (rc != 0) return rc < 0 ? rc : IZB_ERR_SELFCHECK;
    IZB_CUDA(cudaMemset(cmp, 0, 12));
    compare_kernel<<<blocks(n_out), 256>>>(c_tc, c_core, n_out, 0, cmp);
    IZB_CUDA(cudaMemcpy(out, cmp, 12, cudaMemcpyDeviceToHost));
    float err, ref;
    memcpy(&err, &out[1], 4);
    memcpy(&ref, &out[2], 4);
    if (out[0] || !(err <= 1e-5f * ref))
      IZB_FAIL(IZB_ERR_SELFCHECK, "selfcheck: type %d, %s: max|err| %g vs max|ref| %g (%u NaN)", type, mode.what, err, ref, out[0]);
  }
  return IZB_OK;
}
}  // namespace

extern "C" int izb_selfcheck(int device) {
  if (izb_get_tc_ok(device) == 1) return IZB_OK;
  IZB_CUDA(cudaSetDevice(device));
  int verdict = IZB_OK;
  for (int type : {IZB_Q4_K, IZB_Q8_0, IZB_Q5_K, IZB_Q6_K, IZB_IQ4_XS}) {
    verdict = check_form(device, type);
    if (verdict != IZB_OK) break;
  }
  if (verdict != IZB_OK && verdict != IZB_ERR_SELFCHECK) {
    izb_set_tc_ok(device, 0);
    return verdict;
  }
  uint32_t word = 0;
  const int st = izb_device_status(device, &word);
  if (st != IZB_OK && verdict == IZB_OK) { verdict = st; }
  izb_set_tc_ok(device, verdict == IZB_OK ? 1 : 0);
  return verdict;
}

// ---------------------------------------------------------------------------------------------- GEMM without allocation
// izb_gemm_noalloc: the tensor-core GEMM for callers that must not allocate device memory while they run -- a serving
// loop that has handed the whole GPU to its own arena, or code that runs under an allocator it cannot re-enter.  izb_gemm keeps its activation images (the fp16 operand tiles,
// the min-term factors and the gathered scales that act_prepare_kernel writes) in an arena that grows with cudaMalloc;
// this entry point keeps them in a fixed array that is part of the library's device image instead.
//
// The array is a device symbol: in host code its name stands for the symbol, not for an address a kernel could use, so
// the address is looked up with cudaGetSymbolAddress -- once per device, with that device current -- and only that
// pointer is ever handed to a kernel.
namespace {
constexpr size_t kNoAllocBytes = IZB_NOALLOC_SCRATCH_BYTES;  // 24 MiB per GPU that loads the library, held until the process exits
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];
static __device__ __align__(256) uint32_t g_noalloc_status[64];

struct NoAllocDev {
  unsigned char* scratch = nullptr;
  uint32_t* status = nullptr;
};
NoAllocDev g_noalloc_dev[16];
std::mutex g_noalloc_mu;

// Looks the two symbols up for `device` (which must be the current device) the first time it is called for it.
int noalloc_setup(int device, NoAllocDev** out) {
  if (device < 0 || device >= 16) IZB_FAIL(IZB_ERR_ARG, "gemm_noalloc: device %d out of range", device);
  int cur = -1;
  IZB_CUDA(cudaGetDevice(&cur));
  if (cur != device) IZB_FAIL(IZB_ERR_ARG, "gemm_noalloc: device %d must be current (current is %d)", device, cur);
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  NoAllocDev& d = g_noalloc_dev[device];
  if (!d.scratch) {
    void* p = nullptr;
    void* s = nullptr;
    IZB_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    IZB_CUDA(cudaGetSymbolAddress(&s, g_noalloc_status));
    d.status = (uint32_t*)s;
    d.scratch = (unsigned char*)p;
    izb_note_noalloc_status(device, d.status);  // izb_device_status reads (and clears) this word too
  }
  *out = &d;
  return IZB_OK;
}
}  // namespace

extern "C" int izb_gemm_noalloc(const izb_weight* w, int mat, const int8_t* d_aq, const float* d_asc, int M, int Mp, float* d_C,
                                int ldc, int c_off, int acc, uint32_t* d_status, void* stream) {
  if (!w || !d_aq || !d_asc || !d_C) IZB_FAIL(IZB_ERR_ARG, "gemm_noalloc: null pointer");
  if (mat < 0 || mat >= w->n_mats) IZB_FAIL(IZB_ERR_ARG, "gemm_noalloc: matrix %d of %d", mat, w->n_mats);
  if (acc < 0 || acc > 3 || (acc == 3 && !w->gu32)) IZB_FAIL(IZB_ERR_ARG, "gemm_noalloc: store mode %d", acc);
  if (Mp % 16 || w->N % BN || w->K % 256 || M < 1 || M > Mp)
    IZB_FAIL(IZB_ERR_SHAPE, "gemm_noalloc: M=%d Mp=%d N=%d K=%d (need Mp %% 16, N %% 128, K %% 256, 1 <= M <= Mp)", M, Mp, w->N, w->K);
  if (c_off < 0 || ldc < c_off + (acc == 3 ? w->N / 2 : w->N))
    IZB_FAIL(IZB_ERR_SHAPE, "gemm_noalloc: ldc = %d < c_off + output columns = %d", ldc, c_off + (acc == 3 ? w->N / 2 : w->N));
  if (!izb_aligned(d_aq, 16) || !izb_aligned(d_asc, 16) || !izb_aligned(d_C, 16) || ldc % 4 || c_off % 4 || (d_status && !izb_aligned(d_status, 4)))
    IZB_FAIL(IZB_ERR_ALIGN, "gemm_noalloc: aq, asc, C must be 16-byte aligned, ldc and c_off multiples of 4");
  if (w->type == IZB_K16) IZB_FAIL(IZB_ERR_TYPE, "gemm_noalloc: ggml type %d is not taken by the tensor-core kernel", w->ggml_type);
  if (!w->has_tmap) IZB_FAIL(IZB_ERR_CUDA, "gemm_noalloc: the weight has no tensor map (driver entry point missing at creation)");
  const int K = w->K;
  const int n_tiles = (M + BM - 1) / BM;
  const int sps = w->type == IZB_Q4_K ? 5 : 4;
  size_t img_bytes, asc_bytes;
  tc_scratch_bytes(n_tiles, K, sps, &img_bytes, &asc_bytes);
  if (img_bytes + asc_bytes > kNoAllocBytes || n_tiles > 65535)
    IZB_FAIL(IZB_ERR_LIMIT, "gemm_noalloc: M=%d K=%d needs %zu scratch bytes, the fixed array holds %zu (use izb_gemm, or fewer rows per call)",
             M, K, img_bytes + asc_bytes, kNoAllocBytes);
  NoAllocDev* dev = nullptr;
  if (int rc = noalloc_setup(w->device, &dev)) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  // Everything the GEMM reads from the array is rewritten by the pre-pass of the same call (all rows of all its tiles,
  // padding rows as zeros), so nothing stale from an earlier call is ever read; the status word is the one thing that
  // must start at zero.
  uint32_t* status = d_status ? d_status : dev->status;
  IZB_CUDA(cudaMemsetAsync(status, 0, 4, st));
  return run_tc_on(w, mat, d_aq, d_asc, Mp, Mp, nullptr, n_tiles, nullptr, nullptr, M, d_C, ldc, c_off, acc, nullptr, dev->scratch, nullptr, status,
                   st, false);
}

