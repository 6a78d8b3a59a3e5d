// Decode GEMV for 1..8 activation rows: C[t][n] (+)= sum_b asc[b][t] * f(block b of row n), weights read once.
// Bandwidth-bound: no tensor cores; 128-bit streaming weight loads, nibble unpack in registers, dp4a, one warp shuffle
// reduction per output.  Arithmetic of zero/kernels/decode.cl gemv (:913-1034) and gemv_mt (:1581-1694):
//   Q4_K  term = sa * (d * (float)(sc * dot) - dmin * (float)(mn * asum))
//   Q8_0  term = sa * d * (float)dot
// with dot / asum exact int32.  A lane holds a 16-element half of a block, so it adds the term of its half; the sum
// over lanes is a different order of the same f32 terms (the reference leaves that order unspecified as well).
//
// Work split: a warp owns kRows consecutive weight rows for the whole K; the 32 lanes cover 512 weight bytes per step
// (Q4_K: the nibbles of 4 superblocks, lane -> superblock lane/8, 16-byte piece lane%8; Q8_0: 2 superblocks, lane ->
// superblock lane/16, piece lane%16).  The CTA first stages the T activation rows in shared memory, permuted so that
// every lane's operands are one conflict-free 128-bit read, with the per-lane block scales and (Q4_K) the sums of the
// 16 int8 values each lane pairs with a min.
#include "izb_gemv_body.cuh"

int izb_gemv_k16_launch(const izb_weight* w, const uint8_t* raw, const int8_t* aq, const float* asc, int T, int Mp, float* C, int ldc,
                        int c_off, int acc, cudaStream_t st);
int izb_gemv_stream_launch(const izb_weight* w, const uint8_t* raw, const int8_t* aq, const float* asc, int T, int Mp, float* C,
                           int ldc, int c_off, int acc, cudaStream_t st);

bool izb_gemv_stream_fits(const izb_weight* w, int T);
int izb_rows_launch(const izb_weight* w, int mat, const int8_t* aq, const float* asc, int T, int Mp, float* C, int ldc, int c_off, int acc, cudaStream_t st);

namespace {
using namespace izb_gemvk;

template <int QT, int T>
__global__ void __launch_bounds__(kWarps * 32) gemv_kernel(const uint8_t* __restrict__ raw, int N, int K,
                                                           const int8_t* __restrict__ aq, const float* __restrict__ asc, int Mp,
                                                           float* __restrict__ C, int ldc, int c_off, int acc, int spc) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int tok[T];
  if (threadIdx.x < T) tok[threadIdx.x] = threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row0 = (blockIdx.x * kWarps + warp) * kRows;
  float accv[kRows][T];
#pragma unroll
  for (int r = 0; r < kRows; ++r)
#pragma unroll
    for (int t = 0; t < T; ++t) accv[r][t] = 0.0f;
  gemv_body<QT, T>(smem, raw, N, K, aq, asc, Mp, tok, row0, spc, accv);
#pragma unroll
  for (int r = 0; r < kRows; ++r)
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const float v = warp_sum(accv[r][t]);
      const int n = row0 + r;
      if (lane == 0 && n < N) {
        float* c = C + (size_t)t * ldc + c_off + n;
        *c = acc ? *c + v : v;
      }
    }
}

template <int QT, int T>
int launch_qt(const izb_weight* w, const uint8_t* raw, const int8_t* aq, const float* asc, int Mp, float* C, int ldc, int c_off,
              int acc, cudaStream_t st) {
  const int grid = (w->N + kWarps * kRows - 1) / (kWarps * kRows);
  size_t smem = 0;
  const int spc = steps_per_chunk(QT, w->K, T, &smem);
  IZB_SMEM_OPTIN((gemv_kernel<QT, T>), kMaxSmem, w->device);
  IZB_LAUNCH("gemv", st, gemv_kernel<QT, T><<<grid, kWarps * 32, smem, st>>>(raw, w->N, w->K, aq, asc, Mp, C, ldc, c_off, acc, spc));
  return IZB_OK;
}

template <int T>
int launch(const izb_weight* w, const uint8_t* raw, const int8_t* aq, const float* asc, int Mp, float* C, int ldc, int c_off,
           int acc, cudaStream_t st) {
  return w->type == IZB_Q4_K ? launch_qt<IZB_Q4_K, T>(w, raw, aq, asc, Mp, C, ldc, c_off, acc, st)
                             : launch_qt<IZB_Q8_0, T>(w, raw, aq, asc, Mp, C, ldc, c_off, acc, st);
}

// Which of the two ways to the same bits is faster: the matrix instruction's cost does not grow with T but at T = 5, the dot-product kernels' does.
// Measured (us, matrix instruction / dot products, calls back to back with weights that are not in L2; five rows and more behind a quantiser):
//   Q6_K  32000 x 4096 T=1 22/27, T=4 24/52, T=8 38/95; 1024 x 1024 T=1 2.3/2.7, 5120 x 17408 T=1 19/27.  Few row tiles leave most of the chip idle
//         over a long K: 256 x 8192 T=1 5.8/4.9, T=4 6.9/6.4, 256 x 4096 T=1 3.6/3.2, T=2 3.7/3.8, 384 x 8192 T=1 5.8/7.0; 128 x 8192 T=5 11/11, 48 x
//         4096 T=5 7.3/7.9
//   Q4_K  rows that are too long for the dot product's ring: 1024 x 10496 T=1 8.0/13, 4096 x 9472 T=1 8.6/8.2 (fits), T=2 9.4/14, 512 x 12544 T=4 10/14;
//         T = 1 pays in a middle range: 12288 x 2304 7.6/8.3, 12288 x 3840 9.3/10.7, 24576 x 3840 15.3/16.4, 24576 x 5376 21.1/20.2, 8192 x 2816 7.7/6.1;
//         T = 2: 5120 x 1280 3.6/4.0, 5120 x 5376 7.3/8.3, 4096 x 1280 3.5/3.2, 4096 x 2816 4.5/4.4, 4096 x 5376 7.0/6.8, 4096 x 6912 7.1/7.7, 3072 x 8448 8.5/8.2;
//         T = 3: 4096 x 2304 4.4/4.8, 3072 x 2816 4.7/4.5; T = 4: 2560 x 2304 4.4/5.1, 2048 x 2304 3.9/3.5; T >= 5: 1024 x 2048 T=8 4.1/4.2, 34816 x 5120 T=5
//         34/52, T=8 35/76
//         (at up to four rows the kernels for K % 1024 == 0 add in another order: theirs stays)
//   Q8_0  rows that are too long for the ring: 512 x 8192 T=1 7.5/13, T=8 13/21, 1024 x 6144 T=4 7.0/13, 2048 x 5120 T=4 6.7/11; else many row tiles, and while
//         latency, not the copy's rate, is what both take their time for: T = 1 131072 x 1536 35/39, 65536 x 2048 23.5/23.5, 131072 x 2048 45/43, 20480 x
//         2560 10.3/10.9, 32768 x 2560 15.7/15.1, 5120 x 2560 4.4/4.5, 4096 x 2048 3.7/3.3; T = 2: 131072 x 2048 46/50, 32768 x 3072 18.9/19.5 (102 MiB of weights),
//         65536 x 3072 35/34, 16384 x 4096 12.7/13.4 (68), 32768 x 4096 24/23 (136), 24576 x 4352 20.0/20.3 (108), 24576 x 4608 20.8/20.6 (115), 6144 x 4096
//         6.8/6.8; T = 3: 131072 x 5120 112/115, 4096 x 5120 7.2/7.5, 3072 x 4096 5.8/5.6; T = 4: 3072 x 2048 3.6/4.0, 2048 x 1024 2.5/2.3; T >= 5 (a warp holds
//         twice the sums): 1024 x 3072 T=8 6.4/5.0, 4096 x 4096 T=8 8.3/12
bool rows_first(const izb_weight* w, int T) {
  const int N = w->N, K = w->K;
  if (w->type == IZB_K16) return T > 4 ? N >= 128 || K < 8192 : N > 256 || K <= (T == 1 ? 2048 : 4096);
  if (w->type == IZB_Q4_K && T <= 4 && K % 1024 == 0 && N >= 1024) return false;
  if (T > 4 && w->type == IZB_Q4_K) return true;
  if (!izb_gemv_stream_fits(w, T)) return N >= 512;
  if (w->type == IZB_Q4_K)
    return T == 1 ? N >= 12288 && K <= 3840 : T == 2 ? N >= (K <= 6400 ? 5120 : 4096) : N >= (T == 3 ? 4096 : 2560);
  switch (T) {
    case 1: return N >= 5120 && (K <= 1536 || (K <= 2048 && N <= 65536) || (K <= 2560 && N <= 24576));
    case 2: return N >= 6144 && (K <= 2560 || (size_t)N * w->row_bytes <= (size_t)108 << 20);
    case 3: return N >= 4096;
    case 4: return N >= 3072;
    default: return N >= 4096;
  }
}

}  // namespace
extern "C" int izb_gemv(const izb_weight* w, int mat, const int8_t* d_aq, const float* d_asc, int T, int Mp, float* d_C,
                        int ldc, int c_off, int acc, void* stream) {
  if (!w || !d_aq || !d_asc || !d_C) IZB_FAIL(IZB_ERR_ARG, "gemv: null pointer");
  if (mat < 0 || mat >= w->n_mats) IZB_FAIL(IZB_ERR_ARG, "gemv: matrix %d of %d", mat, w->n_mats);
  if (T < 1 || T > 8) IZB_FAIL(IZB_ERR_SHAPE, "gemv: T = %d outside 1..8", T);
  if (Mp < T) IZB_FAIL(IZB_ERR_SHAPE, "gemv: Mp = %d < T = %d", Mp, T);
  if (acc != 0 && acc != 1) IZB_FAIL(IZB_ERR_ARG, "gemv: store mode %d (the GEMV stores or adds, zero/kernels/decode.cl:1031)", acc);
  if (ldc < c_off + w->N && T > 1) IZB_FAIL(IZB_ERR_SHAPE, "gemv: ldc = %d < c_off + N = %d", ldc, c_off + w->N);
  if (!izb_aligned(d_aq, 16)) IZB_FAIL(IZB_ERR_ALIGN, "gemv: aq not 16-byte aligned");
  if (int rc = izb_require_device(w->device, "gemv")) return rc;
  const uint8_t* raw = w->raw + (size_t)mat * w->N * w->row_bytes;
  cudaStream_t st = (cudaStream_t)stream;
  if (rows_first(w, T)) {
    const int rc = izb_rows_launch(w, mat, d_aq, d_asc, T, Mp, d_C, ldc, c_off, acc, st);
    if (rc <= 0) return rc;
  }
  if (w->type == IZB_K16) return izb_gemv_k16_launch(w, raw, d_aq, d_asc, T, Mp, d_C, ldc, c_off, acc, st);
  {  // the streaming kernel takes every call whose staged activations fit in shared memory
    const int rc = izb_gemv_stream_launch(w, raw, d_aq, d_asc, T, Mp, d_C, ldc, c_off, acc, st);
    if (rc <= 0) return rc;
  }
  switch (T) {
    case 1: return launch<1>(w, raw, d_aq, d_asc, Mp, d_C, ldc, c_off, acc, st);
    case 2: return launch<2>(w, raw, d_aq, d_asc, Mp, d_C, ldc, c_off, acc, st);
    case 3: return launch<3>(w, raw, d_aq, d_asc, Mp, d_C, ldc, c_off, acc, st);
    case 4: return launch<4>(w, raw, d_aq, d_asc, Mp, d_C, ldc, c_off, acc, st);
    case 5: return launch<5>(w, raw, d_aq, d_asc, Mp, d_C, ldc, c_off, acc, st);
    case 6: return launch<6>(w, raw, d_aq, d_asc, Mp, d_C, ldc, c_off, acc, st);
    case 7: return launch<7>(w, raw, d_aq, d_asc, Mp, d_C, ldc, c_off, acc, st);
    default: return launch<8>(w, raw, d_aq, d_asc, Mp, d_C, ldc, c_off, acc, st);
  }
}
