// out[M,N] = x[M,K] * w[N,K]^T on the CUDA cores with 32-bit multiply-adds: the
// true 32-bit matrix product (no tensor-core mode of reduced precision), also
// usable with bfloat16 operands as the plain stand-in of the tensor-core kernel.
// Every output element is one chain of fused multiply-adds over k = 0..K-1 in
// order, so a row's result does not depend on which other rows are in the batch.
#include "api.h"
#include "common.cuh"
#include "gemm_f32_tiles.cuh"
#include "gemm_internal.h"

namespace {
constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

template <typename TX, typename TW, typename TO>
__global__ void __launch_bounds__(256) gemm_simt_kernel(TO* __restrict__ out, const TX* __restrict__ x,
                                                        const TW* __restrict__ w, int M, int N, int K, int ldx,
                                                        int ldw, int ldo) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float xs[BK][BM + 4];
  __shared__ float ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid % 16, ty = tid / 16;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    // each thread loads 4 elements of each tile: row = e / BK, k = e % BK
#pragma unroll
    for (int e = tid; e < BM * BK; e += 256) {
      const int r = e / BK, kk = e % BK;
      const int m = m0 + r, k = k0 + kk;
      xs[kk][r] = (m < M && k < K) ? to_f32(x[(size_t)m * ldx + k]) : 0.f;
    }
#pragma unroll
    for (int e = tid; e < BN * BK; e += 256) {
      const int r = e / BK, kk = e % BK;
      const int n = n0 + r, k = k0 + kk;
      ws[kk][r] = (n < N && k < K) ? to_f32(w[(size_t)n * ldw + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = xs[kk][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = ws[kk][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty * TM + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx * TN + j;
      if (n < N) out[(size_t)m * ldo + n] = from_f32<TO>(acc[i][j]);
    }
  }
}

template <typename TX, typename TW, typename TO>
int launch(void* out, const void* x, const void* w, int M, int N, int K, int ldx, int ldw, int ldo,
           cudaStream_t stream) {
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  zi_launch(gemm_simt_kernel<TX, TW, TO>, dim3(grid), dim3(256), 0, stream, (TO*)out, (const TX*)x, (const TW*)w, M, N, K, ldx, ldw, ldo);
  return zi_check_launch("gemm_simt");
}

// ------------------------------------------------------------------ batched and grouped forms
// The same product with three additions, for block-diagonal gates, per-head projections and the
// experts of a mixture:
//   batch    blockIdx.z picks one of `batch` independent products whose operands lie sx, sw, so
//            (and sb for the bias) elements apart;
//   groups   every tile of TM*16 output rows names the weight group (expert) it multiplies with in
//            tile_group[], groups lie group_stride elements apart, the x row of an output row comes
//            from row_src[] (a gather; -1: no row, nothing is stored), and tiles at or beyond
//            *n_tiles_dev do nothing: the sizes are known on the device only;
//   epilogue an optional bias per output column, then ZI_EPI_NONE or ZI_EPI_RELU2 (the square of relu).
// Every output is still one chain of fused multiply-adds over k in order.
template <typename TX, typename TW, typename TO, int TM_>
__global__ void __launch_bounds__(256)
gemm_simt_general_kernel(TO* __restrict__ out, const TX* __restrict__ x, const TW* __restrict__ w, int M, int N, int K,
                         int ldx, int ldw, int ldo, long long sx, long long sw, long long so,
                         const float* __restrict__ bias, long long sb, const int* __restrict__ row_src,
                         const int* __restrict__ tile_group, const int* __restrict__ n_tiles_dev,
                         long long group_stride, int epilogue) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int BM_ = 16 * TM_;
  __shared__ float xs[BK][BM_ + 4];
  __shared__ float ws[BK][BN + 4];
  __shared__ int src_rows[BM_];
  if (n_tiles_dev && (int)blockIdx.y >= *n_tiles_dev) return;
  const int tid = threadIdx.x;
  const int tx = tid % 16, ty = tid / 16;
  const int m0 = blockIdx.y * BM_, n0 = blockIdx.x * BN;
  x += (size_t)blockIdx.z * sx;
  w += (size_t)blockIdx.z * sw;
  out += (size_t)blockIdx.z * so;
  if (bias) bias += (size_t)blockIdx.z * sb;
  if (tile_group) {
    const int e = tile_group[blockIdx.y];
    w += (size_t)e * group_stride;
    if (bias) bias += (size_t)e * N;
  }
  if (tid < BM_) {
    const int m = m0 + tid;
    src_rows[tid] = m < M ? (row_src ? row_src[m] : m) : -1;
  }
  __syncthreads();
  float acc[TM_][TN];
#pragma unroll
  for (int i = 0; i < TM_; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    for (int e = tid; e < BM_ * BK; e += 256) {
      const int r = e / BK, kk = e % BK;
      const int src = src_rows[r], k = k0 + kk;
      xs[kk][r] = (src >= 0 && k < K) ? to_f32(x[(size_t)src * ldx + k]) : 0.f;
    }
#pragma unroll
    for (int e = tid; e < BN * BK; e += 256) {
      const int r = e / BK, kk = e % BK;
      const int n = n0 + r, k = k0 + kk;
      ws[kk][r] = (n < N && k < K) ? to_f32(w[(size_t)n * ldw + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM_], b[TN];
#pragma unroll
      for (int i = 0; i < TM_; ++i) a[i] = xs[kk][ty * TM_ + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = ws[kk][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM_; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM_; ++i) {
    const int m = m0 + ty * TM_ + i;
    if (m >= M || src_rows[ty * TM_ + i] < 0) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx * TN + j;
      if (n >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[n];
      if (epilogue == ZI_EPI_RELU2) {
        v = fmaxf(v, 0.f);
        v *= v;
      }
      out[(size_t)m * ldo + n] = from_f32<TO>(v);
    }
  }
}

template <typename TX, typename TW, typename TO>
int launch_general(void* out, const void* x, const void* w, int M, int N, int K, int ldx, int ldw, int ldo, int batch,
                   long long sx, long long sw, long long so, const float* bias, long long sb, const int* row_src,
                   const int* tile_group, const int* n_tiles_dev, long long group_stride, int epilogue, int small_tiles,
                   cudaStream_t stream) {
  const int bm = small_tiles ? 16 : 64;
  dim3 grid((N + BN - 1) / BN, (M + bm - 1) / bm, batch);
  if (small_tiles)
    zi_launch(gemm_simt_general_kernel<TX, TW, TO, 1>, dim3(grid), dim3(256), 0, stream, (TO*)out, (const TX*)x, (const TW*)w,
              M, N, K, ldx, ldw, ldo, sx, sw, so, bias, sb, row_src, tile_group, n_tiles_dev, group_stride, epilogue);
  else
    zi_launch(gemm_simt_general_kernel<TX, TW, TO, 4>, dim3(grid), dim3(256), 0, stream, (TO*)out, (const TX*)x, (const TW*)w,
              M, N, K, ldx, ldw, ldo, sx, sw, so, bias, sb, row_src, tile_group, n_tiles_dev, group_stride, epilogue);
  return zi_check_launch("gemm_simt (batched or grouped)");
}
}  // namespace

extern "C" int zi_gemm_simt_general(void* out, int out_dtype, const void* x, int x_dtype, const void* w, int w_dtype,
                                    int M, int N, int K, int ldx, int ldw, int ldo, int batch, long long sx,
                                    long long sw, long long so, const float* bias, long long sb, const int* row_src,
                                    const int* tile_group, const int* n_tiles_dev, long long group_stride,
                                    int epilogue, int tile_rows, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || batch <= 0) return 0;
  if (K <= 0) return zi_refuse("gemm: K must be positive, got %d", K);
  if (tile_rows != 16 && tile_rows != 64) return zi_refuse("gemm: tiles have 16 or 64 rows, not %d", tile_rows);
  if (batch > 65535) return zi_refuse("gemm: at most 65535 products in a batch, got %d", batch);
  if (epilogue != ZI_EPI_NONE && epilogue != ZI_EPI_RELU2) return zi_refuse("gemm: unknown epilogue %d", epilogue);
  using bf = __nv_bfloat16;
  const int small = tile_rows == 16;
#define ZI_GENERAL(TX, TW, TO)                                                                                     \
  return launch_general<TX, TW, TO>(out, x, w, M, N, K, ldx, ldw, ldo, batch, sx, sw, so, bias, sb, row_src, tile_group, \
                                    n_tiles_dev, group_stride, epilogue, small, stream)
  const int key = x_dtype * 4 + w_dtype * 2 + out_dtype;
  switch (key) {
    case 0: ZI_GENERAL(float, float, float);
    case 1: ZI_GENERAL(float, float, bf);
    case 2: ZI_GENERAL(float, bf, float);
    case 3: ZI_GENERAL(float, bf, bf);
    case 4: ZI_GENERAL(bf, float, float);
    case 5: ZI_GENERAL(bf, float, bf);
    case 6: ZI_GENERAL(bf, bf, float);
    case 7: ZI_GENERAL(bf, bf, bf);
  }
#undef ZI_GENERAL
  return zi_refuse("gemm: unknown dtype tags x=%d w=%d out=%d", x_dtype, w_dtype, out_dtype);
}

namespace {
// 32-bit operands whose rows start on 16-byte boundaries: which tile (gemm_f32_tiles.cuh).  The line between the tiles is
// how many blocks they make: a chain of K multiply-adds per output cannot be split, so a product is as fast as its
// blocks fill the 148 SMs, and the larger a thread's tile the fewer bytes of shared memory it reads per multiply-add
// (128 bytes a clock and SM feed 4 x 4 outputs a thread at about a third of the multiply-adds' rate, 8 x 8 at half).
// Measured, us on one B200 (rows x columns x K; the plain kernel -> the tile taken; every output's bits are the same):
//   1 x 1024 x 1024  106 -> 5.4      12 x 1024 x 1024  106 -> 8.5     12 x 6144 x 1024  126 -> 14.2   12 x 1024 x 3072  311 -> 21.7
//   30 x 1024 x 1024  11.4           100 x 1024 x 1024  26            512 x 1024 x 1024  101 -> 41    512 x 6144 x 1024  336 -> 187
// The lines lie where a tile's blocks no longer are all resident at once (three an SM of the 16 x 8 and 16 x 16 tiles, four of
// the 64 x 64): 12 x 3072 x 1024 in tiles of 8 | 16 | 32 columns 9.5 | 13.9 | 21, x 3600 15.3 | 14.0 | 20.9, x 7104 19.2 | 15.2 | 16.9,
// x 7500 24.6 | 28.2 | 22.5, x 11840 36.0 | 29.2 | 23.3; 3 x 4096 x 1024 in tiles of 8 | 32 7.1 | 9.8, x 6144 12.2 | 9.7; 24 x 2048 x
// 1024 in tiles of 8 | 16 11.6 | 21.8, x 3072 22.5 | 22.4; 100 x 1024 x 1024 in 32 x 32 tiles 38.  In 32 x 32 | 64 x 64 tiles:
// 512 x 2816 x 1024 106 | 118, 512 x 3072 x 1024 120 | 118, 512 x 4608 x 1024 161 | 118, 300 x 6144 x 1024 144 | 118, 512 x 5632 x 1024
// 200 | 187, 512 x 6144 x 1024 222 | 187, 512 x 1024 x 3072 120 | 342.
constexpr int SMS = 148;
template <typename TO>
int launch_f32(void* out, const float* x, const float* w, int M, int N, int K, int ldx, int ldw, int ldo, int early,
               cudaStream_t stream) {
  const long long blocks32 = (long long)((M + 31) / 32) * ((N + 31) / 32), blocks64 = (long long)((M + 63) / 64) * ((N + 63) / 64);
  if (K % 4 == 0 && (M <= 32 || blocks32 <= SMS)) {
    int* status = zi_internal_status_word();
    if (!status) return zi_refuse("gemm: no device memory for the status word");
#define ZI_FEW(...) return launch_f32_few<F32Few<__VA_ARGS__>, TO>(out, x, w, M, N, K, ldx, ldw, ldo, early, status, stream)
    if (M <= 4) {
      if (N < 32 * SMS) ZI_FEW(4, 8, 1, 1, 256, 4, 7);
      ZI_FEW(4, 32, 2, 1, 128, 4, 7);
    }
    if (M <= 16) {
      if (N <= 24 * SMS) ZI_FEW(16, 8, 2, 1, 256, 3, 3);
      if (N <= 48 * SMS) ZI_FEW(16, 16, 2, 2, 128, 4, 3);
      ZI_FEW(16, 32, 2, 2, 128, 3, 3);
    }
    if (M <= 32) {
      if (N <= 16 * SMS) ZI_FEW(32, 8, 2, 1, 256, 2, 3);
      ZI_FEW(32, 16, 2, 2, 128, 3, 3);
    }
    ZI_FEW(32, 16, 4, 2, 128, 3, 3);
#undef ZI_FEW
  }
  // 64 x 64 tiles: one round of four an SM takes as long as 32 x 32 tiles of 10 an SM; past it they pay again from 4.6 an SM on
  if (blocks64 > 4 * SMS ? 10 * blocks64 >= 46 * SMS : blocks32 > 10 * SMS) return launch_f32_tile<F32Tile<64, 64, 8, 8, 32, 3, 1>, TO>(out, x, w, M, N, K, ldx, ldw, ldo, early, stream);
  return launch_f32_tile<F32Tile<32, 32, 4, 4, 64, 3, 2>, TO>(out, x, w, M, N, K, ldx, ldw, ldo, early, stream);
}
}  // namespace

// early_weights: w is not written by a kernel of this step, so that its first rows may be asked for before the wait for
// the kernels before this one.
extern "C" int zi_gemm_simt(void* out, int out_dtype, const void* x, int x_dtype, const void* w, int w_dtype, int M,
                            int N, int K, int ldx, int ldw, int ldo, int early_weights, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return zi_refuse("gemm: K must be positive, got %d", K);
  using bf = __nv_bfloat16;
  const int key = x_dtype * 4 + w_dtype * 2 + out_dtype;
  // the tiles' grids count rows in blockIdx.y: at most 65,535 blocks of 32
  if ((key == 0 || key == 1) && ((uintptr_t)x | (uintptr_t)w) % 16 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && M <= 65535 * 32) {
    if (key == 0) return launch_f32<float>(out, (const float*)x, (const float*)w, M, N, K, ldx, ldw, ldo, early_weights, stream);
    return launch_f32<bf>(out, (const float*)x, (const float*)w, M, N, K, ldx, ldw, ldo, early_weights, stream);
  }
  switch (key) {
    case 0: return launch<float, float, float>(out, x, w, M, N, K, ldx, ldw, ldo, stream);
    case 1: return launch<float, float, bf>(out, x, w, M, N, K, ldx, ldw, ldo, stream);
    case 2: return launch<float, bf, float>(out, x, w, M, N, K, ldx, ldw, ldo, stream);
    case 3: return launch<float, bf, bf>(out, x, w, M, N, K, ldx, ldw, ldo, stream);
    case 4: return launch<bf, float, float>(out, x, w, M, N, K, ldx, ldw, ldo, stream);
    case 5: return launch<bf, float, bf>(out, x, w, M, N, K, ldx, ldw, ldo, stream);
    case 6: return launch<bf, bf, float>(out, x, w, M, N, K, ldx, ldw, ldo, stream);
    case 7: return launch<bf, bf, bf>(out, x, w, M, N, K, ldx, ldw, ldo, stream);
  }
  return zi_refuse("gemm: unknown dtype tags x=%d w=%d out=%d", x_dtype, w_dtype, out_dtype);
}

ZI_TRACE_SETTER(gemm_simt)
