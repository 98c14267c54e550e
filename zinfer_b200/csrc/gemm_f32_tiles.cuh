// The 32-bit product out[M,N] = x[M,K] * w[N,K]^T for float operands whose rows start on 16-byte boundaries, in tiles
// from 4 x 8 (single tokens) to 64 x 64 (prompts).  As in the plain kernel every output is ONE chain of fused
// multiply-adds over k = 0..K-1 in order, so the tile that computes it does not show in its bits.
#pragma once
#include "common.cuh"
#include "tcgen05_ptx.cuh"

namespace {

// 16 bytes from global to shared memory without passing through registers; bytes past `valid` are filled with zeros.
__device__ __forceinline__ void f32_copy16(float* dst, const float* src, int valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(valid)
               : "memory");
}

template <int BM_, int BN_, int TM_, int TN_, int KC_, int STAGES_, int UNROLL_>
struct F32Tile {
  static constexpr int BM = BM_, BN = BN_, TM = TM_, TN = TN_, KC = KC_, STAGES = STAGES_, UNROLL = UNROLL_;
  static constexpr int THREADS = (BM / TM) * (BN / TN);
  static constexpr int PITCH = KC + 4;           // rows 4 banks apart: eight threads' 16-byte reads of eight rows meet no bank twice
  static constexpr int STAGE = (BM + BN) * PITCH;
  static constexpr size_t SMEM = (size_t)STAGES * STAGE * sizeof(float);
};

// One 16-byte piece along k of a thread's rows of both operands, and its multiply-adds.
template <int TM, int TN>
struct F32Piece {
  float4 a[TM], b[TN];
  template <int GAP_A, int GAP_B>
  __device__ __forceinline__ void read(const float* xs, const float* ws, int p) {
#pragma unroll
    for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(xs + i * GAP_A + p * 4);
#pragma unroll
    for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4*>(ws + j * GAP_B + p * 4);
  }
  __device__ __forceinline__ void multiply(float (&acc)[TM][TN]) const {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
  }
};

// A chunk's pieces (all PIECES of it, or fewer at the end of K) in turn, each read AHEAD pieces before its use: with a warp or
// two a scheduler nothing else hides a shared-memory read's latency, about ten multiply-adds of a chain.
template <int TM, int TN, int GAP_A, int GAP_B, int PIECES, int AHEAD>
__device__ __forceinline__ void f32_chunk(float (&acc)[TM][TN], const float* xs, const float* ws, int pieces) {
  constexpr int RING = AHEAD + 1;
  static_assert(PIECES % RING == 0 && PIECES >= RING, "a chunk is a whole number of rings");
  F32Piece<TM, TN> ring[RING];
  if (pieces == PIECES) {
#pragma unroll
    for (int d = 0; d < AHEAD; ++d) ring[d].template read<GAP_A, GAP_B>(xs, ws, d);
#pragma unroll 1
    for (int p = 0; p < PIECES - RING; p += RING) {
#pragma unroll
      for (int d = 0; d < RING; ++d) {
        ring[(d + AHEAD) % RING].template read<GAP_A, GAP_B>(xs, ws, p + d + AHEAD);
        ring[d].multiply(acc);
      }
    }
    ring[AHEAD].template read<GAP_A, GAP_B>(xs, ws, PIECES - 1);
#pragma unroll
    for (int d = 0; d < RING; ++d) ring[d].multiply(acc);
  } else {
    for (int p = 0; p < pieces; ++p) {
      ring[0].template read<GAP_A, GAP_B>(xs, ws, p);
      ring[0].multiply(acc);
    }
  }
}

// The same for the larger tiles, each piece read one ahead of its use (512 x 6144 x 1024 195 -> 187 us; with the ring above 189,
// and 512 x 1024 x 3072 125 instead of 120).
template <int TM, int TN, int GAP_A, int GAP_B, int PIECES, int UNROLL>
__device__ __forceinline__ void f32_chunk_pairs(float (&acc)[TM][TN], const float* xs, const float* ws, int pieces) {
  F32Piece<TM, TN> even, odd;
  if (pieces == PIECES) {
    even.template read<GAP_A, GAP_B>(xs, ws, 0);
#pragma unroll UNROLL
    for (int p = 0; p < PIECES; p += 2) {
      odd.template read<GAP_A, GAP_B>(xs, ws, p + 1);
      even.multiply(acc);
      if (p + 2 < PIECES) even.template read<GAP_A, GAP_B>(xs, ws, p + 2);
      odd.multiply(acc);
    }
  } else {
    for (int p = 0; p < pieces; ++p) {
      even.template read<GAP_A, GAP_B>(xs, ws, p);
      even.multiply(acc);
    }
  }
}

// Bound by shared memory: a 16-byte read by a warp takes four of the SM's 128-byte clocks whatever the addresses, so the
// plain kernel's one-word reads left the multiply-adds idle most of the time (512 x 6144 x 1024: 336 us, 19 TFLOP/s; now
// 187 us, 34, of the 69 that independent chains of fmaf reach here).  A ring of STAGES chunks of KC columns, filled by
// cp.async; a thread owns TM x TN outputs, rows BM / TM and columns BN / TN apart, and reads both operands as 16-byte pieces along k.  `early`: w is not written by a kernel of this
// step, so its first chunks are requested before the wait for the kernels before this one.
template <typename T, typename TO>
__global__ void __launch_bounds__(T::THREADS)
gemm_f32_tile_kernel(TO* __restrict__ out, const float* __restrict__ x, const float* __restrict__ w, int M, int N, int K,
                     int ldx, int ldw, int ldo, int early) {
  constexpr int BM = T::BM, BN = T::BN, TM = T::TM, TN = T::TN, KC = T::KC, STAGES = T::STAGES, THREADS = T::THREADS;
  constexpr int PITCH = T::PITCH, PIECES = KC / 4, ROWS_M = BM / TM, ROWS_N = BN / TN;
  pdl_launch_dependents();
  extern __shared__ __align__(16) float f32_smem[];
  const int tid = threadIdx.x, tx = tid % ROWS_N, ty = tid / ROWS_N;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int chunks = (K + KC - 1) / KC;

  auto fill = [&](float* dst, const float* src, int rows, int row0, int limit, int ld, int c) {
    for (int e = tid; e < rows * PIECES; e += THREADS) {
      const int r = e / PIECES, k = c * KC + (e % PIECES) * 4;
      const int valid = row0 + r < limit ? min(max(K - k, 0), 4) * 4 : 0;
      f32_copy16(dst + r * PITCH + (e % PIECES) * 4, valid ? src + (size_t)(row0 + r) * ld + k : src, valid);
    }
  };
  auto fill_w = [&](int c) { fill(f32_smem + (c % STAGES) * T::STAGE + BM * PITCH, w, BN, n0, N, ldw, c); };
  auto fill_x = [&](int c) { fill(f32_smem + (c % STAGES) * T::STAGE, x, BM, m0, M, ldx, c); };

  const int ahead = min(STAGES - 1, chunks);
  if (early)
    for (int c = 0; c < ahead; ++c) fill_w(c);
  pdl_wait();
  for (int c = 0; c < STAGES - 1; ++c) {
    if (c < ahead) {
      if (!early) fill_w(c);
      fill_x(c);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  for (int c = 0; c < chunks; ++c) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                       // chunk c has landed for every thread, and chunk c - 1 has been read
    if (c + STAGES - 1 < chunks) {
      fill_w(c + STAGES - 1);
      fill_x(c + STAGES - 1);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* xs = f32_smem + (c % STAGES) * T::STAGE + ty * PITCH;
    const float* ws = f32_smem + (c % STAGES) * T::STAGE + (BM + tx) * PITCH;
    f32_chunk_pairs<TM, TN, ROWS_M * PITCH, ROWS_N * PITCH, PIECES, T::UNROLL>(acc, xs, ws, (min(KC, K - c * KC) + 3) / 4);
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty + i * ROWS_M;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + j * ROWS_N;
      if (n < N) out[(size_t)m * ldo + n] = from_f32<TO>(acc[i][j]);
    }
  }
}

template <typename T, typename TO>
int launch_f32_tile(void* out, const float* x, const float* w, int M, int N, int K, int ldx, int ldw, int ldo, int early,
                    cudaStream_t stream) {
  auto kern = gemm_f32_tile_kernel<T, TO>;
  if (T::SMEM > 48 * 1024 &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::SMEM) != cudaSuccess)
    return zi_refuse("gemm: cannot get %zu bytes of shared memory", T::SMEM);
  const dim3 grid((N + T::BN - 1) / T::BN, (M + T::BM - 1) / T::BM);
  zi_launch(kern, grid, dim3(T::THREADS), T::SMEM, stream, (TO*)out, x, w, M, N, K, ldx, ldw, ldo, early);
  return zi_check_launch("gemm (32-bit tiles)");
}

// ---------------------------------------------------------------------------------------------- few rows
// Up to 32 rows, and more where 32 x 32 tiles would not make a block for every SM: the same tiles with a warp of their own
// for the copies.  One lane per operand row asks for KC columns of it in one untiled bulk copy (both ends on 16-byte
// boundaries, sizes of whole 16 bytes: K % 4 == 0), so the warps that multiply issue nothing but shared-memory reads and
// multiply-adds.  Bound by the chain itself: K dependent multiply-adds of four clocks and the reads that feed them (12 x 1024
// x 1024: 8.5 us, 4 MB of weights; 9.5 with pieces read one ahead; 18 us with copies by the same warps, whose addresses
// cost more issue slots than the product).  One tensor copy a chunk in the place of one bulk copy a row,
// its lines swizzled, was measured too: 11.1 us, for the addresses of the swizzled reads.
template <int BM_, int BN_, int TM_, int TN_, int KC_, int STAGES_, int AHEAD_>
struct F32Few {
  static constexpr int BM = BM_, BN = BN_, TM = TM_, TN = TN_, KC = KC_, STAGES = STAGES_, AHEAD = AHEAD_;
  static constexpr int WORKERS = (BM / TM) * (BN / TN);
  static constexpr int THREADS = WORKERS + 32;
  static constexpr int PITCH = KC + 4;
  static constexpr int STAGE = (BM + BN) * PITCH;
  static constexpr size_t SMEM = (size_t)STAGES * STAGE * sizeof(float) + 2 * STAGES * sizeof(uint64_t);
};

__device__ __forceinline__ void f32_copy_row(float* dst, const float* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src),
               "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

template <typename T, typename TO>
__global__ void __launch_bounds__(T::THREADS)
gemm_f32_few_kernel(TO* __restrict__ out, const float* __restrict__ x, const float* __restrict__ w, int M, int N, int K,
                    int ldx, int ldw, int ldo, int early, int* __restrict__ status) {
  constexpr int BM = T::BM, BN = T::BN, TM = T::TM, TN = T::TN, KC = T::KC, STAGES = T::STAGES, PITCH = T::PITCH;
  constexpr int ROWS_M = BM / TM, ROWS_N = BN / TN;
  pdl_launch_dependents();
  extern __shared__ __align__(16) float f32_smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(f32_smem + (size_t)STAGES * T::STAGE);
  uint64_t* empty = full + STAGES;
  const int tid = threadIdx.x, lane = tid & 31;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int rows_x = min(BM, M - m0), rows_w = min(BN, N - n0);
  const int chunks = (K + KC - 1) / KC;
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], T::WORKERS / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  bool failed = false;
  if (tid >= T::WORKERS) {                 // the copying warp
    auto bytes_of = [&](int c) { return (uint32_t)min(KC, K - c * KC) * 4u; };
    auto copy_w = [&](int c) {
      float* dst = f32_smem + (size_t)(c % STAGES) * T::STAGE + BM * PITCH;
      for (int r = lane; r < rows_w; r += 32) f32_copy_row(dst + r * PITCH, w + (size_t)(n0 + r) * ldw + c * KC, bytes_of(c), &full[c % STAGES]);
    };
    auto copy_x = [&](int c) {
      float* dst = f32_smem + (size_t)(c % STAGES) * T::STAGE;
      for (int r = lane; r < rows_x; r += 32) f32_copy_row(dst + r * PITCH, x + (size_t)(m0 + r) * ldx + c * KC, bytes_of(c), &full[c % STAGES]);
    };
    const int ahead = min(STAGES, chunks);
    if (lane == 0)
      for (int c = 0; c < ahead; ++c) mbar_expect_tx(&full[c], bytes_of(c) * (uint32_t)(rows_x + rows_w));
    __syncwarp();
    if (early)
      for (int c = 0; c < ahead; ++c) copy_w(c);
    pdl_wait();
    for (int c = 0; c < ahead; ++c) {
      if (!early) copy_w(c);
      copy_x(c);
    }
    for (int c = ahead; c < chunks; ++c) {
      if (!warp_mbar_wait(&empty[c % STAGES], ((c / STAGES) & 1) ^ 1)) {
        failed = true;
        break;
      }
      if (lane == 0) mbar_expect_tx(&full[c % STAGES], bytes_of(c) * (uint32_t)(rows_x + rows_w));
      __syncwarp();
      copy_w(c);
      copy_x(c);
    }
    if (failed) {                          // copies in flight land before shared memory is given up
      atomicExch(status, 31);
      for (int i = 0; i < 64; ++i) __nanosleep(10000);
    }
    return;
  }
  pdl_wait();
  const int tx = tid % ROWS_N, ty = tid / ROWS_N;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
  for (int c = 0; c < chunks; ++c) {
    const int s = c % STAGES;
    // (one answer for the warp, here and above: 12 requests' generation 28.8 ms; 28.6 with each lane on its own, and 28.8 again with
    // a note that the lane keeps or the vote behind the chunk)
    if (!warp_mbar_wait(&full[s], (c / STAGES) & 1)) {
      failed = true;
      break;
    }
    const float* xs = f32_smem + (size_t)s * T::STAGE + ty * PITCH;
    const float* ws = f32_smem + (size_t)s * T::STAGE + (BM + tx) * PITCH;
    f32_chunk<TM, TN, ROWS_M * PITCH, ROWS_N * PITCH, KC / 4, T::AHEAD>(acc, xs, ws, min(KC, K - c * KC) / 4);
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[s]);
  }
  if (failed) {
    atomicExch(status, 32);
    for (int i = 0; i < 64; ++i) __nanosleep(10000);
    return;
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty + i * ROWS_M;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + j * ROWS_N;
      if (n < N) out[(size_t)m * ldo + n] = from_f32<TO>(acc[i][j]);
    }
  }
}

template <typename T, typename TO>
int launch_f32_few(void* out, const float* x, const float* w, int M, int N, int K, int ldx, int ldw, int ldo, int early, int* status,
                   cudaStream_t stream) {
  auto kern = gemm_f32_few_kernel<T, TO>;
  if (T::SMEM > 48 * 1024 &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::SMEM) != cudaSuccess)
    return zi_refuse("gemm: cannot get %zu bytes of shared memory", T::SMEM);
  const dim3 grid((N + T::BN - 1) / T::BN, (M + T::BM - 1) / T::BM);
  zi_launch(kern, grid, dim3(T::THREADS), T::SMEM, stream, (TO*)out, x, w, M, N, K, ldx, ldw, ldo, early, status);
  return zi_check_launch("gemm (32-bit, few rows)");
}

}  // namespace
