// Long portions of the recurrences with one decay per key channel and token (linear_attention.cu has the form that walks
// the tokens one by one), in chunks of 64 tokens whose work is matrix products:
//
//     S <- diag(g_t) S ;  u_t = v_t  or  beta_t (v_t - S^T k_t) (delta rule) ;  S <- S + k_t u_t^T ;  o_t = S^T q_t
//
// With G(a, b] the product of the decays of tokens a + 1 .. b (a vector over the key channels) inside a chunk that begins
// from S0, and * the product by channels:
//
//     P_ts = sum_i q_ti k_si G(s, t]_i  for s <= t,    L_ts = beta_t sum_i k_ti k_si G(s, t]_i  for s < t,
//     (I + L) [W | U0] = diag(beta) [k_t * G(0, t] | V] ,   U = U0 - W S0   (without the delta rule U = V),
//     O = (q_t * G(0, t]) S0 + P U ,   S1 = diag(G(0, 64]) S0 + (k_s * G(s, 64])^T U
//
// (the chunked form of "Gated Linear Attention Transformers with Hardware-Efficient Training", Yang et al., 2023, and of
// "Gated Delta Networks", Yang et al., 2024, with the decays of the former).  No quotient and no logarithm of a decay is
// ever taken: the products G are made by multiplying decays, within blocks of 16 tokens pair by pair and between blocks as
// (from s to its block's end) (whole blocks between) (from t's block's begin to t), so decays of any size, zero included,
// only make products small.  The kernels:
//   1. channel_scores  per chunk and head: P, the products k . k, q and k times their decays
//   2. channel_solve   (delta rule) per chunk and head: the triangular system by forward substitution, a thread per column
//   3. channel_walk    per request, head and 16 value channels: the chunks in order, products with the state on the
//                      tensor cores (mma.sync, bfloat16 parts)
// Everything is 32-bit: the tensor cores' operands are split into three bfloat16 parts (all 24 bits of mantissa), the parts'
// products are summed apart, and the state is moved on by 32-bit multiply-adds outside of the tensor cores' accumulators.
// Against 64 bits outputs and states are nearer than the walk's.
//
// A value that is infinite or no number would reach earlier tokens too (zero weights meet it in P U) and infinities would
// not survive the split into parts.  So a block of the walk whose outputs or state come out so takes its request, head and
// value channels again token by token from the state it began with (walk_tokens), as the recurrence is written.
//
// A chunk's place in the workspace: the chunks of the requests that bring two tokens or more, one behind the other.  Requests
// that bring one token are left alone and have no place.
//
// Measured, 2,048 tokens, 8 heads of 128 x 256 (the walk token by token -> chunks): plain form with bfloat16 q, k, v 756 -> 182 us,
// delta rule 833 -> 259 us; one kernel at a time the scores 39 and 48 us, the triangular systems 47, the walk 140 and 185.
// Relative errors of outputs and states against 64 bits, 1e-7 (the walk -> chunks): plain 4.9, 5.8 -> 3.3, 3.6, delta rule
// 2.1, 1.4 -> 1.6, 0.9.  (Two tf32 parts, 22 bits, and rows that took off their terms one by one: 168 and 242 us, but 2.5, 1.7
// with the delta rule, and plain at 8 x 64 tokens 1.65 against the walk's 1.52.)
#include "api.h"
#include "common.cuh"

namespace {

constexpr int RK = 64, SUB = 16, SUBS = RK / SUB;    // tokens per chunk, per block within it
constexpr int RV = 16;                               // value channels per block of the walk
constexpr int KK_PITCH = RK + 4;

struct ChannelJob {
  const void* q;       // [T][G * D]
  const void* k;
  const void* v;       // [T][H * V]
  const float* decay;  // [T][H * D]
  const float* beta;   // [T][H] or null
  int ldq, ldk, ldv, ldg, ldb;
  int qk_dtype;
  float q_scale;
  float* state;
  long long slot_stride;
  int H, G, D, V;
  const int* cu_q;
  const int* state_slots;
  int n_seqs, places;  // places: for whose chunks the workspace has room
  float* out;          // [T][H * V]
  int ldo;
  // workspace, per place and head
  float* qd;           // [RK][D]  q times the decays since the chunk's begin
  float* kd;           // [RK][D]  k times the decays up to the chunk's end
  float* p;            // [RK][RK] P (16 x 16 parts above the diagonal are not written)
  float* gend;         // [D]      the chunk's decays
  float* kk;           // [RK][RK] delta rule only: sum_i k_ti k_si G(s, t]_i for s < t
  float* w;            // [RK][D]  delta rule only: k times the decays since the chunk's begin; then W
  float* u0;           // [RK][V]  delta rule only
};

__device__ __forceinline__ int chunks_of(int qlen) { return qlen > 1 ? (qlen + RK - 1) / RK : 0; }

// The request and chunk at a place, by a whole warp: 32 requests at a time, their chunks counted together.
__device__ __forceinline__ bool channel_chunk(const ChannelJob& j, int place, int& first, int& n) {
  const int lane = threadIdx.x & 31;
  int before = 0;
  for (int s0 = 0; s0 < j.n_seqs; s0 += 32) {
    const int s = s0 + lane;
    int tok0 = 0, qlen = 0;
    if (s < j.n_seqs) {
      tok0 = j.cu_q[s];
      qlen = j.cu_q[s + 1] - tok0;
    }
    const int own = chunks_of(qlen);
    int upto = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += y;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, place < before + upto);
    if (hit) {
      const int src = __ffs(hit) - 1, i = place - before - __shfl_sync(0xffffffffu, upto - own, src);
      first = __shfl_sync(0xffffffffu, tok0, src) + i * RK;
      n = min(RK, __shfl_sync(0xffffffffu, qlen, src) - i * RK);
      return true;
    }
    before += __shfl_sync(0xffffffffu, upto, 31);
  }
  return false;
}
// The place of a request's first chunk, by a whole warp.
__device__ __forceinline__ int first_place(const ChannelJob& j, int seq) {
  int before = 0;
  for (int s = threadIdx.x & 31; s < seq; s += 32) before += chunks_of(j.cu_q[s + 1] - j.cu_q[s]);
  return __reduce_add_sync(0xffffffffu, before);
}

constexpr int SP = RV + 8;                           // pitch of the state and of U, pairs of rows: a fragment's reads fall into 32 banks
constexpr int PP = RK + 8;                           // of P; Q and W have D + 8 (read as pairs along a row), K D + 4 (along a column)

// Two values in three bfloat16 parts each, x in the low halves: 8 bits of mantissa rounded to nearest, then 8 of what is left, then
// the rest, which is no more than 8.  The parts' sum is the value: all 24 bits are there.
__device__ __forceinline__ uint32_t pack_nearest(float x, float y) {
  uint32_t p;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p) : "f"(y), "f"(x));
  return p;
}
__device__ __forceinline__ void three_parts(float x, float y, uint32_t (&p)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    p[i] = pack_nearest(x, y);
    x -= __uint_as_float(p[i] << 16);
    y -= __uint_as_float(p[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ void bf16_mma(float (&d)[4], const uint32_t* a, const uint32_t* b) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void bf16_mma_from_zero(float (&d)[4], const uint32_t* a, const uint32_t* b) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}
// A 16 x 8 result of products of 16 x 16 and 16 x 8 values in three parts: the first parts' products and the others' are summed
// apart, the first parts' 16 at a time (the tensor cores' own sums round down) and then by 32-bit adds.  What is left out,
// the second part times the third and the third times the third, is below 2^-25 of a product.
struct TwoSums {
  float big[4], small[4];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int e = 0; e < 4; ++e) big[e] = small[e] = 0.f;
  }
  __device__ __forceinline__ float sum(int e) const { return big[e] + small[e]; }
  __device__ __forceinline__ void add(const uint32_t (&a)[3][4], const uint32_t (&b)[3][2]) {
    bf16_mma(small, a[2], b[0]);
    bf16_mma(small, a[0], b[2]);
    bf16_mma(small, a[1], b[1]);
    bf16_mma(small, a[1], b[0]);
    bf16_mma(small, a[0], b[1]);
    float d[4];
    bf16_mma_from_zero(d, a[0], b[0]);
#pragma unroll
    for (int e = 0; e < 4; ++e) big[e] += d[e];
  }
};
// A lane's 16 x 16 operand: x[2 i], x[2 i + 1] are neighbours along k of its register i.
__device__ __forceinline__ void left_parts(const float2 (&x)[4], uint32_t (&a)[3][4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t p[3];
    three_parts(x[i].x, x[i].y, p);
#pragma unroll
    for (int n = 0; n < 3; ++n) a[n][i] = p[n];
  }
}
__device__ __forceinline__ float2 pair_at(const float* p) { return *reinterpret_cast<const float2*>(p); }

// ------------------------------------------------------------------------------------------- 1. scores
// Within blocks of 16 tokens pair by pair with 32-bit multiply-adds, between blocks on the tensor cores.
constexpr int SC_THREADS = 256;

template <typename TQ, bool DELTA>
__global__ void __launch_bounds__(SC_THREADS)
channel_scores_kernel(const ChannelJob j) {
  pdl_launch_dependents();
  extern __shared__ __align__(16) float sc[];
  const int place = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, D = j.D, DP = D + 8;
  float* Q = sc;                          // [RK][DP] q; later q times the decays since its block's begin
  float* K = Q + RK * DP;                 // k; later k times the decays up to its block's end
  float* A = K + RK * DP;                 // the decays; later k times the decays since its block's begin
  float* B = A + RK * DP;                 // [SUBS][D] the blocks' decays; then what comes before a block, [SUBS][D]; after it
  float* before = B + SUBS * D;
  float* after = before + SUBS * D;
  pdl_wait();
  int first, n;
  if (!channel_chunk(j, place, first, n)) return;     // uniform in the block
  const int g = h / (j.H / j.G);
  const TQ* q = static_cast<const TQ*>(j.q) + (size_t)first * j.ldq + (size_t)g * D;
  const TQ* k = static_cast<const TQ*>(j.k) + (size_t)first * j.ldk + (size_t)g * D;
  const float* dec = j.decay + (size_t)first * j.ldg + (size_t)h * D;
#pragma unroll 4
  for (int t = warp; t < RK; t += SC_THREADS / 32)
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = lane + 32 * u;
      if (i >= D) break;
      const bool in = t < n;
      Q[t * DP + i] = in ? to_f32(q[(size_t)t * j.ldq + i]) * j.q_scale : 0.f;
      K[t * DP + i] = in ? to_f32(k[(size_t)t * j.ldk + i]) : 0.f;
      A[t * DP + i] = in ? dec[(size_t)t * j.ldg + i] : 1.f;
    }
  __syncthreads();
  const size_t at = (size_t)place * j.H + h;
  float* po = j.p + at * RK * RK;
  float* ko = DELTA ? j.kk + at * RK * RK : nullptr;
  // within a block: a warp takes a key s and walks the block's queries t = s, s + 1, .., four channels a lane; the lanes' shares
  // of all 16 sums are then added together.  The keys are dealt out so that every warp has as many pairs.
#pragma unroll 1
  for (int r = 0; r < RK / 8; ++r) {
    const int s = r * 8 + ((r & 1) ? 7 - warp : warp), b0 = s & ~(SUB - 1), sl = s - b0, i = lane * 4;
    const bool on = i < D;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 ke = on ? *reinterpret_cast<const float4*>(K + s * DP + i) : zero;
    float a[SUB], b[DELTA ? SUB : 1];
#pragma unroll
    for (int u = 0; u < SUB; ++u) {
      a[u] = 0.f;
      if (DELTA) b[u] = 0.f;
      if (u < sl || !on) continue;
      const float4 qt = *reinterpret_cast<const float4*>(Q + (b0 + u) * DP + i);
      if (u > sl) {
        const float4 gt = *reinterpret_cast<const float4*>(A + (b0 + u) * DP + i);
        ke.x *= gt.x; ke.y *= gt.y; ke.z *= gt.z; ke.w *= gt.w;
        if (DELTA) {
          const float4 kt = *reinterpret_cast<const float4*>(K + (b0 + u) * DP + i);
          b[u] = fmaf(kt.x, ke.x, fmaf(kt.y, ke.y, fmaf(kt.z, ke.z, kt.w * ke.w)));
        }
      }
      a[u] = fmaf(qt.x, ke.x, fmaf(qt.y, ke.y, fmaf(qt.z, ke.z, qt.w * ke.w)));
    }
    // halves of the warp trade halves of the sums, then quarters ..: lane l ends with the sum of query l >> 1 (bits reversed)
    auto total = [&](float (&x)[SUB]) {
#pragma unroll
      for (int o = 16, m = SUB / 2; o > 1; o >>= 1, m >>= 1)
#pragma unroll
        for (int u = 0; u < SUB / 2; ++u) {
          if (u >= m) break;
          const float keep = (lane & o) ? x[u + m] : x[u], give = (lane & o) ? x[u] : x[u + m];
          x[u] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
      return x[0] + __shfl_xor_sync(0xffffffffu, x[0], 1);
    };
    const float pa = total(a);
    const int t = b0 + ((lane >> 4) & 1) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1);
    if (!(lane & 1)) po[(size_t)t * RK + s] = pa;       // zero for queries before the key
    if constexpr (DELTA) {
      const float pb = total(b);
      if (!(lane & 1)) ko[(size_t)t * RK + s] = pb;
    }
  }
  __syncthreads();
  // the decays since a block's begin and up to its end, a thread per channel and block
  for (int e = tid; e < SUBS * D; e += SC_THREADS) {
    const int b = e / D, i = e - b * D;
    float gv[SUB], kv[SUB];
#pragma unroll
    for (int u = 0; u < SUB; ++u) {
      gv[u] = A[(b * SUB + u) * DP + i];
      kv[u] = K[(b * SUB + u) * DP + i];
    }
    float run = 1.f;
#pragma unroll
    for (int u = 0; u < SUB; ++u) {
      run *= gv[u];
      Q[(b * SUB + u) * DP + i] *= run;
      if (DELTA) A[(b * SUB + u) * DP + i] = kv[u] * run;
    }
    B[e] = run;
    run = 1.f;
#pragma unroll
    for (int u = SUB - 1; u >= 0; --u) {
      K[(b * SUB + u) * DP + i] = kv[u] * run;
      run *= gv[u];
    }
  }
  __syncthreads();
  for (int i = tid; i < D; i += SC_THREADS) {
    float run = 1.f;
#pragma unroll
    for (int b = 0; b < SUBS; ++b) {
      before[b * D + i] = run;
      run *= B[b * D + i];
    }
    j.gend[at * D + i] = run;
    run = 1.f;
#pragma unroll
    for (int b = SUBS - 1; b >= 0; --b) {
      after[b * D + i] = run;
      run *= B[b * D + i];
    }
  }
  __syncthreads();
  // between blocks b < a, 16 x 16 pairs each, on the tensor cores: the six of q . k, then the six of k . k
  for (int unit = warp; unit < (DELTA ? 12 : 6); unit += SC_THREADS / 32) {
    const int pair = unit % 6, fr = lane >> 2, fk = lane & 3;
    const int a = pair < 3 ? pair + 1 : (pair < 5 ? pair - 1 : 3), b = pair < 3 ? pair : (pair < 5 ? pair - 3 : 0);
    const float* X = (unit < 6 ? Q : A) + (a * SUB + fr) * DP + 2 * fk;
    const float* Y = K + (b * SUB + fr) * DP + 2 * fk;
    TwoSums sum[2];
    sum[0].clear();
    sum[1].clear();
#pragma unroll 1
    for (int c = 0; c < D; c += 16) {
      float2 m[2] = {make_float2(1.f, 1.f), make_float2(1.f, 1.f)};
      for (int w = b + 1; w < a; ++w)                // the whole blocks between
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float2 g = pair_at(B + w * D + c + 8 * i + 2 * fk);
          m[i].x *= g.x;
          m[i].y *= g.y;
        }
      const float2 x[4] = {pair_at(X + c), pair_at(X + 8 * DP + c), pair_at(X + c + 8), pair_at(X + 8 * DP + c + 8)};
      uint32_t xp[3][4];
      left_parts(x, xp);
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        uint32_t yp[3][2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float2 y = pair_at(Y + 8 * n * DP + c + 8 * i);
          uint32_t p[3];
          three_parts(y.x * m[i].x, y.y * m[i].y, p);
#pragma unroll
          for (int t = 0; t < 3; ++t) yp[t][i] = p[t];
        }
        sum[n].add(xp, yp);
      }
    }
    float* to = unit < 6 ? po : ko;
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 4; e += 2)
        *reinterpret_cast<float2*>(to + (size_t)(a * SUB + fr + (e >> 1) * 8) * RK + b * SUB + n * 8 + fk * 2) =
            make_float2(sum[n].sum(e), sum[n].sum(e + 1));
  }
  for (int t = warp; t < RK; t += SC_THREADS / 32) {
    const int i = lane * 4, b = t / SUB;
    if (i >= D) break;
    const float4 fb = *reinterpret_cast<const float4*>(before + b * D + i), fa = *reinterpret_cast<const float4*>(after + b * D + i);
    const float4 qv = *reinterpret_cast<const float4*>(Q + t * DP + i), kv = *reinterpret_cast<const float4*>(K + t * DP + i);
    *reinterpret_cast<float4*>(j.qd + (at * RK + t) * D + i) = make_float4(qv.x * fb.x, qv.y * fb.y, qv.z * fb.z, qv.w * fb.w);
    *reinterpret_cast<float4*>(j.kd + (at * RK + t) * D + i) = make_float4(kv.x * fa.x, kv.y * fa.y, kv.z * fa.z, kv.w * fa.w);
    if (DELTA) {
      const float4 wv = *reinterpret_cast<const float4*>(A + t * DP + i);
      *reinterpret_cast<float4*>(j.w + (at * RK + t) * D + i) = make_float4(wv.x * fb.x, wv.y * fb.y, wv.z * fb.z, wv.w * fb.w);
    }
  }
}

// ------------------------------------------------------------------------------------ 2. the triangular system
// [W | U0] by forward substitution in blocks of 16 rows; a thread holds its column, so that nothing waits for another.  What is
// taken off a row is summed by itself, so that its many small terms are not rounded to the row's own size one by one.
constexpr int SO_COLS = 128;         // columns per block

template <typename TV>
__global__ void __launch_bounds__(SO_COLS)
channel_solve_kernel(const ChannelJob j) {
  pdl_launch_dependents();
  extern __shared__ __align__(16) float so[];
  const int place = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, D = j.D, V = j.V;
  float* L = so;                       // [s][t]
  float* bs = L + RK * KK_PITCH;
  float* xs = bs + RK;                 // [RK][SO_COLS]: this thread's solved rows
  pdl_wait();
  int first, n;
  if (!channel_chunk(j, place, first, n)) return;
  const size_t at = (size_t)place * j.H + h;
  const float* kk = j.kk + at * RK * RK;
  for (int t = tid; t < RK; t += SO_COLS) bs[t] = t < n ? j.beta[(size_t)(first + t) * j.ldb + h] : 0.f;
  __syncthreads();
  for (int e = tid; e < RK * RK; e += SO_COLS) {
    const int t = e / RK, s = e - t * RK;
    L[s * KK_PITCH + t] = s < t ? bs[t] * kk[e] : 0.f;
  }
  __syncthreads();
  const int col = blockIdx.z * SO_COLS + tid;
  const bool on = col < D + V, is_k = col < D;
  float* wo = j.w + at * RK * D + col;
  float* uo = j.u0 + at * RK * V + (col - D);
  const TV* v = static_cast<const TV*>(j.v) + (size_t)first * j.ldv + (size_t)h * V + (col - D);
  auto right = [&](int t) { return !on || t >= n ? 0.f : (is_k ? wo[(size_t)t * D] : to_f32(v[(size_t)t * j.ldv])); };
  float next[SUB];
#pragma unroll
  for (int r = 0; r < SUB; ++r) next[r] = right(r);
#pragma unroll 1
  for (int b = 0; b < RK; b += SUB) {
    float x[SUB], off[SUB];
#pragma unroll
    for (int r = 0; r < SUB; ++r) {
      x[r] = bs[b + r] * next[r];
      off[r] = 0.f;
    }
    if (b + SUB < RK) {
#pragma unroll
      for (int r = 0; r < SUB; ++r) next[r] = right(b + SUB + r);
    }
#pragma unroll 4
    for (int s = 0; s < b; ++s) {
      const float y = xs[s * SO_COLS + tid];
#pragma unroll
      for (int r = 0; r < SUB; r += 4) {
        const float4 l = *reinterpret_cast<const float4*>(L + s * KK_PITCH + b + r);
        off[r] = fmaf(l.x, y, off[r]);
        off[r + 1] = fmaf(l.y, y, off[r + 1]);
        off[r + 2] = fmaf(l.z, y, off[r + 2]);
        off[r + 3] = fmaf(l.w, y, off[r + 3]);
      }
    }
#pragma unroll
    for (int s = 0; s < SUB; ++s) {
      x[s] -= off[s];
#pragma unroll
      for (int r = 0; r < SUB; ++r)
        if (r > s) off[r] = fmaf(L[(b + s) * KK_PITCH + b + r], x[s], off[r]);
    }
#pragma unroll
    for (int r = 0; r < SUB; ++r) {
      xs[(b + r) * SO_COLS + tid] = x[r];
      if (on && is_k) wo[(size_t)(b + r) * D] = x[r];
      if (on && !is_k) uo[(size_t)(b + r) * V] = x[r];
    }
  }
}

// -------------------------------------------------------------------------------------------- 3. the walk
// Two groups of eight warps share a chunk: the first moves the state on (W S, U, Kd^T U), the second reads out (Qd S, P U).
// A warp has 16 tokens (or two times 16 key channels) x 8 value channels.  Bound by instruction issue and by the chain of a
// chunk's two rounds of products and its two barriers, 32 times for 2,048 tokens: the state and U are split into their parts
// once, where they are made.  16 value channels per block put 8 heads of 256 on 128 SMs.  Three bfloat16 parts take six
// products of 16 x 8 x 16, as many as two tf32 parts' three of 16 x 8 x 8, and half the 32-bit adds (three tf32 parts: 249 and 332 us).
constexpr int WK_THREADS = 512;

__device__ __forceinline__ void wk_copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

size_t channel_walk_smem(int D, bool delta) {
  const size_t rows = (size_t)RK * (D + 8), keys = (size_t)RK * (D + 4), p = (size_t)RK * PP;
  return (rows * (delta ? 2 : 1) + 2 * keys + 2 * p + 2 * D + (size_t)3 * (D + RK) / 2 * SP) * sizeof(float);
}

// The recurrence token by token with plain 32-bit multiply-adds, in the walk's own form (linear_attention.cu: read out the decayed
// state, then what the token adds), for value channels v0 .. v0 + RV - 1 of a head, by the whole block: a thread holds the key
// channels tid / RV + 32 r of one value channel.  For portions that hold values which are no numbers; `red` is
// [3][WK_THREADS / 32][RV] of shared memory.
template <typename TV, bool DELTA>
__device__ __noinline__ void walk_tokens(const ChannelJob& j, float* state, float* red, int tok0, int qlen, int h, int v0) {
  constexpr int GROUPS = WK_THREADS / RV, ROWS = 128 / GROUPS, WARPS = WK_THREADS / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, c = tid % RV, col = v0 + c, i0 = tid / RV, g = h / (j.H / j.G);
  const bool on = col < j.V;
  auto key = [&](const void* p, int ld, int t, int i) {
    const size_t at = (size_t)(tok0 + t) * ld + (size_t)g * j.D + i;
    return j.qk_dtype == ZI_F32 ? static_cast<const float*>(p)[at] : to_f32(static_cast<const __nv_bfloat16*>(p)[at]);
  };
  float st[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) st[r] = on && i0 + r * GROUPS < j.D ? state[(size_t)(i0 + r * GROUPS) * j.V + col] : 0.f;
  for (int t = 0; t < qlen; ++t) {
    float kt[ROWS], sum[3] = {0.f, 0.f, 0.f};         // (g S)^T k, (g S)^T q, k . q
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const int i = i0 + r * GROUPS;
      kt[r] = 0.f;
      if (i >= j.D) continue;
      const float qt = key(j.q, j.ldq, t, i) * j.q_scale;
      kt[r] = key(j.k, j.ldk, t, i);
      st[r] *= j.decay[(size_t)(tok0 + t) * j.ldg + (size_t)h * j.D + i];
      if (DELTA) sum[0] = fmaf(st[r], kt[r], sum[0]);
      sum[1] = fmaf(st[r], qt, sum[1]);
      sum[2] = fmaf(kt[r], qt, sum[2]);
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < 3; ++n) {
      sum[n] += __shfl_xor_sync(0xffffffffu, sum[n], RV);
      if (lane < RV) red[(n * WARPS + warp) * RV + c] = sum[n];
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < 3; ++n) {
      sum[n] = 0.f;
      for (int w = 0; w < WARPS; ++w) sum[n] += red[(n * WARPS + w) * RV + c];
    }
    float u = on ? to_f32(static_cast<const TV*>(j.v)[(size_t)(tok0 + t) * j.ldv + (size_t)h * j.V + col]) : 0.f;
    if (DELTA) u = j.beta[(size_t)(tok0 + t) * j.ldb + h] * (u - sum[0]);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) st[r] = fmaf(kt[r], u, st[r]);
    if (on && i0 == 0) j.out[(size_t)(tok0 + t) * j.ldo + (size_t)h * j.V + col] = fmaf(u, sum[2], sum[1]);
  }
#pragma unroll
  for (int r = 0; r < ROWS; ++r)
    if (on && i0 + r * GROUPS < j.D) state[(size_t)(i0 + r * GROUPS) * j.V + col] = st[r];
}

template <typename TV, bool DELTA>
__global__ void __launch_bounds__(WK_THREADS)
channel_walk_kernel(const __grid_constant__ ChannelJob j) {
  pdl_launch_dependents();
  extern __shared__ __align__(16) float wk[];
  const int D = j.D, QP = D + 8, KP = D + 4, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wr = warp & 3, wc = ((warp >> 2) & 1) * 8;
  const bool moves = warp < 8;
  float* Q = wk;                                     // [RK][QP]
  float* W = Q + RK * QP;                            // delta rule only
  float* K = W + (DELTA ? RK * QP : 0);              // twice [RK][KP]
  float* P = K + 2 * RK * KP;                        // twice [RK][PP]
  float* E = P + 2 * RK * PP;                        // twice [D]: the chunk's decays
  uint32_t* S = reinterpret_cast<uint32_t*>(E + 2 * D);       // the state's three parts, pairs of rows, [D / 2][SP] each
  uint32_t* U = S + 3 * D / 2 * SP;                  // U's, [RK / 2][SP] each
  const int seq = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * RV;
  pdl_wait();
  const int tok0 = j.cu_q[seq], qlen = j.cu_q[seq + 1] - tok0;
  if (qlen <= 1) return;
  const int chunks = chunks_of(qlen), place0 = first_place(j, seq);
  if (place0 + chunks > j.places) return;            // more such requests than the caller has counted: no room for their chunks
  float* state = j.state + (size_t)j.state_slots[seq] * j.slot_stride + (size_t)h * D * j.V;
  const int fr = lane >> 2, fk = lane & 3, fc = wc + fk * 2;      // a fragment's row, its channel of eight; a result's column

  const int x4 = lane * 4;                           // copies: a warp a row
  auto load_early = [&](int i) {                     // what the second half of a chunk reads, two buffers
    const size_t at = (size_t)(place0 + i) * j.H + h;
    const int buf = i & 1;
    const float* k = j.kd + at * RK * D;
#pragma unroll
    for (int r = warp; r < RK; r += WK_THREADS / 32) {
      if (x4 >= D) break;
      wk_copy16(K + buf * RK * KP + r * KP + x4, k + r * D + x4);
    }
    const float* p = j.p + at * RK * RK;
#pragma unroll
    for (int e = tid; e < RK * RK / 4; e += WK_THREADS) {
      const int r = e / (RK / 4), s = (e - r * (RK / 4)) * 4;
      if (s < (r & ~(SUB - 1)) + SUB) wk_copy16(P + buf * RK * PP + r * PP + s, p + r * RK + s);
    }
    if (tid * 4 < D) wk_copy16(E + buf * D + tid * 4, j.gend + at * D + tid * 4);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto load_rows = [&](int i) {                      // what its first half reads
    const size_t at = (size_t)(place0 + i) * j.H + h;
    const float* q = j.qd + at * RK * D;
    const float* w = DELTA ? j.w + at * RK * D : nullptr;
#pragma unroll
    for (int r = warp; r < RK; r += WK_THREADS / 32) {
      if (x4 >= D) break;
      wk_copy16(Q + r * QP + x4, q + r * D + x4);
      if (DELTA) wk_copy16(W + r * QP + x4, w + r * D + x4);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load_early(0);
  load_rows(0);

  // A product's results x and y, in columns fc and fc + 1 of row `row`, in three parts `gap` apart, by the whole warp: the lane of
  // the even row of two stores both rows' column fc, the other one their column fc + 1.
  const int odd = fr & 1;
  auto put_parts = [&](uint32_t* to, int gap, int row, float x, float y) {
    const float other = __shfl_xor_sync(0xffffffffu, odd ? x : y, 4);
    uint32_t p[3];
    three_parts(odd ? other : x, odd ? y : other, p);
#pragma unroll
    for (int n = 0; n < 3; ++n) to[n * gap + (row >> 1) * SP + fc + odd] = p[n];
  };
  // the state: key channels (wr + 4 m) 16 .., in the first group's registers as a product's results lie
  float st[2][4] = {};
  auto share_state = [&] {
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int row = (wr + 4 * m) * 16 + fr;
      if (!moves || (wr + 4 * m) * 16 >= D) continue;
      put_parts(S, D / 2 * SP, row, st[m][0], st[m][1]);
      put_parts(S, D / 2 * SP, row + 8, st[m][2], st[m][3]);
    }
  };
  auto each = [&](auto f) {
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      if (!moves || (wr + 4 * m) * 16 >= D) continue;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = (wr + 4 * m) * 16 + fr + (e >> 1) * 8, col = v0 + fc + (e & 1);
        if (col < j.V) f(st[m][e], state + (size_t)row * j.V + col);
      }
    }
  };
  each([](float& x, float* at) { x = *at; });
  share_state();

  // 16 x 16 values times 16 rows of three parts
  auto step = [&](TwoSums& sum, const float2 (&x)[4], const uint32_t* b, int gap) {
    uint32_t ap[3][4], bp[3][2];
    left_parts(x, ap);
#pragma unroll
    for (int n = 0; n < 3; ++n) {
      bp[n][0] = b[n * gap];
      bp[n][1] = b[n * gap + 4 * SP];
    }
    sum.add(ap, bp);
  };
  auto along_row = [&](TwoSums& sum, const float* a, int pitch, const uint32_t* b, int gap) {
    const float2 x[4] = {pair_at(a), pair_at(a + 8 * pitch), pair_at(a + 8), pair_at(a + 8 * pitch + 8)};
    step(sum, x, b, gap);
  };
  auto along_column = [&](TwoSums& sum, const float* a, int pitch, const uint32_t* b, int gap) {
    float2 x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float* p = a + (i >> 1) * 8 * pitch + (i & 1) * 8;
      x[i] = make_float2(p[0], p[pitch]);
    }
    step(sum, x, b, gap);
  };
  const int frag = fk * SP + wc + fr;                // this lane's place in 8 pairs of rows of S or U

  TwoSums sum;
  bool finite = true;                                // the outputs, and at the end the state: neither forgets a value that is no number
  for (int i = 0; i < chunks; ++i) {
    const int n = min(RK, qlen - i * RK), first = tok0 + i * RK, buf = i & 1;
    // what becomes U: asked for now, needed after the product with the state
    float u[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int t = wr * 16 + fr + (e >> 1) * 8, col = v0 + fc + (e & 1);
      u[e] = 0.f;
      if (moves && t < n && col < j.V) {
        u[e] = DELTA ? j.u0[(((size_t)(place0 + i) * j.H + h) * RK + t) * j.V + col]
                     : to_f32(static_cast<const TV*>(j.v)[(size_t)(first + t) * j.ldv + (size_t)h * j.V + col]);
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                  // this chunk's tiles and the state are there
    if (i + 1 < chunks) load_early(i + 1);            // the chunk before is done with these buffers
    sum.clear();
    if (DELTA || !moves) {
      const float* A = (moves ? W : Q) + (wr * 16 + fr) * QP + 2 * fk;
#pragma unroll 2
      for (int c = 0; c < D; c += 16) along_row(sum, A + c, QP, S + c / 2 * SP + frag, D / 2 * SP);
    }
    if (moves) {
#pragma unroll
      for (int e = 0; e < 4; ++e) u[e] = DELTA ? u[e] - sum.sum(e) : u[e];
      put_parts(U, RK / 2 * SP, wr * 16 + fr, u[0], u[1]);
      put_parts(U, RK / 2 * SP, wr * 16 + fr + 8, u[2], u[3]);
    }
    __syncthreads();                                  // U is there; nobody reads Q, W and the state any more
    if (i + 1 < chunks) load_rows(i + 1);
    if (!moves) {
      const float* A = P + buf * RK * PP + (wr * 16 + fr) * PP + 2 * fk;
#pragma unroll 1
      for (int c = 0; c < (wr + 1) * 16; c += 16) along_row(sum, A + c, PP, U + c / 2 * SP + frag, RK / 2 * SP);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = wr * 16 + fr + (e >> 1) * 8, col = v0 + fc + (e & 1);
        const float o = sum.sum(e);
        if (t < n && col < j.V) {
          j.out[(size_t)(first + t) * j.ldo + (size_t)h * j.V + col] = o;
          finite &= isfinite(o);
        }
      }
    } else {
      const float* Kb = K + buf * RK * KP + 2 * fk * KP + fr;
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int c0 = (wr + 4 * m) * 16;
        if (c0 >= D) continue;
        sum.clear();
#pragma unroll 2
        for (int s = 0; s < RK; s += 16) along_column(sum, Kb + s * KP + c0, KP, U + s / 2 * SP + frag, RK / 2 * SP);
        const float g[2] = {E[buf * D + c0 + fr], E[buf * D + c0 + fr + 8]};
#pragma unroll
        for (int e = 0; e < 4; ++e) st[m][e] = fmaf(g[e >> 1], st[m][e], sum.sum(e));
      }
      if (i + 1 < chunks) share_state();
    }
  }
  each([&](float& x, float*) { finite &= isfinite(x); });
  if (__syncthreads_or(!finite)) {
    walk_tokens<TV, DELTA>(j, state, wk, tok0, qlen, h, v0);
    return;
  }
  each([](float& x, float* at) { *at = x; });
}

struct ChannelPlan {
  long long rows, square, ends, values, total;       // floats
};
ChannelPlan channel_plan(int places, int H, int D, int V, int delta) {
  const long long n = (long long)places * H;
  ChannelPlan p;
  p.rows = n * RK * D;
  p.square = n * RK * RK;
  p.ends = n * D;
  p.values = n * RK * V;
  p.total = p.rows * (delta ? 3 : 2) + p.square * (delta ? 2 : 1) + p.ends + (delta ? p.values : 0);
  return p;
}
}  // namespace

extern "C" int zi_channel_recurrence_supported(int D, int V, int H, int G) {
  return D >= 16 && D <= 128 && D % 16 == 0 && V > 0 && H > 0 && G > 0 && H % G == 0 && H <= 65535 && (V + RV - 1) / RV <= 65535;
}
// Chunks of the requests that bring two tokens or more, at most: n_single of the step's n_seqs requests bring one.
static int channel_places(int T, int n_seqs, int n_single) { return (T - n_single) / RK + n_seqs - n_single; }

extern "C" long long zi_channel_recurrence_workspace_floats(int T, int n_seqs, int n_single, int H, int D, int V, int delta) {
  return channel_plan(channel_places(T, n_seqs, n_single), H, D, V, delta).total;
}

// The portions of two tokens and more of a step; the n_single requests that bring one token are left alone.  decay: float32 [T][H * D],
// between 0 and 1; beta: step sizes [T][H], with the delta rule and only there; q and k of one type, v of its own;
// workspace: zi_channel_recurrence_workspace_floats, 16-byte aligned.
extern "C" int zi_channel_recurrence(float* out, int ldo, const void* q, int ldq, const void* k, int ldk, int qk_dtype, const void* v,
                                     int ldv, int v_dtype, const float* decay, int ldg, const float* beta, int ldb, float q_scale,
                                     float* state, long long slot_stride, int T, int H, int G, int D, int V, int delta, const int* cu_q,
                                     const int* state_slots, int n_seqs, int n_single, float* workspace, cudaStream_t stream) {
  if (T <= 0 || n_seqs <= 0) return 0;
  if (n_single < 0 || n_single > n_seqs || n_single > T) return zi_refuse("channel_recurrence: %d of %d requests bring one token", n_single, n_seqs);
  const int places = channel_places(T, n_seqs, n_single);
  if (places == 0) return 0;
  if (!zi_channel_recurrence_supported(D, V, H, G)) return zi_refuse("channel_recurrence: %d heads (%d of keys) of %d x %d", H, G, D, V);
  if (!workspace || ((uintptr_t)workspace & 15) || !decay || (delta != 0) != (beta != nullptr))
    return zi_refuse("channel_recurrence: needs decays, with the delta rule (and only there) steps, and an aligned workspace");
  const ChannelPlan p = channel_plan(places, H, D, V, delta);
  ChannelJob j = {};
  j.q = q; j.k = k; j.v = v; j.decay = decay; j.beta = beta;
  j.ldq = ldq; j.ldk = ldk; j.ldv = ldv; j.ldg = ldg; j.ldb = ldb; j.qk_dtype = qk_dtype; j.q_scale = q_scale;
  j.state = state; j.slot_stride = slot_stride; j.H = H; j.G = G; j.D = D; j.V = V;
  j.cu_q = cu_q; j.state_slots = state_slots; j.n_seqs = n_seqs; j.places = places; j.out = out; j.ldo = ldo;
  float* at = workspace;
  j.qd = at; at += p.rows;
  j.kd = at; at += p.rows;
  if (delta) { j.w = at; at += p.rows; }
  j.p = at; at += p.square;
  if (delta) { j.kk = at; at += p.square; }
  j.gend = at; at += p.ends;
  if (delta) j.u0 = at;
  auto launch = [&](auto kern, dim3 grid, int threads, size_t smem, const char* what) {
    if (smem > 48 * 1024 && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return zi_refuse("%s: cannot get %zu bytes of shared memory", what, smem);
    zi_launch(kern, grid, dim3(threads), smem, stream, j);
    return zi_check_launch(what);
  };
  const size_t score_smem = ((size_t)3 * RK * (D + 8) + 3 * SUBS * D) * sizeof(float);
  const size_t solve_smem = ((size_t)RK * KK_PITCH + RK + (size_t)RK * SO_COLS) * sizeof(float);
  int rc = 0;
  ZI_DISPATCH_DTYPE(qk_dtype, TQ, {
    rc = launch(delta ? channel_scores_kernel<TQ, true> : channel_scores_kernel<TQ, false>, dim3(places, H), SC_THREADS, score_smem, "channel_scores");
  });
  if (rc) return rc;
  ZI_DISPATCH_DTYPE(v_dtype, TV, {
    if (delta) {
      rc = launch(channel_solve_kernel<TV>, dim3(places, H, (D + V + SO_COLS - 1) / SO_COLS), SO_COLS, solve_smem, "channel_solve");
      if (rc) return rc;
    }
    rc = launch(delta ? channel_walk_kernel<TV, true> : channel_walk_kernel<TV, false>, dim3(n_seqs, H, (V + RV - 1) / RV), WK_THREADS,
                channel_walk_smem(D, delta != 0), "channel_walk");
  });
  return rc;
}

ZI_TRACE_SETTER(channel_recurrence)
