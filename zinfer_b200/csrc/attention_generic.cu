// Causal attention of query tokens against the paged cache, for any mix of prompt
// portions and single decoded tokens, any head size up to 256 in steps of 2, any
// number of heads and groups, with an optional window that may also keep a request's
// first tokens visible (keep_first).  32-bit arithmetic on the
// CUDA cores (exact expf); the storage type alone differs between the float32 path
// and the plain bfloat16 path.  A query row visits its keys in ascending order in
// tiles aligned to multiples of BK, so its result does not depend on how the
// request was cut into steps or on what else is in the batch.
//
// Grid: (query tile of BQ tokens of one request, query head).  Pages are
// [page][kv head][offset][d]; the key at position j of request s lies in page
// block_tables[s][j / page_size] at offset j % page_size.
#include "api.h"
#include "common.cuh"

namespace {
constexpr int BQ = 16, BK = 32, THREADS = 128, ROWS_PER_WARP = BQ / (THREADS / 32);

// Values may have another size than keys and may lie in the key rows themselves (a latent cache whose row
// serves as key and, in its first dv columns, as value): dv value columns are read from rows of
// v_row elements in `vcache`; the output has dv columns per head.  MAXJ * 32 bounds dv.
// With a window, query i sees key j <= i if i - j < window or j < keep_first.  With pooled blocks (pool.per > 0) it also
// sees one key and value for every block of `per` tokens that lies wholly before its window: entry b of the request's
// pooled pages, if b per + per - 1 <= i - window.  They are walked first; all keys share one softmax.
// Changes to the score, each off unless given: softcap c (s <- c tanh(s / c) after the scale), dist_bias
// [heads][n_dist] (a bias by the distance i - j, distances from n_dist - 1 on share the last entry; added after
// the cap), sink_logit [heads] (exp(sink_logit[h]) joins head h's denominator; it has no value).
template <typename T, int MAXJ>
__global__ void __launch_bounds__(THREADS)
paged_attention_kernel(T* __restrict__ out, int out_stride, const T* __restrict__ q, int q_stride,
                       const T* __restrict__ kcache, const T* __restrict__ vcache,
                       const int* __restrict__ block_tables, int bt_stride, const int* __restrict__ cu_q,
                       const int* __restrict__ kv_lens, const int* __restrict__ tile_seq,
                       const int* __restrict__ tile_q0, int nq, int nkv, int d, int page_size, int window,
                       float scale, int dv, int v_row, int skip_from, int skip_single, float sink, int keep_first,
                       const float* __restrict__ sink_logit, float softcap, const float* __restrict__ dist_bias,
                       int n_dist, const PooledKeys pool) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ float smem[];
  float* Qs = smem;                   // [BQ][d]
  float* Ks = Qs + BQ * d;            // [BK][d+1]
  float* Vs = Ks + BK * (d + 1);      // [BK][dv]
  float* Ss = Vs + BK * dv;           // [BQ][BK]

  const int seq = tile_seq[blockIdx.x], q0 = tile_q0[blockIdx.x];
  const int h = blockIdx.y, kvh = h / (nq / nkv);
  const int tok0 = cu_q[seq], qlen = cu_q[seq + 1] - tok0, kvlen = kv_lens[seq];
  const int ctx = kvlen - qlen;  // tokens of this request already in the cache before this step
  const int nqv = min(BQ, qlen - q0);
  if (nqv <= 0 || (skip_from > 0 && qlen >= skip_from) || (skip_single && qlen == 1)) return;
  const int first_pos = ctx + q0, last_pos = first_pos + nqv - 1;
  const int kv_begin = window > 0 ? max(0, first_pos - window + 1) : 0;
  const int kv_end = last_pos + 1;
  // keys [0, keep_end) lie before the window and stay visible; the tiles between them and the window are skipped
  const int keep_end = window > 0 ? min(keep_first, kv_begin) : 0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int* bt = block_tables + (size_t)seq * bt_stride;

  for (int e = tid; e < BQ * d; e += THREADS) {
    const int r = e / d, c = e % d;
    Qs[e] = r < nqv ? to_f32(q[(size_t)(tok0 + q0 + r) * q_stride + (size_t)h * d + c]) : 0.f;
  }

  float m[ROWS_PER_WARP], l[ROWS_PER_WARP], acc[ROWS_PER_WARP][MAXJ];
#pragma unroll
  for (int i = 0; i < ROWS_PER_WARP; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
#pragma unroll
    for (int j = 0; j < MAXJ; ++j) acc[i][j] = 0.f;
  }

  const int n_pooled = pooled_visible(pool, last_pos, window);          // what the tile's last query sees
  const T* kpool = static_cast<const T*>(pool.k);
  const T* vpool = static_cast<const T*>(pool.v);
  const int* pbt = pool.block_tables + (size_t)seq * pool.bt_stride;
  // tiles of pooled entries first (ahead > 0), then the tokens'
  int ahead = (n_pooled + BK - 1) / BK, kt = ahead > 0 ? 0 : (keep_end > 0 ? 0 : (kv_begin / BK) * BK);
  for (; ahead > 0 || kt < kv_end; kt += BK) {
    const bool of_blocks = ahead > 0;
    if (!of_blocks && kt >= keep_end && kt + BK <= kv_begin) {   // a tile wholly between the kept first tokens and the window
      kt = (kv_begin / BK) * BK - BK;
      continue;
    }
    __syncthreads();  // previous tile fully consumed (also orders the Q load the first time)
    for (int e = tid; e < BK * d; e += THREADS) {
      const int kk = e / d, c = e % d;
      const int j = kt + kk;
      float kval = 0.f;
      if (of_blocks) {
        const int page = j < n_pooled ? pbt[j / page_size] : -1;
        if (page >= 0) kval = to_f32(kpool[(((size_t)page * nkv + kvh) * page_size + (j % page_size)) * d + c]);
      } else if ((j >= kv_begin || j < keep_end) && j < kv_end) {
        const int page = bt[j / page_size];
        if (page >= 0) kval = to_f32(kcache[(((size_t)page * nkv + kvh) * page_size + (j % page_size)) * d + c]);
      }
      Ks[kk * (d + 1) + c] = kval;
    }
    for (int e = tid; e < BK * dv; e += THREADS) {
      const int kk = e / dv, c = e % dv;
      const int j = kt + kk;
      float vval = 0.f;
      if (of_blocks) {
        const int page = j < n_pooled ? pbt[j / page_size] : -1;
        if (page >= 0) vval = to_f32(vpool[(((size_t)page * nkv + kvh) * page_size + (j % page_size)) * dv + c]);
      } else if ((j >= kv_begin || j < keep_end) && j < kv_end) {
        const int page = bt[j / page_size];
        if (page >= 0) vval = to_f32(vcache[(((size_t)page * nkv + kvh) * page_size + (j % page_size)) * v_row + c]);
      }
      Vs[e] = vval;
    }
    __syncthreads();

    float alpha[ROWS_PER_WARP];
#pragma unroll
    for (int i = 0; i < ROWS_PER_WARP; ++i) {
      const int r = warp * ROWS_PER_WARP + i;
      alpha[i] = 1.f;
      if (r >= nqv) continue;  // uniform within the warp
      const int pos = first_pos + r, j = kt + lane;
      const float* qr = Qs + r * d;
      const float* kr = Ks + lane * (d + 1);
      float s = 0.f;
      for (int c = 0; c < d; ++c) s = fmaf(qr[c], kr[c], s);
      s *= scale;
      if (softcap > 0.f) s = softcap * tanhf(s / softcap);
      const bool visible = of_blocks ? j < pooled_visible(pool, pos, window)
                                     : j <= pos && (window <= 0 || j > pos - window || j < keep_first);
      if (!visible) s = -INFINITY;
      else if (dist_bias) s += dist_bias[(size_t)h * n_dist + min(pos - j, n_dist - 1)];   // not scaled, not capped
      const float m_new = fmaxf(m[i], warp_max(s));
      float p = 0.f;
      if (m_new != -INFINITY) {
        p = visible ? expf(s - m_new) : 0.f;
        alpha[i] = expf(m[i] - m_new);  // exp(-inf) = 0 on the first visible tile
      }
      l[i] = l[i] * alpha[i] + warp_sum(p);
      m[i] = m_new;
      Ss[r * BK + lane] = p;
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < ROWS_PER_WARP; ++i) {
      const int r = warp * ROWS_PER_WARP + i;
      if (r >= nqv) continue;
#pragma unroll
      for (int j = 0; j < MAXJ; ++j) acc[i][j] *= alpha[i];
      for (int kk = 0; kk < BK; ++kk) {
        const float p = Ss[r * BK + kk];
#pragma unroll
        for (int j = 0; j < MAXJ; ++j) {
          const int c = lane + 32 * j;
          if (c < dv) acc[i][j] = fmaf(p, Vs[kk * dv + c], acc[i][j]);
        }
      }
    }
    if (of_blocks && --ahead == 0) kt = (keep_end > 0 ? 0 : (kv_begin / BK) * BK) - BK;   // on with the tokens
  }
#pragma unroll
  for (int i = 0; i < ROWS_PER_WARP; ++i) {
    const int r = warp * ROWS_PER_WARP + i;
    if (r >= nqv) continue;
    // a sink: `sink` keys whose score is 0 and which have no value, counted in the denominator only
    // a learned sink: exp(sink_logit[h]) in the denominator, neither scaled nor capped
    const float inv = 1.0f / (sink_logit ? l[i] + expf(sink_logit[h] - m[i]) : (sink > 0.f ? l[i] + sink * expf(-m[i]) : l[i]));
    T* o = out + (size_t)(tok0 + q0 + r) * out_stride + (size_t)h * dv;
#pragma unroll
    for (int j = 0; j < MAXJ; ++j) {
      const int c = lane + 32 * j;
      if (c < dv) o[c] = from_f32<T>(acc[i][j] * inv);
    }
  }
}

// The same attention for float pages in its plain form (no sink, cap, bias by distance, kept first tokens or pooled
// blocks; values of the keys' size D): a block takes the HG query heads (up to four) that share a kv head for one tile
// of BQ tokens, so that a key tile is fetched once for all of them, by cp.async into two buffers, and a thread works on
// several rows and columns at once, reading shared memory in 16-byte pieces.  Every row's arithmetic is that of the
// kernel above, operation for operation (one chain over the head's channels, one softmax step per tile of BK keys in
// the same order, one chain over a tile's keys), so both give the same bits.
// Bound by shared-memory reads in prompts and by the chain of a tile's steps for single tokens.  Measured, 16 heads of 64
// over 4 kv heads: prompts of 354 and 158 tokens 281 -> 101 us, 12 requests with prompts of 46 to 134 tokens through
// prompts and 24 decoded tokens each 113 -> 23 us a launch.  A short prompt of one request has a quarter of the plain kernel's
// blocks and gains all the same: 16 tokens 21 -> 13 us, 64 tokens 47 -> 21.
template <int D, int HG>
struct F32Attention {
  static constexpr int ROWS = BQ * HG, KP = D + 4, SP = BK + 4;         // pitches: rows four banks apart
  static constexpr int CG = D / 4, RG = THREADS / CG > ROWS ? ROWS : THREADS / CG, RPT = ROWS / RG;
  static constexpr int WR = ROWS / (THREADS / 32);                       // softmax rows per warp
  static constexpr size_t SMEM = (size_t)(ROWS * KP + 2 * BK * (KP + D) + ROWS * SP + ROWS) * sizeof(float);
};

template <int D, int HG>
__global__ void __launch_bounds__(THREADS)
paged_attention_f32_kernel(float* __restrict__ out, int out_stride, const float* __restrict__ q, int q_stride,
                           const float* __restrict__ kcache, const float* __restrict__ vcache,
                           const int* __restrict__ block_tables, int bt_stride, const int* __restrict__ cu_q,
                           const int* __restrict__ kv_lens, const int* __restrict__ tile_seq, const int* __restrict__ tile_q0,
                           int nq, int nkv, int page_size, int window, float scale) {
  using L = F32Attention<D, HG>;
  constexpr int ROWS = L::ROWS, KP = L::KP, SP = L::SP, CG = L::CG, RG = L::RG, RPT = L::RPT, WR = L::WR, PIECES = D / 4;
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float smem[];
  float* Qs = smem;                         // [ROWS][KP], row = head * BQ + token
  float* Ks = Qs + ROWS * KP;               // [2][BK][KP]
  float* Vs = Ks + 2 * BK * KP;             // [2][BK][D]
  float* Ss = Vs + 2 * BK * D;              // [ROWS][SP]
  float* As = Ss + ROWS * SP;               // [ROWS]: what the row's sums so far are multiplied by

  const int seq = tile_seq[blockIdx.x], q0 = tile_q0[blockIdx.x];
  const int group = nq / nkv, parts = (group + HG - 1) / HG;
  const int kvh = blockIdx.y / parts, h0 = kvh * group + (blockIdx.y % parts) * HG;
  const int heads = min(HG, (kvh + 1) * group - h0);
  const int tok0 = cu_q[seq], qlen = cu_q[seq + 1] - tok0, kvlen = kv_lens[seq];
  const int nqv = min(BQ, qlen - q0);
  if (nqv <= 0) return;
  const int first_pos = kvlen - qlen + q0, kv_end = first_pos + nqv;
  const int kv_begin = window > 0 ? max(0, first_pos - window + 1) : 0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int* bt = block_tables + (size_t)seq * bt_stride;
  const bool single = nqv == 1;

  for (int e = tid; e < ROWS * PIECES; e += THREADS) {
    const int r = e / PIECES, c = (e % PIECES) * 4, head = r / BQ, t = r % BQ;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < nqv && head < heads) v = *reinterpret_cast<const float4*>(q + (size_t)(tok0 + q0 + t) * q_stride + (size_t)(h0 + head) * D + c);
    *reinterpret_cast<float4*>(Qs + r * KP + c) = v;
  }
  auto fill = [&](int kt, int buf) {
#pragma unroll
    for (int e = tid; e < BK * PIECES; e += THREADS) {
      const int kk = e / PIECES, c = (e % PIECES) * 4, j = kt + kk;
      int page = -1;
      if (j >= kv_begin && j < kv_end) page = bt[j / page_size];
      const size_t at = page >= 0 ? (((size_t)page * nkv + kvh) * page_size + (j % page_size)) * D + c : 0;
      const int valid = page >= 0 ? 16 : 0;      // the rest of the piece is filled with zeros
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(Ks + (buf * BK + kk) * KP + c)),
                   "l"(kcache + at), "r"(valid) : "memory");
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(Vs + (buf * BK + kk) * D + c)),
                   "l"(vcache + at), "r"(valid) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  float m[WR], l[WR];
#pragma unroll
  for (int i = 0; i < WR; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
  }
  // rows ag + i RG, columns cg 4 .. + 3; for a single token: row warp * BQ (a head a warp), columns lane + 32 j in acc[0]
  float acc[RPT][4];
#pragma unroll
  for (int i = 0; i < RPT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  const int cg = tid % CG, rg = tid / CG;

  int kt = (kv_begin / BK) * BK, buf = 0;
  fill(kt, 0);
  for (; kt < kv_end; kt += BK, buf ^= 1) {
    __syncthreads();                        // the buffer that is filled next has been read
    if (kt + BK < kv_end) {
      fill(kt + BK, buf ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const float* K0 = Ks + buf * BK * KP;
    const float* V0 = Vs + buf * BK * D;
    if (single) {
      if (warp < heads) {
        const float* qr = Qs + warp * BQ * KP;
        const float* kr = K0 + lane * KP;
        float s = 0.f;
#pragma unroll 8
        for (int c = 0; c < D; c += 4) {
          const float4 a = *reinterpret_cast<const float4*>(qr + c), b = *reinterpret_cast<const float4*>(kr + c);
          s = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s))));
        }
        Ss[warp * BQ * SP + lane] = s;
      }
    } else {
      // thread: token tid / 8 of every head, keys tid % 8 + 8 j
      const float* qr = Qs + (tid >> 3) * KP;
      const float* kr = K0 + (tid & 7) * KP;
      float s[HG][4];
#pragma unroll
      for (int i = 0; i < HG; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 2
      for (int c = 0; c < D; c += 4) {
        float4 a[HG], b[4];
#pragma unroll
        for (int i = 0; i < HG; ++i) a[i] = *reinterpret_cast<const float4*>(qr + i * BQ * KP + c);
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(kr + j * 8 * KP + c);
#pragma unroll
        for (int i = 0; i < HG; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) s[i][j] = fmaf(a[i].w, b[j].w, fmaf(a[i].z, b[j].z, fmaf(a[i].y, b[j].y, fmaf(a[i].x, b[j].x, s[i][j]))));
      }
#pragma unroll
      for (int i = 0; i < HG; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) Ss[(i * BQ + (tid >> 3)) * SP + (tid & 7) + 8 * j] = s[i][j];
    }
    __syncthreads();
    // a warp's rows in turn, a key per lane
#pragma unroll
    for (int i = 0; i < WR; ++i) {
      const int r = warp * WR + i, t = r % BQ;
      if (t >= nqv || r / BQ >= heads) continue;          // uniform within the warp
      const int pos = first_pos + t, j = kt + lane;
      float s = Ss[r * SP + lane] * scale;
      const bool visible = j <= pos && (window <= 0 || j > pos - window);
      if (!visible) s = -INFINITY;
      const float m_new = fmaxf(m[i], warp_max(s));
      float p = 0.f, alpha = 1.f;
      if (m_new != -INFINITY) {
        p = visible ? expf(s - m_new) : 0.f;
        alpha = expf(m[i] - m_new);
      }
      l[i] = l[i] * alpha + warp_sum(p);
      m[i] = m_new;
      Ss[r * SP + lane] = p;
      if (lane == 0) As[r] = alpha;
    }
    __syncthreads();
    if (single) {
      if (warp < heads) {
        const float alpha = As[warp * BQ];
        const float* pr = Ss + warp * BQ * SP;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int c = lane + 32 * j;
          if (c < D) {
            float a = acc[0][j] * alpha;
#pragma unroll 8
            for (int kk = 0; kk < BK; ++kk) a = fmaf(pr[kk], V0[kk * D + c], a);
            acc[0][j] = a;
          }
        }
      }
    } else if (rg < RG) {
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        const float alpha = As[rg + i * RG];
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] *= alpha;
      }
#pragma unroll 2
      for (int kk = 0; kk < BK; kk += 4) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = *reinterpret_cast<const float4*>(V0 + (kk + u) * D + cg * 4);
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          const float4 p = *reinterpret_cast<const float4*>(Ss + (rg + i * RG) * SP + kk);
          acc[i][0] = fmaf(p.w, v[3].x, fmaf(p.z, v[2].x, fmaf(p.y, v[1].x, fmaf(p.x, v[0].x, acc[i][0]))));
          acc[i][1] = fmaf(p.w, v[3].y, fmaf(p.z, v[2].y, fmaf(p.y, v[1].y, fmaf(p.x, v[0].y, acc[i][1]))));
          acc[i][2] = fmaf(p.w, v[3].z, fmaf(p.z, v[2].z, fmaf(p.y, v[1].z, fmaf(p.x, v[0].z, acc[i][2]))));
          acc[i][3] = fmaf(p.w, v[3].w, fmaf(p.z, v[2].w, fmaf(p.y, v[1].w, fmaf(p.x, v[0].w, acc[i][3]))));
        }
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < WR; ++i)
    if (lane == 0) As[warp * WR + i] = 1.0f / l[i];
  __syncthreads();
  if (single) {
    if (warp < heads) {
      const float inv = As[warp * BQ];
      float* o = out + (size_t)(tok0 + q0) * out_stride + (size_t)(h0 + warp) * D;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (lane + 32 * j < D) o[lane + 32 * j] = acc[0][j] * inv;
    }
    return;
  }
  if (rg >= RG) return;
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int r = rg + i * RG, t = r % BQ, head = r / BQ;
    if (t >= nqv || head >= heads) continue;
    const float inv = As[r];
    float* o = out + (size_t)(tok0 + q0 + t) * out_stride + (size_t)(h0 + head) * D + cg * 4;
    *reinterpret_cast<float4*>(o) = make_float4(acc[i][0] * inv, acc[i][1] * inv, acc[i][2] * inv, acc[i][3] * inv);
  }
}

template <int D, int HG>
int launch_f32_attention(float* out, int out_stride, const float* q, int q_stride, const float* kcache, const float* vcache,
                         const int* block_tables, int bt_stride, const int* cu_q, const int* kv_lens, const int* tile_seq,
                         const int* tile_q0, int n_tiles, int nq, int nkv, int page_size, int window, float scale, cudaStream_t stream) {
  auto kern = paged_attention_f32_kernel<D, HG>;
  constexpr size_t bytes = F32Attention<D, HG>::SMEM;
  if (bytes > 48 * 1024 && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess)
    return zi_refuse("paged_attention: cannot get %zu bytes of shared memory", bytes);
  const int group = nq / nkv;
  zi_launch(kern, dim3(n_tiles, nkv * ((group + HG - 1) / HG)), dim3(THREADS), bytes, stream, out, out_stride, q, q_stride, kcache, vcache,
            block_tables, bt_stride, cu_q, kv_lens, tile_seq, tile_q0, nq, nkv, page_size, window, scale);
  return zi_check_launch("paged_attention (32-bit)");
}
}  // namespace

extern "C" int zi_paged_attention_tile_rows() { return BQ; }

extern "C" int zi_paged_attention(void* out, int out_stride, const void* q, int q_stride, int dtype,
                                  const void* kcache, const void* vcache, const int* block_tables, int bt_stride,
                                  const int* cu_q, const int* kv_lens, const int* tile_seq, const int* tile_q0,
                                  int n_tiles, int nq, int nkv, int d, int page_size, int window, float scale,
                                  cudaStream_t stream) {
  return zi_paged_attention_v(out, out_stride, q, q_stride, dtype, kcache, vcache, block_tables, bt_stride, cu_q, kv_lens,
                              tile_seq, tile_q0, n_tiles, nq, nkv, d, d, d, page_size, window, scale, 0, 0, stream);
}

extern "C" int zi_paged_attention_v(void* out, int out_stride, const void* q, int q_stride, int dtype,
                                    const void* kcache, const void* vcache, const int* block_tables, int bt_stride,
                                    const int* cu_q, const int* kv_lens, const int* tile_seq, const int* tile_q0,
                                    int n_tiles, int nq, int nkv, int d, int dv, int v_row, int page_size, int window,
                                    float scale, int skip_from, int skip_single, cudaStream_t stream) {
  return zi_paged_attention_sink(out, out_stride, q, q_stride, dtype, kcache, vcache, block_tables, bt_stride, cu_q, kv_lens,
                                 tile_seq, tile_q0, n_tiles, nq, nkv, d, dv, v_row, page_size, window, scale, skip_from,
                                 skip_single, 0.f, stream);
}

extern "C" int zi_paged_attention_sink(void* out, int out_stride, const void* q, int q_stride, int dtype,
                                       const void* kcache, const void* vcache, const int* block_tables, int bt_stride,
                                       const int* cu_q, const int* kv_lens, const int* tile_seq, const int* tile_q0,
                                       int n_tiles, int nq, int nkv, int d, int dv, int v_row, int page_size, int window,
                                       float scale, int skip_from, int skip_single, float sink, cudaStream_t stream) {
  return zi_paged_attention_mask(out, out_stride, q, q_stride, dtype, kcache, vcache, block_tables, bt_stride, cu_q, kv_lens,
                                 tile_seq, tile_q0, n_tiles, nq, nkv, d, dv, v_row, page_size, window, 0, scale, skip_from,
                                 skip_single, sink, stream);
}

// The general form: a sink, values of any size (dv columns of rows of v_row elements), and a window that
// keeps the first keep_first tokens of a request visible.
extern "C" int zi_paged_attention_mask(void* out, int out_stride, const void* q, int q_stride, int dtype,
                                       const void* kcache, const void* vcache, const int* block_tables, int bt_stride,
                                       const int* cu_q, const int* kv_lens, const int* tile_seq, const int* tile_q0,
                                       int n_tiles, int nq, int nkv, int d, int dv, int v_row, int page_size, int window,
                                       int keep_first, float scale, int skip_from, int skip_single, float sink,
                                       cudaStream_t stream) {
  return zi_paged_attention_mods(out, out_stride, q, q_stride, dtype, kcache, vcache, block_tables, bt_stride, cu_q, kv_lens,
                                 tile_seq, tile_q0, n_tiles, nq, nkv, d, dv, v_row, page_size, window, keep_first, scale,
                                 skip_from, skip_single, sink, nullptr, 0.f, nullptr, 0, nullptr, nullptr, nullptr, 0, 0, stream);
}

// The same with the changes to the score (a learned sink per head, a cap, a bias by distance), and with pooled keys and
// values: pages of one entry per pool_per tokens beside the window's tokens (0: none).
extern "C" int zi_paged_attention_mods(void* out, int out_stride, const void* q, int q_stride, int dtype,
                                       const void* kcache, const void* vcache, const int* block_tables, int bt_stride,
                                       const int* cu_q, const int* kv_lens, const int* tile_seq, const int* tile_q0,
                                       int n_tiles, int nq, int nkv, int d, int dv, int v_row, int page_size, int window,
                                       int keep_first, float scale, int skip_from, int skip_single, float sink,
                                       const float* sink_logit, float softcap, const float* dist_bias, int n_dist,
                                       const void* kpool, const void* vpool, const int* pool_tables, int pool_bt_stride,
                                       int pool_per, cudaStream_t stream) {
  if (n_tiles <= 0) return 0;
  if (!(softcap >= 0.f)) return zi_refuse("paged_attention: the cap on the scores must not be negative");
  if (dist_bias && n_dist <= 0) return zi_refuse("paged_attention: a bias by distance needs a table");
  if (sink_logit && sink != 0.f) return zi_refuse("paged_attention: a learned sink and a counted sink exclude each other");
  if (keep_first < 0) return zi_refuse("paged_attention: %d kept first tokens", keep_first);
  if (!(sink >= 0.f)) return zi_refuse("paged_attention: the sink's weight must not be negative");
  constexpr int WIDE = 20;   // value columns up to 640 (latent caches); 8 serves every ordinary head size
  if (d <= 0 || d > 32 * WIDE) return zi_refuse("paged_attention: head_dim %d is outside 1..%d", d, 32 * WIDE);
  if (dv <= 0 || dv > 32 * WIDE || v_row < dv) return zi_refuse("paged_attention: %d value columns of rows of %d, keys of %d", dv, v_row, d);
  if (nkv <= 0 || nq % nkv) return zi_refuse("paged_attention: %d query heads do not divide into %d kv heads", nq, nkv);
  if (page_size <= 0) return zi_refuse("paged_attention: page_size %d", page_size);
  if (pool_per > 0 && (!kpool || !vpool || !pool_tables || window <= 0 || dist_bias || v_row != dv))
    return zi_refuse("paged_attention: pooled keys go with a window, pages of their own and no bias by distance");
  // Float pages in the plain form, rows on 16-byte boundaries, the head sizes that real models use: the kernel for groups of heads.
  const bool aligned = ((uintptr_t)out | (uintptr_t)q | (uintptr_t)kcache | (uintptr_t)vcache) % 16 == 0 && out_stride % 4 == 0 && q_stride % 4 == 0;
  if (dtype == ZI_F32 && aligned && dv == d && v_row == d && (d == 16 || d == 32 || d == 64 || d == 128) && !skip_from && !skip_single &&
      sink == 0.f && !sink_logit && softcap == 0.f && !dist_bias && !keep_first && pool_per <= 0) {
    const int group = nq / nkv;
#define ZI_F32_ATTENTION(D, HG)                                                                                                  \
  return launch_f32_attention<D, HG>((float*)out, out_stride, (const float*)q, q_stride, (const float*)kcache, (const float*)vcache, \
                                     block_tables, bt_stride, cu_q, kv_lens, tile_seq, tile_q0, n_tiles, nq, nkv, page_size, window, \
                                     scale, stream)
#define ZI_F32_HEADS(D)                                        \
  do {                                                         \
    if (group == 1) ZI_F32_ATTENTION(D, 1);                    \
    if (group == 2) ZI_F32_ATTENTION(D, 2);                    \
    ZI_F32_ATTENTION(D, 4);                                    \
  } while (0)
    if (d == 16) ZI_F32_HEADS(16);
    if (d == 32) ZI_F32_HEADS(32);
    if (d == 64) ZI_F32_HEADS(64);
    ZI_F32_HEADS(128);
#undef ZI_F32_HEADS
#undef ZI_F32_ATTENTION
  }
  const PooledKeys pool = {kpool, vpool, pool_tables, pool_bt_stride, pool_per, d, dv};
  const size_t smem = (size_t)(BQ * d + BK * (d + 1) + BK * dv + BQ * BK) * sizeof(float);
  dim3 grid(n_tiles, nq);
#define ZI_LAUNCH_ATTN(J)                                                                                          \
  do {                                                                                                             \
    auto kern = paged_attention_kernel<TT, J>;                                                                     \
    if (smem > 48 * 1024) {                                                                                        \
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);          \
      if (e != cudaSuccess) return zi_refuse("paged_attention: cannot get %zu bytes of shared memory", smem);      \
    }                                                                                                              \
    zi_launch(kern, dim3(grid), dim3(THREADS), smem, stream, (TT*)out, out_stride, (const TT*)q, q_stride,         \
              (const TT*)kcache, (const TT*)vcache, block_tables, bt_stride, cu_q, kv_lens, tile_seq, tile_q0, nq, \
              nkv, d, page_size, window, scale, dv, v_row, skip_from, skip_single, sink, keep_first, sink_logit,    \
              softcap, dist_bias, n_dist, pool);                                                                       \
  } while (0)
  ZI_DISPATCH_DTYPE(dtype, TT, {
    if (dv <= 256) ZI_LAUNCH_ATTN(8);
    else ZI_LAUNCH_ATTN(WIDE);
  });
#undef ZI_LAUNCH_ATTN
  return zi_check_launch("paged_attention");
}

ZI_TRACE_SETTER(attention_generic)
