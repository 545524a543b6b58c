// The two delta rules (one decay a head, or one a key channel) over portions of prompts, in chunks of 32 tokens and
// 32-bit throughout.  With G_t[c] the product of a chunk's decays of channel c up to and with token t, S0 the matrix
// (dim x vdim) before the chunk, and products of decays only (never quotients, so nothing can overflow),
//     A[t][s] = beta_t sum_c k_t[c] k_s[c] g_{s+1}[c] .. g_t[c]   (s < t)
//     (I + A) W = beta G k,   (I + A) U0 = beta v                 (the same triangle, solved by substitution)
//     U = U0 - W S0;   o_t = (G_t q_t) S0 + sum_{s<=t} M[t][s] u_s,   M[t][s] = sum_c q_t[c] k_s[c] g_{s+1}[c] .. g_t[c]
//     S32 = G_31 S0 + sum_s (g_{s+1} .. g_31 k_s) u_s^T
// Everything but the lines with S0 is the same work for every chunk whatever came before it, and is done for all
// chunks at once; what stays one after another is two products of 32 x 128 with the matrix and one back, whose
// columns are independent and are cut over blocks.  A decay a head is the same with equal channels.
//
//   delta_chunk_prepare   a block a (chunk, head): the short convolution over time with silu (its inputs straight from
//                         the stacked product, and from the kept inputs in front of a portion), unit vectors, decays,
//                         then A, M, W, U0 and the scaled queries and keys as one record.  The sums between tokens of
//                         unlike eighths of a chunk are plain products of rows that were scaled up to the eighth's edge;
//                         inside an eighth the decays are multiplied in key by key
//   delta_chunk_scan      a block a (16 columns of a head's matrix, request): the chunks one after another.  The 64 x
//                         128 rows of W and G q meet the columns in 4 x 4 register tiles, k cut over four pairs of warps;
//                         the next chunk's record is on its way (cp.async) while this one is worked through
//
// A request's chunks are counted from its portion's first row; the record of chunk c of request r lies at place
// q_start[r] / 32 + r + c (no two the same, and known without a pass over the other requests).
#include "common.cuh"

#define DC_TOKENS 32
#define DC_DIM 128                        // lanes of a key, zeros behind the head's own
#define DC_COLS 16                        // columns of a scan block
#define DC_MAX_TAPS 16
#define DC_PREPARE_THREADS 256
#define DC_SCAN_THREADS 256
constexpr int kDcStride = DC_DIM + 4;     // of rows that several lanes read at once, 16 bytes each
constexpr int kDcPairs = DC_TOKENS + 4;   // of A's and M's rows
// a record, in floats: W, G q, decayed k (32 x 128 each), M (32 x 32), G_31 (128), U0 (32 x vdim)
constexpr int kDcQ = DC_TOKENS * DC_DIM, kDcK = 2 * kDcQ, kDcM = 3 * kDcQ, kDcG = kDcM + DC_TOKENS * DC_TOKENS,
              kDcU = kDcG + DC_DIM;

__device__ __forceinline__ float dc_sigmoid(float v) { return 1.0f / (1.0f + expf(-v)); }
__device__ __forceinline__ float dc_softplus(float v) { return v > 20.f ? v : log1pf(expf(v)); }

struct DeltaChunkArgs {
  const void* proj;          // the stacked input product [T, ld]: q, k, v at qkv_at, the projection behind beta at b_at
  int ld, qkv_at, b_at;
  const void* decay;         // what stands in front of the decays' softplus: columns decay_at .. of [T, decay_ld]
  int decay_ld, decay_at;    // (one a head, or dim a head)
  const float* conv_w;       // [channels, taps]
  const float* a_log;        // [heads]
  const float* dt_bias;      // [heads] or [heads * dim]
  const float* state;        // the kept inputs at conv_off of a request's slot
  long long state_stride;
  const int* q_start;
  const int* state_slot;
  float* records;
  float q_scale;
  int groups, heads, dim, vdim, taps, conv_off, n_requests;
};

// T: type of proj (and of `decay` where it is one a head: the same product's columns)
template <typename T, bool BY_CHANNEL>
__global__ void __launch_bounds__(DC_PREPARE_THREADS, 2) delta_chunk_prepare_kernel(const DeltaChunkArgs a) {
  extern __shared__ __align__(16) float dc_raw[];
  float* q_s = dc_raw;                                  // [32][132] each
  float* k_s = q_s + DC_TOKENS * kDcStride;
  float* g_s = k_s + DC_TOKENS * kDcStride;
  float* r_s = g_s + DC_TOKENS * kDcStride;             // keys decayed up to the next eighth's edge
  float* l_s = r_s + DC_TOKENS * kDcStride;             // an eighth's keys, then its queries, decayed from its edge on
  float* a_s = l_s + 16 * kDcStride;                    // [32][36]
  float* m_s = a_s + DC_TOKENS * kDcPairs;              // [32][36]
  float* beta_s = m_s + DC_TOKENS * kDcPairs;           // [32]
  const int place = blockIdx.x, h = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the request whose chunks lie around this place: the last one that begins at or before it
  int r = -1;
  for (int i0 = 0; i0 < a.n_requests; i0 += 32) {
    const int i = i0 + lane;
    r += __popc(__ballot_sync(0xffffffffu, i < a.n_requests && a.q_start[i] / DC_TOKENS + i <= place));
  }
  const int start = r >= 0 ? a.q_start[r] : 0;
  const int at0 = r >= 0 ? (place - start / DC_TOKENS - r) * DC_TOKENS : 0;      // the chunk's first token's place in its portion
  const int t0 = start + at0;
  const int n_here = r >= 0 ? min(DC_TOKENS, a.q_start[r + 1] - t0) : 0;
  pdl_wait();
  pdl_launch();
  if (n_here <= 0) return;
  const int group = h / (a.heads / a.groups);
  const int channels = 2 * a.groups * a.dim + a.heads * a.vdim;
  const float* kept = a.state + (size_t)a.state_slot[r] * a.state_stride + a.conv_off;
  const T* proj = static_cast<const T*>(a.proj);
  float* rec = a.records + ((size_t)place * a.heads + h) * (size_t)(kDcU + DC_TOKENS * a.vdim);

  // ---- convolution and silu: a channel a thread, down the chunk's tokens ----
  auto convolve = [&](int ch, float (&y)[DC_TOKENS]) {
    const T* in = proj + a.qkv_at + ch;
    const float* w = a.conv_w + (size_t)ch * a.taps;
    // an input `back` places before the portion's start is the kept one that many from the end
    auto input = [&](int at) {
      return at >= 0 ? to_float(in[(size_t)(start + at) * a.ld]) : kept[(size_t)(a.taps - 1 + at) * channels + ch];
    };
    if (a.taps == 4) {
      const float w0 = w[0], w1 = w[1], w2 = w[2], w3 = w[3];
      float x0 = input(at0 - 3), x1 = input(at0 - 2), x2 = input(at0 - 1);
#pragma unroll
      for (int t = 0; t < DC_TOKENS; ++t) y[t] = t < n_here ? to_float(in[(size_t)(t0 + t) * a.ld]) : 0.f;
#pragma unroll
      for (int t = 0; t < DC_TOKENS; ++t) {
        const float x3 = y[t];
        const float v = fmaf(w3, x3, fmaf(w2, x2, fmaf(w1, x1, w0 * x0)));
        y[t] = t < n_here ? v * dc_sigmoid(v) : 0.f;
        x0 = x1; x1 = x2; x2 = x3;
      }
    } else {
#pragma unroll
      for (int t = 0; t < DC_TOKENS; ++t) {
        float v = 0.f;
        if (t < n_here)
          for (int j = 0; j < a.taps; ++j) v = fmaf(w[j], input(at0 + t - (a.taps - 1 - j)), v);
        y[t] = v * dc_sigmoid(v);
      }
    }
  };
  float col[DC_TOKENS];                                 // threads 128 ..: a column of v, later of U0; below: of W
  if (threadIdx.x < DC_DIM) {
    const int l = threadIdx.x;
#pragma unroll 1
    for (int which = 0; which < 2; ++which) {
      float* dst = which ? k_s : q_s;
      if (l < a.dim) {
        convolve((which ? a.groups + group : group) * a.dim + l, col);
      } else {
#pragma unroll
        for (int t = 0; t < DC_TOKENS; ++t) col[t] = 0.f;
      }
#pragma unroll
      for (int t = 0; t < DC_TOKENS; ++t) dst[t * kDcStride + l] = col[t];
    }
  } else {
    const int j = threadIdx.x - DC_DIM;
    if (j < a.vdim) {
      convolve(2 * a.groups * a.dim + h * a.vdim + j, col);
    } else {
#pragma unroll
      for (int t = 0; t < DC_TOKENS; ++t) col[t] = 0.f;
    }
  }
  // ---- decays and beta; A and M start as zeros ----
  {
    const float rate = expf(a.a_log[h]);
    if (BY_CHANNEL) {
      const float* pre = static_cast<const float*>(a.decay) + a.decay_at + h * a.dim;
      for (int i = threadIdx.x; i < DC_TOKENS * DC_DIM; i += DC_PREPARE_THREADS) {
        const int t = i / DC_DIM, l = i % DC_DIM;
        g_s[t * kDcStride + l] = t < n_here && l < a.dim
            ? expf(-rate * dc_softplus(pre[(size_t)(t0 + t) * a.decay_ld + l] + a.dt_bias[h * a.dim + l])) : 1.f;
      }
    } else {
      const T* pre = static_cast<const T*>(a.decay) + a.decay_at + h;
      for (int t = warp; t < DC_TOKENS; t += DC_PREPARE_THREADS / 32) {
        const float g = t < n_here ? expf(-rate * dc_softplus(to_float(pre[(size_t)(t0 + t) * a.decay_ld]) + a.dt_bias[h])) : 1.f;
        *reinterpret_cast<float4*>(g_s + t * kDcStride + lane * 4) = make_float4(g, g, g, g);
      }
    }
    if (threadIdx.x < DC_TOKENS)
      beta_s[threadIdx.x] = threadIdx.x < n_here ? dc_sigmoid(to_float(proj[(size_t)(t0 + threadIdx.x) * a.ld + a.b_at + h])) : 0.f;
    for (int i = threadIdx.x; i < 2 * DC_TOKENS * kDcPairs; i += DC_PREPARE_THREADS) a_s[i] = 0.f;
  }
  __syncthreads();
  // ---- unit vectors: a warp a row, four lanes of it a thread ----
  for (int row = warp; row < 2 * DC_TOKENS; row += DC_PREPARE_THREADS / 32) {
    const bool key = row >= DC_TOKENS;
    float4* at = reinterpret_cast<float4*>((key ? k_s : q_s) + (row % DC_TOKENS) * kDcStride) + lane;
    float4 v = *at;
    const float unit = 1.0f / sqrtf(warp_sum(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w) + 1e-6f) * (key ? 1.f : a.q_scale);
    v.x *= unit; v.y *= unit; v.z *= unit; v.w *= unit;
    *at = v;
    if (key) reinterpret_cast<float4*>(r_s + (row % DC_TOKENS) * kDcStride)[lane] = v;
  }
  __syncthreads();
  // ---- A and M, eight tokens' rows at a time ----
#pragma unroll 1
  for (int e = 0; e < DC_TOKENS; e += 8) {
    {                                                   // the eight's rows, decayed from its first token on
      const int l = threadIdx.x & (DC_DIM - 1);
      const float* src = threadIdx.x < DC_DIM ? k_s : q_s;
      float* dst = l_s + (threadIdx.x < DC_DIM ? 0 : 8) * kDcStride;
      float upto = 1.f;
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        upto *= g_s[(e + t) * kDcStride + l];
        dst[t * kDcStride + l] = upto * src[(e + t) * kDcStride + l];
      }
    }
    {
      // pairs inside the eight: warp w takes token e + w as the key and all eight tokens as the other, those before it
      // with nothing; the sixteen sums cross the lanes together, in 8 + 4 + 2 + 1 exchanges and a last one
      float sums[16];
      float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const float4 kt = reinterpret_cast<const float4*>(k_s + (e + t) * kDcStride)[lane];
        const float4 qt = reinterpret_cast<const float4*>(q_s + (e + t) * kDcStride)[lane];
        const float4 g = reinterpret_cast<const float4*>(g_s + (e + t) * kDcStride)[lane];
        if (t == warp) p = kt;
        else { p.x *= g.x; p.y *= g.y; p.z *= g.z; p.w *= g.w; }
        sums[t] = fmaf(p.x, kt.x, p.y * kt.y) + fmaf(p.z, kt.z, p.w * kt.w);
        sums[8 + t] = fmaf(p.x, qt.x, p.y * qt.y) + fmaf(p.z, qt.z, p.w * qt.w);
      }
#pragma unroll
      for (int width = 8; width > 0; width >>= 1) {        // lanes with the bit keep the upper half of what is left
        const bool upper = lane & (2 * width);
#pragma unroll
        for (int i = 0; i < width; ++i) {
          const float got = __shfl_xor_sync(0xffffffffu, upper ? sums[i] : sums[i + width], 2 * width);
          sums[i] = (upper ? sums[i + width] : sums[i]) + got;
        }
      }
      sums[0] += __shfl_xor_sync(0xffffffffu, sums[0], 1);
      // lanes 2 i, 2 i + 1 hold sum i: keys with token i, then queries
      const int t = (lane >> 1) & 7;
      if (!(lane & 1)) {
        if (lane < 16) {
          if (t > warp) a_s[(e + t) * kDcPairs + e + warp] = sums[0] * beta_s[e + t];
        } else if (t >= warp) {
          m_s[(e + t) * kDcPairs + e + warp] = sums[0];
        }
      }
    }
    __syncthreads();
    {                                                   // the eight against every token before it
      const int t = lane & 7, s = warp * 4 + (lane >> 3);
      if (s < e) {
        const float* kl = l_s + t * kDcStride;
        const float* ql = kl + 8 * kDcStride;
        const float* rs = r_s + s * kDcStride;
        float kk[2] = {0.f, 0.f}, qk[2] = {0.f, 0.f};
#pragma unroll 4
        for (int l = 0; l < DC_DIM; l += 4) {
          const float4 x = *reinterpret_cast<const float4*>(kl + l), y = *reinterpret_cast<const float4*>(ql + l);
          const float4 z = *reinterpret_cast<const float4*>(rs + l);
          kk[0] = fmaf(x.x, z.x, kk[0]); kk[1] = fmaf(x.y, z.y, kk[1]);
          kk[0] = fmaf(x.z, z.z, kk[0]); kk[1] = fmaf(x.w, z.w, kk[1]);
          qk[0] = fmaf(y.x, z.x, qk[0]); qk[1] = fmaf(y.y, z.y, qk[1]);
          qk[0] = fmaf(y.z, z.z, qk[0]); qk[1] = fmaf(y.w, z.w, qk[1]);
        }
        a_s[(e + t) * kDcPairs + s] = (kk[0] + kk[1]) * beta_s[e + t];
        m_s[(e + t) * kDcPairs + s] = qk[0] + qk[1];
      }
    }
    __syncthreads();
    {                                                   // the keys so far, decayed over this eight
      const int l = threadIdx.x & (DC_DIM - 1), half = threadIdx.x / DC_DIM;
      float behind = 1.f;
#pragma unroll
      for (int t = 7; t >= 0; --t) {
        if ((t & 1) == half) r_s[(e + t) * kDcStride + l] *= behind;
        behind *= g_s[(e + t) * kDcStride + l];
      }
      for (int s = half; s < e; s += 2) r_s[s * kDcStride + l] *= behind;
    }
    __syncthreads();
  }
  // ---- (I + A) W = beta G k and (I + A) U0 = beta v, a column a thread; the scaled queries on the way ----
  if (threadIdx.x < DC_DIM) {
    float upto = 1.f;
#pragma unroll
    for (int t = 0; t < DC_TOKENS; ++t) {
      upto *= g_s[t * kDcStride + threadIdx.x];
      rec[kDcQ + t * DC_DIM + threadIdx.x] = upto * q_s[t * kDcStride + threadIdx.x];
      col[t] = beta_s[t] * (upto * k_s[t * kDcStride + threadIdx.x]);
    }
    rec[kDcG + threadIdx.x] = upto;
  } else {
#pragma unroll
    for (int t = 0; t < DC_TOKENS; ++t) col[t] *= beta_s[t];
  }
#pragma unroll
  for (int t = 1; t < DC_TOKENS; ++t) {
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int s = 0; s < t; s += 4) {
      const float4 x = *reinterpret_cast<const float4*>(a_s + t * kDcPairs + s);
      sum[0] = fmaf(x.x, col[s], sum[0]);
      if (s + 1 < t) sum[1] = fmaf(x.y, col[s + 1], sum[1]);
      if (s + 2 < t) sum[2] = fmaf(x.z, col[s + 2], sum[2]);
      if (s + 3 < t) sum[3] = fmaf(x.w, col[s + 3], sum[3]);
    }
    col[t] -= (sum[0] + sum[1]) + (sum[2] + sum[3]);
  }
  if (threadIdx.x < DC_DIM) {
#pragma unroll
    for (int t = 0; t < DC_TOKENS; ++t) rec[t * DC_DIM + threadIdx.x] = col[t];
  } else if (threadIdx.x - DC_DIM < a.vdim) {
#pragma unroll
    for (int t = 0; t < DC_TOKENS; ++t) rec[kDcU + t * a.vdim + threadIdx.x - DC_DIM] = col[t];
  }
  for (int i = threadIdx.x; i < DC_TOKENS * DC_DIM / 4; i += DC_PREPARE_THREADS) {
    const int t = i / (DC_DIM / 4), l = i % (DC_DIM / 4) * 4;
    *reinterpret_cast<float4*>(rec + kDcK + t * DC_DIM + l) = *reinterpret_cast<const float4*>(r_s + t * kDcStride + l);
  }
  for (int i = threadIdx.x; i < DC_TOKENS * DC_TOKENS; i += DC_PREPARE_THREADS)
    rec[kDcM + i] = m_s[i / DC_TOKENS * kDcPairs + i % DC_TOKENS];
}
constexpr int kDcPrepareSmem = (4 * DC_TOKENS * kDcStride + 16 * kDcStride + 2 * DC_TOKENS * kDcPairs + DC_TOKENS) * 4;

// ---- the chunks one after another --------------------------------------------------------------------------------
// a stage, in floats: W and G q (64 x 132), decayed k (32 x 128), M (32 x 36), G_31 (128), U0 (32 x 16)
constexpr int kDsK = 2 * DC_TOKENS * kDcStride, kDsM = kDsK + DC_TOKENS * DC_DIM, kDsG = kDsM + DC_TOKENS * kDcPairs,
              kDsU = kDsG + DC_DIM, kDsStage = kDsU + DC_TOKENS * DC_COLS;
// behind the two stages: the columns of S [128][16], the four partial sums [4][64][16], U [32][16]
constexpr int kDsFloats = 2 * kDsStage + DC_DIM * DC_COLS + 4 * 2 * DC_TOKENS * DC_COLS + DC_TOKENS * DC_COLS;

__device__ __forceinline__ void dc_copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

__global__ void __launch_bounds__(DC_SCAN_THREADS, 1)
delta_chunk_scan_kernel(const float* __restrict__ records, int heads, int vdim, float* __restrict__ state,
                        long long state_stride, const int* __restrict__ q_start, const int* __restrict__ state_slot,
                        float* __restrict__ o_out) {
  extern __shared__ __align__(16) float ds_raw[];
  float* s_s = ds_raw + 2 * kDsStage;
  float* part_s = s_s + DC_DIM * DC_COLS;
  float* u_s = part_s + 4 * 2 * DC_TOKENS * DC_COLS;
  const int r = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * DC_COLS;
  const int first = q_start[r], n = q_start[r + 1] - first;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_wait();
  pdl_launch();
  if (n <= 0) return;
  const int chunks = (n + DC_TOKENS - 1) / DC_TOKENS;
  const size_t record = (size_t)(kDcU + DC_TOKENS * vdim);
  const float* base = records + ((size_t)(first / DC_TOKENS + r) * heads + h) * record;
  auto fetch = [&](int c) {
    if (c < chunks) {
      const float* src = base + (size_t)c * heads * record;
      float* dst = ds_raw + (c & 1) * kDsStage;
      for (int i = threadIdx.x; i < 2 * DC_TOKENS * DC_DIM / 4; i += DC_SCAN_THREADS)
        dc_copy16(dst + i / (DC_DIM / 4) * kDcStride + i % (DC_DIM / 4) * 4, src + i * 4);
      for (int i = threadIdx.x; i < DC_TOKENS * DC_DIM / 4; i += DC_SCAN_THREADS)
        dc_copy16(dst + kDsK + i * 4, src + kDcK + i * 4);
      dc_copy16(dst + kDsM + threadIdx.x / (DC_TOKENS / 4) * kDcPairs + threadIdx.x % (DC_TOKENS / 4) * 4,
                src + kDcM + threadIdx.x * 4);
      if (threadIdx.x < DC_DIM / 4) dc_copy16(dst + kDsG + threadIdx.x * 4, src + kDcG + threadIdx.x * 4);
      if (threadIdx.x >= 128) {
        const int i = threadIdx.x - 128, t = i / (DC_COLS / 4), l = i % (DC_COLS / 4) * 4;
        dc_copy16(dst + kDsU + t * DC_COLS + l, src + kDcU + t * vdim + col0 + l);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  static_assert(DC_SCAN_THREADS == DC_TOKENS * DC_TOKENS / 4 && DC_TOKENS * DC_COLS / 4 == 128, "a copy a thread");
  fetch(0);
  // this thread's share of the matrix: rows row .. + 3 of columns 2 pair, 2 pair + 1
  const int row = ((warp & 3) * 8 + lane / 4) * 4, pair = (warp >> 2) * 4 + lane % 4;
  float* mine = state + (size_t)state_slot[r] * state_stride + ((size_t)h * vdim + col0 + 2 * pair) * DC_DIM + row;
  float S[4][2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const float4 v = *reinterpret_cast<const float4*>(mine + j * DC_DIM);
    S[0][j] = v.x; S[1][j] = v.y; S[2][j] = v.z; S[3][j] = v.w;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<float2*>(s_s + (row + i) * DC_COLS + 2 * pair) = make_float2(S[i][0], S[i][1]);

  for (int c = 0; c < chunks; ++c) {
    const float* stage = ds_raw + (c & 1) * kDsStage;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                     // the record and the matrix are in place
    fetch(c + 1);                                        // into the stage that the chunk before has left
    {
      // rows of W (even warps) and of G q (odd ones) times the columns: lanes k0 .. k0 + 31, rows group + 8 i
      const int k0 = (warp >> 1) * 32, group = lane >> 2, cols = (lane & 3) * 4;
      const float* x_s = stage + ((warp & 1) * DC_TOKENS + group) * kDcStride;
      float acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll
      for (int k = k0; k < k0 + 32; k += 4) {
        float4 x[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const float4*>(x_s + i * 8 * kDcStride + k);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          const float4 y = *reinterpret_cast<const float4*>(s_s + (k + kk) * DC_COLS + cols);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float v = kk == 0 ? x[i].x : kk == 1 ? x[i].y : kk == 2 ? x[i].z : x[i].w;
            acc[i][0] = fmaf(v, y.x, acc[i][0]);
            acc[i][1] = fmaf(v, y.y, acc[i][1]);
            acc[i][2] = fmaf(v, y.z, acc[i][2]);
            acc[i][3] = fmaf(v, y.w, acc[i][3]);
          }
        }
      }
      float* to = part_s + (((warp >> 1) * 2 + (warp & 1)) * DC_TOKENS + group) * DC_COLS + cols;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float4*>(to + i * 8 * DC_COLS) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    }
    __syncthreads();
    // a row (of W for the first half of the threads, of G q for the second) and four columns a thread
    const int t = (threadIdx.x >> 2) & (DC_TOKENS - 1), cols = (threadIdx.x & 3) * 4;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 v = *reinterpret_cast<const float4*>(part_s + (i * 2 * DC_TOKENS + (threadIdx.x >> 2)) * DC_COLS + cols);
      sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
    }
    if (threadIdx.x < 128) {
      const float4 v = *reinterpret_cast<const float4*>(stage + kDsU + t * DC_COLS + cols);
      *reinterpret_cast<float4*>(u_s + t * DC_COLS + cols) = make_float4(v.x - sum.x, v.y - sum.y, v.z - sum.z, v.w - sum.w);
    }
    __syncthreads();
    if (threadIdx.x >= 128) {
      const float* m_row = stage + kDsM + t * kDcPairs;          // zeros behind the diagonal
#pragma unroll 4
      for (int s = 0; s < DC_TOKENS; s += 4) {
        const float4 x = *reinterpret_cast<const float4*>(m_row + s);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 u = *reinterpret_cast<const float4*>(u_s + (s + i) * DC_COLS + cols);
          const float v = i == 0 ? x.x : i == 1 ? x.y : i == 2 ? x.z : x.w;
          sum.x = fmaf(v, u.x, sum.x); sum.y = fmaf(v, u.y, sum.y);
          sum.z = fmaf(v, u.z, sum.z); sum.w = fmaf(v, u.w, sum.w);
        }
      }
      const int token = c * DC_TOKENS + t;
      if (token < n)
        *reinterpret_cast<float4*>(o_out + ((size_t)(first + token) * heads + h) * vdim + col0 + cols) = sum;
    }
    // the matrix moves on by the chunk
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float g = stage[kDsG + row + i];
      S[i][0] *= g;
      S[i][1] *= g;
    }
#pragma unroll 8
    for (int s = 0; s < DC_TOKENS; ++s) {
      const float4 k = *reinterpret_cast<const float4*>(stage + kDsK + s * DC_DIM + row);
      const float2 u = *reinterpret_cast<const float2*>(u_s + s * DC_COLS + 2 * pair);
      S[0][0] = fmaf(k.x, u.x, S[0][0]); S[0][1] = fmaf(k.x, u.y, S[0][1]);
      S[1][0] = fmaf(k.y, u.x, S[1][0]); S[1][1] = fmaf(k.y, u.y, S[1][1]);
      S[2][0] = fmaf(k.z, u.x, S[2][0]); S[2][1] = fmaf(k.z, u.y, S[2][1]);
      S[3][0] = fmaf(k.w, u.x, S[3][0]); S[3][1] = fmaf(k.w, u.y, S[3][1]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      *reinterpret_cast<float2*>(s_s + (row + i) * DC_COLS + 2 * pair) = make_float2(S[i][0], S[i][1]);
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
    *reinterpret_cast<float4*>(mine + j * DC_DIM) = make_float4(S[0][j], S[1][j], S[2][j], S[3][j]);
}

// ---- launchers ---------------------------------------------------------------------------------------------------
// Whether heads of these sizes run in chunks: keys that fill a column of 128 lanes, values in whole blocks of columns.
TOKB200_API int tokb200_delta_chunks_supported(int dim, int vdim) {
  return dim > 64 && dim <= DC_DIM && vdim > 0 && vdim <= 128 && vdim % DC_COLS == 0;
}

// Floats of the records of a step.
TOKB200_API long long tokb200_delta_chunk_floats(int n_rows, int n_requests, int heads, int vdim) {
  return ((long long)n_rows / DC_TOKENS + n_requests) * heads * (kDcU + DC_TOKENS * vdim);
}

// The shared memory of a kernel, allowed once a device.
template <typename K>
static int dc_allow(K* kernel, int bytes, bool (&done)[64]) {
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return TOKB200_BAD_SIZE;
  if (!done[device]) {
    const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (err != cudaSuccess) return (int)err;
    done[device] = true;
  }
  return TOKB200_OK;
}

template <typename T, bool BY_CHANNEL>
static int dc_prepare(const DeltaChunkArgs& args, dim3 grid, cudaStream_t stream) {
  static bool done[64] = {};
  const int status = dc_allow(delta_chunk_prepare_kernel<T, BY_CHANNEL>, kDcPrepareSmem, done);
  if (status != TOKB200_OK) return status;
  return launch_dependent(delta_chunk_prepare_kernel<T, BY_CHANNEL>, grid, dim3(DC_PREPARE_THREADS),
                          (size_t)kDcPrepareSmem, stream, args);
}

TOKB200_API int tokb200_delta_chunk_prepare(const void* proj, int proj_dtype, int ld, int qkv_at, int b_at,
                                            const void* decay, int decay_ld, int decay_at, int by_channel, int groups,
                                            int heads, int dim, int vdim, int taps, const float* conv_w,
                                            const float* a_log, const float* dt_bias, const float* state,
                                            long long state_stride, int conv_off, const int* q_start,
                                            const int* state_slot, int n_rows, int n_requests, float* records,
                                            cudaStream_t stream) {
  if (n_rows <= 0 || n_requests <= 0) return TOKB200_OK;
  if (groups <= 0 || heads <= 0 || heads % groups || heads > 65535 || taps < 1 || taps > DC_MAX_TAPS ||
      !tokb200_delta_chunks_supported(dim, vdim))
    return TOKB200_BAD_SIZE;
  if (((uintptr_t)records & 15)) return TOKB200_BAD_ALIGNMENT;
  const DeltaChunkArgs args = {proj, ld, qkv_at, b_at, decay, decay_ld, decay_at, conv_w, a_log, dt_bias, state,
                               state_stride, q_start, state_slot, records, 1.0f / sqrtf((float)dim), groups, heads, dim,
                               vdim, taps, conv_off, n_requests};
  const dim3 grid(n_rows / DC_TOKENS + n_requests, heads);
  if (by_channel) return proj_dtype == TOKB200_F32 ? dc_prepare<float, true>(args, grid, stream) : TOKB200_BAD_DTYPE;
  if (proj_dtype == TOKB200_F32) return dc_prepare<float, false>(args, grid, stream);
  if (proj_dtype == TOKB200_BF16) return dc_prepare<__nv_bfloat16, false>(args, grid, stream);
  return TOKB200_BAD_DTYPE;
}

TOKB200_API int tokb200_delta_chunk_scan(const float* records, int heads, int dim, int vdim, float* state,
                                         long long state_stride, const int* q_start, const int* state_slot,
                                         int n_requests, float* o_out, cudaStream_t stream) {
  if (n_requests <= 0) return TOKB200_OK;
  if (heads <= 0 || heads > 65535 || n_requests > 65535 || !tokb200_delta_chunks_supported(dim, vdim))
    return TOKB200_BAD_SIZE;
  if ((((uintptr_t)records | (uintptr_t)state | (uintptr_t)o_out) & 15) || state_stride % 4) return TOKB200_BAD_ALIGNMENT;
  constexpr int bytes = kDsFloats * (int)sizeof(float);
  static bool done[64] = {};
  const int status = dc_allow(delta_chunk_scan_kernel, bytes, done);
  if (status != TOKB200_OK) return status;
  return launch_dependent(delta_chunk_scan_kernel, dim3(vdim / DC_COLS, heads, n_requests), dim3(DC_SCAN_THREADS),
                          (size_t)bytes, stream, records, heads, vdim, state, state_stride, q_start, state_slot, o_out);
}
