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
//                         then A, M, W, U0 and the scaled queries and keys as one record.  Pairs of tokens in different
//                         halves of 32, 16 or 8 tokens are plain products of rows that were decayed to and from the
//                         middle; inside four the decays are multiplied in key by key
//   delta_chunk_scan      a block a (16 or 32 columns of a head's matrix, request): the chunks one after another.  The 64
//                         x 128 rows of W and G q meet the columns on the tensor cores (mma.sync), every 32-bit value as
//                         three bfloat16 pieces that add up to it; the next chunk's pieces are on their way (cp.async, each
//                         thread its own) while this one is worked through
//
// The scan is one chain: a chunk's products need the matrix that the chunk before left.  Counters at 2,048 tokens: shared
// memory's pipe busy 53 % of the time, the tensor cores 30 %; with FMA register tiles that pipe was busy 62 % and the scan of
// 16 heads took 162 us where it now takes 111.  The prepare kernel is bound by latency, not by a pipe (instructions issue 39 %
// of the time, two blocks of eight warps an SM by shared memory): short loops over copied inputs for the convolution
// and the decays, eight tokens' loads and exponentials side by side, made it faster (105 -> 94 us by head at 2,048, 239 -> 221 by
// channel over four prompts); half of all its code in loops, tried on an earlier form of it, slower (88.7 -> 100 us).  Measured
// (16 heads of 128 x 128, both kernels and the kept inputs between them, us; in front the FMA tiles): a prompt of 2,048
// tokens 254 -> 197 with one decay a head and 272 -> 209 with one a channel, four prompts of 5,100 in all 537 -> 479.  Error
// against 64 bits (2-norm, 2,048 tokens at memories of tens to hundreds), outputs and 32-bit states, FMA tiles / here: 1.89e-7 /
// 1.85e-7 and 2.03e-7 / 1.85e-7, by channel 1.94e-7 / 1.87e-7 and 2.55e-7 / 2.33e-7.  A record takes 95 KB at 128 values.
//
// A request's chunks are counted from its portion's first row; the record of chunk c of request r lies at place
// q_start[r] / 32 + r + c (no two the same, and known without a pass over the other requests).
#include "common.cuh"
#include "exact_mma.cuh"

#define DC_TOKENS 32
#define DC_DIM 128                        // lanes of a key, zeros behind the head's own
#define DC_COLS 16                        // columns of a narrow scan block (wide ones: 32)
#define DC_MAX_TAPS 16
#define DC_PREPARE_THREADS 256
constexpr int kDcStride = DC_DIM + 4;     // of rows that several lanes read at once, 16 bytes each
constexpr int kDcPairs = DC_TOKENS + 4;   // of A's and M's rows
// a record, in floats: W over G q (64 x 128), then decayed k (32 x 128), as pieces in the order in which a lane of a product
// takes them ([16 channels][tile][piece][lane] of 16 bytes, see exact_mma.cuh); M (32 x 32), G_31 (128), U0 (32 x vdim)
constexpr int kDcK = 8 * 4 * 3 * 128, kDcM = kDcK + 8 * 2 * 3 * 128, kDcG = kDcM + DC_TOKENS * DC_TOKENS, kDcU = kDcG + DC_DIM;

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
  int quads;                 // 32-bit rows whose pieces of four channels lie on 16 bytes
};

// N sums of every lane over LANES neighbouring lanes, all N together: lanes give away the half of their sums that the
// other side of the exchange keeps.  N >= LANES: lane i of the LANES ends with sums i N / LANES .. in front; N < LANES: with
// sum i N / LANES (rounded down) in front.
template <int N, int LANES, int KEEP>
__device__ __forceinline__ void dc_exchange(float (&sums)[KEEP], int lane) {
  if constexpr (LANES > 1) {
    if constexpr (N > 1) {
      const bool upper = lane & (LANES / 2);
#pragma unroll
      for (int i = 0; i < N / 2; ++i) {
        const float got = __shfl_xor_sync(0xffffffffu, upper ? sums[i] : sums[i + N / 2], LANES / 2);
        sums[i] = (upper ? sums[i + N / 2] : sums[i]) + got;
      }
      dc_exchange<N / 2, LANES / 2>(sums, lane);
    } else {
      sums[0] += __shfl_xor_sync(0xffffffffu, sums[0], LANES / 2);
      dc_exchange<1, LANES / 2>(sums, lane);
    }
  }
}
template <int V> struct dc_int { static constexpr int value = V; };

// T: type of proj (and of `decay` where it is one a head: the same product's columns)
template <typename T, bool BY_CHANNEL>
__global__ void __launch_bounds__(DC_PREPARE_THREADS, 2) delta_chunk_prepare_kernel(const DeltaChunkArgs a) {
  extern __shared__ __align__(16) float dc_raw[];
  float* q_s = dc_raw;                                  // [32][132] each
  float* k_s = q_s + DC_TOKENS * kDcStride;
  float* g_s = k_s + DC_TOKENS * kDcStride;
  float* l_s = g_s + DC_TOKENS * kDcStride;             // keys, then queries, of upper halves, decayed from the edge on
  float* r_s = l_s + DC_TOKENS * kDcStride;             // keys of lower halves, decayed up to the edge
  float* a_s = r_s + 16 * kDcStride;                    // [32][36]
  float* m_s = a_s + DC_TOKENS * kDcPairs;              // [32][36]
  float* beta_s = m_s + DC_TOKENS * kDcPairs;           // [32]
  float* v_s = beta_s + DC_TOKENS;                      // [32][132]
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

  const int l = threadIdx.x & (DC_DIM - 1), half = threadIdx.x / DC_DIM;
  // ---- convolution and silu, a channel a thread: threads 0 .. 127 take q and the first half of k's tokens, the others v
  // and the second half.  The inputs come to where the results will lie, four channels a copy where they lie on 16 bytes; a
  // thread then takes eight tokens at a time, all read before the first is written, so that eight chains of exponential and
  // quotient run side by side (one by one a token took 195 cycles, a quarter of the block's time) ----
  const int a_lanes = half ? a.vdim : a.dim;
  const int a_ch = half ? 2 * a.groups * a.dim + h * a.vdim + l : group * a.dim + l, k_ch = (a.groups + group) * a.dim + l;
  const int k0 = half * (DC_TOKENS / 2);
  float* a_to = (half ? v_s : q_s) + l;
  // an input `back` places before the portion's start is the kept one that many from the end
  auto input = [&](int ch, int at) {
    return at >= 0 ? to_float(proj[(size_t)(start + at) * a.ld + a.qkv_at + ch]) : kept[(size_t)(a.taps - 1 + at) * channels + ch];
  };
  if constexpr (sizeof(T) == 4) {
    auto copy = [](float* to, const float* from, bool in, auto bytes) {
      constexpr int n = decltype(bytes)::value;
      if constexpr (n == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from),
                     "r"(in ? 16 : 0) : "memory");
      else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from),
                     "r"(in ? 4 : 0) : "memory");
    };
    auto bring = [&](float* to, const float* from, int ld, int lanes) {       // 32 rows
      if (a.quads) {
#pragma unroll
        for (int t = warp; t < DC_TOKENS; t += DC_PREPARE_THREADS / 32) {
          const bool in = lane * 4 < lanes && t < n_here;
          copy(to + t * kDcStride + lane * 4, from + (in ? (size_t)t * ld + lane * 4 : 0), in, dc_int<16>());
        }
      } else {
#pragma unroll 8
        for (int t = half; t < DC_TOKENS; t += 2) {
          const bool in = l < lanes && t < n_here;
          copy(to + t * kDcStride + l, from + (in ? (size_t)t * ld + l : 0), in, dc_int<4>());
        }
      }
    };
    const float* row = proj + (size_t)t0 * a.ld + a.qkv_at;
    bring(q_s, row + group * a.dim, a.ld, a.dim);
    bring(k_s, row + (a.groups + group) * a.dim, a.ld, a.dim);
    bring(v_s, row + 2 * a.groups * a.dim + h * a.vdim, a.ld, a.vdim);
    if (BY_CHANNEL)
      bring(g_s, static_cast<const float*>(a.decay) + (size_t)t0 * a.decay_ld + a.decay_at + h * a.dim, a.decay_ld, a.dim);
  } else {
#pragma unroll 8
    for (int t = 0; t < DC_TOKENS; ++t)
      a_to[t * kDcStride] = l < a_lanes && t < n_here ? to_float(proj[(size_t)(t0 + t) * a.ld + a.qkv_at + a_ch]) : 0.f;
#pragma unroll 8
    for (int t = k0; t < k0 + DC_TOKENS / 2; ++t)
      k_s[t * kDcStride + l] = l < a.dim && t < n_here ? to_float(proj[(size_t)(t0 + t) * a.ld + a.qkv_at + k_ch]) : 0.f;
  }
  float pre[4];
  if (!BY_CHANNEL) {
    const T* raw = static_cast<const T*>(a.decay) + a.decay_at + h;
#pragma unroll
    for (int i = 0; i < 4; ++i) pre[i] = warp + 8 * i < n_here ? to_float(raw[(size_t)(t0 + warp + 8 * i) * a.decay_ld]) : 0.f;
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  auto silu = [](float v) { return v * dc_sigmoid(v); };
  if (a.taps == 4) {
    float aw[4], kw[4], ax[3], kx[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      ax[j] = l < a_lanes ? input(a_ch, at0 - 3 + j) : 0.f;
      kx[j] = k0 < n_here && l < a.dim ? input(k_ch, at0 + k0 - 3 + j) : 0.f;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      aw[j] = l < a_lanes ? a.conv_w[(size_t)a_ch * 4 + j] : 0.f;
      kw[j] = l < a.dim ? a.conv_w[(size_t)k_ch * 4 + j] : 0.f;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll 1
    for (int i = 0; i < 6; ++i) {                        // four times eight tokens of q or v, twice of k
      const bool of_k = i >= 4;
      const int from = of_k ? k0 + (i - 4) * 8 : i * 8;
      float* at = (of_k ? k_s + l : a_to) + from * kDcStride;
      if (i == 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) aw[j] = kw[j];
#pragma unroll
        for (int j = 0; j < 3; ++j) ax[j] = kx[j];
      }
      float x[11];
#pragma unroll
      for (int j = 0; j < 3; ++j) x[j] = ax[j];
#pragma unroll
      for (int j = 0; j < 8; ++j) x[3 + j] = at[j * kDcStride];
#pragma unroll
      for (int j = 0; j < 3; ++j) ax[j] = x[8 + j];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        x[j] = silu(fmaf(aw[3], x[3 + j], fmaf(aw[2], x[2 + j], fmaf(aw[1], x[1 + j], aw[0] * x[j]))));
#pragma unroll
      for (int j = 0; j < 8; ++j) at[j * kDcStride] = from + j < n_here ? x[j] : 0.f;
    }
  } else {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    auto sum = [&](int ch, int t) {
      float v = 0.f;
      for (int j = 0; j < a.taps; ++j) v = fmaf(a.conv_w[(size_t)ch * a.taps + j], input(ch, at0 + t - (a.taps - 1 - j)), v);
      return silu(v);
    };
#pragma unroll 1
    for (int t = 0; t < DC_TOKENS; ++t) a_to[t * kDcStride] = t < n_here && l < a_lanes ? sum(a_ch, t) : 0.f;
#pragma unroll 1
    for (int t = k0; t < k0 + DC_TOKENS / 2; ++t) k_s[t * kDcStride + l] = t < n_here && l < a.dim ? sum(k_ch, t) : 0.f;
  }
  // ---- decays and beta; A and M start as zeros ----
  {
    const float rate = expf(a.a_log[h]);
    if (BY_CHANNEL) {
      const float shift = l < a.dim ? a.dt_bias[h * a.dim + l] : 0.f;
#pragma unroll 1
      for (int i = half; i < DC_TOKENS; i += 16) {       // eight at a time, side by side as above
        float* at = g_s + i * kDcStride + l;
        float x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = at[2 * j * kDcStride];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = expf(-rate * dc_softplus(x[j] + shift));
#pragma unroll
        for (int j = 0; j < 8; ++j) at[2 * j * kDcStride] = i + 2 * j < n_here && l < a.dim ? x[j] : 1.f;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = warp + 8 * i;
        const float g = t < n_here ? expf(-rate * dc_softplus(pre[i] + a.dt_bias[h])) : 1.f;
        *reinterpret_cast<float4*>(g_s + t * kDcStride + lane * 4) = make_float4(g, g, g, g);
      }
    }
    if (threadIdx.x < DC_TOKENS)
      beta_s[threadIdx.x] = threadIdx.x < n_here ? dc_sigmoid(to_float(proj[(size_t)(t0 + threadIdx.x) * a.ld + a.b_at + h])) : 0.f;
    for (int i = threadIdx.x; i < 2 * DC_TOKENS * kDcPairs; i += DC_PREPARE_THREADS) a_s[i] = 0.f;
  }
  __syncthreads();
  // ---- unit vectors: a warp a row, four lanes of it a thread ----
  {
    constexpr int kRows = 2 * DC_TOKENS / (DC_PREPARE_THREADS / 32);
    float4 v[kRows];
    float sum[kRows];
    auto at = [&](int i) {                               // four rows of q, four of k
      return reinterpret_cast<float4*>((i < kRows / 2 ? q_s : k_s) + (i % (kRows / 2) * 8 + warp) * kDcStride) + lane;
    };
#pragma unroll
    for (int i = 0; i < kRows; ++i) v[i] = *at(i);
#pragma unroll
    for (int i = 0; i < kRows; ++i) sum[i] = v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < kRows; ++i) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], o);
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const float unit = 1.0f / sqrtf(sum[i] + 1e-6f) * (i < kRows / 2 ? a.q_scale : 1.f);
      *at(i) = make_float4(v[i].x * unit, v[i].y * unit, v[i].z * unit, v[i].w * unit);
    }
  }
  __syncthreads();
  // ---- A and M: pairs whose tokens a block of 2 w tokens' middle parts, w = 16, 8, 4, as products of rows that were
  // decayed to and from that middle; 4 x 4 pairs of both matrices a thread over a share of the lanes ----
  auto level = [&](auto width) {
    constexpr int w = decltype(width)::value;
    // token `i` of the 16 in lower halves; + w: its like in the upper half
    auto token = [](int i) { return (i / w) * 2 * w + i % w; };
    if (!half) {
#pragma unroll
      for (int i = 0; i < 16; i += w) {
        float upto = 1.f;
#pragma unroll
        for (int j = i; j < i + w; ++j) {
          const int t = token(j) + w;
          upto *= g_s[t * kDcStride + l];
          l_s[j * kDcStride + l] = upto * k_s[t * kDcStride + l];
          l_s[(16 + j) * kDcStride + l] = upto * q_s[t * kDcStride + l];
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < 16; i += w) {
        float behind = 1.f;
#pragma unroll
        for (int j = i + w - 1; j >= i; --j) {
          const int t = token(j);
          r_s[j * kDcStride + l] = behind * k_s[t * kDcStride + l];
          behind *= g_s[t * kDcStride + l];
        }
      }
    }
    __syncthreads();
    constexpr int kAcross = w / 4, kTiles = 16 / w * kAcross * kAcross, kLanes = w == 16 ? 16 : 32;
    const int tile = threadIdx.x / kLanes, slice = threadIdx.x % kLanes;
    if (tile < kTiles) {                                // whole warps
      const int t4 = tile / (kAcross * kAcross) * w + tile / kAcross % kAcross * 4;      // rows of l_s, of r_s
      const int s4 = tile / (kAcross * kAcross) * w + tile % kAcross * 4;
      float sums[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) sums[i] = 0.f;
#pragma unroll
      for (int c = 0; c < DC_DIM; c += kLanes * 4) {
        float4 z[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) z[j] = *reinterpret_cast<const float4*>(r_s + (s4 + j) * kDcStride + c + slice * 4);
#pragma unroll
        for (int i = 0; i < 8; ++i) {                   // four keys, four queries
          const float4 x = *reinterpret_cast<const float4*>(l_s + (i / 4 * 16 + t4 + i % 4) * kDcStride + c + slice * 4);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float& v = sums[i * 4 + j];
            v = fmaf(x.x, z[j].x, v); v = fmaf(x.y, z[j].y, v);
            v = fmaf(x.z, z[j].z, v); v = fmaf(x.w, z[j].w, v);
          }
        }
      }
      dc_exchange<32, kLanes>(sums, lane);
#pragma unroll
      for (int e = 0; e < 32 / kLanes; ++e) {
        const int i = slice * (32 / kLanes) + e;        // the sum this lane holds
        const int t = token(t4 + i / 4 % 4) + w, s = token(s4 + i % 4);
        if (i < 16) a_s[t * kDcPairs + s] = sums[e] * beta_s[t];
        else m_s[t * kDcPairs + s] = sums[e];
      }
    }
  };
  level(dc_int<16>());
  __syncthreads();
  level(dc_int<8>());
  __syncthreads();
  level(dc_int<4>());
  {
    // pairs inside four tokens, a warp the four: token s's key decayed on from token to token
    const int e = warp * 4;
    float4 k[4], q[4], g[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      k[i] = reinterpret_cast<const float4*>(k_s + (e + i) * kDcStride)[lane];
      q[i] = reinterpret_cast<const float4*>(q_s + (e + i) * kDcStride)[lane];
      g[i] = reinterpret_cast<const float4*>(g_s + (e + i) * kDcStride)[lane];
    }
    float sums[16];                                     // of (t, s): the query's for s <= t at 4 t + s, the key's for s < t at 4 s + t
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      float4 p = k[s];
#pragma unroll
      for (int t = s; t < 4; ++t) {
        if (t > s) {
          p.x *= g[t].x; p.y *= g[t].y; p.z *= g[t].z; p.w *= g[t].w;
          sums[4 * s + t] = fmaf(p.x, k[t].x, p.y * k[t].y) + fmaf(p.z, k[t].z, p.w * k[t].w);
        }
        sums[4 * t + s] = fmaf(p.x, q[t].x, p.y * q[t].y) + fmaf(p.z, q[t].z, p.w * q[t].w);
      }
    }
    dc_exchange<16, 32>(sums, lane);
    const int i = lane >> 1, x = i >> 2, y = i & 3;
    if (!(lane & 1)) {
      if (y <= x) m_s[(e + x) * kDcPairs + e + y] = sums[0];
      else a_s[(e + y) * kDcPairs + e + x] = sums[0] * beta_s[e + y];
    }
  }
  __syncthreads();
  // ---- (I + A) W = beta G k and (I + A) U0 = beta v, a column of both a thread of the first half (a row of A is read
  // once for the two); the second half scales the queries and keys and writes M meanwhile ----
  float col[DC_TOKENS], other[DC_TOKENS];
  if (!half) {
    float upto = 1.f;
#pragma unroll
    for (int t = 0; t < DC_TOKENS; ++t) {
      const float beta = beta_s[t];
      upto *= g_s[t * kDcStride + l];
      col[t] = beta * (upto * k_s[t * kDcStride + l]);
      other[t] = beta * v_s[t * kDcStride + l];
    }
  }
  __syncthreads();                                       // the keys' rows are read
  if (!half) {
#pragma unroll
    for (int t = 1; t < DC_TOKENS; ++t) {
      float sum[2] = {0.f, 0.f}, more[2] = {0.f, 0.f};
#pragma unroll
      for (int s = 0; s < t; s += 4) {
        const float4 x = *reinterpret_cast<const float4*>(a_s + t * kDcPairs + s);
        sum[0] = fmaf(x.x, col[s], sum[0]); more[0] = fmaf(x.x, other[s], more[0]);
        if (s + 1 < t) { sum[1] = fmaf(x.y, col[s + 1], sum[1]); more[1] = fmaf(x.y, other[s + 1], more[1]); }
        if (s + 2 < t) { sum[0] = fmaf(x.z, col[s + 2], sum[0]); more[0] = fmaf(x.z, other[s + 2], more[0]); }
        if (s + 3 < t) { sum[1] = fmaf(x.w, col[s + 3], sum[1]); more[1] = fmaf(x.w, other[s + 3], more[1]); }
      }
      col[t] -= sum[0] + sum[1];
      other[t] -= more[0] + more[1];
    }
#pragma unroll
    for (int t = 0; t < DC_TOKENS; ++t) l_s[t * kDcStride + l] = col[t];
    if (l < a.vdim) {
#pragma unroll
      for (int t = 0; t < DC_TOKENS; ++t) rec[kDcU + t * a.vdim + l] = other[t];
    }
  } else {
    float upto = 1.f, behind = 1.f;
#pragma unroll
    for (int t = 0; t < DC_TOKENS; ++t) {
      upto *= g_s[t * kDcStride + l];
      q_s[t * kDcStride + l] *= upto;
    }
    rec[kDcG + l] = upto;
#pragma unroll
    for (int t = DC_TOKENS - 1; t >= 0; --t) {
      k_s[t * kDcStride + l] *= behind;
      behind *= g_s[t * kDcStride + l];
    }
    for (int i = l; i < DC_TOKENS * DC_TOKENS; i += DC_DIM) rec[kDcM + i] = m_s[i / DC_TOKENS * kDcPairs + i % DC_TOKENS];
  }
  __syncthreads();
  // ---- W, G q and the decayed keys in pieces, six tiles a warp: channels 16 w on, of 16 rows or of 16 tokens ----
  const int g = lane >> 2, c = lane & 3;
#pragma unroll
  for (int e = 0; e < 6; ++e) {
    unsigned p[3][4];
    uint4* to;
    if (e < 4) {
      const float* from = (e < 2 ? l_s : q_s) + ((e & 1) * 16 + g) * kDcStride + warp * 16 + 2 * c;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 v = *reinterpret_cast<const float2*>(from + (i & 1) * 8 * kDcStride + (i >> 1) * 8);
        xm_cut(v.x, v.y, p[0][i], p[1][i], p[2][i]);
      }
      to = reinterpret_cast<uint4*>(rec) + (warp * 4 + e) * 3 * 32 + lane;
    } else {
      const float* from = k_s + ((e - 4) * 16 + 2 * c) * kDcStride + warp * 16 + g;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float* at = from + (i & 1) * 8 * kDcStride + (i >> 1) * 8;
        xm_cut(at[0], at[kDcStride], p[0][i], p[1][i], p[2][i]);
      }
      to = reinterpret_cast<uint4*>(rec + kDcK) + (warp * 2 + e - 4) * 3 * 32 + lane;
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) to[q * 32] = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
  }
}
constexpr int kDcPrepareSmem = (5 * DC_TOKENS * kDcStride + 16 * kDcStride + 2 * DC_TOKENS * kDcPairs + DC_TOKENS) * 4;

// ---- the chunks one after another --------------------------------------------------------------------------------
// The products run on the tensor cores with their operands in exact pieces (exact_mma.cuh).
//   warps 0 .. 7    channels 16 w .. + 15 of the block's columns of S, transposed, in the layout of a product's result, which
//                   is that of the next product's second operand.  W and G q times S over their channels, the eight partial
//                   sums through shared memory, U; then S = G S + K^T U
//   warps 8 .. 11   bring the next chunk's M, G_31 and U0 (cp.async), and finish G q S + M U: plain multiply-adds over the
//                   tokens up to a row's own (an infinity or a NaN behind it is not this row's)
// A chunk of 16 columns takes 3,300 cycles (4,900 with multiply-adds, whose reads of shared memory bounded it): the tensor
// pipe's own 1,150, and the two meetings of all warps, whose sums and cuts lie one behind the other.  us, a scan of 16 heads
// of 128 x 128: one prompt of 2,048 tokens 162 -> 112, four of 5,100 in all 322 -> 245.  Pieces straight from memory to
// registers a chunk ahead instead of two chunks ahead through shared memory: 128; 32-bit records, cut by the helping warps: 216.
#define DT_THREADS 384
#define DT_HELPERS 128
#define DT_PITCH 40                       // floats between columns of U: no two lanes of a load on one bank
// a stage, in floats: M (32 x 36), G_31 (128), U0 (32 x COLS)
constexpr int kDtG = DC_TOKENS * kDcPairs, kDtU = kDtG + DC_DIM;
constexpr int kDtPieces = kDcM * 4;       // bytes of a record's pieces
template <int COLS> struct DtShape {
  static constexpr int kStage = kDtU + DC_TOKENS * COLS;
  static constexpr int kPart = 3 * kStage;                                  // [8][64][16] partial sums
  static constexpr int kUs = kPart + 8 * 64 * 16;                           // [2][COLS][DT_PITCH]
  static constexpr int kOs = kUs + 2 * COLS * DT_PITCH;                     // [2][32][COLS + 4]
  static constexpr int kRing = kOs + 2 * DC_TOKENS * (COLS + 4);            // [2] chunks' pieces, a lane's places in eighteens
  static constexpr int kSmem = kRing * 4 + 2 * kDtPieces;
};

// A number of a record's pieces: they add up to it (a NaN where it is one; W, G q and K hold no infinities, their rows being
// products of decays, of unit vectors and of what the substitution makes of them).
__device__ __forceinline__ float dt_whole(const float* tile, int lane, int i) {       // tile: [piece][lane][8]
  const __nv_bfloat16* p = reinterpret_cast<const __nv_bfloat16*>(tile) + lane * 8 + i;
  return (__bfloat162float(p[0]) + __bfloat162float(p[256])) + __bfloat162float(p[512]);
}
// The same portion in plain multiply-adds, all threads of the block, for numbers that have no pieces (an infinity in the matrix
// or in U, numbers that round to one in 16 bits, and what then comes of them): slow, and replaces nothing but what the pieces
// left as no finite number.  Inlined in small loops: a call, which is never made, cost the fast walk 2
// to 4 %.  `mine`: the block's columns of the matrix in memory, as they were before the portion; what lies behind the portion's
// last token, or behind a row's own, takes no part.  s_s: [128][COLS] floats, behind it the matrix as the pieces left it, of that
// form, and U [32][COLS].
template <int COLS>
__device__ __forceinline__ void dt_scan_plain(float* s_s, const float* __restrict__ rec, size_t record_ld, int n, int vdim, int col0,
                                           float* __restrict__ mine, float* __restrict__ o_out, size_t o_ld) {
  const float* end_s = s_s + DC_DIM * COLS;
  float* u_s = s_s + 2 * DC_DIM * COLS;
#pragma unroll 1
  for (int i = threadIdx.x; i < DC_DIM * COLS; i += DT_THREADS) s_s[i] = mine[(size_t)(i % COLS) * DC_DIM + i / COLS];
  __syncthreads();
#pragma unroll 1
  for (int t0 = 0; t0 < n; t0 += DC_TOKENS, rec += record_ld) {
    const int here = min(DC_TOKENS, n - t0);
    auto product = [&](int row, int c) {                 // a row of W (0 .. 31) or G q (32 .. 63) times a column
      const int lane = (row & 7) * 4, high = row >> 3 & 1;
      float sum = 0.f;
#pragma unroll 1
      for (int k = 0; k < DC_DIM; ++k)
        sum = fmaf(dt_whole(rec + (k / 16 * 4 + row / 16) * 384, lane + (k & 7) / 2, ((k >> 3 & 1) * 2 + high) * 2 + (k & 1)),
                   s_s[k * COLS + c], sum);
      return sum;
    };
#pragma unroll 1
    for (int i = threadIdx.x; i < here * COLS; i += DT_THREADS) {
      const int t = i / COLS, c = i % COLS;
      u_s[i] = rec[kDcU + t * vdim + col0 + c] - product(t, c);
    }
    __syncthreads();
#pragma unroll 1
    for (int i = threadIdx.x; i < here * COLS; i += DT_THREADS) {
      const int t = i / COLS, c = i % COLS;
      float* to = o_out + (size_t)(t0 + t) * o_ld + c;
      if (*to - *to == 0.f) continue;
      float sum = product(DC_TOKENS + t, c);
#pragma unroll 1
      for (int s = 0; s <= t; ++s) sum = fmaf(rec[kDcM + t * DC_TOKENS + s], u_s[s * COLS + c], sum);
      *to = sum;
    }
    __syncthreads();
#pragma unroll 1
    for (int i = threadIdx.x; i < DC_DIM * COLS; i += DT_THREADS) {
      const int k = i / COLS, c = i % COLS;
      float more = 0.f;
#pragma unroll 1
      for (int t = 0; t < here; ++t)
        more = fmaf(dt_whole(rec + kDcK + (k / 16 * 2 + t / 16) * 384, (k & 7) * 4 + (t & 7) / 2,
                             ((k >> 3 & 1) * 2 + (t >> 3 & 1)) * 2 + (t & 1)), u_s[t * COLS + c], more);
      s_s[i] = fmaf(rec[kDcG + k], s_s[i], more);
    }
    __syncthreads();
  }
#pragma unroll 1
  for (int i = threadIdx.x; i < DC_DIM * COLS; i += DT_THREADS)
    mine[(size_t)(i % COLS) * DC_DIM + i / COLS] = end_s[i] - end_s[i] == 0.f ? end_s[i] : s_s[i];
}

template <int COLS>
__global__ void __launch_bounds__(DT_THREADS, 1)
delta_chunk_scan_kernel(const float* __restrict__ records, int heads, int vdim, float* __restrict__ state,
                        long long state_stride, const int* __restrict__ q_start, const int* __restrict__ state_slot,
                        float* __restrict__ o_out) {
  using S = DtShape<COLS>;
  constexpr int kHalves = COLS / 16;
  extern __shared__ __align__(16) float dt_raw[];
  float* part_s = dt_raw + S::kPart;
  const int r = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * COLS;
  const int first = q_start[r], n = q_start[r + 1] - first;
  // the warp's number through a shuffle: the compiler sees that the roles do not diverge
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int g = lane >> 2, c = lane & 3;                 // of a product's layout: row (or column) and pair
  pdl_wait();
  pdl_launch();
  if (n <= 0) return;
  const int chunks = (n + DC_TOKENS - 1) / DC_TOKENS;
  const size_t record = (size_t)(kDcU + DC_TOKENS * vdim);
  const float* base = records + ((size_t)(first / DC_TOKENS + r) * heads + h) * record;
  bool wild;                                             // a result of the pieces is no finite number

  if (warp < 8) {
    float* mine = state + (size_t)state_slot[r] * state_stride + ((size_t)h * vdim + col0 + g) * DC_DIM + warp * 16 + 2 * c;
    float s[kHalves][2][4];                              // columns g and g + 8 of a half, channels 8 j + 2 c, + 1
#pragma unroll
    for (int e = 0; e < kHalves; ++e)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; i += 2)
          *reinterpret_cast<float2*>(&s[e][j][i]) = *reinterpret_cast<const float2*>(mine + (e * 16 + i * 4) * DC_DIM + j * 8);
    // The pieces of a record that a lane takes are its own alone: copied two chunks ahead to places of shared memory that no
    // other thread touches.
    const unsigned ring = (unsigned)__cvta_generic_to_shared(dt_raw + S::kRing) + (warp * 18 * 32 + lane) * 16;
    auto fetch = [&](int chunk) {
      if (chunk < chunks) {
        const float* src = base + (size_t)chunk * heads * record + lane * 4;
        const unsigned to = ring + (chunk & 1) * kDtPieces;
#pragma unroll
        for (int i = 0; i < 18; ++i) {
          const float* from = i < 12 ? src + (warp * 12 + i) * 128 : src + kDcK + (warp * 6 + i - 12) * 128;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + i * 512), "l"(from) : "memory");
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto piece = [&](int chunk, int i, unsigned (&v)[4]) {
      asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                   : "r"(ring + (chunk & 1) * kDtPieces + i * 512) : "memory");
    };
    fetch(0);
    fetch(1);
    __syncthreads();                                     // the first stage is in place
    for (int chunk = 0; chunk < chunks; ++chunk) {
      const float* stage = dt_raw + chunk % 3 * S::kStage;
      float* u_s = dt_raw + S::kUs + (chunk & 1) * COLS * DT_PITCH;
      float* o_s = dt_raw + S::kOs + (chunk & 1) * DC_TOKENS * (COLS + 4);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      unsigned a[4][3][4];                               // W and G q: tile of 16 rows, piece
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int p = 0; p < 3; ++p) piece(chunk, m * 3 + p, a[m][p]);
#pragma unroll
      for (int e = 0; e < kHalves; ++e) {
        unsigned b[2][3][2];                             // S as second operand, columns 0 .. 7 and 8 .. 15 of the half
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) xm_cut(s[e][j][2 * i], s[e][j][2 * i + 1], b[i][0][j], b[i][1][j], b[i][2][j]);
        float d[4][2][4] = {}, low[4][2][4] = {};
        xm_products(d, low, a, b);
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            // columns in eights change places where two rows of one bank would meet
            const int at = (warp * 64 + m * 16 + g) * 16 + ((i * 8) ^ ((g >> 1 & 1) * 8)) + 2 * c;
#pragma unroll
            for (int j = 0; j < 4; ++j) d[m][i][j] += low[m][i][j];
            *reinterpret_cast<float2*>(part_s + at) = make_float2(d[m][i][0], d[m][i][1]);
            *reinterpret_cast<float2*>(part_s + at + 8 * 16) = make_float2(d[m][i][2], d[m][i][3]);
          }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        const int row = threadIdx.x >> 2, q = (threadIdx.x & 3) * 4;
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < 8; ++w) {
          const float4 v = *reinterpret_cast<const float4*>(part_s + (w * 64 + row) * 16 + (q ^ ((row >> 1 & 1) * 8)));
          sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
        }
        if (row < DC_TOKENS) {
          const float4 v = *reinterpret_cast<const float4*>(stage + kDtU + row * COLS + e * 16 + q);
          float* to = u_s + (e * 16 + q) * DT_PITCH + row;
          to[0] = v.x - sum.x; to[DT_PITCH] = v.y - sum.y; to[2 * DT_PITCH] = v.z - sum.z; to[3 * DT_PITCH] = v.w - sum.w;
        } else {
          *reinterpret_cast<float4*>(o_s + (row - DC_TOKENS) * (COLS + 4) + e * 16 + q) = sum;
        }
        if (e + 1 < kHalves) asm volatile("bar.sync 1, 256;" ::: "memory");
      }
      __syncthreads();                                   // U and G q S are in place, and the next stage
      // the matrix moves on by the chunk
      float2 decay[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) decay[j] = *reinterpret_cast<const float2*>(stage + kDtG + warp * 16 + j * 8 + 2 * c);
      float more[kHalves][2][4] = {}, low[kHalves][2][4] = {};
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        unsigned k[2][3][2];                             // keys of 16 tokens: [eight channels][piece]
#pragma unroll
        for (int p = 0; p < 3; ++p) {
          unsigned v[4];
          piece(chunk, 12 + t * 3 + p, v);
          k[0][p][0] = v[0]; k[0][p][1] = v[1]; k[1][p][0] = v[2]; k[1][p][1] = v[3];
        }
        unsigned u[kHalves][3][4];                       // U transposed: columns g, g + 8 of tokens 2 c, + 1 and 8 behind
#pragma unroll
        for (int e = 0; e < kHalves; ++e)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 v = *reinterpret_cast<const float2*>(u_s + (e * 16 + g + (i & 1) * 8) * DT_PITCH + t * 16 + 2 * c + (i >> 1) * 8);
            xm_cut(v.x, v.y, u[e][0][i], u[e][1][i], u[e][2][i]);
          }
        xm_products(more, low, u, k);
      }
      fetch(chunk + 2);
#pragma unroll
      for (int e = 0; e < kHalves; ++e)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int i = 0; i < 4; ++i) s[e][j][i] = fmaf(i & 1 ? decay[j].y : decay[j].x, s[e][j][i], more[e][j][i] + low[e][j][i]);
    }
    float zero = 0.f;                                    // a NaN where one of them is no finite number, which then stays so
#pragma unroll
    for (int e = 0; e < kHalves; ++e)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) zero = fmaf(s[e][j][i], 0.f, zero);
    wild = __syncthreads_or(!(zero == 0.f));
#pragma unroll
    for (int e = 0; e < kHalves; ++e)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; i += 2)
          if (wild) {
            float* to = dt_raw + (DC_DIM + warp * 16 + 2 * c + 8 * j) * COLS + e * 16 + i * 4 + g;
            to[0] = s[e][j][i];
            to[COLS] = s[e][j][i + 1];
          } else {
            *reinterpret_cast<float2*>(mine + (e * 16 + i * 4) * DC_DIM + j * 8) = *reinterpret_cast<const float2*>(&s[e][j][i]);
          }
  } else {
    const int id = threadIdx.x - 256;
    float zero = 0.f;                                    // as above, of the outputs
    auto fetch = [&](int chunk) {                        // M, G_31 and U0
      if (chunk < chunks) {
        const float* src = base + (size_t)chunk * heads * record;
        float* to = dt_raw + chunk % 3 * S::kStage;
        auto copy = [&](float* dst, const float* from) {
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(from) : "memory");
        };
#pragma unroll
        for (int i = id; i < DC_TOKENS * DC_TOKENS / 4; i += DT_HELPERS) copy(to + i / 8 * kDcPairs + i % 8 * 4, src + kDcM + i * 4);
        if (id < DC_DIM / 4) copy(to + kDtG + id * 4, src + kDcG + id * 4);
#pragma unroll
        for (int i = id; i < DC_TOKENS * COLS / 4; i += DT_HELPERS)
          copy(to + kDtU + i * 4, src + kDcU + i / (COLS / 4) * vdim + col0 + i % (COLS / 4) * 4);
      }
    };
    const int t = id >> 2, col = id & 3;                 // of G q S + M U: a row, columns col + 4 i
    auto outputs = [&](int chunk) {
      const float* m_row = dt_raw + chunk % 3 * S::kStage + t * kDcPairs;
      const float* u_s = dt_raw + S::kUs + (chunk & 1) * COLS * DT_PITCH + col * DT_PITCH;
      const float* o_s = dt_raw + S::kOs + (chunk & 1) * DC_TOKENS * (COLS + 4) + t * (COLS + 4) + col;
      float sum[COLS / 4];
#pragma unroll
      for (int i = 0; i < COLS / 4; ++i) sum[i] = o_s[4 * i];
#pragma unroll
      for (int s0 = 0; s0 < DC_TOKENS; s0 += 4) {
        if (s0 > t) break;
        const float4 m = *reinterpret_cast<const float4*>(m_row + s0);
#pragma unroll
        for (int i = 0; i < COLS / 4; ++i) {
          const float4 u = *reinterpret_cast<const float4*>(u_s + 4 * i * DT_PITCH + s0);
          sum[i] = fmaf(m.x, u.x, sum[i]);
          if (s0 + 1 <= t) sum[i] = fmaf(m.y, u.y, sum[i]);
          if (s0 + 2 <= t) sum[i] = fmaf(m.z, u.z, sum[i]);
          if (s0 + 3 <= t) sum[i] = fmaf(m.w, u.w, sum[i]);
        }
      }
      const int token = chunk * DC_TOKENS + t;
      if (token < n) {
        float* to = o_out + ((size_t)(first + token) * heads + h) * vdim + col0 + col;
#pragma unroll
        for (int i = 0; i < COLS / 4; ++i) {
          to[4 * i] = sum[i];
          zero = fmaf(sum[i], 0.f, zero);
        }
      }
    };
    fetch(0);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    for (int chunk = 0; chunk < chunks; ++chunk) {
      fetch(chunk + 1);                                  // three stages: what the one before the last held is read by now
      if (chunk > 0) outputs(chunk - 1);
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
    }
    outputs(chunks - 1);
    wild = __syncthreads_or(!(zero == 0.f));
  }
  if (wild)
    dt_scan_plain<COLS>(dt_raw, base, heads * record, n, vdim, col0,
                        state + (size_t)state_slot[r] * state_stride + ((size_t)h * vdim + col0) * DC_DIM,
                        o_out + ((size_t)first * heads + h) * vdim + col0, (size_t)heads * vdim);
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
                               vdim, taps, conv_off, n_requests,
                               (dim | vdim | ld | qkv_at | (by_channel ? decay_ld | decay_at : 0)) % 4 == 0 &&
                                   (((uintptr_t)proj | (by_channel ? (uintptr_t)decay : 0)) & 15) == 0};
  const dim3 grid(n_rows / DC_TOKENS + n_requests, heads);
  if (by_channel) return proj_dtype == TOKB200_F32 ? dc_prepare<float, true>(args, grid, stream) : TOKB200_BAD_DTYPE;
  if (proj_dtype == TOKB200_F32) return dc_prepare<float, false>(args, grid, stream);
  if (proj_dtype == TOKB200_BF16) return dc_prepare<__nv_bfloat16, false>(args, grid, stream);
  return TOKB200_BAD_DTYPE;
}

template <int COLS>
static int dc_scan(const float* records, int heads, int vdim, float* state, long long state_stride, const int* q_start,
                   const int* state_slot, int n_requests, float* o_out, cudaStream_t stream) {
  constexpr int bytes = DtShape<COLS>::kSmem;
  static bool done[64] = {};
  const int status = dc_allow(delta_chunk_scan_kernel<COLS>, bytes, done);
  if (status != TOKB200_OK) return status;
  return launch_dependent(delta_chunk_scan_kernel<COLS>, dim3(vdim / COLS, heads, n_requests), dim3(DT_THREADS),
                          (size_t)bytes, stream, records, heads, vdim, state, state_stride, q_start, state_slot, o_out);
}

// `columns`: of a block, 16 or 32; 0: by the number of blocks.
TOKB200_API int tokb200_delta_chunk_scan(const float* records, int heads, int dim, int vdim, float* state,
                                         long long state_stride, const int* q_start, const int* state_slot,
                                         int n_requests, float* o_out, int columns, cudaStream_t stream) {
  if (n_requests <= 0) return TOKB200_OK;
  if (heads <= 0 || heads > 65535 || n_requests > 65535 || !tokb200_delta_chunks_supported(dim, vdim))
    return TOKB200_BAD_SIZE;
  if ((((uintptr_t)records | (uintptr_t)state | (uintptr_t)o_out) & 15) || state_stride % 4) return TOKB200_BAD_ALIGNMENT;
  // Wide blocks do a column's work in less time but are half as many: taken where narrow ones would need a second turn on
  // 148 SMs (us of both kernels, narrow / wide: 16 heads of one request of 2,048 tokens 212 / 296, of sixteen of 128 223 /
  // 206, of one of 512 and 63 single ones 306 / 264, of eight of 512 371 / 371).
  const bool wide = columns ? columns == 32 : (long long)vdim / DC_COLS * heads * n_requests > 148;
  if (columns && columns != 16 && columns != 32) return TOKB200_BAD_SIZE;
  if (wide && vdim % 32 == 0)
    return dc_scan<32>(records, heads, vdim, state, state_stride, q_start, state_slot, n_requests, o_out, stream);
  return dc_scan<16>(records, heads, vdim, state, state_stride, q_start, state_slot, n_requests, o_out, stream);
}
