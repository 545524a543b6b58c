// The selective state-space recurrence with a scalar decay a head over portions of prompts, in chunks of 32 tokens and
// 32-bit throughout:
//     S <- a S + dt B x^T,   y = S^T C + D x,   a = exp(-exp(A_log) dt),   dt = softplus(raw + dt_bias)
// With G_t the product of a chunk's decays up to and with token t and S0 the matrix (N x P) before the chunk,
//     y_t = G_t S0^T C_t + sum_{s<=t} M[t][s] x_s + D x_t,   M[t][s] = (a_{s+1} .. a_t) (C_t . B_s) dt_s
//     S32 = G_31 S0 + sum_s (a_{s+1} .. a_31 dt_s) B_s x_s^T
// (products of decays only, never quotients: nothing can overflow).
//
//   ssd_chunk_prepare   a block a (chunk, group): C_t . B_s once for all heads of the group, and C and B in pieces; then a
//                       head a warp: steps, decays, M, G and the weights of the state's sum as one record
//   ssd_chunk_scan      a block a (32 columns of a head's matrix, request): the chunks one after another, the products with
//                       the matrix on the tensor cores with their operands in exact pieces (exact_mma.cuh).  A warp has 16
//                       channels of the matrix: the rows of C times them, whose sums over the warps meet in shared memory,
//                       then the matrix moves on; four more warps bring the next chunk, cut its weighted x and finish the
//                       rows of the one before
//
// The tensor pipe is busy 41 % of a block's time (counters), the pipe of shared memory 60 %: two warps a scheduler, each
// a chain of reads, cuts, products and sums.  Measured (heads of 64 x 128, us of both kernels, token by token / multiply-adds
// in chunks / here): 64 heads, a prompt of 2,048 tokens 392 / 213 / 149, two of 1,905 and 1,096 611 / 311 / 214; 16 heads,
// 2,048 126 / 198 / 125, four of 1,200 235 / 135 / 97.  Error against 64 bits (2-norm, memories of tens to hundreds of tokens),
// outputs and 32-bit states, multiply-adds in chunks / here: two prompts, 64 heads 1.43e-7 / 1.44e-7 and 1.66e-7 / 1.46e-7, 2,048
// tokens, 16 heads 1.38e-7 / 1.36e-7 and 1.77e-7 / 1.51e-7.  A chunk's records take 4.3 KB a head and 49 KB a group.
//
// A request's chunks are counted from its portion's first row; the record of chunk c of request r lies at place
// q_start[r] / 32 + r + c (no two the same, and known without a pass over the other requests).
#include "common.cuh"
#include "exact_mma.cuh"

#define SC_TOKENS 32
#define SC_DIM 128                        // lanes of B and C, zeros behind the model's own
#define SC_THREADS 256
#define SC_SCAN_THREADS 384
#define SC_COLS 32                        // columns of a scan block
constexpr int kScStride = SC_DIM + 4;     // of rows that several lanes read at once, 16 bytes each
constexpr int kScPairs = SC_TOKENS + 4;   // of M's rows
// a record, in floats: M (32 x 32), G (32), the weights of the state's sum (32)
constexpr int kScG = SC_TOKENS * SC_TOKENS, kScR = kScG + SC_TOKENS, kScRecord = kScR + SC_TOKENS;
// in front of a chunk's records, a group each: its C, then its B, as pieces in the order in which a lane of a product takes
// them ([16 channels][tile][piece][lane] of 16 bytes, see exact_mma.cuh); in floats
constexpr int kScB = 8 * 2 * 3 * 128, kScPieces = 2 * kScB;
__host__ __device__ static inline size_t sc_place(int heads, int groups) {
  return (size_t)groups * kScPieces + (size_t)heads * kScRecord;
}

__device__ __forceinline__ void sc_copy16(float* dst, const float* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 16 : 0) : "memory");
}

// xbc: [T, channels]: x (heads * P), B (groups * N), C (groups * N)
template <typename T>
__global__ void __launch_bounds__(SC_THREADS)
ssd_chunk_prepare_kernel(const float* __restrict__ xbc, int channels, const T* __restrict__ raw, int raw_ld,
                         const float* __restrict__ dt_bias, const float* __restrict__ a_log, int heads, int groups, int P,
                         int N, const int* __restrict__ q_start, int n_requests, float* __restrict__ records) {
  __shared__ __align__(16) float c_s[SC_TOKENS * kScStride], b_s[SC_TOKENS * kScStride], cb_s[SC_TOKENS * kScPairs];
  const int place = blockIdx.x, g = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int r = -1;                             // the request whose chunks lie around this place
  for (int i0 = 0; i0 < n_requests; i0 += 32) {
    const int i = i0 + lane;
    r += __popc(__ballot_sync(0xffffffffu, i < n_requests && q_start[i] / SC_TOKENS + i <= place));
  }
  const int start = r >= 0 ? q_start[r] : 0;
  const int t0 = start + (r >= 0 ? (place - start / SC_TOKENS - r) * SC_TOKENS : 0);
  const int n_here = r >= 0 ? min(SC_TOKENS, q_start[r + 1] - t0) : 0;
  pdl_wait();
  pdl_launch();
  if (n_here <= 0) return;
  for (int i = threadIdx.x; i < 2 * SC_TOKENS * (SC_DIM / 4); i += SC_THREADS) {
    const int which = i / (SC_TOKENS * (SC_DIM / 4)), t = i / (SC_DIM / 4) % SC_TOKENS, l = i % (SC_DIM / 4) * 4;
    const bool in = t < n_here && l < N;
    const float* src = xbc + (in ? (size_t)(t0 + t) * channels + (size_t)heads * P + (size_t)(which * groups + g) * N + l : 0);
    sc_copy16((which ? c_s : b_s) + t * kScStride + l, src, in);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  {
    const int t = threadIdx.x >> 3, s0 = threadIdx.x & 7;
    float4 dot[4];                        // four chains a sum: a single one of 128 rounds twice as much
#pragma unroll
    for (int i = 0; i < 4; ++i) dot[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int l = 0; l < SC_DIM; l += 4) {
      const float4 x = *reinterpret_cast<const float4*>(c_s + t * kScStride + l);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 y = *reinterpret_cast<const float4*>(b_s + (s0 + 8 * i) * kScStride + l);
        dot[i].x = fmaf(x.x, y.x, dot[i].x); dot[i].y = fmaf(x.y, y.y, dot[i].y);
        dot[i].z = fmaf(x.z, y.z, dot[i].z); dot[i].w = fmaf(x.w, y.w, dot[i].w);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) cb_s[t * kScPairs + s0 + 8 * i] = (dot[i].x + dot[i].y) + (dot[i].z + dot[i].w);
  }
  __syncthreads();
  float* at_place = records + (size_t)place * sc_place(heads, groups);
  {
    const int row = lane >> 2, pair = (lane & 3) * 2;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      unsigned p[3][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (e < 2) {                      // 16 rows of C, 16 channels
          const float2 v = *reinterpret_cast<const float2*>(c_s + (e * 16 + row + (i & 1) * 8) * kScStride + warp * 16 + pair + (i >> 1) * 8);
          xm_cut(v.x, v.y, p[0][i], p[1][i], p[2][i]);
        } else {                          // 16 tokens of B, twice eight channels
          const float* v = b_s + ((e - 2) * 16 + pair + (i & 1) * 8) * kScStride + warp * 16 + (i >> 1) * 8 + row;
          xm_cut(v[0], v[kScStride], p[0][i], p[1][i], p[2][i]);
        }
      }
      uint4* to = reinterpret_cast<uint4*>(at_place + (size_t)g * kScPieces + (e < 2 ? 0 : kScB)) + (warp * 2 + (e & 1)) * 3 * 32 + lane;
#pragma unroll
      for (int q = 0; q < 3; ++q) to[q * 32] = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
    }
  }
  const int share = heads / groups;
  for (int j = warp; j < share; j += SC_THREADS / 32) {
    const int h = g * share + j;
    float* rec = at_place + (size_t)groups * kScPieces + (size_t)h * kScRecord;
    float dt = 0.f, keep = 1.f;           // this lane's token
    if (lane < n_here) {
      const float v = to_float(raw[(size_t)(t0 + lane) * raw_ld + h]) + dt_bias[h];
      dt = v > 20.f ? v : log1pf(expf(v));
      keep = expf(-expf(a_log[h]) * dt);
    }
    float upto = keep, behind = 1.f;      // a_0 .. a_t, and a_{t+1} .. a_31
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float other = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto *= other;
    }
    float between = 0.f;                  // lane s: a_{s+1} .. a_t, from t = s on
#pragma unroll
    for (int t = 0; t < SC_TOKENS; ++t) {
      const float a = __shfl_sync(0xffffffffu, keep, t);
      between = t == lane ? 1.f : between * a;
      rec[t * SC_TOKENS + lane] = t >= lane ? cb_s[t * kScPairs + lane] * between * dt : 0.f;
    }
    behind = between;
    rec[kScG + lane] = upto;
    rec[kScR + lane] = behind * dt;
  }
}

__device__ __forceinline__ void sc_add(float4& a, float v, const float4& b) {
  a.x = fmaf(v, b.x, a.x); a.y = fmaf(v, b.y, a.y); a.z = fmaf(v, b.z, a.z); a.w = fmaf(v, b.w, a.w);
}

// a stage, in bytes: the weighted x as pieces ([half of the columns][16 tokens][piece][lane] of 16 bytes), then x (32 x 32),
// M (32 x 36) and G (32) as floats
constexpr int kSsX = 4 * 3 * 512, kSsM = kSsX + SC_TOKENS * SC_COLS * 4, kSsG = kSsM + SC_TOKENS * kScPairs * 4,
              kSsStage = kSsG + SC_TOKENS * 4;
// behind the three stages: the eight partial sums of C S [8][32][32] of two chunks
constexpr int kSsPart = 3 * kSsStage, kSsRing = kSsPart + 2 * 8 * SC_TOKENS * SC_COLS * 4 /* two chunks' pieces */,
              kSsBytes = kSsRing + 2 * kScPieces * 4;

// The same portion in plain multiply-adds, all threads of the block, for numbers that have no pieces (an infinity in the matrix,
// in B, C or x, numbers that round to one in 16 bits, and what then comes of them): slow, and replaces nothing but what the pieces
// left as no finite number.  `mine`: the block's columns of the matrix in memory, as they were before the portion; end_s: as the
// pieces left them ([128][32], as s_s); what lies behind the portion's last token, or behind a row's own, takes no part.  Inlined
// in small loops: a call, which is never made, cost the fast walk 2 to 4 %.
__device__ __forceinline__ void sc_scan_plain(float* s_s, const float* end_s, const float* __restrict__ x_in, const float* __restrict__ b_in,
                                           const float* __restrict__ c_in, int channels, const float* __restrict__ rec, size_t place,
                                           float d, int n, int N, float* __restrict__ mine, float* __restrict__ y_out, size_t y_ld) {
#pragma unroll 1
  for (int i = threadIdx.x; i < N * SC_COLS; i += SC_SCAN_THREADS) s_s[i] = mine[(size_t)(i % SC_COLS) * N + i / SC_COLS];
  __syncthreads();
#pragma unroll 1
  for (int t0 = 0; t0 < n; t0 += SC_TOKENS, rec += place) {
    const int here = min(SC_TOKENS, n - t0);
    const float* x = x_in + (size_t)t0 * channels;
#pragma unroll 1
    for (int i = threadIdx.x; i < here * SC_COLS; i += SC_SCAN_THREADS) {
      const int t = i / SC_COLS, c = i % SC_COLS;
      float* to = y_out + (size_t)(t0 + t) * y_ld + c;
      if (*to - *to == 0.f) continue;
      float sum = 0.f, acc = 0.f;
#pragma unroll 1
      for (int l = 0; l < N; ++l) sum = fmaf(c_in[(size_t)(t0 + t) * channels + l], s_s[l * SC_COLS + c], sum);
#pragma unroll 1
      for (int s = 0; s <= t; ++s) acc = fmaf(rec[t * SC_TOKENS + s], x[(size_t)s * channels + c], acc);
      acc = fmaf(d, x[(size_t)t * channels + c], acc);
      *to = fmaf(rec[kScG + t], sum, acc);
    }
    __syncthreads();
#pragma unroll 1
    for (int i = threadIdx.x; i < N * SC_COLS; i += SC_SCAN_THREADS) {
      const int l = i / SC_COLS, c = i % SC_COLS;
      float v = rec[kScG + SC_TOKENS - 1] * s_s[i];
#pragma unroll 1
      for (int s = 0; s < here; ++s)
        v = fmaf(b_in[(size_t)(t0 + s) * channels + l], rec[kScR + s] * x[(size_t)s * channels + c], v);
      s_s[i] = v;
    }
    __syncthreads();
  }
#pragma unroll 1
  for (int i = threadIdx.x; i < N * SC_COLS; i += SC_SCAN_THREADS)
    mine[(size_t)(i % SC_COLS) * N + i / SC_COLS] = end_s[i] - end_s[i] == 0.f ? end_s[i] : s_s[i];
}

__global__ void __launch_bounds__(SC_SCAN_THREADS, 1)
ssd_chunk_scan_kernel(const float* __restrict__ xbc, int channels, const float* __restrict__ records,
                      const float* __restrict__ skip, int heads, int groups, int P, int N, float* __restrict__ state,
                      long long state_stride, const int* __restrict__ q_start, const int* __restrict__ state_slot,
                      float* __restrict__ y_out) {
  extern __shared__ __align__(16) unsigned char ss_raw[];
  const int r = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * SC_COLS;
  const int first = q_start[r], n = q_start[r + 1] - first;
  // the warp's number through a shuffle: the compiler sees that the roles do not diverge
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int g = lane >> 2, c = lane & 3;                 // of a product's layout: row (or column) and pair
  pdl_wait();
  pdl_launch();
  if (n <= 0) return;
  const int chunks = (n + SC_TOKENS - 1) / SC_TOKENS;
  const size_t place = sc_place(heads, groups);
  const float* here = records + (size_t)(first / SC_TOKENS + r) * place;
  const float* base = here + (size_t)groups * kScPieces + (size_t)h * kScRecord;
  bool wild;                                             // a result of the pieces is no finite number
  float* end_s = reinterpret_cast<float*>(ss_raw) + SC_DIM * SC_COLS;      // then the matrix as the pieces left it

  if (warp < 8) {
    // ---- channels 16 w .. + 15 of the columns of S, transposed, as results and second operands of products lie ----
    const float* pieces = here + (size_t)(h / (heads / groups)) * kScPieces;
    const int channel = warp * 16 + 2 * c;
    float* mine = state + (size_t)state_slot[r] * state_stride + ((size_t)h * P + col0 + g) * N + channel;
    float s[2][2][4];                                    // columns g and g + 8 of a half, channels 8 j + 2 c, + 1
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; i += 2)
          *reinterpret_cast<float2*>(&s[e][j][i]) =
              channel + 8 * j < N ? *reinterpret_cast<const float2*>(mine + (size_t)(e * 16 + i * 4) * N + j * 8) : make_float2(0.f, 0.f);
    // The pieces of C and B that a lane takes are its own alone: copied two chunks ahead to places of shared memory that no
    // other thread touches.
    const unsigned ring = (unsigned)__cvta_generic_to_shared(ss_raw + kSsRing) + (warp * 12 * 32 + lane) * 16;
    auto fetch = [&](int chunk) {
      if (chunk < chunks) {
        const float* src = pieces + (size_t)chunk * place + lane * 4;
        const unsigned to = ring + (chunk & 1) * kScPieces * 4;
#pragma unroll
        for (int i = 0; i < 12; ++i) {
          const float* from = src + (i < 6 ? 0 : kScB) + (warp * 6 + i % 6) * 128;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + i * 512), "l"(from) : "memory");
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto piece = [&](int chunk, int i, unsigned (&v)[4]) {
      asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                   : "r"(ring + (chunk & 1) * kScPieces * 4 + i * 512) : "memory");
    };
    fetch(0);
    fetch(1);
    __syncthreads();                                     // the first stage is in place
    for (int chunk = 0; chunk < chunks; ++chunk) {
      const unsigned char* stage = ss_raw + chunk % 3 * kSsStage;
      float* part_s = reinterpret_cast<float*>(ss_raw + kSsPart) + (chunk & 1) * 8 * SC_TOKENS * SC_COLS;
      // the rows of C times the columns, over this warp's channels
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      unsigned a[2][3][4];                               // C: tile of 16 rows, piece
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int p = 0; p < 3; ++p) piece(chunk, m * 3 + p, a[m][p]);
      unsigned b[4][3][2];                               // eight columns each
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int j = 0; j < 2; ++j)
          xm_cut(s[e >> 1][j][2 * (e & 1)], s[e >> 1][j][2 * (e & 1) + 1], b[e][0][j], b[e][1][j], b[e][2][j]);
      float d[2][4][4] = {}, low[2][4][4] = {};
      xm_products(d, low, a, b);
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          // columns in eights change places so that the rows of a store lie on different banks
          const int row = m * 16 + g, at = (warp * SC_TOKENS + row) * SC_COLS + ((e ^ (row & 3)) * 8) + 2 * c;
#pragma unroll
          for (int i = 0; i < 4; ++i) d[m][e][i] += low[m][e][i];
          *reinterpret_cast<float2*>(part_s + at) = make_float2(d[m][e][0], d[m][e][1]);
          *reinterpret_cast<float2*>(part_s + at + 8 * SC_COLS) = make_float2(d[m][e][2], d[m][e][3]);
        }
      // the matrix moves on by the chunk
      const float all = *reinterpret_cast<const float*>(stage + kSsG + (SC_TOKENS - 1) * 4);
      const uint4* u_s = reinterpret_cast<const uint4*>(stage) + lane;
      float more[2][2][4] = {}, low_more[2][2][4] = {};
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        unsigned u[2][3][4], k[2][3][2];                 // B of 16 tokens: [eight channels][piece]
#pragma unroll
        for (int p = 0; p < 3; ++p) {
          unsigned v[4];
          piece(chunk, 6 + t * 3 + p, v);
          k[0][p][0] = v[0]; k[0][p][1] = v[1]; k[1][p][0] = v[2]; k[1][p][1] = v[3];
        }
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(u[e][p]) = u_s[((e * 2 + t) * 3 + p) * 32];
        xm_products(more, low_more, u, k);
      }
      fetch(chunk + 2);
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int i = 0; i < 4; ++i) s[e][j][i] = fmaf(all, s[e][j][i], more[e][j][i] + low_more[e][j][i]);
      __syncthreads();                                   // the partial sums and the next stage are in place
    }
    float zero = 0.f;                                    // a NaN where one of them is no finite number, which then stays so
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) zero = fmaf(s[e][j][i], 0.f, zero);
    wild = __syncthreads_or(!(zero == 0.f));
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; i += 2)
          if (wild) {
            float* to = end_s + (channel + 8 * j) * SC_COLS + e * 16 + i * 4 + g;
            to[0] = s[e][j][i];
            to[SC_COLS] = s[e][j][i + 1];
          } else if (channel + 8 * j < N) {
            *reinterpret_cast<float2*>(mine + (size_t)(e * 16 + i * 4) * N + j * 8) = *reinterpret_cast<const float2*>(&s[e][j][i]);
          }
  } else {
    const int w = warp - 8, id = threadIdx.x - 256;
    float zero = 0.f;                                    // as above, of the outputs
    const float* x_in = xbc + (size_t)h * P + col0;
    const float d = skip[h];
    const int t = id >> 3, c4 = (id & 7) * 4;            // of x, M and the outputs: rows t and t + 16, four columns
    float uu[8], weight[4];                              // columns g, g + 8 of half w / 2, tokens 16 (w % 2) + 2 c, + 1 and 8 behind
    auto load = [&](int chunk) {
      const float* rec = base + (size_t)chunk * place;
      const size_t at0 = (size_t)(first + chunk * SC_TOKENS) * channels;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int row = (w & 1) * 16 + 2 * c + (i & 1) + (i >> 2) * 8, col = (w >> 1) * 16 + g + (i >> 1 & 1) * 8;
        uu[i] = chunk * SC_TOKENS + row < n ? x_in[at0 + (size_t)row * channels + col] : 0.f;
        if (!(i & 2)) weight[(i & 1) + (i >> 2) * 2] = rec[kScR + row];       // used a chunk later, as is x
      }
    };
    auto put = [&](int chunk) {
      unsigned char* stage = ss_raw + chunk % 3 * kSsStage;
      const float* rec = base + (size_t)chunk * place;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int row = t + 16 * e;
        const bool in = chunk * SC_TOKENS + row < n;
        sc_copy16(reinterpret_cast<float*>(stage + kSsX + (row * SC_COLS + c4) * 4),
                  x_in + (in ? (size_t)(first + chunk * SC_TOKENS + row) * channels + c4 : 0), in);
        sc_copy16(reinterpret_cast<float*>(stage + kSsM + (row * kScPairs + c4) * 4), rec + row * SC_TOKENS + c4, true);
      }
      if (id < SC_TOKENS / 4) sc_copy16(reinterpret_cast<float*>(stage + kSsG + id * 16), rec + kScG + id * 4, true);
      unsigned p[3][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        xm_cut(weight[i & 2] * uu[2 * i], weight[(i & 2) + 1] * uu[2 * i + 1], p[0][i], p[1][i], p[2][i]);
      uint4* to = reinterpret_cast<uint4*>(stage) + w * 3 * 32 + lane;
#pragma unroll
      for (int q = 0; q < 3; ++q) to[q * 32] = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
    };
    auto outputs = [&](int chunk) {
      const unsigned char* stage = ss_raw + chunk % 3 * kSsStage;
      const float* part_s = reinterpret_cast<const float*>(ss_raw + kSsPart) + (chunk & 1) * 8 * SC_TOKENS * SC_COLS;
      const float* m_row = reinterpret_cast<const float*>(stage + kSsM) + t * kScPairs;
      const float4* x_s = reinterpret_cast<const float4*>(stage + kSsX) + (id & 7);
      float4 sum[2], acc[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        sum[e] = acc[e] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 v = *reinterpret_cast<const float4*>(part_s + (i * SC_TOKENS + t + 16 * e) * SC_COLS + (c4 ^ ((t & 3) * 8)));
          sum[e].x += v.x; sum[e].y += v.y; sum[e].z += v.z; sum[e].w += v.w;
        }
      }
      // what comes behind a row's own token is left out, not added with weight 0: an infinity or a NaN there is not this row's
#pragma unroll
      for (int s0 = 0; s0 < SC_TOKENS; s0 += 4) {
        float4 m[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) m[e] = *reinterpret_cast<const float4*>(m_row + 16 * e * kScPairs + s0);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 v = x_s[(s0 + i) * 8];
#pragma unroll
          for (int e = 0; e < 2; ++e)
            if (s0 + i <= 16 * e || (s0 + i < 16 * e + 16 && s0 + i <= t + 16 * e))
              sc_add(acc[e], i == 0 ? m[e].x : i == 1 ? m[e].y : i == 2 ? m[e].z : m[e].w, v);
        }
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int row = t + 16 * e, token = chunk * SC_TOKENS + row;
        sc_add(acc[e], d, x_s[row * 8]);
        sc_add(acc[e], *reinterpret_cast<const float*>(stage + kSsG + row * 4), sum[e]);
        if (token < n) {
          *reinterpret_cast<float4*>(y_out + ((size_t)(first + token) * heads + h) * P + col0 + c4) = acc[e];
          zero = fmaf(acc[e].x, 0.f, fmaf(acc[e].y, 0.f, fmaf(acc[e].z, 0.f, fmaf(acc[e].w, 0.f, zero))));
        }
      }
    };
    load(0);
    put(0);
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (chunks > 1) load(1);
    __syncthreads();
    for (int chunk = 0; chunk < chunks; ++chunk) {
      if (chunk + 1 < chunks) {                          // three stages: what the one before the last held is read by now
        put(chunk + 1);
        if (chunk + 2 < chunks) load(chunk + 2);
      }
      if (chunk > 0) outputs(chunk - 1);
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
    }
    outputs(chunks - 1);
    wild = __syncthreads_or(!(zero == 0.f));
  }
  if (wild) {
    const float* x_in = xbc + (size_t)first * channels;
    const float* b_in = x_in + (size_t)heads * P + (size_t)(h / (heads / groups)) * N;
    sc_scan_plain(reinterpret_cast<float*>(ss_raw), end_s, x_in + (size_t)h * P + col0, b_in, b_in + (size_t)groups * N, channels, base, place,
                  skip[h], n, N, state + (size_t)state_slot[r] * state_stride + ((size_t)h * P + col0) * N,
                  y_out + ((size_t)first * heads + h) * P + col0, (size_t)heads * P);
  }
}

// ---- launchers -----------------------------------------------------------------------------------------------------
// Whether the recurrence of these sizes runs in chunks.
TOKB200_API int tokb200_ssd_chunks_supported(int P, int N) {
  return N > 64 && N <= SC_DIM && N % 4 == 0 && P > 0 && P % SC_COLS == 0;
}

// Floats of the records of a step.
TOKB200_API long long tokb200_ssd_chunk_floats(int n_rows, int n_requests, int heads, int groups) {
  return ((long long)n_rows / SC_TOKENS + n_requests) * (long long)sc_place(heads, groups);
}

TOKB200_API int tokb200_ssd_chunks(const float* xbc, int channels, const void* proj, int proj_dtype, int ld, int dt_at,
                                   const float* dt_bias, const float* a_log, const float* skip, int heads, int groups,
                                   int P, int N, float* state, long long stride, const int* q_start, const int* state_slot,
                                   int n_rows, int n_requests, float* y, float* records, cudaStream_t stream) {
  if (n_rows <= 0 || n_requests <= 0) return TOKB200_OK;
  if (heads <= 0 || groups <= 0 || heads % groups || heads > 65535 || n_requests > 65535 ||
      channels != heads * P + 2 * groups * N || !tokb200_ssd_chunks_supported(P, N))
    return TOKB200_BAD_SIZE;
  if ((((uintptr_t)xbc | (uintptr_t)state | (uintptr_t)y | (uintptr_t)records) & 15) || stride % 4) return TOKB200_BAD_ALIGNMENT;
  static bool done[64] = {};
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return TOKB200_BAD_SIZE;
  if (!done[device]) {
    const cudaError_t err = cudaFuncSetAttribute(ssd_chunk_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSsBytes);
    if (err != cudaSuccess) return (int)err;
    done[device] = true;
  }
  const dim3 grid(n_rows / SC_TOKENS + n_requests, groups);
  int status = TOKB200_BAD_DTYPE;
  if (proj_dtype == TOKB200_F32)
    status = launch_dependent(ssd_chunk_prepare_kernel<float>, grid, dim3(SC_THREADS), 0, stream, xbc, channels,
                              (const float*)proj + dt_at, ld, dt_bias, a_log, heads, groups, P, N, q_start, n_requests, records);
  else if (proj_dtype == TOKB200_BF16)
    status = launch_dependent(ssd_chunk_prepare_kernel<__nv_bfloat16>, grid, dim3(SC_THREADS), 0, stream, xbc, channels,
                              (const __nv_bfloat16*)proj + dt_at, ld, dt_bias, a_log, heads, groups, P, N, q_start, n_requests,
                              records);
  if (status != TOKB200_OK) return status;
  return launch_dependent(ssd_chunk_scan_kernel, dim3(P / SC_COLS, heads, n_requests), dim3(SC_SCAN_THREADS),
                          (size_t)kSsBytes, stream, xbc, channels, records, skip, heads, groups, P, N, state, stride, q_start,
                          state_slot, y);
}
