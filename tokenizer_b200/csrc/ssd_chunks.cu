// The selective state-space recurrence with a scalar decay a head over portions of prompts, in chunks of 32 tokens and
// 32-bit throughout:
//     S <- a S + dt B x^T,   y = S^T C + D x,   a = exp(-exp(A_log) dt),   dt = softplus(raw + dt_bias)
// With G_t the product of a chunk's decays up to and with token t and S0 the matrix (N x P) before the chunk,
//     y_t = G_t S0^T C_t + sum_{s<=t} M[t][s] x_s + D x_t,   M[t][s] = (a_{s+1} .. a_t) (C_t . B_s) dt_s
//     S32 = G_31 S0 + sum_s (a_{s+1} .. a_31 dt_s) B_s x_s^T
// (products of decays only, never quotients: nothing can overflow).
//
//   ssd_chunk_prepare   a block a (chunk, group): C_t . B_s once for all heads of the group, then a head a warp: steps,
//                       decays, M, G and the weights of the state's sum as one record
//   ssd_chunk_scan      a block a (32 columns of a head's matrix, request): the chunks one after another.  The 32 rows of C
//                       meet the columns in 8 x 8 register tiles, lanes cut over 16 half warps; then half of the threads
//                       move the matrix on (8 x 4 of it each, in registers) while the others finish the chunk's rows.  The
//                       next chunk's B, C, x and record are on their way (cp.async) meanwhile
//
// The scan is bound by reads of shared memory (counters: the pipe that brings them back busy 66 % of the time, the FMA pipe
// 44 %; a tile of R x C costs R + C cycles of the 128 bytes a cycle that come back, and R C / 4
// of the multiply-adds): hence the large tiles.  Measured (heads of 64 x 128, us, token by token / here): 64 heads, a prompt
// of 2,048 tokens 307 / 214, two of 1,905 and 1,096 412 / 312; with tiles of 4 x 4 it was 301 and 441.
//
// A request's chunks are counted from its portion's first row; the record of chunk c of request r lies at place
// q_start[r] / 32 + r + c (no two the same, and known without a pass over the other requests).
#include "common.cuh"

#define SC_TOKENS 32
#define SC_DIM 128                        // lanes of B and C, zeros behind the model's own
#define SC_THREADS 256
#define SC_COLS 32                        // columns of a scan block
constexpr int kScStride = SC_DIM + 4;     // of rows that several lanes read at once, 16 bytes each
constexpr int kScPairs = SC_TOKENS + 4;   // of M's rows
// a record, in floats: M (32 x 32), G (32), the weights of the state's sum (32)
constexpr int kScG = SC_TOKENS * SC_TOKENS, kScR = kScG + SC_TOKENS, kScRecord = kScR + SC_TOKENS;

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
  const int share = heads / groups;
  for (int j = warp; j < share; j += SC_THREADS / 32) {
    const int h = g * share + j;
    float* rec = records + ((size_t)place * heads + h) * kScRecord;
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

// a stage, in floats: C (32 x 132), B (32 x 128), M (32 x 36), G and the weights (32 each), x (32 x 32)
constexpr int kSsB = SC_TOKENS * kScStride, kSsM = kSsB + SC_TOKENS * SC_DIM, kSsG = kSsM + SC_TOKENS * kScPairs,
              kSsR = kSsG + SC_TOKENS, kSsX = kSsR + SC_TOKENS, kSsStage = kSsX + SC_TOKENS * SC_COLS;
// behind the two stages: the columns of S [128][32], the eight partial sums [8][32][32], the weighted x [32][32]
constexpr int kSsBytes = (2 * kSsStage + SC_DIM * SC_COLS + 8 * SC_TOKENS * SC_COLS + SC_TOKENS * SC_COLS) * 4;

template <bool V> struct sc_bool { static constexpr bool value = V; };

__device__ __forceinline__ void sc_add(float4& a, float v, const float4& b) {
  a.x = fmaf(v, b.x, a.x); a.y = fmaf(v, b.y, a.y); a.z = fmaf(v, b.z, a.z); a.w = fmaf(v, b.w, a.w);
}

__global__ void __launch_bounds__(SC_THREADS, 1)
ssd_chunk_scan_kernel(const float* __restrict__ xbc, int channels, const float* __restrict__ records,
                      const float* __restrict__ skip, int heads, int groups, int P, int N, float* __restrict__ state,
                      long long state_stride, const int* __restrict__ q_start, const int* __restrict__ state_slot,
                      float* __restrict__ y_out) {
  extern __shared__ __align__(16) float ss_raw[];
  float* s_s = ss_raw + 2 * kSsStage;
  float* part_s = s_s + SC_DIM * SC_COLS;
  float* u_s = part_s + 8 * SC_TOKENS * SC_COLS;
  const int r = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * SC_COLS;
  const int first = q_start[r], n = q_start[r + 1] - first;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_wait();
  pdl_launch();
  if (n <= 0) return;
  const int chunks = (n + SC_TOKENS - 1) / SC_TOKENS;
  const float* base = records + ((size_t)(first / SC_TOKENS + r) * heads + h) * kScRecord;
  const int g = h / (heads / groups);
  const float* b_in = xbc + (size_t)heads * P + (size_t)g * N;
  const float* c_in = b_in + (size_t)groups * N;
  // t and c4: of the 32 x 32 numbers of x, of its weighted copy and of M, four neighbours a thread
  const int t = threadIdx.x >> 3, c4 = (threadIdx.x & 7) * 4;
  auto fetch = [&](int c) {
    if (c < chunks) {
      float* dst = ss_raw + (c & 1) * kSsStage;
      const int t0 = c * SC_TOKENS, tb = threadIdx.x / (SC_DIM / 4), l = threadIdx.x % (SC_DIM / 4) * 4;
#pragma unroll
      for (int i = 0; i < SC_TOKENS; i += SC_THREADS / (SC_DIM / 4)) {
        const bool in = t0 + tb + i < n && l < N;
        const size_t at = in ? (size_t)(first + t0 + tb + i) * channels + l : 0;
        sc_copy16(dst + (tb + i) * kScStride + l, c_in + at, in);
        sc_copy16(dst + kSsB + (tb + i) * SC_DIM + l, b_in + at, in);
      }
      const float* rec = base + (size_t)c * heads * kScRecord;
      sc_copy16(dst + kSsM + t * kScPairs + c4, rec + threadIdx.x * 4, true);
      if (threadIdx.x < 16) sc_copy16(dst + kSsG + threadIdx.x * 4, rec + kScG + threadIdx.x * 4, true);
      const bool in = t0 + t < n;
      sc_copy16(dst + kSsX + threadIdx.x * 4, xbc + (in ? (size_t)(first + t0 + t) * channels + (size_t)h * P + col0 + c4 : 0), in);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  static_assert(SC_THREADS * 4 == SC_TOKENS * SC_TOKENS && SC_TOKENS == SC_COLS, "a copy a thread");
  fetch(0);
  // threads 0 .. 127: rows row .. + 7 of columns c4 .. + 3 of the matrix
  const bool owner = threadIdx.x < 128;
  const int row = t * 8;
  float* mine = state + (size_t)state_slot[r] * state_stride + ((size_t)h * P + col0 + c4) * N + row;
  float4 S[8];                                           // a row's four columns each
  if (owner) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float4 v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        v[j] = row + 4 * e < N ? *reinterpret_cast<const float4*>(mine + (size_t)j * N + 4 * e) : make_float4(0.f, 0.f, 0.f, 0.f);
      S[4 * e] = make_float4(v[0].x, v[1].x, v[2].x, v[3].x);
      S[4 * e + 1] = make_float4(v[0].y, v[1].y, v[2].y, v[3].y);
      S[4 * e + 2] = make_float4(v[0].z, v[1].z, v[2].z, v[3].z);
      S[4 * e + 3] = make_float4(v[0].w, v[1].w, v[2].w, v[3].w);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) *reinterpret_cast<float4*>(s_s + (row + i) * SC_COLS + c4) = S[i];
  }
  const float d = skip[h];

  for (int c = 0; c < chunks; ++c) {
    const float* stage = ss_raw + (c & 1) * kSsStage;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                     // the chunk and the matrix are in place
    fetch(c + 1);                                        // into the stage that the chunk before has left
    float zero;
    {
      const float w = stage[kSsR + t];
      const float4 x = *reinterpret_cast<const float4*>(stage + kSsX + threadIdx.x * 4);
      *reinterpret_cast<float4*>(u_s + threadIdx.x * 4) = make_float4(w * x.x, w * x.y, w * x.z, w * x.w);
      zero = fmaf(x.x, 0.f, x.y * 0.f) + fmaf(x.z, 0.f, x.w * 0.f);      // a NaN where one of them is no number
    }
    {
      // the rows of C times the columns, lanes k0 .. k0 + 7 a half warp: rows group + 4 i, columns cols .. + 3 and
      // cols + 16 .. + 19
      const int k0 = warp * 16 + (lane >> 4) * 8, group = (lane >> 2) & 3, cols = (lane & 3) * 4;
      const float* x_s = stage + group * kScStride;
      float acc[8][8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
#pragma unroll
      for (int k = k0; k < k0 + 8; k += 4) {
        float4 x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = *reinterpret_cast<const float4*>(x_s + i * 4 * kScStride + k);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          const float4 lo = *reinterpret_cast<const float4*>(s_s + (k + kk) * SC_COLS + cols);
          const float4 hi = *reinterpret_cast<const float4*>(s_s + (k + kk) * SC_COLS + 16 + cols);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float v = kk == 0 ? x[i].x : kk == 1 ? x[i].y : kk == 2 ? x[i].z : x[i].w;
            acc[i][0] = fmaf(v, lo.x, acc[i][0]); acc[i][1] = fmaf(v, lo.y, acc[i][1]);
            acc[i][2] = fmaf(v, lo.z, acc[i][2]); acc[i][3] = fmaf(v, lo.w, acc[i][3]);
            acc[i][4] = fmaf(v, hi.x, acc[i][4]); acc[i][5] = fmaf(v, hi.y, acc[i][5]);
            acc[i][6] = fmaf(v, hi.z, acc[i][6]); acc[i][7] = fmaf(v, hi.w, acc[i][7]);
          }
        }
      }
      const bool upper = lane & 16;                      // the half warps' sums meet: the upper one keeps i = 4 .. 7
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
          v[j] = (upper ? acc[i + 4][j] : acc[i][j]) + __shfl_xor_sync(0xffffffffu, upper ? acc[i][j] : acc[i + 4][j], 16);
        float* to = part_s + (warp * SC_TOKENS + group + 4 * i + (upper ? 16 : 0)) * SC_COLS + cols;
        *reinterpret_cast<float4*>(to) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4*>(to + 16) = make_float4(v[4], v[5], v[6], v[7]);
      }
    }
    const bool wild = __syncthreads_or(!(zero == 0.f));      // the chunk's x holds infinities or NaN
    if (owner) {
      // the matrix moves on by the chunk
      const float all = stage[kSsG + SC_TOKENS - 1];
#pragma unroll
      for (int i = 0; i < 8; ++i) S[i] = make_float4(S[i].x * all, S[i].y * all, S[i].z * all, S[i].w * all);
#pragma unroll 8
      for (int s = 0; s < SC_TOKENS; ++s) {
        const float4 lo = *reinterpret_cast<const float4*>(stage + kSsB + s * SC_DIM + row);
        const float4 hi = *reinterpret_cast<const float4*>(stage + kSsB + s * SC_DIM + row + 4);
        const float4 u = *reinterpret_cast<const float4*>(u_s + s * SC_COLS + c4);
        sc_add(S[0], lo.x, u); sc_add(S[1], lo.y, u); sc_add(S[2], lo.z, u); sc_add(S[3], lo.w, u);
        sc_add(S[4], hi.x, u); sc_add(S[5], hi.y, u); sc_add(S[6], hi.z, u); sc_add(S[7], hi.w, u);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) *reinterpret_cast<float4*>(s_s + (row + i) * SC_COLS + c4) = S[i];
    } else {
      // rows t - 16 and t, four columns of each
      const int at[2] = {t - 16, t};
      float4 sum[2], acc[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        sum[e] = acc[e] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 v = *reinterpret_cast<const float4*>(part_s + (i * SC_TOKENS + at[e]) * SC_COLS + c4);
          sum[e].x += v.x; sum[e].y += v.y; sum[e].z += v.z; sum[e].w += v.w;
        }
      }
      // M is 0 behind a row's own token; where an infinity or a NaN stands there it is left out, not added with weight 0
      auto rows = [&](auto all) {
#pragma unroll
        for (int s = 0; s < SC_TOKENS; s += 4) {
          float4 m[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) m[e] = *reinterpret_cast<const float4*>(stage + kSsM + at[e] * kScPairs + s);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 x = *reinterpret_cast<const float4*>(stage + kSsX + (s + i) * SC_COLS + c4);
#pragma unroll
            for (int e = 0; e < 2; ++e)
              if (decltype(all)::value || s + i <= at[e])
                sc_add(acc[e], i == 0 ? m[e].x : i == 1 ? m[e].y : i == 2 ? m[e].z : m[e].w, x);
          }
        }
      };
      if (wild) rows(sc_bool<false>());
      else rows(sc_bool<true>());
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int token = c * SC_TOKENS + at[e];
        sc_add(acc[e], d, *reinterpret_cast<const float4*>(stage + kSsX + at[e] * SC_COLS + c4));
        sc_add(acc[e], stage[kSsG + at[e]], sum[e]);
        if (token < n) *reinterpret_cast<float4*>(y_out + ((size_t)(first + token) * heads + h) * P + col0 + c4) = acc[e];
      }
    }
  }
  if (owner) {
#pragma unroll
    for (int e = 0; e < 2; ++e)
      if (row + 4 * e < N) {
        const float4* v = S + 4 * e;
        *reinterpret_cast<float4*>(mine + 4 * e) = make_float4(v[0].x, v[1].x, v[2].x, v[3].x);
        *reinterpret_cast<float4*>(mine + (size_t)N + 4 * e) = make_float4(v[0].y, v[1].y, v[2].y, v[3].y);
        *reinterpret_cast<float4*>(mine + (size_t)2 * N + 4 * e) = make_float4(v[0].z, v[1].z, v[2].z, v[3].z);
        *reinterpret_cast<float4*>(mine + (size_t)3 * N + 4 * e) = make_float4(v[0].w, v[1].w, v[2].w, v[3].w);
      }
  }
}

// ---- launchers -----------------------------------------------------------------------------------------------------
// Whether the recurrence of these sizes runs in chunks.
TOKB200_API int tokb200_ssd_chunks_supported(int P, int N) {
  return N > 64 && N <= SC_DIM && N % 4 == 0 && P > 0 && P % SC_COLS == 0;
}

// Floats of the records of a step.
TOKB200_API long long tokb200_ssd_chunk_floats(int n_rows, int n_requests, int heads) {
  return ((long long)n_rows / SC_TOKENS + n_requests) * heads * kScRecord;
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
  return launch_dependent(ssd_chunk_scan_kernel, dim3(P / SC_COLS, heads, n_requests), dim3(SC_THREADS),
                          (size_t)kSsBytes, stream, xbc, channels, records, skip, heads, groups, P, N, state, stride, q_start,
                          state_slot, y);
}
