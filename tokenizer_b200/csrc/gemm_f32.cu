// True 32-bit matrix product C[M,N] = A[M,K] W[N,K]^T (+ bias) where K is below 768, no multiple of 4 or the operands do not
// lie on 16 bytes (the others go to the tensor cores in exact pieces, gemm_f32_tcgen05.cu, whose error is the smaller one there):
// plain FMA in float, no tensor cores and no reduced-precision mode.  Each output
// element sums its K products in index order, so a row's result does not depend
// on how many other rows are in the batch, nor on the tile the element falls into.
//
// A block of 16 x 16 threads computes TM * 16 rows x 128 columns, TM x 8 sums a thread.  Per step of k a thread reads TM
// numbers of A and 8 of W, by 16-byte loads and a step ahead of their use, for 8 TM multiply-adds (paired ones,
// fma.rn.f32x2, measured half as fast).  Bound by issue: four of five slots are taken, the FMA pipe and the pipe of shared
// memory are busy 70 % of the time each (counters, 777 x 9,728 x 896, tiles of 128 rows).  Operands are staged k-major, 16 of k at a time, the next piece's
// global loads in registers while this one is multiplied.
#include "common.cuh"

#define TILE_N 128
#define TILE_K 16
#define GEMM_THREADS 256

// VEC: K and lda are whole 4s and both bases lie on 16 bytes (16-byte loads along k)
template <int TM, bool VEC>
__global__ void __launch_bounds__(GEMM_THREADS, TM == 8 ? 2 : 3)
gemm_f32_kernel(const float* __restrict__ a, const float* __restrict__ w,
                const float* __restrict__ bias, float* __restrict__ c, int M, int N, int K,
                int lda, int ldc) {
  constexpr int TILE_M = TM * 16;
  constexpr int kAStride = TILE_M + 4, kWStride = TILE_N + 4;
  // 16-byte pieces of k a thread loads a step
  constexpr int kAPieces = (TILE_M * TILE_K / 4 + GEMM_THREADS - 1) / GEMM_THREADS;
  constexpr int kWPieces = TILE_N * TILE_K / 4 / GEMM_THREADS;
  __shared__ __align__(16) float a_s[2][TILE_K * kAStride];
  __shared__ __align__(16) float w_s[2][TILE_K * kWStride];
  const int m0 = blockIdx.y * TILE_M, n0 = blockIdx.x * TILE_N;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  float acc[TM][8];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;

  float4 a_r[kAPieces], w_r[kWPieces];
  auto load4 = [&](const float* base, int row, int rows, int ld, int k) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < rows) {
      const float* src = base + (size_t)row * ld + k;
      if (VEC) {
        if (k < K) v = *reinterpret_cast<const float4*>(src);
      } else {
        if (k < K) v.x = src[0];
        if (k + 1 < K) v.y = src[1];
        if (k + 2 < K) v.z = src[2];
        if (k + 3 < K) v.w = src[3];
      }
    }
    return v;
  };
  auto fetch = [&](int k0) {
#pragma unroll
    for (int e = 0; e < kAPieces; ++e) {
      const int idx = threadIdx.x + e * GEMM_THREADS, row = idx / (TILE_K / 4);
      if (TILE_M * TILE_K / 4 % GEMM_THREADS == 0 || row < TILE_M) a_r[e] = load4(a, m0 + row, M, lda, k0 + idx % (TILE_K / 4) * 4);
    }
#pragma unroll
    for (int e = 0; e < kWPieces; ++e) {
      const int idx = threadIdx.x + e * GEMM_THREADS;
      w_r[e] = load4(w, n0 + idx / (TILE_K / 4), N, K, k0 + idx % (TILE_K / 4) * 4);
    }
  };
  auto put = [&](int buf) {
#pragma unroll
    for (int e = 0; e < kAPieces; ++e) {
      const int idx = threadIdx.x + e * GEMM_THREADS, row = idx / (TILE_K / 4);
      float* to = &a_s[buf][idx % (TILE_K / 4) * 4 * kAStride + row];
      if (TILE_M * TILE_K / 4 % GEMM_THREADS == 0 || row < TILE_M) {
        to[0] = a_r[e].x; to[kAStride] = a_r[e].y; to[2 * kAStride] = a_r[e].z; to[3 * kAStride] = a_r[e].w;
      }
    }
#pragma unroll
    for (int e = 0; e < kWPieces; ++e) {
      const int idx = threadIdx.x + e * GEMM_THREADS;
      float* to = &w_s[buf][idx % (TILE_K / 4) * 4 * kWStride + idx / (TILE_K / 4)];
      to[0] = w_r[e].x; to[kWStride] = w_r[e].y; to[2 * kWStride] = w_r[e].z; to[3 * kWStride] = w_r[e].w;
    }
  };

  fetch(0);
  put(0);
  __syncthreads();
  const int steps = (K + TILE_K - 1) / TILE_K;
  for (int s = 0; s < steps; ++s) {
    const int buf = s & 1;
    if (s + 1 < steps) fetch((s + 1) * TILE_K);
    const float* a_b = &a_s[buf][ty * TM];
    const float* w_b = &w_s[buf][tx * 4];
    // a step of k's operands: TM of A, and columns tx * 4 .. + 3 and 64 + tx * 4 .. + 3 of W (neighbouring threads read
    // neighbouring 16 bytes)
    float av[2][TM], wv[2][8];
    auto operands = [&](int kk, int to) {
#pragma unroll
      for (int i = 0; i < TM; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(a_b + kk * kAStride + i);
        av[to][i] = v.x; av[to][i + 1] = v.y; av[to][i + 2] = v.z; av[to][i + 3] = v.w;
      }
#pragma unroll
      for (int j = 0; j < 8; j += 4) {
        const float4 v = *reinterpret_cast<const float4*>(w_b + kk * kWStride + j * 16);
        wv[to][j] = v.x; wv[to][j + 1] = v.y; wv[to][j + 2] = v.z; wv[to][j + 3] = v.w;
      }
    };
    operands(0, 0);
#pragma unroll
    for (int kk = 0; kk < TILE_K; ++kk) {
      if (kk + 1 < TILE_K) operands(kk + 1, (kk + 1) & 1);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(av[kk & 1][i], wv[kk & 1][j], acc[i][j]);
    }
    if (s + 1 < steps) put(buf ^ 1);      // its last readers passed the barrier of the step before
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty * TM + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int n = n0 + (j / 4) * 64 + tx * 4 + j % 4;
      if (n < N) c[(size_t)m * ldc + n] = acc[i][j] + (bias ? bias[n] : 0.f);
    }
  }
}

template <int TM>
static int launch_f32(const float* a, const float* w, const float* bias, float* c, int M, int N, int K, int lda, int ldc,
                      bool vec, cudaStream_t stream) {
  dim3 grid((N + TILE_N - 1) / TILE_N, (M + TM * 16 - 1) / (TM * 16));
  if (grid.y > 65535) return TOKB200_BAD_SIZE;
  if (vec) gemm_f32_kernel<TM, true><<<grid, GEMM_THREADS, 0, stream>>>(a, w, bias, c, M, N, K, lda, ldc);
  else gemm_f32_kernel<TM, false><<<grid, GEMM_THREADS, 0, stream>>>(a, w, bias, c, M, N, K, lda, ldc);
  return tokb200_launch_status();
}

// Few rows, or too few tiles of the kind above for the device: tiles of 4 R rows x 32 columns by 128 threads, a warp's
// lanes are the columns and each warp keeps R rows (w + 4 i).  With few rows bound by latency: pieces of 32 of k come
// through a ring of cp.async stages, so that several are on their way while one is multiplied.  With many bound by reads of
// shared memory (its pipe busy 90 % at 777 x 896 x 4,864 in tiles of 32 rows, the FMA pipe 36 %).
#define FEW_N 32
#define FEW_K 32
#define FEW_THREADS 128

__device__ __forceinline__ void f32_copy16(float* dst, const float* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 16 : 0) : "memory");
}

template <int R, bool VEC>
__global__ void __launch_bounds__(FEW_THREADS)
gemm_f32_few_kernel(const float* __restrict__ a, const float* __restrict__ w,
                    const float* __restrict__ bias, float* __restrict__ c, int M, int N, int K,
                    int lda, int ldc) {
  constexpr int kRows = 4 * R, kStages = R == 16 ? 3 : 4, kStride = FEW_K + 4;
  __shared__ __align__(16) float a_s[kStages][kRows * kStride];
  __shared__ __align__(16) float w_s[kStages][FEW_N * kStride];
  const int m0 = blockIdx.y * kRows, n0 = blockIdx.x * FEW_N;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto piece = [&](float* to, const float* base, int row, int rows, int ld, int k) {
    const bool in = row < rows && k < K;
    const float* src = base + (in ? (size_t)row * ld + k : 0);
    if (VEC) {
      f32_copy16(to, src, in);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) to[i] = in && k + i < K ? src[i] : 0.f;
    }
  };
  auto fetch = [&](int step) {
    const int buf = step % kStages, k0 = step * FEW_K;
#pragma unroll
    for (int e = threadIdx.x; e < FEW_N * FEW_K / 4; e += FEW_THREADS)
      piece(&w_s[buf][e / (FEW_K / 4) * kStride + e % (FEW_K / 4) * 4], w, n0 + e / (FEW_K / 4), N, K,
            k0 + e % (FEW_K / 4) * 4);
#pragma unroll
    for (int e = threadIdx.x; e < kRows * FEW_K / 4; e += FEW_THREADS)
      piece(&a_s[buf][e / (FEW_K / 4) * kStride + e % (FEW_K / 4) * 4], a, m0 + e / (FEW_K / 4), M, lda,
            k0 + e % (FEW_K / 4) * 4);
  };
  float acc[R];
#pragma unroll
  for (int i = 0; i < R; ++i) acc[i] = 0.f;
  const int steps = (K + FEW_K - 1) / FEW_K;
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < steps) fetch(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();                    // step s is in place, and everybody is done with the buffer fetched into next
    if (s + kStages - 1 < steps) fetch(s + kStages - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* w_b = &w_s[s % kStages][lane * kStride];
    const float* a_b = &a_s[s % kStages][warp * kStride];
#pragma unroll
    for (int k = 0; k < FEW_K; k += 4) {
      const float4 x = *reinterpret_cast<const float4*>(w_b + k);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const float4 y = *reinterpret_cast<const float4*>(a_b + 4 * i * kStride + k);
        acc[i] = fmaf(y.x, x.x, acc[i]);
        acc[i] = fmaf(y.y, x.y, acc[i]);
        acc[i] = fmaf(y.z, x.z, acc[i]);
        acc[i] = fmaf(y.w, x.w, acc[i]);
      }
    }
  }
  const int n = n0 + lane;
  if (n >= N) return;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int m = m0 + warp + 4 * i;
    if (m < M) c[(size_t)m * ldc + n] = acc[i] + (bias ? bias[n] : 0.f);
  }
}

template <int R>
static int launch_f32_few(const float* a, const float* w, const float* bias, float* c, int M, int N, int K, int lda,
                          int ldc, bool vec, cudaStream_t stream) {
  dim3 grid((N + FEW_N - 1) / FEW_N, (M + 4 * R - 1) / (4 * R));
  if (grid.y > 65535) return TOKB200_BAD_SIZE;
  if (vec) gemm_f32_few_kernel<R, true><<<grid, FEW_THREADS, 0, stream>>>(a, w, bias, c, M, N, K, lda, ldc);
  else gemm_f32_few_kernel<R, false><<<grid, FEW_THREADS, 0, stream>>>(a, w, bias, c, M, N, K, lda, ldc);
  return tokb200_launch_status();
}

// `form`: the tile, an index into `forms` below; -1: by the rule.
TOKB200_API int tokb200_gemm_f32(const float* a, const float* w, const float* bias, float* c,
                                 int M, int N, int K, int lda, int ldc, int form, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return TOKB200_OK;
  if (K <= 0 || lda < K || ldc < N) return TOKB200_BAD_SIZE;
  if (M > 64LL * 65535) return TOKB200_BAD_SIZE;
  // Every form gives the same bits, so the choice is one of time alone: measured, a lone tile on an SM takes `first`
  // cycles a step of k and every further one `more` (at 777 rows, us of forms 0 1 3: 9,728 x 896 343 / 371 / 536, 896 x
  // 4,864 506 / 367 / 292, 1,152 x 896 97 / 72 / 77); the form with the least time for the SM that gets the most wins.
  struct Form { int rows, columns; float first, more; };
  static const Form forms[] = {{128, 128, 191.f, 180.f}, {64, 128, 136.f, 108.f}, {64, 32, 53.f, 35.f}, {32, 32, 30.f, 21.f},
                               {16, 32, 24.f, 12.f}, {4, 32, 15.6f, 7.3f}};
  const long long sms = 148;
  int best = -1;
  double least = 0.;
  for (int i = 0; i < (int)(sizeof(forms) / sizeof(forms[0])); ++i) {
    const long long down = (M + forms[i].rows - 1) / forms[i].rows;
    const long long tiles = down * ((N + forms[i].columns - 1) / forms[i].columns);
    if (down > 65535) continue;
    const double time = forms[i].first + (double)((tiles + sms - 1) / sms - 1) * forms[i].more;
    if (best < 0 || time < least) { best = i; least = time; }
  }
  if (form >= (int)(sizeof(forms) / sizeof(forms[0]))) return TOKB200_BAD_SIZE;
  if (form >= 0) best = form;
  const bool vec = K % 4 == 0 && lda % 4 == 0 && ((((uintptr_t)a) | ((uintptr_t)w)) & 15) == 0;
  switch (best) {
    case 0: return launch_f32<8>(a, w, bias, c, M, N, K, lda, ldc, vec, stream);
    case 1: return launch_f32<4>(a, w, bias, c, M, N, K, lda, ldc, vec, stream);
    case 2: return launch_f32_few<16>(a, w, bias, c, M, N, K, lda, ldc, vec, stream);
    case 3: return launch_f32_few<8>(a, w, bias, c, M, N, K, lda, ldc, vec, stream);
    case 4: return launch_f32_few<4>(a, w, bias, c, M, N, K, lda, ldc, vec, stream);
    default: return launch_f32_few<1>(a, w, bias, c, M, N, K, lda, ldc, vec, stream);
  }
}
