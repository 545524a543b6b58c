// Attention over the paged cache for any batch of rows: portions of prompts and
// single decoded tokens alike.  Row t belongs to request row_req[t] and sits at
// absolute position pos[t]; it attends to the keys of its request at positions
// lo..pos[t] (lo = 0, or pos - window when the layer has a window: a key is
// hidden when key + window < query), all read from the cache, where this step's
// own keys were written before the launch.
//
// This is the general kernel: any head size, any number of heads and groups,
// both precisions.  One block per (row, query head); keys are processed in
// fixed chunks of ATT_CHUNK counted from lo, so a row's arithmetic depends only on
// its own position and window, never on the batch around it.  Scores, the
// running maximum, the exponentials and the weighted sum are 32-bit.
//
// `keep_first` (> 0): the sequence's first keys that stay visible although the window has passed them.  They
// are walked in front of the others: key i of the walk is i for the kept ones and lo + i - kept behind them.
//
// `sink` (optional, one float32 per query head): a learned score without key or value that
// takes part in the softmax's denominator once, unscaled: the running maximum starts at it
// and the running sum at 1.  `softcap` (> 0): a score s becomes softcap * tanh(s / softcap) before
// the softmax.
#include "common.cuh"

#define ATT_THREADS 128
#define ATT_CHUNK 128
#define ATT_MAX_HEAD_DIM 1024

template <typename T>
__global__ void __launch_bounds__(ATT_THREADS)
paged_attention_generic_kernel(const T* __restrict__ q, const T* __restrict__ k_pool,
                               const T* __restrict__ v_pool, T* __restrict__ out,
                               const int* __restrict__ block_table, int table_stride,
                               const int* __restrict__ row_req, const int* __restrict__ pos,
                               int nh, int nkv, int d, int page, int window, int chunk, int keep_first, float scale,
                               const float* __restrict__ sink, float softcap) {
  extern __shared__ float smem[];
  float* q_s = smem;                 // d
  float* p_s = smem + d;             // ATT_CHUNK
  int* slot_s = (int*)(p_s + ATT_CHUNK);  // ATT_CHUNK
  __shared__ float scratch[33];

  const int t = blockIdx.x, h = blockIdx.y;
  const int r = row_req[t];
  if (r < 0) return;
  const int p = pos[t];
  const int kvh = h / (nh / nkv);
  const int lo = first_key_with_kept(first_visible_key(p, window, chunk), keep_first);
  const int kept = kept_first_keys(lo, keep_first);
  const int n_keys = p - lo + 1 + kept;
  const int* table = block_table + (size_t)r * table_stride;

  const T* q_row = q + ((size_t)t * nh + h) * d;
  for (int i = threadIdx.x; i < d; i += ATT_THREADS) q_s[i] = to_float(q_row[i]);
  __syncthreads();

  float m = sink ? sink[h] : -INFINITY, l = sink ? 1.f : 0.f;
  float acc[ATT_MAX_HEAD_DIM / ATT_THREADS];
#pragma unroll
  for (int i = 0; i < ATT_MAX_HEAD_DIM / ATT_THREADS; ++i) acc[i] = 0.f;

  for (int c0 = 0; c0 < n_keys; c0 += ATT_CHUNK) {
    const int at = c0 + (int)threadIdx.x;
    const bool live = at < n_keys;
    const int key = at < kept ? at : lo + at - kept;
    float s = -INFINITY;
    int slot = -1;
    if (live) {
      const int pg = table[key / page];
      slot = pg * page + key % page;
      const T* k_row = k_pool + ((size_t)slot * nkv + kvh) * d;
      float dot = 0.f;
      for (int i = 0; i < d; ++i) dot += q_s[i] * to_float(k_row[i]);
      s = dot * scale;
      if (softcap > 0.f) s = softcap * tanhf(s / softcap);
    }
    const float c_max = block_max(s, scratch);
    const float m_new = fmaxf(m, c_max);
    const float e = live ? expf(s - m_new) : 0.f;
    p_s[threadIdx.x] = e;
    slot_s[threadIdx.x] = slot;
    const float c_sum = block_sum(e, scratch);  // contains the barrier that publishes p_s
    const float corr = expf(m - m_new);         // 0 on the first chunk (m = -inf)
    l = l * corr + c_sum;
    m = m_new;
    const int n = min(ATT_CHUNK, n_keys - c0);
#pragma unroll
    for (int i = 0; i < ATT_MAX_HEAD_DIM / ATT_THREADS; ++i) {
      const int dim = threadIdx.x + i * ATT_THREADS;
      if (dim < d) {
        float a = acc[i] * corr;
        for (int j = 0; j < n; ++j)
          a += p_s[j] * to_float(v_pool[((size_t)slot_s[j] * nkv + kvh) * d + dim]);
        acc[i] = a;
      }
    }
    __syncthreads();  // p_s and slot_s are rewritten by the next chunk
  }
  T* o_row = out + ((size_t)t * nh + h) * d;
#pragma unroll
  for (int i = 0; i < ATT_MAX_HEAD_DIM / ATT_THREADS; ++i) {
    const int dim = threadIdx.x + i * ATT_THREADS;
    if (dim < d) o_row[dim] = from_float<T>(acc[i] / l);
  }
}

TOKB200_API int tokb200_paged_attention_generic(
    const void* q, const void* k_pool, const void* v_pool, void* out, int dtype,
    const int* block_table, int table_stride, const int* row_req, const int* pos, int n_rows,
    int nh, int nkv, int d, int page, int window, int chunk, int keep_first, float scale, const float* sink,
    float softcap, cudaStream_t stream) {
  if (n_rows <= 0) return TOKB200_OK;
  if (d <= 0 || d > ATT_MAX_HEAD_DIM || nh <= 0 || nkv <= 0 || nh % nkv || page <= 0 ||
      nh > 65535)
    return TOKB200_BAD_SIZE;
  const size_t smem = (size_t)(d + 2 * ATT_CHUNK) * sizeof(float);
  dim3 grid(n_rows, nh);
  if (dtype == TOKB200_F32)
    paged_attention_generic_kernel<float><<<grid, ATT_THREADS, smem, stream>>>(
        (const float*)q, (const float*)k_pool, (const float*)v_pool, (float*)out, block_table,
        table_stride, row_req, pos, nh, nkv, d, page, window, chunk, keep_first, scale, sink, softcap);
  else if (dtype == TOKB200_BF16)
    paged_attention_generic_kernel<__nv_bfloat16><<<grid, ATT_THREADS, smem, stream>>>(
        (const __nv_bfloat16*)q, (const __nv_bfloat16*)k_pool, (const __nv_bfloat16*)v_pool,
        (__nv_bfloat16*)out, block_table, table_stride, row_req, pos, nh, nkv, d, page, window,
        chunk, keep_first, scale, sink, softcap);
  else
    return TOKB200_BAD_DTYPE;
  return tokb200_launch_status();
}

// ---- portions of prompts in 32-bit ------------------------------------------------------------------------------
// The same arithmetic, key by key and sum by sum (a row's bits are those of the kernel above, whatever tile it falls
// into), for tiles of up to 64 consecutive rows of one request whose keys all begin at 0 (no window, no chunk) and
// heads of 64 or 128 lanes.  A block takes a tile and a query head: a chunk's 128 keys and values are staged in shared
// memory once for the tile's rows instead of being read by every row.  256 threads, 16 x 16: thread (ty, tx) keeps rows
// 4 ty .. + 3, in the first product keys tx + 16 i (a warp sum's butterfly over 32 keys is then one addition inside the
// thread and four exchanges), in the second lanes 4 tx .. of the head, with K of the next chunk on its way during the second
// product and V during the first.  A block an SM, so eight warps: neither pipe is full (777 tokens, 14 heads of 64: FMA 32 %,
// shared memory 40 %), warps wait for shared memory and for results, and 182 blocks leave most of a second turn empty.
#define ATT_TILE_ROWS 64

__device__ __forceinline__ void att_copy16(float* dst, const float* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 16 : 0) : "memory");
}

template <int D>
constexpr int att_tiles_smem() {
  return (ATT_TILE_ROWS * D + 2 * ATT_CHUNK * (D + 4) + ATT_CHUNK * (ATT_TILE_ROWS + 4)) * (int)sizeof(float);
}

template <int D>
__global__ void __launch_bounds__(256, 1)
paged_attention_f32_tiles_kernel(const float* __restrict__ q, const float* __restrict__ k_pool,
                                 const float* __restrict__ v_pool, float* __restrict__ out,
                                 const int* __restrict__ block_table, int table_stride,
                                 const int* __restrict__ row_req, const int* __restrict__ pos,
                                 const int* __restrict__ tiles, int nh, int nkv, int page, float scale,
                                 const float* __restrict__ sink, float softcap) {
  constexpr int kStride = D + 4, kPStride = ATT_TILE_ROWS + 4, kLanes = D / 16;
  extern __shared__ __align__(16) float att_raw[];
  float* q_s = att_raw;                                   // [64][D]
  float* k_s = q_s + ATT_TILE_ROWS * D;                   // [128][D + 4]
  float* v_s = k_s + ATT_CHUNK * kStride;                 // [128][D + 4]
  float* p_s = v_s + ATT_CHUNK * kStride;                 // [128][64 + 4], a key's probabilities for all rows
  const int h = blockIdx.x, row0 = tiles[2 * blockIdx.y], n_rows = tiles[2 * blockIdx.y + 1];
  if (n_rows <= 0) return;
  const int r_id = row_req[row0];
  if (r_id < 0) return;
  const int pos0 = pos[row0], pos_last = pos0 + n_rows - 1;
  const int kvh = h / (nh / nkv);
  const int* table = block_table + (size_t)r_id * table_stride;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;

  auto fetch = [&](float* to, const float* pool, int c0) {
    for (int e = threadIdx.x; e < ATT_CHUNK * (D / 4); e += 256) {
      const int t = e / (D / 4), c = e % (D / 4) * 4, key = c0 + t;
      const bool in = key <= pos_last;
      const size_t at = in ? ((size_t)(table[key / page] * page + key % page) * nkv + kvh) * D + c : 0;
      att_copy16(to + t * kStride + c, pool + at, in);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int e = threadIdx.x; e < ATT_TILE_ROWS * (D / 4); e += 256) {
    const int t = e / (D / 4), c = e % (D / 4) * 4;
    att_copy16(q_s + t * D + c, q + ((size_t)(row0 + (t < n_rows ? t : 0)) * nh + h) * D + c, t < n_rows);
  }
  fetch(k_s, k_pool, 0);                                   // q rides with the first keys
  fetch(v_s, v_pool, 0);

  const bool busy = ty * 4 < n_rows;                       // threads without a row only stage
  float m[4], l[4], acc[4][kLanes];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m[i] = sink ? sink[h] : -INFINITY;
    l[i] = sink ? 1.f : 0.f;
#pragma unroll
    for (int j = 0; j < kLanes; ++j) acc[i][j] = 0.f;
  }
  for (int c0 = 0; c0 <= pos_last; c0 += ATT_CHUNK) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();                                       // the chunk's keys (and q) are in place
    if (__any_sync(0xffffffffu, busy)) {
      float s[4][8];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) s[i][j] = 0.f;
#pragma unroll 2
      for (int c = 0; c < D; c += 4) {
        float4 x[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const float4*>(q_s + (ty * 4 + i) * D + c);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 y = *reinterpret_cast<const float4*>(k_s + (tx + 16 * j) * kStride + c);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            s[i][j] = fmaf(x[i].x, y.x, s[i][j]);
            s[i][j] = fmaf(x[i].y, y.y, s[i][j]);
            s[i][j] = fmaf(x[i].z, y.z, s[i][j]);
            s[i][j] = fmaf(x[i].w, y.w, s[i][j]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int p = pos0 + ty * 4 + i;
        float top = -INFINITY;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float v = s[i][j] * scale;
          if (softcap > 0.f) v = softcap * tanhf(v / softcap);
          s[i][j] = c0 + tx + 16 * j <= p ? v : -INFINITY;
          top = fmaxf(top, s[i][j]);
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        const float m_new = fmaxf(m[i], top);
        float sums[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
#pragma unroll
          for (int j = 2 * g; j < 2 * g + 2; ++j) s[i][j] = c0 + tx + 16 * j <= p ? expf(s[i][j] - m_new) : 0.f;
          sums[g] = s[i][2 * g] + s[i][2 * g + 1];
#pragma unroll
          for (int o = 8; o > 0; o >>= 1) sums[g] += __shfl_xor_sync(0xffffffffu, sums[g], o);
        }
        const float sum = (sums[0] + sums[2]) + (sums[1] + sums[3]);
        if (c0 <= p) {                                     // a row whose keys ended before this chunk stays as it is
          const float corr = expf(m[i] - m_new);
          l[i] = fmaf(l[i], corr, sum);
          m[i] = m_new;
#pragma unroll
          for (int j = 0; j < kLanes; ++j) acc[i][j] *= corr;
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j)
        *reinterpret_cast<float4*>(p_s + (tx + 16 * j) * kPStride + ty * 4) = make_float4(s[0][j], s[1][j], s[2][j], s[3][j]);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                       // values and probabilities are in place, the keys are done with
    if (c0 + ATT_CHUNK <= pos_last) fetch(k_s, k_pool, c0 + ATT_CHUNK);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    if (busy) {
      // rows 4 ty .. + 3 see n, n + 1, n + 2, n + 3 of the chunk's keys: a key that a row does not see is left out, not
      // added with weight 0
      const int n = pos0 + ty * 4 - c0 + 1;
      const int common = min(max(n, 0), ATT_CHUNK), most = min(max(n + 3, 0), ATT_CHUNK);
      auto value = [&](int j, float (&y)[kLanes]) {
#pragma unroll
        for (int e = 0; e < kLanes; e += 4) {
          const float4 v = *reinterpret_cast<const float4*>(v_s + j * kStride + e * 16 + tx * 4);
          y[e] = v.x; y[e + 1] = v.y; y[e + 2] = v.z; y[e + 3] = v.w;
        }
      };
#pragma unroll 4
      for (int j = 0; j < common; ++j) {
        const float4 x = *reinterpret_cast<const float4*>(p_s + j * kPStride + ty * 4);
        float y[kLanes];
        value(j, y);
#pragma unroll
        for (int e = 0; e < kLanes; ++e) {
          acc[0][e] = fmaf(x.x, y[e], acc[0][e]);
          acc[1][e] = fmaf(x.y, y[e], acc[1][e]);
          acc[2][e] = fmaf(x.z, y[e], acc[2][e]);
          acc[3][e] = fmaf(x.w, y[e], acc[3][e]);
        }
      }
      for (int j = common; j < most; ++j) {
        float y[kLanes];
        value(j, y);
#pragma unroll
        for (int i = 1; i < 4; ++i)
          if (j < n + i) {
            const float x = p_s[j * kPStride + ty * 4 + i];
#pragma unroll
            for (int e = 0; e < kLanes; ++e) acc[i][e] = fmaf(x, y[e], acc[i][e]);
          }
      }
    }
    __syncthreads();                                       // values and probabilities are done with
    if (c0 + ATT_CHUNK <= pos_last) fetch(v_s, v_pool, c0 + ATT_CHUNK);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (ty * 4 + i >= n_rows) continue;
    float* o_row = out + ((size_t)(row0 + ty * 4 + i) * nh + h) * D;
#pragma unroll
    for (int e = 0; e < kLanes; e += 4)
      *reinterpret_cast<float4*>(o_row + e * 16 + tx * 4) =
          make_float4(acc[i][e] / l[i], acc[i][e + 1] / l[i], acc[i][e + 2] / l[i], acc[i][e + 3] / l[i]);
  }
}

template <int D>
static int launch_f32_tiles(const float* q, const float* k_pool, const float* v_pool, float* out, const int* block_table,
                            int table_stride, const int* row_req, const int* pos, const int* tiles, int n_tiles, int nh,
                            int nkv, int page, float scale, const float* sink, float softcap, cudaStream_t stream) {
  static bool configured[64] = {};
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return TOKB200_BAD_SIZE;
  if (!configured[device]) {
    cudaError_t err = cudaFuncSetAttribute(paged_attention_f32_tiles_kernel<D>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, att_tiles_smem<D>());
    if (err != cudaSuccess) return (int)err;
    configured[device] = true;
  }
  paged_attention_f32_tiles_kernel<D><<<dim3(nh, n_tiles), 256, att_tiles_smem<D>(), stream>>>(
      q, k_pool, v_pool, out, block_table, table_stride, row_req, pos, tiles, nh, nkv, page, scale, sink, softcap);
  return tokb200_launch_status();
}

// tiles: [n_tiles][2] = (first row, rows) of consecutive rows of one request, rows <= 64 (0: none)
TOKB200_API int tokb200_paged_attention_f32_tiles(
    const float* q, const float* k_pool, const float* v_pool, float* out, const int* block_table, int table_stride,
    const int* row_req, const int* pos, const int* tiles, int n_tiles, int nh, int nkv, int d, int page, float scale,
    const float* sink, float softcap, cudaStream_t stream) {
  if (n_tiles <= 0) return TOKB200_OK;
  if (nh <= 0 || nkv <= 0 || nh % nkv || page <= 0 || n_tiles > 65535) return TOKB200_BAD_SIZE;
  if (((uintptr_t)q | (uintptr_t)k_pool | (uintptr_t)v_pool | (uintptr_t)out) & 15) return TOKB200_BAD_ALIGNMENT;
  if (d == 64)
    return launch_f32_tiles<64>(q, k_pool, v_pool, out, block_table, table_stride, row_req, pos, tiles, n_tiles, nh, nkv,
                                page, scale, sink, softcap, stream);
  if (d == 128)
    return launch_f32_tiles<128>(q, k_pool, v_pool, out, block_table, table_stride, row_req, pos, tiles, n_tiles, nh, nkv,
                                 page, scale, sink, softcap, stream);
  return TOKB200_BAD_SIZE;
}
