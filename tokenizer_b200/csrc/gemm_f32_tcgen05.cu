// True 32-bit matrix product C[M,N] = A[M,K] W[N,K]^T (+ bias) on the fifth-generation tensor cores: every operand is cut
// into three bfloat16 numbers that add up to it exactly (8 + 8 + 8 bits and signs), and of the nine products of pieces the
// six that reach 2^-24 of the whole are added up in 32-bit:
//
//     x w = x0 w0 + (x1 w0 + x0 w1) + (x2 w0 + x1 w1 + x0 w2) + what is below 2^-24
//
// The tensor core cuts a sum's low bits off instead of rounding, so no sum is left to it for long: each of the three orders
// has an accumulator of its own, which starts at zero every 256 of k and is added to registers in plain 32-bit.  An
// element's value depends on its row, its weight row and K alone: the chunks of 256, the order of the sums and the cut of k
// into groups follow from K, never from the batch or the tile.
//
//   * eight converter warps bring 32-bit tiles from global memory into registers a stage ahead, cut them and write three
//     planes of 128 weight rows and NT batch rows x 64 into shared memory (128-byte swizzled, as TMA would);
//   * one warp issues tcgen05.mma (M = 128 weight rows, K = 16): three a step of 16, N = 3 NT, 2 NT and NT;
//   * eight drain warps add a chunk's accumulators (double-buffered in tensor memory) to their registers and write the
//     outputs, 32 neighbouring weight rows a warp.
//
// One block an SM walks segments (a tile of outputs, a group of at most 10 stages of k).  Either a block takes a tile's
// groups one after another and adds each to the output, or the groups go to different blocks as partial sums that
// `gemm_f32_sum_kernel` adds in the same order, which gives the same bits.
//
// Measured (one B200, us, this / the kernel of multiply-adds): 777 rows of 1,152 x 896 21 / 71, 896 x 896 16 / 57, 9,728 x 896
// 104 / 343 (131 TFLOP/s), 896 x 4,864 56 / 291; one row of the same 9.6 / 9.0, 9.6 / 9.0, 14.0 / 14.9, 13.1 / 39.8,
// and of the vocabulary's 151,936 x 896 137 / 118 (to four rows; 8 rows 141 / 217, 16 147 / 214), of 17,920 x 1,536 30.5 / 28.6, 37,888
// x 3,584 125 / 123: few rows of a wide weight wait for the converters, which have one stage of 32 KB an SM on its way.  A whole
// step of one row gains (24 layers of the first four and the vocabulary 1,250 / 1,870), and a row must meet the same kernel
// in every batch, so the line is drawn by k alone.  Error
// against 64 bits (2-norm, normal numbers) 2.1e-7 / 5.3e-7 at k = 896, 2.2e-7 / 1.25e-6 at 4,864; from k = 768 on it is the
// smaller one for numbers of one sign too (896: 3.2e-7 / 4.4e-7; 512: 3.8e-7 / 3.5e-7), which is where `ops.gemm_f32` draws
// the line.  A stage of 80 rows takes 1,270 ns: the products alone 745, the cutting alone 735 (both bound by shared memory,
// 190 KB a stage), the loads alone 540; chunks of 128 of k, whose accumulators are read twice as often, 1,520.  Two
// things that counted: a row's 32 bytes in one load (140 -> 128 us at 9,728 x 896) and loads of the output in front of
// the adds to it, eight at a time (the drain alone took 47 us of 148).
//
// An operand that is an infinity, a NaN or rounds to an infinity in 16 bits has no such pieces (its last one is a NaN), and a
// product just below the largest number may lie above it in its first pieces: outputs that come out as no finite number are
// computed anew by a chain of multiply-adds.  Numbers below 2^-109 keep an absolute error of 2^-133.  Every wait on an mbarrier is
// bounded.
#include "common.cuh"

#define FS_K 64
#define FS_W_ROWS 128
#define FS_CONVERT 256                 // threads that convert, behind the 256 that drain
#define FS_UNIT (FS_CONVERT / 8)       // rows they convert at a time
#define FS_DRAIN 256
#define FS_THREADS (FS_CONVERT + FS_DRAIN + 32)
#define FS_GROUP 10                    // stages of k a group has at most
#define FS_CHUNK 4                     // stages whose products the tensor core adds up before they go to registers
#define FS_WAIT_LIMIT (1u << 17)       // polls of up to 20 us each: seconds in all

__device__ int fs_error_flag = 0;

__device__ __forceinline__ unsigned fs_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void fs_bar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(fs_smem(bar)), "r"(count));
}
__device__ __forceinline__ void fs_arrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(fs_smem(bar)) : "memory");
}
__device__ __forceinline__ bool fs_try(unsigned long long* bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n.reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
      "selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done) : "r"(fs_smem(bar)), "r"(parity), "r"(20000u) : "memory");
  return done != 0;
}
__device__ __noinline__ bool fs_wait_long(unsigned long long* bar, unsigned parity) {
  for (unsigned spin = 0; spin < FS_WAIT_LIMIT; ++spin)
    if (fs_try(bar, parity)) return true;
  atomicExch(&fs_error_flag, 1);
  tokb200_report_error(TOKB200_LIB_GEMM_F32_TCGEN05, 1);
  return false;
}
// false when the limit ran out
__device__ __forceinline__ bool fs_wait(unsigned long long* bar, unsigned parity) {
  return fs_try(bar, parity) || fs_wait_long(bar, parity);
}
__device__ __forceinline__ bool fs_elect() {
  unsigned lead;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(lead));
  return lead != 0;
}
// K-major tile with 128-byte swizzle, rows of 128 bytes, 8-row groups 1,024 bytes apart
__device__ __forceinline__ unsigned long long fs_desc(unsigned smem_address) {
  return (unsigned long long)((smem_address & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void fs_mma(unsigned tmem_d, unsigned long long a_desc, unsigned long long b_desc, unsigned idesc,
                                       unsigned accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
      ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void fs_commit(unsigned long long* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
               ::"r"(fs_smem(bar)) : "memory");
}
__device__ __forceinline__ void fs_tmem_load(unsigned taddr, unsigned (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr) : "memory");
}
__device__ __forceinline__ void fs_tmem_load(unsigned taddr, unsigned (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}

template <int NT> struct FsShape {
  static constexpr int kPlaneW = FS_W_ROWS * 128, kPlaneA = NT * 128;          // bytes
  static constexpr int kStage = 3 * (kPlaneW + kPlaneA);
  static constexpr int kStages = NT <= 16 ? 4 : NT <= 64 ? 3 : 2;
  static constexpr int kPitch = NT == 16 ? 64 : NT == 32 ? 128 : 256;          // columns of a buffer, of which 3 NT are used
  static constexpr int kSmem = kStages * kStage + 1024 /* alignment slack */ + 256 /* barriers */;
};

struct FsProblem {
  const float* a;
  const float* w;
  const float* bias;        // may be null
  float* out;               // [M, N], or partial sums [groups, M, N]
  int M, N, K;
  int across;               // tiles along the batch
  int tiles, groups, group_stages, stages;
  int split;                // the groups go to different blocks
  int wide;                 // rows of both operands lie on 32 bytes
};

// the block's i-th segment; false behind its last
__device__ __forceinline__ bool fs_segment(const FsProblem& p, int i, int& tile, int& group) {
  if (p.split) {
    const long long q = blockIdx.x + (long long)i * gridDim.x;
    if (q >= (long long)p.tiles * p.groups) return false;
    tile = (int)(q / p.groups);
    group = (int)(q % p.groups);
  } else {
    const long long t = blockIdx.x + (long long)(i / p.groups) * gridDim.x;
    if (t >= p.tiles) return false;
    tile = (int)t;
    group = i % p.groups;
  }
  return true;
}

// eight numbers into three planes of eight bfloat16, each piece to the nearest (the second and third are of either sign)
__device__ __forceinline__ void fs_cut(const float4& x, const float4& y, uint4& p0, uint4& p1, uint4& p2) {
  const float v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
  unsigned b0[4], b1[4], b2[4];
  auto pack = [](float lo, float hi) {
    __nv_bfloat162 pair = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<unsigned*>(&pair);
  };
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    b0[i] = pack(v[2 * i], v[2 * i + 1]);
    const float lo = v[2 * i] - __uint_as_float(b0[i] << 16), hi = v[2 * i + 1] - __uint_as_float(b0[i] & 0xffff0000u);  // exact
    b1[i] = pack(lo, hi);
    b2[i] = pack(lo - __uint_as_float(b1[i] << 16), hi - __uint_as_float(b1[i] & 0xffff0000u));                          // exact
  }
  p0 = make_uint4(b0[0], b0[1], b0[2], b0[3]);
  p1 = make_uint4(b1[0], b1[1], b1[2], b1[3]);
  p2 = make_uint4(b2[0], b2[1], b2[2], b2[3]);
}

template <int NT>
__global__ void __launch_bounds__(FS_THREADS, 1) gemm_f32_tcgen05_kernel(const FsProblem p) {
  using S = FsShape<NT>;
  constexpr int kW = FS_W_ROWS / FS_UNIT, kUnits = kW + (NT + FS_UNIT - 1) / FS_UNIT;      // the weight's, then the batch's
  extern __shared__ unsigned char fs_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(fs_raw) + 1023) & ~(uintptr_t)1023);
  unsigned long long* full = reinterpret_cast<unsigned long long*>(tiles + S::kStages * S::kStage);
  unsigned long long* empty = full + S::kStages;
  unsigned long long* sums_full = empty + S::kStages;    // [2]
  unsigned long long* sums_empty = sums_full + 2;
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(sums_empty + 2);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::kStages; ++s) { fs_bar_init(&full[s], FS_CONVERT / 32); fs_bar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { fs_bar_init(&sums_full[b], 1); fs_bar_init(&sums_empty[b], FS_DRAIN / 32); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == (FS_DRAIN + FS_CONVERT) / 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(fs_smem(tmem_slot)), "r"((unsigned)(2 * S::kPitch)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  pdl_wait();
  pdl_launch();

  if (warp < FS_DRAIN / 32) {
    // ---- drain: warp w has lanes 32 (w % 4) .. + 31 (weight rows) and one half of the batch's columns ----
    constexpr int kCols = NT / 2, kPiece = 8;
    const int quarter = warp & 3, half = (warp >> 2) * kCols;
    const unsigned mine = tmem + ((unsigned)(quarter * 32) << 16) + half;
    unsigned turn = 0;
    bool sound = true;
    for (int i = 0, tile, group; sound && fs_segment(p, i, tile, group); ++i) {
      float acc[kCols];
#pragma unroll
      for (int j = 0; j < kCols; ++j) acc[j] = 0.f;
      const int kb0 = group * p.group_stages, kb1 = min(p.stages, kb0 + p.group_stages);
      for (int kb = kb0; kb < kb1; kb += FS_CHUNK, ++turn) {
        const int b = turn & 1;
        // the lanes come here one by one, from polls and from stores that some of them skip: the loads want all of them at once
        if (!__all_sync(0xffffffffu, fs_wait(&sums_full[b], (turn >> 1) & 1))) { sound = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int c = 0; c < kCols; c += kPiece) {
          unsigned large[kPiece], middle[kPiece], small[kPiece];
          fs_tmem_load(mine + b * S::kPitch + c, large);
          fs_tmem_load(mine + b * S::kPitch + NT + c, middle);
          fs_tmem_load(mine + b * S::kPitch + 2 * NT + c, small);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < kPiece; ++j)
            acc[c + j] += __uint_as_float(large[j]) + (__uint_as_float(middle[j]) + __uint_as_float(small[j]));
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) fs_arrive(&sums_empty[b]);
      }
      if (!sound) break;
      const int n = tile / p.across * FS_W_ROWS + quarter * 32 + lane, m0 = tile % p.across * NT + half;
      const bool first = p.split || group == 0, last = !p.split && group == p.groups - 1;
      if (n >= p.N) continue;
      const float shift = last && p.bias ? p.bias[n] : 0.f;          // nothing changes by 0 but the sign of a zero
      float* out = p.out + (p.split ? (size_t)group * p.M * p.N : 0) + (size_t)m0 * p.N + n;
      bool odd = false;
#pragma unroll
      for (int c = 0; c < kCols; c += 8) {               // loads of eight rows at once: each is a trip to L2
        float before[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) before[j] = !first && m0 + c + j < p.M ? out[(size_t)(c + j) * p.N] : 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (m0 + c + j >= p.M) continue;
          const float v = acc[c + j];
          if (v - v == 0.f) out[(size_t)(c + j) * p.N] = first ? v + shift : (before[j] + v) + shift;
          else odd = true;
        }
      }
      if (odd) {                       // an operand without pieces, a product of pieces beyond the largest number, or truly no finite one
        unsigned long long which = 0;
#pragma unroll
        for (int j = 0; j < kCols; ++j) which |= (unsigned long long)(m0 + j < p.M && !(acc[j] - acc[j] == 0.f)) << j;
#pragma unroll 1
        for (int j = 0; j < kCols; ++j) {
          if (!(which >> j & 1)) continue;
          const float *x = p.a + (size_t)(m0 + j) * p.K, *y = p.w + (size_t)n * p.K;
          float v = 0.f;
          for (int k = kb0 * FS_K; k < min(p.K, kb1 * FS_K); ++k) v = fmaf(x[k], y[k], v);
          float* to = out + (size_t)j * p.N;
          *to = first ? v + shift : (*to + v) + shift;
        }
      }
    }
  } else if (warp < (FS_DRAIN + FS_CONVERT) / 32) {
    // ---- converters: eight neighbouring threads a row of 64, FS_UNIT rows at a time ----
    const int id = threadIdx.x - FS_DRAIN, r8 = id >> 3, k8 = (id & 7) * 8;
    const unsigned place = r8 * 128 + (((id & 7) ^ (r8 & 7)) << 4);
    int ahead = 0, tile, group;                          // the segment and stage that is loaded
    bool more = fs_segment(p, 0, tile, group);
    int kb = group * p.group_stages, end = min(p.stages, kb + p.group_stages);
    int n_at = tile / p.across * FS_W_ROWS + r8, m_at = tile % p.across * NT + r8;
    float4 v[kUnits][2];
    // rows behind the last one are the last one again: nobody stores what becomes of them
    auto from = [&](int u) {
      return u < kW ? p.w + (size_t)min(n_at + u * FS_UNIT, p.N - 1) * p.K
                    : p.a + (size_t)min(m_at + (u - kW) * FS_UNIT, p.M - 1) * p.K;
    };
    // 32 bytes in one load: a unit's two halves would be two of a warp's few outstanding-load counters
    auto load = [&](int u) {
      asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];" : "=f"(v[u][0].x), "=f"(v[u][0].y), "=f"(v[u][0].z),
                   "=f"(v[u][0].w), "=f"(v[u][1].x), "=f"(v[u][1].y), "=f"(v[u][1].z), "=f"(v[u][1].w)
                   : "l"(from(u) + kb * FS_K + k8));
    };
    auto load_end = [&](int u) {
      const int k = kb * FS_K + k8;
      const float4* src = reinterpret_cast<const float4*>(from(u) + k);
      v[u][0] = v[u][1] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (k < p.K) v[u][0] = src[0];
      if (k + 4 < p.K) v[u][1] = src[1];
    };
    auto cut = [&](int u, unsigned char* stage) {
      if (u >= kW && (u - kW + 1) * FS_UNIT > NT && r8 >= NT % FS_UNIT) return;         // a last unit of fewer rows
      uint4 p0, p1, p2;
      fs_cut(v[u][0], v[u][1], p0, p1, p2);
      unsigned char* to = stage + (u < kW ? u * FS_UNIT * 128 : 3 * S::kPlaneW + (u - kW) * FS_UNIT * 128);
      *reinterpret_cast<uint4*>(to) = p0;
      *reinterpret_cast<uint4*>(to + (u < kW ? S::kPlaneW : S::kPlaneA)) = p1;
      *reinterpret_cast<uint4*>(to + 2 * (u < kW ? S::kPlaneW : S::kPlaneA)) = p2;
    };
#pragma unroll
    for (int u = 0; u < kUnits; ++u) load_end(u);
    for (unsigned turn = 0; more; ++turn) {
      const int s = turn % S::kStages;
      if (++kb >= end) {
        more = fs_segment(p, ++ahead, tile, group);
        if (more) {
          kb = group * p.group_stages;
          end = min(p.stages, kb + p.group_stages);
          n_at = tile / p.across * FS_W_ROWS + r8;
          m_at = tile % p.across * NT + r8;
        }
      }
      if (!fs_wait(&empty[s], (turn / S::kStages & 1) ^ 1)) break;
      unsigned char* stage = tiles + s * S::kStage + place;
      if (more && p.wide && (kb + 1) * FS_K <= p.K) {
#pragma unroll
        for (int u = 0; u < kUnits; ++u) { cut(u, stage); load(u); }
      } else if (more) {
#pragma unroll
        for (int u = 0; u < kUnits; ++u) { cut(u, stage); load_end(u); }
      } else {
#pragma unroll
        for (int u = 0; u < kUnits; ++u) cut(u, stage);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // the tensor core reads through the other proxy
      __syncwarp();
      if (lane == 0) fs_arrive(&full[s]);
    }
  } else {
    // ---- products: the whole warp walks the stages, so that descriptors stay in uniform registers, one lane issues.  A
    // batch tile's three planes lie behind one another, so w0 x0, w0 x1, w0 x2 are one instruction of N = 3 NT; w1 x0 and
    // w1 x1 add to the last two blocks of columns, w2 x0 to the last ----
    auto shape = [](int n) { return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(n >> 3) << 17) | ((unsigned)(FS_W_ROWS >> 4) << 24); };
    unsigned turn = 0, chunk = 0;
    bool sound = true;
    for (int i = 0, tile, group; sound && fs_segment(p, i, tile, group); ++i) {
      const int kb0 = group * p.group_stages, kb1 = min(p.stages, kb0 + p.group_stages);
      for (int kb = kb0; kb < kb1; ++kb, ++turn) {
        const int s = turn % S::kStages, b = chunk & 1;
        const bool fresh = (kb - kb0) % FS_CHUNK == 0, done = (kb - kb0) % FS_CHUNK == FS_CHUNK - 1 || kb == kb1 - 1;
        bool there = fs_wait(&full[s], turn / S::kStages & 1);
        if (fresh) there = there && fs_wait(&sums_empty[b], (chunk >> 1 & 1) ^ 1);
        if (!__all_sync(0xffffffffu, there)) { sound = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const unsigned base = fs_smem(tiles) + s * S::kStage, sums = tmem + b * S::kPitch;
        const unsigned long long w = fs_desc(base), x = fs_desc(base + 3 * S::kPlaneW);
        constexpr int kNext = S::kPlaneW / 16;           // from plane to plane, as descriptors count
        if (fs_elect()) {
#pragma unroll
          for (int k = 0; k < FS_K / 16; ++k) {
            fs_mma(sums, w + 2 * k, x + 2 * k, shape(3 * NT), !fresh || k != 0);
            fs_mma(sums + NT, w + kNext + 2 * k, x + 2 * k, shape(2 * NT), 1);
            fs_mma(sums + 2 * NT, w + 2 * kNext + 2 * k, x + 2 * k, shape(NT), 1);
          }
          fs_commit(&empty[s]);
          if (done) fs_commit(&sums_full[b]);
        }
        __syncwarp();
        chunk += done;
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == (FS_DRAIN + FS_CONVERT) / 32) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((unsigned)(2 * S::kPitch)) : "memory");
  }
}

// the groups' partial sums in order, then the bias: what a block that takes all groups of a tile does
template <int V>
__global__ void gemm_f32_sum_kernel(const float* __restrict__ part, const float* __restrict__ bias, float* __restrict__ out,
                                    long long count, int N, int groups) {
  pdl_wait();
  pdl_launch();
  const long long at = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * V;
  if (at >= count) return;
  float v[V];
  if (V == 4) *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(part + at);
  else v[0] = part[at];
#pragma unroll 4
  for (int g = 1; g < groups; ++g) {
    const float* src = part + g * count + at;
    if (V == 4) {
      const float4 x = *reinterpret_cast<const float4*>(src);
      v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
    } else {
      v[0] += *src;
    }
  }
  if (bias) {
#pragma unroll
    for (int j = 0; j < V; ++j) v[j] += bias[at % N + j];
  }
  if (V == 4) *reinterpret_cast<float4*>(out + at) = *reinterpret_cast<float4*>(v);
  else out[at] = v[0];
}

template <int NT>
static int fs_launch(const FsProblem& p, int sms, cudaStream_t stream) {
  static const cudaError_t ready = cudaFuncSetAttribute(gemm_f32_tcgen05_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                        FsShape<NT>::kSmem);
  if (ready != cudaSuccess) return (int)ready;
  const long long units = (long long)p.tiles * (p.split ? p.groups : 1);
  return launch_dependent(gemm_f32_tcgen05_kernel<NT>, dim3((unsigned)(units < sms ? units : sms)), dim3(FS_THREADS),
                          FsShape<NT>::kSmem, stream, p);
}

// stages of k in groups of one length (the last may be shorter, none is empty)
static int fs_groups(int stages, int* group_stages) {
  const int groups = (stages + FS_GROUP - 1) / FS_GROUP;
  *group_stages = (stages + groups - 1) / groups;
  return (stages + *group_stages - 1) / *group_stages;
}

static const int fs_rows[] = {16, 32, 48, 64, 80};

// The tile (an index into fs_rows) and whether the groups go to different blocks, for a product of these sizes.
TOKB200_API int tokb200_gemm_f32_tcgen05_plan(int M, int N, int K, int* tile, int* split, int* groups) {
  if (M <= 0 || N <= 0 || K <= 0) return TOKB200_BAD_SIZE;
  const int sms = 148, stages = (K + FS_K - 1) / FS_K;
  int group;
  *groups = fs_groups(stages, &group);
  // measured cycles of a stage, and of a segment's start and end; the second kernel's start and traffic
  static const double stage_cycles[] = {2000., 2050., 2150., 2300., 2430.};
  double least = -1.;
  for (int i = 0; i < 5; ++i) {
    const long long tiles = (long long)((N + FS_W_ROWS - 1) / FS_W_ROWS) * ((M + fs_rows[i] - 1) / fs_rows[i]);
    for (int s = 0; s < (*groups > 1 ? 2 : 1); ++s) {
      const double bytes = 8. * *groups * M * N;
      if (s && (tiles > 2 * sms || bytes > (64 << 20))) continue;
      const long long units = s ? tiles * *groups : tiles;
      const double time = (double)((units + sms - 1) / sms) * ((s ? group : stages) * stage_cycles[i] + 2500.) +
                          (s ? 4500. + bytes / 2600. : 0.);
      if (least < 0. || time < least) { least = time; *tile = i; *split = s; }
    }
  }
  return TOKB200_OK;
}

// `partials`: [groups, M, N] where `split`.  K a multiple of 4, a and w on 16 bytes.
TOKB200_API int tokb200_gemm_f32_tcgen05(const float* a, const float* w, const float* bias, float* c, float* partials, int M,
                                         int N, int K, int tile, int split, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return TOKB200_OK;
  if (K <= 0 || K % 4 || tile < 0 || tile >= 5) return TOKB200_BAD_SIZE;
  if (((((uintptr_t)a) | ((uintptr_t)w)) & 15) != 0) return TOKB200_BAD_ALIGNMENT;
  FsProblem p = {};
  p.a = a; p.w = w; p.M = M; p.N = N; p.K = K;
  p.stages = (K + FS_K - 1) / FS_K;
  p.groups = fs_groups(p.stages, &p.group_stages);
  p.split = split && p.groups > 1;
  p.wide = K % 8 == 0 && ((((uintptr_t)a) | ((uintptr_t)w)) & 31) == 0;
  if (p.split && partials == nullptr) return TOKB200_BAD_SIZE;
  p.bias = p.split ? nullptr : bias;
  p.out = p.split ? partials : c;
  p.across = (M + fs_rows[tile] - 1) / fs_rows[tile];
  const long long tiles = (long long)((N + FS_W_ROWS - 1) / FS_W_ROWS) * p.across;
  if (tiles > 0x7fffffff / 2) return TOKB200_BAD_SIZE;
  p.tiles = (int)tiles;
  const int sms = 148;
  int status;
  switch (tile) {
    case 0: status = fs_launch<16>(p, sms, stream); break;
    case 1: status = fs_launch<32>(p, sms, stream); break;
    case 2: status = fs_launch<48>(p, sms, stream); break;
    case 3: status = fs_launch<64>(p, sms, stream); break;
    default: status = fs_launch<80>(p, sms, stream); break;
  }
  if (status != TOKB200_OK || !p.split) return status;
  const long long count = (long long)M * N;
  const bool wide = N % 4 == 0 && ((((uintptr_t)partials) | ((uintptr_t)c)) & 15) == 0;
  const long long blocks = (count / (wide ? 4 : 1) + 255) / 256;
  if (blocks > 0x7fffffff) return TOKB200_BAD_SIZE;
  return wide ? launch_dependent(gemm_f32_sum_kernel<4>, dim3((unsigned)blocks), dim3(256), 0, stream, partials, bias, c, count, N, p.groups)
              : launch_dependent(gemm_f32_sum_kernel<1>, dim3((unsigned)blocks), dim3(256), 0, stream, partials, bias, c, count, N, p.groups);
}

TOKB200_API int tokb200_gemm_f32_tcgen05_error(void) {
  int value = 0, zero = 0;
  cudaMemcpyFromSymbol(&value, fs_error_flag, sizeof(int));
  cudaMemcpyToSymbol(fs_error_flag, &zero, sizeof(int));
  return value;
}
