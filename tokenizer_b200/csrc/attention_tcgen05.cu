// Attention for portions of prompts on the fifth-generation tensor cores
// (bfloat16, tcgen05 with the scores, the probabilities and the weighted values in tensor memory).
//
// A block takes a tile of up to 128 consecutive rows of one request and runs TWO lanes of work on it, so
// that the tensor core has one lane's products to do while the other lane's softmax runs:
//   * side by side: lane 0 and lane 1 are two query heads of one key/value head.  Both walk the same key
//     blocks, and a block's keys and values are brought into shared memory once for both;
//   * split: both lanes are the same query head, lane 0 walks the key blocks 0, 2, 4 ..., lane 1 the blocks
//     1, 3, 5 ...; their sums meet at the end.  For a group's odd head, and for all heads of a step with few
//     blocks of work, which is then cut twice as fine.
// The block owns its SM (all 512 columns of tensor memory: per lane a score buffer and an accumulator).  Its
// roles, all of them walking the same sequence of key and value tiles (128 keys each) through a ring of
// shared-memory buffers:
//   * two loader warps, tile by tile in turn, bring the tiles from the cache pages with TMA, a copy per run of
//     keys inside one page (any page size that is a multiple of 8), in the 128-byte swizzled layout the tensor
//     core reads; runs without a visible key come as zeros (coordinates behind the pool).  A run of VALUES that
//     the tile sees in part is copied by the warp itself with zeros for the others, whatever the cache holds
//     there (a zero probability times a stored infinity would be a NaN; keys need no such care, a score is
//     replaced, not multiplied, where it is masked).  Other page sizes: both warps copy every tile themselves,
//     together;
//   * one warp issues, lane by lane in turn, P V of a block and S = Q K^T of the lane's next block
//     (tcgen05.mma, M = 128 rows, N = 128 keys; P is the A operand straight from tensor memory, V the B
//     operand in MN-major form, which is how the cache stores it: a key per row);
//   * 256 threads a lane, two a row, run the softmax: 64 of the row's scores each in one tcgen05.ld, the
//     maximum shared through shared memory, exponentials and sum in registers, the probabilities back to tensor
//     memory as bfloat16.  The accumulator stays in tensor memory over the whole walk; the reference maximum
//     follows the true one lazily: only when the maximum has grown by more than 2^8 since it was set are the
//     sum and the accumulator rescaled, which happens a few times per row; probabilities stay below 2^8.
// Measured (28 heads over 4 of 128 lanes, one prompt, us): 8,192 tokens 1,547 -> 456 (311 -> 1,054 TFLOP/s), 2,048 126 ->
// 47; 14 heads over 2 of 64: 346 -> 198 and 36.8 -> 24.7.  The form before it took one tile and one head a block, and its
// loader waited for a block's copies before it asked for the next.  What bounds it now: a step of the two lanes takes
// 4,200 cycles at 128 lanes, of which the tensor core 2,300 and each lane's softmax 1,900 (the exponentials alone 1,024 of
// MUFU), the rest the hand-offs between them; scores asked for while the softmax still runs (probabilities through shared
// memory at 128 lanes) measured slower, 590 us: both lanes' softmaxes then run at once and slow one another.
// Everything but q, k, v, p and the output is 32-bit.  Every wait is bounded; when one runs out an error flag
// is set and all roles fall through to the common exit, where tensor memory is given back.
//
// `keep_first` (> 0): the sequence's first keys that stay visible although the window has passed them; the
// blocks that hold them are walked in front of the others.
//
// HEAD_DIM is a compile-time size (64 or 128), -DHEAD_DIM=...
#include <cuda.h>

#include "common.cuh"

#ifndef HEAD_DIM
#define HEAD_DIM 64
#endif
static_assert(HEAD_DIM == 64 || HEAD_DIM == 128, "head size");

#define FA_ROWS 128
#define FA_KEYS 128
#define FA_SOFTMAX_WARPS 16             // eight a lane
#define FA_LOADER_WARPS 2               // 19 warps in all leave 96 registers a thread
#define FA_THREADS ((FA_SOFTMAX_WARPS + FA_LOADER_WARPS + 1) * 32)
#define FA_BUFFERS (HEAD_DIM == 64 ? 8 : 5)
#define FA_WAIT_LIMIT (1u << 17)      // polls of up to 20 us each: seconds in all
#define FA_RESCALE_AT 8.0f            // log2 units the maximum may lead its reference by
constexpr int kDBlocks = HEAD_DIM / 64;           // 64-lane pieces of the head (128 bytes a row)
constexpr int kSubTile = 128 * 128;               // bytes of a [128 x 64] bfloat16 swizzled tile
constexpr int kTmemCols = 512;
// Tensor memory: scores of the lanes at 0 and 128, accumulators at 256 and 384.  The probabilities (64 columns a
// lane) lie behind the accumulators of 64 columns; accumulators of 128 leave no room, and they take the first half
// of the lane's scores, which are in registers by then (the lane's next scores then wait for its P V).
constexpr bool kPOnScores = HEAD_DIM == 128;
constexpr int kPFirst = kPOnScores ? 0 : 256 + HEAD_DIM;
constexpr int kHalfKeys = FA_KEYS / 2;            // of a block, that a softmax thread owns

__device__ int fa_error_flag = 0;


// shared memory: q of the two lanes | ring of key and value tiles (each a whole number of 16 KB sub-tiles), then
// what a row's threads tell one another, then the barriers
constexpr int kTileBytes = kDBlocks * kSubTile;
constexpr int kStatBytes = 2 * 2 * FA_ROWS * 4;
constexpr int kBarBytes = (2 * FA_BUFFERS + 7) * 8 + 8;     // the barriers, where tensor memory lies, whether a wait ran out
constexpr int kFaSmem = 2 * kTileBytes + FA_BUFFERS * kTileBytes + kStatBytes + kBarBytes;
static_assert(kFaSmem > 116 * 1024 && kFaSmem <= 227 * 1024, "one block an SM: it takes all of tensor memory");

extern __shared__ __align__(1024) unsigned char fa_raw[];      // swizzle atoms: 1024-byte aligned

__device__ __forceinline__ unsigned fa_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
// the word that a wait that ran out sets
__device__ __forceinline__ unsigned fa_gave_up_at() { return fa_smem(fa_raw) + (unsigned)(kFaSmem - 4); }
__device__ __forceinline__ void fa_mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(fa_smem(bar)), "r"(count));
}
__device__ __forceinline__ void fa_mbar_arrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(fa_smem(bar)) : "memory");
}
__device__ __forceinline__ bool fa_mbar_wait(unsigned long long* bar, unsigned parity) {
  const unsigned addr = fa_smem(bar);
  // the thread sleeps in hardware until the phase completes or the hint runs out, so
  // waiting warps do not take issue slots from working ones
  const unsigned suspend_ns = 20000u;
  // Unrolled, and with the report of a wait that ran out at each of its two dozen places, this loop made half of the
  // kernel's 115 KB of code.  Behind a layer's other kernels that code starts cold, and its misses stand in a row: one
  // portion of 128 tokens behind 256 MB of other traffic took 16.1 us (14 heads of 64) and 17.3 (12 of 128), and 9.3 and
  // 11.8 with this, loops of the loaders kept as loops and the block's start in the order it has now; 2,048 tokens 36.4 ->
  // 28.1 and 36.7 -> 32.3.
#pragma unroll 1
  for (unsigned spin = 0; spin < FA_WAIT_LIMIT; ++spin) {
    unsigned done;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done) : "r"(addr), "r"(parity), "r"(suspend_ns) : "memory");
    if (done) return true;
  }
  asm volatile("st.shared.u32 [%0], 1;" ::"r"(fa_gave_up_at()) : "memory");      // reported at the block's end
  return false;
}
// byte offset of element (row, 16-byte piece c) in a [rows x 64] bfloat16 tile with 128-byte swizzle
__device__ __forceinline__ int swz(int row, int c) {
  return (row >> 3) * 1024 + (row & 7) * 128 + ((c ^ (row & 7)) << 4);
}
__device__ __forceinline__ bool fa_elect() {
  unsigned one;
  asm volatile("{\n.reg .pred p;\n.reg .b32 r;\nelect.sync r|p, 0xffffffff;\nselp.b32 %0, 1, 0, p;\n}\n" : "=r"(one));
  return one != 0;
}
// Matrix descriptors of tiles of 128-byte swizzled rows, 8-row groups 1024 bytes apart (stride offset); the low word is
// the tile's address in 16 bytes and the leading offset, which steps inside a tile only add to.
//   K-major (q, k): no leading offset;  MN-major (v: a key per 128-byte row of 64 lanes): 64-lane pieces of the head
//   one sub-tile apart
constexpr unsigned kDescHigh = 64u | (1u << 14) | (2u << 29);
constexpr unsigned kDescK = 1u << 16, kDescV = (unsigned)(kSubTile >> 4) << 16;
// the product of a K-major a and b
__device__ __forceinline__ void fa_mma(unsigned tmem_d, unsigned a_at, unsigned b_at, unsigned idesc, bool accumulate) {
  asm volatile(
      "{\n.reg .pred p;\n.reg .b64 a, b;\nsetp.ne.b32 p, %4, 0;\nmov.b64 a, {%1, %5};\nmov.b64 b, {%2, %5};\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n}\n"
      ::"r"(tmem_d), "r"(a_at | kDescK), "r"(b_at | kDescK), "r"(idesc), "r"((unsigned)accumulate), "r"(kDescHigh)
      : "memory");
}
// the first operand from tensor memory (16 bits, two to a column: a product's 16 lanes of k are 8 columns)
__device__ __forceinline__ void fa_mma_ts(unsigned tmem_d, unsigned tmem_a, unsigned b_at, unsigned idesc,
                                          bool accumulate) {
  asm volatile(
      "{\n.reg .pred p;\n.reg .b64 b;\nsetp.ne.b32 p, %4, 0;\nmov.b64 b, {%2, %5};\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %3, p;\n}\n"
      ::"r"(tmem_d), "r"(tmem_a), "r"(b_at | kDescV), "r"(idesc), "r"((unsigned)accumulate), "r"(kDescHigh)
      : "memory");
}
__device__ __forceinline__ void fa_commit(unsigned long long* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
               ::"r"(fa_smem(bar)) : "memory");
}
// columns of this thread's row, waited for in the same statement (nothing may use a register before the wait)
__device__ __forceinline__ void fa_tmem_load64(unsigned taddr, float (&v)[64]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x64.b32 {"
      "%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15"
      ",%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31"
      ",%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47"
      ",%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63"
      "}, [%64];\n"
      "tcgen05.wait::ld.sync.aligned;\n"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
        "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]),
        "=f"(v[16]), "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]),
        "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31]),
        "=f"(v[32]), "=f"(v[33]), "=f"(v[34]), "=f"(v[35]), "=f"(v[36]), "=f"(v[37]), "=f"(v[38]), "=f"(v[39]),
        "=f"(v[40]), "=f"(v[41]), "=f"(v[42]), "=f"(v[43]), "=f"(v[44]), "=f"(v[45]), "=f"(v[46]), "=f"(v[47]),
        "=f"(v[48]), "=f"(v[49]), "=f"(v[50]), "=f"(v[51]), "=f"(v[52]), "=f"(v[53]), "=f"(v[54]), "=f"(v[55]),
        "=f"(v[56]), "=f"(v[57]), "=f"(v[58]), "=f"(v[59]), "=f"(v[60]), "=f"(v[61]), "=f"(v[62]), "=f"(v[63])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void fa_tmem_load16(unsigned taddr, float (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {"
      "%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15"
      "}, [%16];\n"
      "tcgen05.wait::ld.sync.aligned;\n"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
        "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void fa_tmem_store16(unsigned taddr, const float (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {"
      "%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16"
      "};\n"
      :: "r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]),
        "f"(v[8]), "f"(v[9]), "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15])
      : "memory");
}
__device__ __forceinline__ void fa_tmem_store32(unsigned taddr, const unsigned (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {"
      "%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16"
      ",%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32"
      "};\n"
      :: "r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
        "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
        "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}
// two 32-bit values in one 64-bit register, for the packed arithmetic of sm_100
__device__ __forceinline__ unsigned long long fa_pack2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void fa_unpack2(unsigned long long v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ unsigned long long fa_fma2(unsigned long long a, unsigned long long b,
                                                      unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long fa_add2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float fa_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void fa_copy16(void* dst, const void* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(fa_smem(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void fa_expect(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fa_smem(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void fa_tma(void* dst, const CUtensorMap* map, unsigned long long* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(fa_smem(dst)), "l"(map), "r"(fa_smem(bar)), "r"(x), "r"(y) : "memory");
}

template <bool CAPPED>
__global__ void __launch_bounds__(FA_THREADS, 1)
attention_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                         const __grid_constant__ CUtensorMap map_v, const __nv_bfloat16* __restrict__ k_pool,
                         const __nv_bfloat16* __restrict__ v_pool, __nv_bfloat16* __restrict__ out,
                         const int* __restrict__ block_table, int table_stride,
                         const int* __restrict__ row_req, const int* __restrict__ pos,
                         const int* __restrict__ tiles, int n_tiles, int nh, int nkv, int page, int run,
                         int pool_rows, int split_all, int window, int chunk, int keep_first, float scale_log2,
                         const float* __restrict__ sink, float cap_in, float cap_out) {
  unsigned char* q_s = fa_raw;                                   // lane 0, lane 1
  unsigned char* ring = q_s + 2 * kTileBytes;
  float* stat_s = reinterpret_cast<float*>(ring + FA_BUFFERS * kTileBytes);   // [lane][half][row]
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(ring + FA_BUFFERS * kTileBytes + kStatBytes);
  unsigned long long* full = bars;                               // [buffers]: a tile is in place
  unsigned long long* empty = full + FA_BUFFERS;                 // [buffers]: commit of its last reader
  unsigned long long* s_full = empty + FA_BUFFERS;               // [2], commit of Q K^T
  unsigned long long* p_ready = s_full + 2;                      // [2], an arrival per softmax warp of the lane
  unsigned long long* pv_done = p_ready + 2;                     // [2], commit of P V
  unsigned long long* q_full = pv_done + 2;
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(q_full + 1);

  // heads run fastest over the grid so that the tiles with the most keys (first in
  // `tiles`) of all heads are placed first
  const int tile = blockIdx.y, group = nh / nkv;
  const int pairs = (group + 1) / 2;
  const int kvh = split_all ? blockIdx.x / group : blockIdx.x / pairs;
  const int h0 = split_all ? blockIdx.x : kvh * group + (blockIdx.x % pairs) * 2;
  const bool split = split_all || h0 + 1 == (kvh + 1) * group;     // a group's odd head is split
  // through a shuffle, so that the compiler can see it is the same for the whole warp: the roles are then no divergent
  // branches and may keep such values in uniform registers (28 heads of 128, 8,192
  // tokens: 548 -> 456 us, 2,048: 58 -> 47; 14 heads of 64, 2,048 tokens: 27.6 -> 24.7)
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  // What needs nothing of the step comes first: the trips to memory for the step's rows, one behind the other, then lie
  // beside the maps' way into the SM and the claim on tensor memory, not in front of them.
  constexpr int kMmaWarp = FA_SOFTMAX_WARPS + FA_LOADER_WARPS;
  const bool by_tma = run > 0;            // runs of keys inside one page, 8 to 128 of them

  if (warp == FA_SOFTMAX_WARPS && lane < 3)      // the maps themselves are memory: on their way before the first copy
    asm volatile("prefetch.tensormap [%0];" ::"l"(lane == 0 ? &map_q : lane == 1 ? &map_k : &map_v) : "memory");
  if (threadIdx.x == 0) {
    for (int i = 0; i < FA_BUFFERS; ++i) {
      fa_mbar_init(&full[i], by_tma ? 1 : FA_LOADER_WARPS);
      fa_mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      fa_mbar_init(&s_full[i], 1);
      fa_mbar_init(&p_ready[i], FA_SOFTMAX_WARPS / 2);
      fa_mbar_init(&pv_done[i], 1);
    }
    fa_mbar_init(q_full, 1);
    tmem_slot[1] = 0;                            // no wait has run out
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(fa_smem(tmem_slot)), "r"((unsigned)kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  const int row0 = tiles[2 * tile], n_rows = tiles[2 * tile + 1];
  const int r_id = row_req[row0], pos_row0 = pos[row0];
  // uniform over the block; a misaligned base (never seen) is reported instead of used
  const bool aligned = (fa_smem(fa_raw) & 1023u) == 0;
  if (!aligned && threadIdx.x == 0) {
    atomicExch(&fa_error_flag, 2);
    tokb200_report_error(TOKB200_LIB_ATTENTION_TCGEN05, 2);
  }
  const bool live = aligned && tile < n_tiles && r_id >= 0 && n_rows > 0;
  const int pos0 = live ? pos_row0 : 0;
  const int pos_last = pos0 + n_rows - 1;
  const int lo_first = first_visible_key(pos0, window, chunk);
  const int lo_last = first_visible_key(pos_last, window, chunk);
  const int kb_first = lo_first / FA_KEYS * FA_KEYS;
  // blocks of kept keys that lie before the first block of the window
  const int n_kept = min((keep_first + FA_KEYS - 1) / FA_KEYS, kb_first / FA_KEYS);
  const int n_blocks = live ? n_kept + (pos_last - kb_first) / FA_KEYS + 1 : 0;
  auto first_of = [&](int b) { return b < n_kept ? b * FA_KEYS : kb_first + (b - n_kept) * FA_KEYS; };
  // what a lane walks: its step b is block `block_of(lane, b)`
  auto steps_of = [&](int l) { return split ? (n_blocks + 1 - l) / 2 : n_blocks; };
  auto block_of = [&](int l, int b) { return split ? 2 * b + l : b; };
  // the ring's sequence of tiles: K0 V0 K1 V1 ... side by side, K0 K1 V0 K2 V1 K3 ... split (in the order of their
  // use; a split walk's place for the keys behind the last block stays empty, nothing comes behind it in its buffer)
  auto k_place = [&](int b) { return split ? (b < 2 ? b : 2 * b - 1) : 2 * b; };
  auto v_place = [&](int b) { return split ? 2 * b + 2 : 2 * b + 1; };
  // and back: whether a place holds values, and of which block (n_blocks or more: it stays empty)
  auto of_values = [&](int n) { return split ? n >= 2 && n % 2 == 0 : n % 2 == 1; };
  auto block_at = [&](int n) { return !split ? n / 2 : n < 2 ? n : n % 2 == 0 ? n / 2 - 1 : (n + 1) / 2; };
  const int* table = block_table + (size_t)(live ? r_id : 0) * table_stride;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  pdl_wait();

  if (live && warp >= FA_SOFTMAX_WARPS && warp < kMmaWarp) {
    // ---------------- loaders ----------------
    const int loader = warp - FA_SOFTMAX_WARPS;
    if (loader == 0 && lane == 0) {      // rows behind the tile belong to others or lie behind q (zeros): nobody stores theirs
      const int n_q = split ? 1 : 2;
      fa_expect(q_full, (unsigned)(n_q * kTileBytes));
      for (int i = 0; i < n_q; ++i)
#pragma unroll
        for (int c = 0; c < kDBlocks; ++c)
          fa_tma(q_s + i * kTileBytes + c * kSubTile, &map_q, q_full, (h0 + i) * HEAD_DIM + c * 64, row0);
    }
    __syncwarp();
    const int n_places = v_place(n_blocks - 1) + 1;
    auto visible = [&](int key) { return (key >= lo_first || key < keep_first) && key <= pos_last; };
    if (by_tma) {
      // The loader warps take the places in turn; where a place's runs lie is looked up while the place before it is
      // waited for and copied (one warp that did one after the other took 1,900 cycles a tile of 32 KB, and the
      // products waited for keys for two fifths of a split walk).
      const int runs = FA_KEYS / run;                    // at most 16: a lane each
      // a place's block and whether it is values; this lane's run of keys: its pool row (behind the pool: zeros), and
      // whether the tile sees some or all of it
      struct Place { int b, y; bool values, some, all; };
      auto locate = [&](int n) {
        Place at;
        at.values = of_values(n);
        at.b = block_at(n);
        at.y = pool_rows;
        at.some = at.all = false;
        if (n < n_places && at.b < n_blocks && lane < runs) {
          const int key0 = first_of(at.b) + lane * run, last = key0 + run - 1;
          at.some = key0 <= pos_last && (last >= lo_first || key0 < keep_first);
          at.all = last <= pos_last && (key0 >= lo_first || last < keep_first);
          if (at.some) at.y = table[key0 / page] * page + key0 % page;
        }
        return at;
      };
      int n = loader;
      Place next = locate(n);
#pragma unroll 1
      for (; n < n_places; n += FA_LOADER_WARPS) {
        const Place at = next;
        next = locate(n + FA_LOADER_WARPS);
        if (at.b >= n_blocks) continue;
        const int buf = n % FA_BUFFERS, use = n / FA_BUFFERS;
        if (use > 0 && !__all_sync(0xffffffffu, fa_mbar_wait(&empty[buf], (use - 1) & 1))) break;
        unsigned char* dst = ring + buf * kTileBytes;
        const unsigned mixed = __ballot_sync(0xffffffffu, at.values && at.some && !at.all);
        if (mixed) {                                     // values seen in part: zeros for the others
#pragma unroll 1
          for (unsigned left = mixed; left; left &= left - 1) {
            const int i = __ffs(left) - 1;
            const int row = __shfl_sync(0xffffffffu, at.y, i), first = first_of(at.b) + i * run;
#pragma unroll 1
            for (int e = lane; e < run * (HEAD_DIM / 8); e += 32) {
              const int t = e / (HEAD_DIM / 8), c = e % (HEAD_DIM / 8);
              uint4 piece = make_uint4(0u, 0u, 0u, 0u);
              if (visible(first + t))
                piece = *reinterpret_cast<const uint4*>(v_pool + ((size_t)(row + t) * nkv + kvh) * HEAD_DIM + c * 8);
              *reinterpret_cast<uint4*>(dst + (c / 8) * kSubTile + swz(i * run + t, c % 8)) = piece;
            }
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
        }
        if (lane == 0) fa_expect(&full[buf], (unsigned)(kTileBytes - __popc(mixed) * run * HEAD_DIM * 2));
        __syncwarp();
        if (lane < runs && !(mixed >> lane & 1u)) {
#pragma unroll
          for (int c = 0; c < kDBlocks; ++c)
            fa_tma(dst + c * kSubTile + lane * run * 128, at.values ? &map_v : &map_k, &full[buf],
                   kvh * HEAD_DIM + c * 64, at.y);
        }
        __syncwarp();
      }
      // every copy has landed before the block gives its shared memory back, whatever became of its readers (the places
      // that nothing came behind in their buffers)
      const int end = min(n, n_places);
#pragma unroll 1
      for (int i = loader; i < end; i += FA_LOADER_WARPS)
        if (i >= end - FA_BUFFERS && locate(i).b < n_blocks)
          fa_mbar_wait(&full[i % FA_BUFFERS], (i / FA_BUFFERS) & 1);
    } else {
      // Pages of other sizes: each warp copies half of every tile's rows (cp.async, 16 bytes a lane, a row's lanes side by
      // side), kLag places on their way at a time; before a place is asked for, the one kLag before it is waited for and
      // announced.  Plain loads, whose values a thread had to hold, kept 8 of them in flight a thread (2,048 tokens, cold
      // caches, us, plain loads / now / pages of 16 by TMA: pages of 20 keys, 28 heads of 128 211 / 70 / 59, 14 of 64 114 / 38
      // / 28; pages of 5 keys 223 / 70 and 127 / 38).  A place that is not announced yet is never one that the release of a
      // buffer still waits for: kLag < the buffers (side by side a place is read out only when the one behind it has been
      // announced too).
      constexpr int kLag = HEAD_DIM == 64 ? 4 : 3, kRowPieces = HEAD_DIM / 8, kRowsAtOnce = 32 / kRowPieces;
      static_assert(kLag < FA_BUFFERS, "a buffer's release may wait for the place behind it");
      // a place's block, and of this lane's two keys of the warp's half their pages (-1: not seen) and places in them
      struct Copy { int b, page_at[2], in_page[2]; };
      auto look_up = [&](int n) {
        Copy at;
        at.b = n < n_places ? block_at(n) : n_blocks;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int key = first_of(at.b) + loader * 64 + i * 32 + lane;
          at.in_page[i] = key % page;
          at.page_at[i] = at.b < n_blocks && visible(key) ? table[key / page] : -1;
        }
        return at;
      };
      auto announce = [&](int n) {                       // this thread's copies of place n have landed
        if (block_at(n) < n_blocks) {
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) fa_mbar_arrive(&full[n % FA_BUFFERS]);
        }
      };
      bool ok = true;
      Copy next = look_up(0);
#pragma unroll 1
      for (int n = 0; n < n_places; ++n) {
        const Copy at = next;
        next = look_up(n + 1);
        if (n >= kLag) {
          asm volatile("cp.async.wait_group %0;" ::"n"(kLag - 1) : "memory");
          announce(n - kLag);
        }
        if (at.b < n_blocks) {
          const int buf = n % FA_BUFFERS, use = n / FA_BUFFERS;
          if (use > 0 && !__all_sync(0xffffffffu, fa_mbar_wait(&empty[buf], (use - 1) & 1))) { ok = false; break; }
          unsigned char* dst = ring + buf * kTileBytes;
          const int c = lane % kRowPieces;
          const unsigned char* pool =
              reinterpret_cast<const unsigned char*>((of_values(n) ? v_pool : k_pool) + kvh * HEAD_DIM + c * 8);
          const unsigned row_bytes = (unsigned)nkv * HEAD_DIM * 2;
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const int mine = at.page_at[half] < 0 ? -1 : at.page_at[half] * page + at.in_page[half];
#pragma unroll 8
            for (int i = 0; i < 32; i += kRowsAtOnce) {
              const int t = half * 32 + i + lane / kRowPieces;              // of the warp's half of the tile
              const int row = __shfl_sync(0xffffffffu, mine, t % 32);
              fa_copy16(dst + (c / 8) * kSubTile + swz(loader * 64 + t, c % 8),
                        pool + (size_t)(unsigned)(row < 0 ? 0 : row) * row_bytes, row >= 0);
            }
          }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      if (ok)
#pragma unroll 1
        for (int n = max(0, n_places - kLag); n < n_places; ++n) announce(n);
      if (loader == 0) fa_mbar_wait(q_full, 0);          // q's copies are TMA's all the same
    }
  } else if (live && warp == kMmaWarp) {
    // ---------------- products ----------------
    // The whole warp goes through the waits, so that everything the instructions take is the same for all of it and
    // lies in uniform registers, and one thread issues: with one thread in the loop alone an instruction took 120
    // cycles to issue, twice what the tensor core takes for it.
    const bool leader = fa_elect();
    constexpr unsigned idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(FA_KEYS >> 3) << 17) |
                                 ((unsigned)(FA_ROWS >> 4) << 24);
    constexpr unsigned idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) /* v is MN-major */ |
                                 ((unsigned)(HEAD_DIM >> 3) << 17) | ((unsigned)(FA_ROWS >> 4) << 24);
    const unsigned q_at = (fa_smem(q_s) & 0x3FFFFu) >> 4, ring_at = (fa_smem(ring) & 0x3FFFFu) >> 4;
    auto wait = [&](unsigned long long* bar, int parity) {
      return (bool)__all_sync(0xffffffffu, fa_mbar_wait(bar, (unsigned)parity));
    };
    auto wait_place = [&](int n) { return wait(&full[n % FA_BUFFERS], (n / FA_BUFFERS) & 1); };
    // S = Q K^T of lane l's step b, 16 lanes of the head at a time
    auto scores = [&](int l, int b) {
      const int buf = k_place(block_of(l, b)) % FA_BUFFERS;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned a_at = q_at + (unsigned)((split ? 0 : l) * (kTileBytes >> 4));
      const unsigned b_at = ring_at + (unsigned)(buf * (kTileBytes >> 4));
      const unsigned s_t = tmem_base + (unsigned)(l * 128);
      if (leader) {
#pragma unroll 1
        for (int kk = 0; kk < HEAD_DIM / 16; ++kk) {
          const unsigned off = (unsigned)((kk / 4) * (kSubTile >> 4) + 2 * (kk % 4));
          fa_mma(s_t, a_at + off, b_at + off, idesc_s, kk != 0);
        }
        fa_commit(&s_full[l]);
        if (split || l == 1) fa_commit(&empty[buf]);
      }
      __syncwarp();
    };
    bool ok = wait(q_full, 0);
    for (int l = 0; ok && l < 2; ++l)
      if (steps_of(l) > 0 && (ok = wait_place(k_place(block_of(l, 0))))) scores(l, 0);
    const int most = steps_of(0);
    for (int b = 0; ok && b < most; ++b) {
      for (int l = 0; ok && l < 2; ++l) {
        if (b >= steps_of(l)) continue;
        const int place = v_place(block_of(l, b)), buf = place % FA_BUFFERS;
        ok = wait_place(place) && wait(&p_ready[l], b & 1);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // P V over the block's keys, 16 at a time: p advances 8 columns, v two 8-key groups
        const unsigned p_t = tmem_base + (unsigned)(kPFirst + l * 128), o_t = tmem_base + 256u + (unsigned)(l * 128);
        const unsigned b_at = ring_at + (unsigned)(buf * (kTileBytes >> 4));
        if (leader) {
#pragma unroll 1
          for (int kk = 0; kk < FA_KEYS / 16; ++kk)
            fa_mma_ts(o_t, p_t + (unsigned)(kk * 8), b_at + (unsigned)(kk * 128), idesc_o, b > 0 || kk != 0);
          fa_commit(&pv_done[l]);
          if (split || l == 1) fa_commit(&empty[buf]);
        }
        __syncwarp();
        if (b + 1 < steps_of(l)) {
          // the lane's scores were read before p_ready; where p lies on them, its reader has to be through
          ok = wait_place(k_place(block_of(l, b + 1))) && (!kPOnScores || wait(&pv_done[l], b & 1));
          if (ok) scores(l, b + 1);
        }
      }
    }
  } else if (live && warp < FA_SOFTMAX_WARPS) {
    // ---------------- softmax: two threads a row, 64 of a block's keys each ----------------
    const int l = warp >> 3, half = (warp >> 2) & 1;
    const int r = (warp & 3) * 32 + lane;
    const int h = split ? h0 : h0 + l;
    const int p_row = pos0 + min(r, n_rows - 1);            // rows past the tile repeat its last row
    const int lo_row = first_visible_key(p_row, window, chunk);
    const unsigned lane_base = ((unsigned)((warp & 3) * 32) << 16);
    const unsigned my_s = tmem_base + lane_base + (unsigned)(l * 128);
    const unsigned my_p = my_s + (unsigned)(kPFirst + half * (kHalfKeys / 2));
    const unsigned my_o = my_s + 256u;
    // the two threads of a row (of neighbouring warps of the lane) meet at a barrier of their 64
    float* my_stat = stat_s + (l * 2 + half) * FA_ROWS + r;
    const float* other_stat = stat_s + (l * 2 + 1 - half) * FA_ROWS + r;
    auto meet = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + l * 4 + (warp & 3)) : "memory"); };
    const int steps = steps_of(l);
    float m_ref = -INFINITY, l_run = 0.f;     // reference maximum (raw score units, the row's) and running sum (this half's)
    bool ok = true;
    for (int b = 0; b < steps; ++b) {
      const int kb = first_of(block_of(l, b)) + half * kHalfKeys;
      // behind a wait that ran out a warp goes on through its steps without waiting, so that it meets its partner as
      // often as that one does
      ok = __all_sync(0xffffffffu, ok && fa_mbar_wait(&s_full[l], b & 1));
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float s[kHalfKeys];
      fa_tmem_load64(my_s + (unsigned)(half * kHalfKeys), s);
      if (CAPPED) {      // a cap on the scores: times the scale, the squashed raw product is cap * tanh(score / cap)
#pragma unroll
        for (int j = 0; j < kHalfKeys; ++j) s[j] = softcap_raw(s[j], cap_in, cap_out);
      }
      if (kb + kHalfKeys - 1 > pos0 || kb < lo_last) {
#pragma unroll
        for (int j = 0; j < kHalfKeys; ++j) {
          const int key = kb + j;
          s[j] = (key <= p_row && (key >= lo_row || key < keep_first)) ? s[j] : -INFINITY;
        }
      }
      float m8[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) m8[i] = fmaxf(s[i], s[8 + i]);
#pragma unroll
      for (int j = 16; j < kHalfKeys; j += 8)
#pragma unroll
        for (int i = 0; i < 8; ++i) m8[i] = fmaxf(m8[i], s[j + i]);
      float m_blk = fmaxf(fmaxf(fmaxf(m8[0], m8[1]), fmaxf(m8[2], m8[3])), fmaxf(fmaxf(m8[4], m8[5]), fmaxf(m8[6], m8[7])));
      // the other half's maximum (its slot is written again only behind the next scores, which wait for both
      // halves' probabilities, so one slot a thread is enough)
      *my_stat = m_blk;
      if (kPOnScores) asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      meet();
      if (kPOnScores) asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      m_blk = fmaxf(m_blk, *other_stat);
      // the reference moves only when the maximum has run away from it
      const bool move = m_blk > -INFINITY &&
                        (m_ref == -INFINITY || (m_blk - m_ref) * scale_log2 > FA_RESCALE_AT);
      float factor = 1.f;
      if (move) {
        factor = m_ref == -INFINITY ? 0.f : fa_exp2((m_ref - m_blk) * scale_log2);
        m_ref = m_blk;
        l_run *= factor;
      }
      // probabilities, their sum, and the bfloat16 copy for the second product; two columns an instruction
      // where the hardware has it (scale and shift, the sum).  Masked scores are -inf: probability 0.
      const float m_scaled = m_ref == -INFINITY ? 0.f : m_ref * scale_log2;
      const unsigned long long scale2 = fa_pack2(scale_log2, scale_log2), shift2 = fa_pack2(-m_scaled, -m_scaled);
      unsigned long long sum2[4] = {0ull, 0ull, 0ull, 0ull};
      unsigned p[kHalfKeys / 2];
#pragma unroll
      for (int j = 0; j < kHalfKeys; j += 2) {
        float x0, x1;
        fa_unpack2(fa_fma2(fa_pack2(s[j], s[j + 1]), scale2, shift2), x0, x1);
        x0 = fa_exp2(x0);
        x1 = fa_exp2(x1);
        sum2[(j >> 1) & 3] = fa_add2(sum2[(j >> 1) & 3], fa_pack2(x0, x1));
        const __nv_bfloat162 pair = __floats2bfloat162_rn(x0, x1);
        p[j >> 1] = *reinterpret_cast<const unsigned*>(&pair);
      }
      float sum_even, sum_odd;
      fa_unpack2(fa_add2(fa_add2(sum2[0], sum2[1]), fa_add2(sum2[2], sum2[3])), sum_even, sum_odd);
      l_run += sum_even + sum_odd;
      // The scores of this block were committed behind the lane's P V of the block before: p is free.  Where p lies
      // on the scores, it takes the first half's columns, which both halves have read before they met.
      fa_tmem_store32(my_p, p);
      // a rescaling waits for the last block's P V, which writes the accumulator; each half takes half of its lanes
      if (b > 0 && __any_sync(0xffffffffu, move)) {
        ok = __all_sync(0xffffffffu, ok && fa_mbar_wait(&pv_done[l], (b - 1) & 1));
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
        for (int c0 = half * (HEAD_DIM / 2); c0 < (half + 1) * (HEAD_DIM / 2); c0 += 16) {
          float acc[16];
          fa_tmem_load16(my_o + (unsigned)c0, acc);
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[j] *= factor;
          fa_tmem_store16(my_o + (unsigned)c0, acc);
        }
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (ok && lane == 0) fa_mbar_arrive(&p_ready[l]);                    // one arrival a warp
    }
    // ---------------- the row's output ----------------
    if (steps > 0) ok = ok && fa_mbar_wait(&pv_done[l], (steps - 1) & 1);
    const int other_steps = split ? steps_of(1 - l) : 0;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    *my_stat = l_run;                        // both halves' sums (the maxima were read before the last P V)
    meet();
    const float l_all = l_run + *other_stat;
    float m_all = m_ref, weight = 1.f, weight_other = 0.f, den = l_all;
    if (split) {
      meet();                                // read before the slots are written again
      *my_stat = half ? l_all : m_ref;
      // the other lane's threads have seen its last P V done when they come here
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      asm volatile("bar.sync 9, %0;" ::"n"(FA_SOFTMAX_WARPS * 32) : "memory");
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float m_other = stat_s[(1 - l) * 2 * FA_ROWS + r], l_other = stat_s[((1 - l) * 2 + 1) * FA_ROWS + r];
      m_all = fmaxf(m_ref, m_other);
      weight = m_ref == -INFINITY ? 0.f : fa_exp2((m_ref - m_all) * scale_log2);
      weight_other = m_other == -INFINITY ? 0.f : fa_exp2((m_other - m_all) * scale_log2);
      den = weight * l_all + weight_other * l_other;
    }
    // a sink takes part in the denominator once, unscaled (it has no key and no value)
    if (sink && m_all > -INFINITY) den += exp2f(sink[h] * 1.4426950408889634f - m_all * scale_log2);
    if (__all_sync(0xffffffffu, ok)) {
      const float inv = 1.0f / den;
      // a thread writes its half of the head; split, its quarter, from both accumulators (one without a step was
      // never written)
      const int width = split ? HEAD_DIM / 4 : HEAD_DIM / 2, first = (split ? l * 2 + half : half) * width;
      __nv_bfloat16* dst = out + ((size_t)(row0 + min(r, n_rows - 1)) * nh + h) * HEAD_DIM;
#pragma unroll 1
      for (int c0 = first; c0 < first + width; c0 += 16) {
        float acc[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = 0.f;
        if (steps > 0) {
          float part[16];
          fa_tmem_load16(my_o + (unsigned)c0, part);
#pragma unroll
          for (int i = 0; i < 16; ++i) acc[i] = weight * part[i];
        }
        if (other_steps > 0) {
          float part[16];
          fa_tmem_load16(tmem_base + lane_base + 256u + (unsigned)((1 - l) * 128 + c0), part);
#pragma unroll
          for (int i = 0; i < 16; ++i) acc[i] = fmaf(weight_other, part[i], acc[i]);
        }
        if (r < n_rows) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint4 piece;
            unsigned* w = reinterpret_cast<unsigned*>(&piece);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              __nv_bfloat162 pair = __floats2bfloat162_rn(acc[8 * c + 2 * e] * inv, acc[8 * c + 2 * e + 1] * inv);
              w[e] = *reinterpret_cast<unsigned*>(&pair);
            }
            *reinterpret_cast<uint4*>(dst + c0 + c * 8) = piece;
          }
        }
      }
    }
  }
  // ---------------- common exit ----------------
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  pdl_launch();
  if (threadIdx.x == 0 && tmem_slot[1] != 0) {
    atomicExch(&fa_error_flag, 1);
    tokb200_report_error(TOKB200_LIB_ATTENTION_TCGEN05, 1);
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"((unsigned)kTmemCols) : "memory");
  }
}

TOKB200_API int tokb200_attention_tcgen05_head_dim() { return HEAD_DIM; }

TOKB200_API int tokb200_attention_tcgen05_error(void) {
  int flag = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&flag, fa_error_flag, sizeof(int)) != cudaSuccess) return -1;
  if (flag) cudaMemcpyToSymbol(fa_error_flag, &zero, sizeof(int));
  return flag;
}

// ---- host side ----------------------------------------------------------------
typedef CUresult (*FaEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                               const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                               CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static FaEncodeFn fa_encode() {
  static const FaEncodeFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<FaEncodeFn>(p);
  }();
  return fn;
}

// A map over row-major [rows, lanes] bfloat16, boxes of box_rows x 64 lanes, 128-byte swizzle, zeros outside.
static int fa_map(CUtensorMap* map, const void* base, long long rows, long long lanes, int box_rows) {
  const FaEncodeFn fn = fa_encode();
  if (!fn) return TOKB200_BAD_SIZE;
  const cuuint64_t dims[2] = {(cuuint64_t)lanes, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)lanes * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  const cuuint32_t elem[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? TOKB200_OK : TOKB200_BAD_ALIGNMENT;
}

// tiles: [n_tiles][2] = (first row, rows) of consecutive rows of one request, rows <= 128.  `q_rows`, `pool_rows`: rows
// of q and of the pools.  `split`: 1 cuts every head's key blocks over the two lanes, 0 puts heads side by side.
TOKB200_API int tokb200_attention_tcgen05(
    const void* q, const void* k_pool, const void* v_pool, void* out, const int* block_table,
    int table_stride, const int* row_req, const int* pos, const int* tiles, int n_tiles, int q_rows, int pool_rows,
    int nh, int nkv, int d, int page, int window, int chunk, int keep_first, float scale, const float* sink,
    float softcap, int split, cudaStream_t stream) {
  if (n_tiles <= 0) return TOKB200_OK;
  if (d != HEAD_DIM || nh <= 0 || nkv <= 0 || nh % nkv || page <= 0 || keep_first < 0 || q_rows <= 0 || pool_rows <= 0)
    return TOKB200_BAD_SIZE;
  if (((uintptr_t)q | (uintptr_t)k_pool | (uintptr_t)v_pool | (uintptr_t)out) & 15)
    return TOKB200_BAD_ALIGNMENT;
  static bool configured[64] = {};
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return TOKB200_BAD_SIZE;
  if (!configured[device]) {
    cudaError_t err = cudaFuncSetAttribute(attention_tcgen05_kernel<false>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, kFaSmem);
    if (err == cudaSuccess)
      err = cudaFuncSetAttribute(attention_tcgen05_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFaSmem);
    if (err != cudaSuccess) return (int)err;
    configured[device] = true;
  }
  if (n_tiles > 65535) return TOKB200_BAD_SIZE;
  // keys that lie together in a page whatever the block: the largest power of two that divides the page, up to a block
  int run = page & -page;
  run = run > FA_KEYS ? FA_KEYS : run < 8 ? 0 : run;
  CUtensorMap map_q, map_k, map_v;
  int status = fa_map(&map_q, q, q_rows, (long long)nh * HEAD_DIM, FA_ROWS);
  if (status == TOKB200_OK) status = fa_map(&map_k, k_pool, pool_rows, (long long)nkv * HEAD_DIM, run ? run : 8);
  if (status == TOKB200_OK) status = fa_map(&map_v, v_pool, pool_rows, (long long)nkv * HEAD_DIM, run ? run : 8);
  if (status != TOKB200_OK) return status;
  const int pairs = nkv * ((nh / nkv + 1) / 2);
  dim3 grid(split ? nh : pairs, n_tiles);
  // This kernel starts strictly after its predecessor.  Started early (its blocks allocating tensor
  // memory and waiting while the rotary kernel before it still runs), with the product after it
  // started early as well, about one step in a hundred of some 1,800 prompt tokens came out with
  // a few rows wrong (bitwise comparison of repeated identical steps; never with either of the
  // two early starts taken away, nor with this kernel alone or between two products).  The cause
  // has not been found; the early start saved about two microseconds a layer.  All of that was seen with the
  // kernel's form of one tile and head a block; this one has not been started early.
  return launch_ordered(false, softcap > 0.f ? attention_tcgen05_kernel<true> : attention_tcgen05_kernel<false>, grid,
                        dim3(FA_THREADS), (size_t)kFaSmem, stream, map_q, map_k,
                        map_v, (const __nv_bfloat16*)k_pool, (const __nv_bfloat16*)v_pool, (__nv_bfloat16*)out,
                        block_table, table_stride, row_req, pos, tiles, n_tiles, nh, nkv, page, run, pool_rows, split,
                        window, chunk, keep_first, scale * 1.4426950408889634f, sink,
                        softcap > 0.f ? scale / softcap : 0.f, softcap > 0.f ? softcap / scale : 0.f);
}
