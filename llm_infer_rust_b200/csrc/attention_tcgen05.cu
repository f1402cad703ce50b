// Causal prefill attention over the paged bfloat16 cache on the fifth-generation tensor cores, head size 128.
//
// A CTA serves 128 query vectors: 128 / group consecutive tokens of one row x the `group` query heads of one KV
// head (row r of the tile = token r / group, head r mod group).  It walks the visible keys in blocks of 128:
//   S = Q K^T      tcgen05.mma, M 128, N 128 (keys), K 16 x 8; Q and K are K-major tiles in the 128-byte swizzle
//                  (Q is written there by the softmax warps, K arrives by TMA); S lands in one of TWO score
//                  buffers in tensor memory, so the scores of block i + 1 are computed under the softmax of block i;
//   softmax        four warps, one thread per query row: two passes over the row of S in tensor memory
//                  (tcgen05.ld): the row maximum, then exp2 and the row sum; the bfloat16 probabilities go back
//                  into tensor memory (tcgen05.st), two to a column, over the first half of the scores they
//                  came from.  The further forms (soft-cap, weights in two terms, blocks, sinks, differences) have
//                  eight warps and two threads a row, each with its half of the scores in registers (softmax_half);
//                  the two-tile kernel one thread a row, one score buffer a tile and the whole row in registers after
//                  one pass, and its P V begins with the first 64 keys' weights (softmax_row);
//   O += P V       tcgen05.mma with the A operand in tensor memory, M 128, N 128 (head dims), K 16 x 8,
//                  accumulating in tensor memory over all blocks; V is used as it lies in the cache (keys x dims,
//                  the dims contiguous: an MN-major B operand).  The tensor pipe runs the MMAs of one thread in
//                  the order of issue, so the scores of block i + 2 overwrite the buffer only behind P V of block i.
//                  The probabilities are taken relative to a reference maximum that is raised only when a row's
//                  maximum has grown by more than 2^8 (then the row's thread rescales its O in tensor memory,
//                  tcgen05.ld / st, once P V of the block before is finished); a stale reference is exact, since
//                  the row sum uses the same one.
// Two warps (one in the two-tile kernel) fetch K blocks (ring of three) and V blocks (ring of two) by TMA, a page's
// box each in turn; one warp owns tensor memory and issues the MMAs.  Semantics as attention.cu (reference: src/models/attention/backend.rs:1455-1498): causal
// mask, optional window, scale as a parameter, softmax in float.  Value rows at or beyond what the tile may see are
// zeroed in shared memory before they are used.  Every wait is bounded by the clock; on a time-out the error word
// is flagged and every path still reaches the end, where tensor memory is given back.
#include <cuda.h>
#include <math.h>
#include <string.h>

#include <initializer_list>

#include "common.cuh"
#include "pairs.cuh"

#ifndef HEAD_DIM
#define HEAD_DIM 128
#endif
static_assert(HEAD_DIM == 128, "the tcgen05 attention kernel is written for head size 128");

typedef __nv_bfloat16 bf16;
constexpr int D = 128;
constexpr int BQ = 128;                  // query vectors per CTA
constexpr int BKV = 128;                 // keys per block
constexpr int HALF = BKV * 128;          // bytes of a [128 rows x 64 columns] half tile
constexpr int TILE = 2 * HALF;           // bytes of a [128 x 128] bfloat16 tile
constexpr int K_STAGES = 3, V_STAGES = 2;
// Warps that issue the copies: warp 0 and the warps behind the softmax warps.  Measured (kernel alone, pages of 16 keys):
// the one-tile kernel with 1 / 2 / 4 / 8 copy warps: 48.1 / 43.3 / 43.7 / 45.3 us at 2,048 tokens x 16 heads and 594 /
// 740 / 709 / 673 TFLOP/s at 16,384 x 32; the two-tile kernel, which fetches half as much a query: 892 / 886 / 869 / 801.
constexpr int COPY_WARPS = 2;
constexpr int PAIR_COPY_WARPS = 1;
constexpr int THREADS = 192 + 32 * (COPY_WARPS - 1);   // one tile per CTA: warp 0 copies, warp 1 MMA, warps 2-5 softmax, warps 6.. copy
constexpr int PAIR_THREADS = 320 + 32 * (PAIR_COPY_WARPS - 1);   // two tiles per CTA: four more softmax warps (2-9), warps 10.. copy
constexpr int TMEM_COLS = 512;           // S buffers (and P in their first 64 columns): columns 0..127 and 128..255; O: 256..383
constexpr float RESCALE_STEP = 8.0f;     // the reference maximum follows only growth beyond 2^8

// Shared memory: V stages, K stages, Q (each tile 32 KB), then the barriers.
constexpr int V_OFF = 0, K_OFF = V_STAGES * TILE, Q_OFF = K_OFF + K_STAGES * TILE, BAR_OFF = Q_OFF + TILE;
constexpr int N_BARS = 2 * K_STAGES + 2 * V_STAGES + 2 + 4;
constexpr int TBL_ENTRIES = 2048;         // page numbers of a row that the copy warp keeps in shared memory (the rest it reads as before)
constexpr int TBL_OFF = BAR_OFF + (N_BARS + 1) * 8;      // (one more slot holds the tensor-memory address)
constexpr int SMEM_BYTES = TBL_OFF + TBL_ENTRIES * 4;
constexpr int SHAPED_THREADS = THREADS + 128;             // two softmax threads a row
constexpr int XCH_OFF = (SMEM_BYTES + 15) / 16 * 16;      // what they exchange: [4][2] flags, then [2][2][128] floats
constexpr int SHAPED_SMEM_BYTES = XCH_OFF + 32 + 4 * BQ * 4;
static_assert(1024 + SHAPED_SMEM_BYTES <= 227 * 1024, "shared memory of one CTA");

__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
// All lanes of a warp wait and agree on the outcome: the collective tensor-memory loads that follow need the
// warp whole, also when a wait has run out.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, int* err) {
  const bool mine = mbar_wait(bar, parity, err);
  return __all_sync(0xffffffffu, mine ? 1 : 0) != 0;
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n"
               ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y) : "memory");
}
// K-major tile in the 128-byte swizzle: 8-row groups 1024 bytes apart, leading byte offset unused (1).
__device__ __forceinline__ uint64_t desc_k_major(uint32_t addr) {
  const uint32_t lo = ((addr >> 4) & 0x3FFFu) | (1u << 16);
  const uint32_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);
  return (static_cast<uint64_t>(hi) << 32) | lo;
}
// MN-major tile in the 128-byte swizzle (rows = k, 64 MN elements = 128 bytes contiguous): 8-row groups 1024 bytes
// apart (stride byte offset), the next 64 MN elements HALF bytes further (leading byte offset).
__device__ __forceinline__ uint64_t desc_mn_major(uint32_t addr) {
  const uint32_t lo = ((addr >> 4) & 0x3FFFu) | (static_cast<uint32_t>(HALF >> 4) << 16);
  const uint32_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);
  return (static_cast<uint64_t>(hi) << 32) | lo;
}
// float accumulator, bfloat16 operands, M 128, N 128; B is K-major for S = Q K^T and MN-major for P V.
constexpr uint32_t kDescQK = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
constexpr uint32_t kDescPV = kDescQK | (1u << 16);

__device__ __forceinline__ void umma(uint32_t tmem_c, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
               ::"r"(tmem_c), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
// The A operand from tensor memory: 16-bit elements packed two to a column (k = 2c, 2c + 1 in column c of lane m).
__device__ __forceinline__ void umma_a_tmem(uint32_t tmem_c, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
               ::"r"(tmem_c), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
// True in one lane of a whole warp.  The warp that issues products walks along as a whole and only the instruction itself is one
// lane's: what comes before it is then the same in every lane for all the compiler knows, and descriptors are made in uniform
// registers, where the instruction takes them.  (From one lane's own registers a product took 100 cycles to issue, so 35: 8,192 tokens x
// 16 heads 299 -> 275 us.)
__device__ __forceinline__ bool elect_one() {
  uint32_t is;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.b32 %0, 1, 0, p;\n}\n" : "=r"(is));
  return is != 0;
}
__device__ __forceinline__ int same_in_warp(int v) { return __shfl_sync(0xffffffffu, v, 0); }
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
               "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
               "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                 "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                 "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
// 64 consecutive columns of this thread's lane, in one load and one wait.
__device__ __forceinline__ void tmem_ld64(uint32_t taddr, float (&v)[64]) {
  uint32_t r[64];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x64.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, %48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%64];\n"
               "tcgen05.wait::ld.sync.aligned;\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]), "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]), "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]), "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]), "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
               : "r"(taddr) : "memory");
#pragma unroll
  for (int i = 0; i < 64; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float (&v)[32]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
               "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
               "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};\n"
               ::"r"(taddr), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])),
                 "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])),
                 "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
                 "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])), "r"(__float_as_uint(v[15])),
                 "r"(__float_as_uint(v[16])), "r"(__float_as_uint(v[17])), "r"(__float_as_uint(v[18])), "r"(__float_as_uint(v[19])),
                 "r"(__float_as_uint(v[20])), "r"(__float_as_uint(v[21])), "r"(__float_as_uint(v[22])), "r"(__float_as_uint(v[23])),
                 "r"(__float_as_uint(v[24])), "r"(__float_as_uint(v[25])), "r"(__float_as_uint(v[26])), "r"(__float_as_uint(v[27])),
                 "r"(__float_as_uint(v[28])), "r"(__float_as_uint(v[29])), "r"(__float_as_uint(v[30])), "r"(__float_as_uint(v[31]))
               : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
}
// 32 columns of this thread's lane from 32 registers; the caller waits (tcgen05.wait::st) before it tells anyone.
__device__ __forceinline__ void tmem_st32_raw(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
               "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
               "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};\n"
               ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
                 "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
                 "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
                 "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
               : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n"
               ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
               "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n"
               ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
                 "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
               "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
               "tcgen05.wait::ld.sync.aligned;\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                 "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
               : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ float fast_exp2(float x) {      // 2^x, one special-function instruction (-inf gives 0)
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

// Byte offset of (row r, 16-byte chunk c of 16) inside a [128 x 128] bfloat16 tile of two swizzled halves.
__device__ __forceinline__ int swz(int r, int c) { return (c >> 3) * HALF + r * 128 + (((c & 7) ^ (r & 7)) << 4); }

// ---------------------------------------------------------------------------------------------------------------
// What the softmax threads of both kernels do.  A thread owns one query row: lane r of tensor memory.

// The row's Q vector into its K-major tile in the 128-byte swizzle (zeros for a row that is not used), chunks
// c_lo .. c_lo + CHUNKS - 1 of 16.
template <int CHUNKS>
__device__ __forceinline__ void write_q_row(unsigned char* q_tile, const bf16* src, int r, bool used, int c_lo) {
#pragma unroll
  for (int i = 0; i < CHUNKS; ++i) {
    const int c = c_lo + i;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (used) v = *reinterpret_cast<const uint4*>(src + c * 8);
    *reinterpret_cast<uint4*>(q_tile + swz(r, c)) = v;
  }
  proxy_fence();
}

// Row r of an MN-major value tile (128 dims in two halves of 128 bytes), chunks c_lo .. c_lo + CHUNKS - 1 of 16 set to zero.
template <int CHUNKS>
__device__ __forceinline__ void zero_value_row(unsigned char* v_tile, int r, int c_lo) {
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int c = c_lo; c < c_lo + CHUNKS; ++c) *reinterpret_cast<uint4*>(v_tile + (c >> 3) * HALF + r * 128 + (c & 7) * 16) = zero;
}

struct RowState {
  float m_ref = -INFINITY;     // reference maximum (log2 units): follows the row's maximum in steps of RESCALE_STEP
  float l_run = 0.0f;          // sum of the probabilities relative to it
};

// One block of 128 keys for this thread's row.  The scores lie in the 128 columns from s_base on; the bfloat16
// probabilities go back over the first 64 of them, two to a column (the A operand of P V), and are in tensor memory
// when the function returns.  The row sees keys lo_key .. hi_key (none: hi_key -1).  `block` counts the row's blocks from 0; P V of block - 1 commits to `pv_done`.  Every
// phase of that barrier is waited for here, in order: before the accumulator at o_base is rescaled (the row's
// maximum grew by more than the step), else at the end, when that product has long finished.  A wait by parity
// cannot tell "phase b - 1 is not finished" from "phase b - 2 is not finished": a waiter that skipped a phase
// would pass at once.  Returns false when a wait ran out.
__device__ __forceinline__ bool softmax_block(uint32_t s_base, uint32_t o_base, int first_key, int lo_key, int hi_key,
                                              bool masked, float scale_log2, int block, uint64_t* pv_done, RowState& st,
                                              int* err) {
  tc_fence_after();
  // pass 1: the row's maximum over the block's visible keys (of the raw scores; the scale is positive)
  float mx = -INFINITY;
#pragma unroll 1
  for (int c = 0; c < 2; ++c) {
    float v[64];
    tmem_ld64(s_base + c * 64, v);
    if (masked) {
#pragma unroll
      for (int e = 0; e < 64; ++e) {
        const int key = first_key + c * 64 + e;
        const bool vis = key >= lo_key && key <= hi_key;
        mx = fmaxf(mx, vis ? v[e] : -INFINITY);
      }
    } else {
      float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};      // four chains instead of one
#pragma unroll
      for (int e = 0; e < 64; e += 4) {
        m4[0] = fmaxf(m4[0], v[e]); m4[1] = fmaxf(m4[1], v[e + 1]); m4[2] = fmaxf(m4[2], v[e + 2]); m4[3] = fmaxf(m4[3], v[e + 3]);
      }
      mx = fmaxf(mx, fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])));
    }
  }
  mx = hi_key >= 0 ? mx * scale_log2 : -INFINITY;
  // The reference follows the maximum when it grew by more than the step (or there was none yet).
  const bool raise = mx > st.m_ref + RESCALE_STEP || (st.m_ref == -INFINITY && mx > -INFINITY);
  const float m_new = raise ? mx : st.m_ref;
  const float corr = raise ? (st.m_ref == -INFINITY ? 0.0f : exp2f(st.m_ref - m_new)) : 1.0f;
  const float base = m_new == -INFINITY ? 0.0f : m_new;
  bool pv_seen = block == 0;
  // The accumulator may be rescaled only between two products: P V of the block before has to be finished.
  if (block > 0 && __any_sync(0xffffffffu, raise ? 1 : 0)) {
    if (!mbar_wait_warp(pv_done, (block - 1) & 1, err)) return false;
    pv_seen = true;
    tc_fence_after();
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
      float o[32];
      tmem_ld32(o_base + c * 32, o);
#pragma unroll
      for (int e = 0; e < 32; ++e) o[e] *= corr;
      tmem_st32(o_base + c * 32, o);
    }
  }
  st.l_run = st.l_run * corr;
  st.m_ref = m_new;
  // pass 2: probabilities relative to the reference and their sum; those of columns 64c .. 64c + 63 go back into
  // tensor memory over the scores that were just read (columns 32c .. 32c + 31)
  const float neg_base = hi_key >= 0 ? -base : -INFINITY;      // a row that is not used gets zeros
  float sum4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 1
  for (int c = 0; c < 2; ++c) {
    float v[64];
    tmem_ld64(s_base + c * 64, v);
    if (masked) {
#pragma unroll
      for (int e = 0; e < 64; ++e) {
        const int key = first_key + c * 64 + e;
        const bool vis = key >= lo_key && key <= hi_key;
        v[e] = vis ? fast_exp2(fmaf(v[e], scale_log2, neg_base)) : 0.0f;
      }
    } else {
#pragma unroll
      for (int e = 0; e < 64; ++e) v[e] = fast_exp2(fmaf(v[e], scale_log2, neg_base));
    }
    uint32_t pr[32];
#pragma unroll
    for (int e = 0; e < 64; e += 2) {
      sum4[(e >> 1) & 3] += v[e] + v[e + 1];
      __nv_bfloat162 two = __floats2bfloat162_rn(v[e], v[e + 1]);
      pr[e >> 1] = *reinterpret_cast<uint32_t*>(&two);
    }
    tmem_st32_raw(s_base + c * 32, pr);
  }
  st.l_run += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
  tmem_wait_st();                                      // P is in tensor memory
  return pv_seen || mbar_wait_warp(pv_done, (block - 1) & 1, err);
}

// The two-tile kernel's block: all 128 scores in registers (one load of the row, where softmax_block waits for four), and the
// products with the values begin when half of the weights stand: `half_done` is called behind the first 64 keys' weights.
// S of a block is issued behind P V of the block before it, so whoever has seen these scores may touch the accumulator:
// pv_done is not asked.  A tile walks a chain of its own latencies (measured with softmax_block, SM cycles a block at 8,192
// tokens: 2,040 until the next scores stand, 2,700 in the softmax, 1,720 of those behind the maximum, for 1,024 of
// special-function work), so what shortens the chain counts: 8,192 tokens x 16 heads 340 -> 302 us, 16,384 x 32 2,165 us
// (1,015 TFLOP/s).  Behind the maximum the thread's issue slots are the chain, so scale and sum take two scores an instruction
// (with the MMAs issued by a whole warp: 275 -> 265 us, 3,000 tokens 58.6 -> 56.8; from the two before both, 16,384 x 32 2,283 -> 2,171).
// The weights are added up as softmax_block adds them, a pair's two and then pairs into four sums, so that both kernels give the
// same bits: which of them runs follows from the other rows of the step.  (Every weight into a sum of its own place, one addition less
// in the chain, was 264 us.)  Two threads a row, which pay for the further forms below, were slower here (483 us: sixteen warps leave
// 96 registers a thread, so the scores are read twice).
__device__ __forceinline__ void tmem_ld32_begin(uint32_t taddr, float (&v)[32]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
               "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
               "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
                 "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]),
                 "=f"(v[16]), "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]),
                 "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
               : "r"(taddr));
}
template <typename F>
__device__ __forceinline__ void softmax_row(uint32_t s_base, uint32_t o_base, int first_key, int lo_key, int hi_key, bool masked,
                                            float scale_log2, int block, RowState& st, const F& half_done) {
  tc_fence_after();
  float v[4][32];
#pragma unroll
  for (int c = 0; c < 4; ++c) tmem_ld32_begin(s_base + c * 32, v[c]);
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int e = 0; e < 32; ++e) asm volatile("" : "+f"(v[c][e]));      // (used only behind the wait)
  if (masked) {
    const int lo = lo_key - first_key, hi = hi_key - first_key;
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int e = 0; e < 32; ++e) v[c][e] = c * 32 + e >= lo && c * 32 + e <= hi ? v[c][e] : -INFINITY;
  }
  float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int e = 0; e < 32; ++e) m4[e & 3] = fmaxf(m4[e & 3], v[c][e]);
  const float raw = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
  const float mx = hi_key >= 0 ? raw * scale_log2 : -INFINITY;
  const bool raise = mx > st.m_ref + RESCALE_STEP || (st.m_ref == -INFINITY && mx > -INFINITY);
  const float m_new = raise ? mx : st.m_ref;
  if (__any_sync(0xffffffffu, raise ? 1 : 0)) {
    const float corr = raise ? (st.m_ref == -INFINITY ? 0.0f : exp2f(st.m_ref - m_new)) : 1.0f;
    st.l_run *= corr;
    if (block > 0) {
#pragma unroll 1
      for (int c = 0; c < 8; ++c) {
        uint32_t o[16];
        tmem_ld16(o_base + c * 16, o);
#pragma unroll
        for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * corr);
        tmem_st16(o_base + c * 16, o);
      }
      tmem_wait_st();
    }
  }
  st.m_ref = m_new;
  const float neg_base = hi_key < 0 ? -INFINITY : m_new == -INFINITY ? 0.0f : -m_new;      // a row that is not used gets zeros
  f32x2 sums[2] = {0, 0};
  const f32x2 scale2 = twice(scale_log2), base2 = twice(neg_base);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t pr[16];
#pragma unroll
    for (int i = 0; i < 16; i += 2) {                  // two pairs of weights a turn: (a0, b0), (a1, b1)
      float a0, b0, a1, b1;
      unpack2(fma2(pack2(v[c][2 * i], v[c][2 * i + 1]), scale2, base2), a0, b0);
      unpack2(fma2(pack2(v[c][2 * i + 2], v[c][2 * i + 3]), scale2, base2), a1, b1);
      a0 = fast_exp2(a0);
      b0 = fast_exp2(b0);
      a1 = fast_exp2(a1);
      b1 = fast_exp2(b1);
      sums[(i >> 1) & 1] = add2(sums[(i >> 1) & 1], add2(pack2(a0, a1), pack2(b0, b1)));
      const __nv_bfloat162 p0 = __floats2bfloat162_rn(a0, b0), p1 = __floats2bfloat162_rn(a1, b1);
      pr[i] = *reinterpret_cast<const uint32_t*>(&p0);
      pr[i + 1] = *reinterpret_cast<const uint32_t*>(&p1);
    }
    tmem_st16(s_base + c * 16, pr);
    if (c == 1) {
      tmem_wait_st();
      half_done();
    }
  }
  float sum4[4];
  unpack2(sums[0], sum4[0], sum4[1]);
  unpack2(sums[1], sum4[2], sum4[3]);
  st.l_run += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
  tmem_wait_st();                                      // P is in tensor memory
}

// ---- The further forms of a score and of what is stored, for the builds of the one-tile kernel that know them (SHAPED):
//   cap_log2 > 0       score <- cap tanh(score * scale / cap), in log2 units (tanh_in = scale / cap);
//   split              a weight enters the product with the values as two bfloat16 terms, the rounded weight (in the first
//                      64 columns of its score buffer) and what the rounding left (in the other 64): twice the P V;
//   chunk C > 0        the query at position p also sees only keys from p - p % C on;
//   sinks              exp(sinks[head]) joins the softmax's denominator;
//   diff_* (DIFF)      query vectors are pairs, neighbouring rows 2j and 2j + 1 the two maps of one head: what is stored is
//                      o / sqrt(mean(o^2) + eps) * gain, o = a_(2j) - lambda a_(2j + 1), in float until then.
struct ScoreShape {
  float cap_log2, tanh_in;
  int split, chunk;
  const float* sinks;
  float diff_lambda, diff_gain, diff_eps;
};
// cap_log2 tanh(s tanh_in) + shift, with tanh(x) = 1 - 2 / (e^(2x) + 1): two special-function instructions.
__device__ __forceinline__ float capped(const ScoreShape& f, float s, float shift) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(fast_exp2(s * (f.tanh_in * 2.8853900817779268f)) + 1.0f));
  return fmaf(-2.0f * f.cap_log2, r, f.cap_log2 + shift);
}
// The same of two scores; NaN stays NaN, a masked score (-inf) does not stay masked.
__device__ __forceinline__ f32x2 capped2(const ScoreShape& f, f32x2 s, float shift) {
  float a, b;
  unpack2(mul2(s, twice(f.tanh_in * 2.8853900817779268f)), a, b);
  unpack2(add2(pack2(fast_exp2(a), fast_exp2(b)), twice(1.0f)), a, b);
  asm("rcp.approx.ftz.f32 %0, %0;\n" : "+f"(a));
  asm("rcp.approx.ftz.f32 %0, %0;\n" : "+f"(b));
  return fma2(twice(-2.0f * f.cap_log2), pack2(a, b), twice(f.cap_log2 + shift));
}

// These forms cost several times the instructions of the plain one, so there a row has TWO threads: thread c = 0, 1 of a row
// takes columns 64 c .. 64 c + 63 of its scores (one load; they stay in registers) and of its accumulator; the two warps
// that hold the same 32 rows exchange their maxima and meet at a barrier of their own, behind which both have read their
// scores, so that the weights' terms may overwrite all 128 columns.  `xch`: [2 parities][2 threads of a row][128 rows] floats,
// `failed`: [2 parities] flags of this quarter.  A warp whose wait has run out still comes to the next barrier (ok: false);
// behind that one both know and both leave, so that nobody is waited for in vain.  Meetings take turns with the parity: what
// was written before one is read before the next, and written again only behind that.
// (One thread a row, the scores read twice as in softmax_block: weights in two terms 104 us at 2,048 tokens x 16 heads,
// 1,263 at 8,192; two threads 43 and 426.  The mma.sync kernel that served these forms: 139 and 1,363; soft-capped 152 and
// 1,515 against 60 and 666; differences over a window of 1,024 159 and 716 against 72 and 309.)
struct HalfRows {
  float* xch;
  volatile int* failed;
  int c, r, quarter;
  // Both warps of the quarter arrive; returns the partner's value.  `left`: one of the two had failed.
  __device__ __forceinline__ float meet(float mine, int parity, bool ok, bool& left) const {
    float* buf = xch + parity * 2 * BQ;
    buf[c * BQ + r] = mine;
    if (!ok) failed[parity] = 1;
    tc_fence_before();
    asm volatile("bar.sync %0, 64;\n" ::"r"(2 + quarter) : "memory");
    tc_fence_after();
    left = failed[parity] != 0;
    return buf[(c ^ 1) * BQ + r];
  }
};

// 2^exponent(scores) of 64 scores, two at a time, their sum added to sums (a pair's two weights first, then pairs into four sums); the weights and (split) what their rounding left into
// tensor memory.  Multiply-adds and sums take two an instruction.
template <typename F>
__device__ __forceinline__ void store_weights(const float (&v)[64], uint32_t p_base, bool split, f32x2 (&sums)[2], const F& exponent) {
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    uint32_t pr[8], rest[8];
#pragma unroll
    for (int i = 0; i < 8; i += 2) {                   // two pairs of weights a turn: (a0, b0), (a1, b1)
      const int e = h * 16 + 2 * i;
      float a0, b0, a1, b1;
      unpack2(exponent(v[e], v[e + 1]), a0, b0);
      unpack2(exponent(v[e + 2], v[e + 3]), a1, b1);
      const f32x2 a = pack2(fast_exp2(a0), fast_exp2(a1)), b = pack2(fast_exp2(b0), fast_exp2(b1));
      sums[(i >> 1) & 1] = add2(sums[(i >> 1) & 1], add2(a, b));
      unpack2(a, a0, a1);
      unpack2(b, b0, b1);
      const __nv_bfloat162 p0 = __floats2bfloat162_rn(a0, b0), p1 = __floats2bfloat162_rn(a1, b1);
      pr[i] = *reinterpret_cast<const uint32_t*>(&p0);
      pr[i + 1] = *reinterpret_cast<const uint32_t*>(&p1);
      unpack2(fma2(pack2(__uint_as_float(pr[i] << 16), __uint_as_float(pr[i + 1] << 16)), twice(-1.0f), a), a0, a1);
      unpack2(fma2(pack2(__uint_as_float(pr[i] & 0xffff0000u), __uint_as_float(pr[i + 1] & 0xffff0000u)), twice(-1.0f), b), b0, b1);
      const __nv_bfloat162 r0 = __floats2bfloat162_rn(a0, b0), r1 = __floats2bfloat162_rn(a1, b1);
      rest[i] = *reinterpret_cast<const uint32_t*>(&r0);
      rest[i + 1] = *reinterpret_cast<const uint32_t*>(&r1);
    }
    tmem_st8(p_base + h * 8, pr);
    if (split) tmem_st8(p_base + 64 + h * 8, rest);
  }
}

// As softmax_block, for this thread's 64 keys of the block; `ok` is what came before (a warp whose wait failed passes false),
// `left` as in HalfRows.
__device__ __forceinline__ bool softmax_half(bool ok, uint32_t s_base, uint32_t o_base, int first_key, int lo_key, int hi_key,
                                             bool masked, float scale_log2, const ScoreShape& shape, int block,
                                             uint64_t* pv_done, const HalfRows& rows, RowState& st, bool& left, int* err) {
  tc_fence_after();
  float v[64];
  float mx = -INFINITY;
  if (ok) {
    tmem_ld64(s_base + rows.c * 64, v);
    if (masked) {
      const int lo = lo_key - first_key - rows.c * 64, hi = hi_key - first_key - rows.c * 64;
#pragma unroll
      for (int e = 0; e < 64; ++e) v[e] = e >= lo && e <= hi ? v[e] : -INFINITY;
    }
    float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int e = 0; e < 64; ++e) m4[e & 3] = fmaxf(m4[e & 3], v[e]);
    mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
  }
  mx = fmaxf(mx, rows.meet(mx, block & 1, ok, left));
  if (!ok || left) return false;
  const bool cap = shape.cap_log2 > 0.0f;
  if (hi_key < 0) mx = -INFINITY;
  else if (cap) mx = mx > -INFINITY ? capped(shape, mx, 0.0f) : mx;      // (the cap rises with the score)
  else mx *= scale_log2;
  const bool raise = mx > st.m_ref + RESCALE_STEP || (st.m_ref == -INFINITY && mx > -INFINITY);
  const float m_new = raise ? mx : st.m_ref;
  const float corr = raise ? (st.m_ref == -INFINITY ? 0.0f : exp2f(st.m_ref - m_new)) : 1.0f;
  bool pv_seen = block == 0;
  if (block > 0 && __any_sync(0xffffffffu, raise ? 1 : 0)) {
    if (!mbar_wait_warp(pv_done, (block - 1) & 1, err)) return false;
    pv_seen = true;
    tc_fence_after();
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      float o[32];
      tmem_ld32(o_base + rows.c * 64 + h * 32, o);
#pragma unroll
      for (int e = 0; e < 32; ++e) o[e] *= corr;
      tmem_st32(o_base + rows.c * 64 + h * 32, o);
    }
  }
  st.m_ref = m_new;
  const float neg_base = hi_key < 0 ? -INFINITY : m_new == -INFINITY ? 0.0f : -m_new;      // a row that is not used gets zeros
  f32x2 sums[2] = {0, 0};
  const uint32_t p_base = s_base + rows.c * 32;
  if (!cap)
    store_weights(v, p_base, shape.split, sums, [&](float x, float y) { return fma2(pack2(x, y), twice(scale_log2), twice(neg_base)); });
  else if (!masked)
    store_weights(v, p_base, shape.split, sums, [&](float x, float y) { return capped2(shape, pack2(x, y), neg_base); });
  else
    store_weights(v, p_base, shape.split, sums, [&](float x, float y) {
      float a, b;
      unpack2(capped2(shape, pack2(x, y), neg_base), a, b);
      return pack2(x == -INFINITY ? x : a, y == -INFINITY ? y : b);
    });
  float sum4[4];
  unpack2(sums[0], sum4[0], sum4[1]);
  unpack2(sums[1], sum4[2], sum4[3]);
  st.l_run = st.l_run * corr + ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));
  tmem_wait_st();                                      // P is in tensor memory
  return pv_seen || mbar_wait_warp(pv_done, (block - 1) & 1, err);
}

// The finished row: the accumulator over the row's sum, as bfloat16, chunks c_lo .. c_hi - 1 of 32 columns.  (Every lane of the
// warp takes part in the loads, also those whose row is not used.)
__device__ __forceinline__ void store_output(uint32_t o_base, bf16* dst, float l_run, bool used, int c_lo, int c_hi) {
  tc_fence_after();
  const float inv = l_run > 0.0f ? 1.0f / l_run : 0.0f;
#pragma unroll 1
  for (int c = c_lo; c < c_hi; ++c) {
    float o[32];
    tmem_ld32(o_base + c * 32, o);
    if (used) {
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4) {
        __align__(16) bf16 y[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) y[e] = __float2bfloat16_rn(o[q4 * 8 + e] * inv);
        *reinterpret_cast<uint4*>(dst + c * 32 + q4 * 8) = *reinterpret_cast<const uint4*>(y);
      }
    }
  }
  tc_fence_before();
}

// The finished pair of rows 2j (even lanes) and 2j + 1: a head's two maps, their difference normed over its 128 values, this
// thread's 64 columns of it (the even lane stores the first 16 of 32, the odd lane the others).  `dst`: the head's place.
__device__ __forceinline__ void store_difference(uint32_t o_base, bf16* dst, float l_run, bool used, const ScoreShape& f,
                                                 const HalfRows& rows, int parity) {
  tc_fence_after();
  const int odd = threadIdx.x & 1;
  const float inv = l_run > 0.0f ? 1.0f / l_run : 0.0f, w = odd ? -f.diff_lambda * inv : inv;
  float d[64];
  tmem_ld64(o_base + rows.c * 64, d);
  float ss = 0.0f;
#pragma unroll
  for (int e = 0; e < 64; ++e) {
    d[e] *= w;
    d[e] += __shfl_xor_sync(0xffffffffu, d[e], 1);
    ss = fmaf(d[e], d[e], ss);
  }
  bool left;
  ss += rows.meet(ss, parity, true, left);
  const float gain = f.diff_gain / sqrtf(ss / static_cast<float>(D) + f.diff_eps);
  if (used) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      __align__(16) bf16 y[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) y[e] = __float2bfloat16_rn((odd ? d[c * 32 + 16 + e] : d[c * 32 + e]) * gain);
      uint4* to = reinterpret_cast<uint4*>(dst + rows.c * 64 + c * 32 + odd * 16);
      to[0] = reinterpret_cast<const uint4*>(y)[0];
      to[1] = reinterpret_cast<const uint4*>(y)[1];
    }
  }
  tc_fence_before();
}

// SHAPED: the forms of ScoreShape, with DIFF the difference of two maps, and two softmax threads a row (warps 2-9, the second
// copy warp behind them); the plain build carries none of that code.
template <bool SHAPED, bool DIFF>
__global__ void __launch_bounds__(SHAPED ? SHAPED_THREADS : THREADS, 1)
prefill_tcgen05_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                       const bf16* __restrict__ q, bf16* __restrict__ out, const int* __restrict__ block_table,
                       int table_stride, const int* __restrict__ cu_q, const int* __restrict__ kv_len,
                       const int* __restrict__ prefix_len, const int* __restrict__ rows, int nh, int nkv, int page_size,
                       int box_rows, int window, float scale_log2, const ScoreShape shape, int* err) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* k_full = reinterpret_cast<uint64_t*>(sm + BAR_OFF);      // [3]
  uint64_t* k_empty = k_full + K_STAGES;                             // [3]
  uint64_t* v_full = k_empty + K_STAGES;                             // [2]
  uint64_t* v_empty = v_full + V_STAGES;                             // [2]
  uint64_t* s_full = v_empty + V_STAGES;                             // [2]
  uint64_t* q_full = s_full + 2;
  uint64_t* p_full = q_full + 1;                                     // [2]: one per score buffer, so that a softmax that runs
  uint64_t* pv_done = p_full + 2;                                    //      a block ahead can never lap the MMA thread's wait
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pv_done + 1);
  constexpr int SOFTMAX_WARPS = SHAPED ? 8 : 4;

  const int warp = same_in_warp(threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < K_STAGES; ++s) { mbar_init(k_full + s, 1); mbar_init(k_empty + s, 1); }
    for (int s = 0; s < V_STAGES; ++s) { mbar_init(v_full + s, 1); mbar_init(v_empty + s, 1); }
    mbar_init(s_full, 1);
    mbar_init(s_full + 1, 1);
    mbar_init(q_full, SOFTMAX_WARPS);
    mbar_init(p_full, SOFTMAX_WARPS);
    mbar_init(p_full + 1, SOFTMAX_WARPS);
    mbar_init(pv_done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    if (SHAPED)
      for (int f = 0; f < 8; ++f) reinterpret_cast<int*>(sm + XCH_OFF)[f] = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = same_in_warp(*tmem_slot);
  pdl_launch_dependents();
  pdl_wait();                                  // q, the step's index arrays and the newest keys and values come from earlier kernels

  // Grid: x = KV head, y = row, z = tile order.  CTAs start in the order x, y, z, and a row's last tiles see the
  // most keys: every row's heaviest tiles start first, over all heads, and the light ones fill the gaps behind them.
  const int row = rows[blockIdx.y];
  const int kvh = blockIdx.x;
  const int group = nh / nkv, head0 = kvh * group;
  const int tile_tokens = BQ / group;
  const int q_begin = cu_q[row], q_len = cu_q[row + 1] - q_begin;
  const int tile = (q_len + tile_tokens - 1) / tile_tokens - 1 - static_cast<int>(blockIdx.z);
  const bool active = tile >= 0;               // (an idle CTA still walks to the end, where tensor memory is freed)
  const int tok0 = active ? tile * tile_tokens : 0;
  const int ntok = active ? min(tile_tokens, q_len - tok0) : 0;
  const int prefix = prefix_len[row];
  const int kv_end = active ? min(kv_len[row], prefix + tok0 + ntok) : 0;
  const int p_lo = prefix + tok0;
  int k_begin = window > 0 ? max(0, p_lo - window + 1) : 0;
  if (SHAPED && shape.chunk > 0) k_begin = max(k_begin, p_lo - p_lo % shape.chunk);
  k_begin -= k_begin % BKV;
  const int nblk = same_in_warp(active ? (kv_end - k_begin + BKV - 1) / BKV : 0);
  const int* table = block_table + static_cast<size_t>(row) * table_stride;

  if (warp == 0 || warp >= 2 + SOFTMAX_WARPS) {
    // ---- copies: COPY_WARPS warps share a block's sub-blocks (box_rows keys each): warp c's lane l fetches the
    // sub-blocks c + COPY_WARPS l, ...  (One SM takes in more through boxes that several warps issue than through
    // as many from one warp: 34 to 37 against 23 GB/s in a probe that only copies pages of 16 keys; all copy warps
    // walk the same stages and wait for the same barriers, the first announces a stage's bytes.  A box that lands
    // before its stage's bytes are announced is no harm: the phase cannot end before the announcing arrival.)
    // Keys run one block further ahead than values (three stages against two): S of block i + 2 is wanted
    // while block i is still in the softmax.
    // The row's page numbers for this tile's keys come into shared memory first: a copy then does not begin with a
    // load from global memory whose answer it needs for its address.
    const int cw = warp == 0 ? 0 : warp - 1 - SOFTMAX_WARPS;
    bool ok = true;
    int* tbl = reinterpret_cast<int*>(sm + TBL_OFF);
    const int first_page = k_begin / page_size;
    const int n_pages = min(TBL_ENTRIES, (kv_end + page_size - 1) / page_size - first_page);
    for (int t = cw * 32 + lane; t < n_pages; t += 32 * COPY_WARPS) tbl[t] = table[first_page + t];
    asm volatile("bar.sync 1, %0;\n" ::"n"(32 * COPY_WARPS) : "memory");      // (the copy warps only)
    auto fetch = [&](const CUtensorMap* map, unsigned char* dst, uint64_t* bar, int first_key) {
      const int n_sub = (min(BKV, kv_end - first_key) + box_rows - 1) / box_rows;
      proxy_fence();
      if (cw == 0 && lane == 0) mbar_expect_tx(bar, static_cast<uint32_t>(n_sub) * 2u * box_rows * 128u);
      __syncwarp();
      for (int j = cw + COPY_WARPS * lane; j < n_sub; j += 32 * COPY_WARPS) {
        const int key0 = first_key + j * box_rows;
        const int pi = key0 / page_size - first_page;
        const int page = pi < TBL_ENTRIES ? tbl[pi] : table[first_page + pi];
        const int y = (page * nkv + kvh) * page_size + key0 % page_size;
        tma_load_2d(dst + j * box_rows * 128, map, 0, y, bar);
        tma_load_2d(dst + HALF + j * box_rows * 128, map, 64, y, bar);
      }
    };
    auto wait_all = [&](uint64_t* bar, uint32_t parity) {        // every lane waits, then the warp agrees
      const bool mine = mbar_wait(bar, parity, err);
      return __all_sync(0xffffffffu, mine ? 1 : 0) != 0;
    };
    int ik = 0;                                                  // next key block to fetch
    for (int i = 0; i < nblk && ok; ++i) {
      for (; ik < nblk && ik <= i + K_STAGES - 1 && ok; ++ik) {
        const int s = ik % K_STAGES, use = ik / K_STAGES;
        if (use > 0) ok = wait_all(k_empty + s, (use - 1) & 1);
        if (ok) fetch(&kmap, sm + K_OFF + s * TILE, k_full + s, k_begin + ik * BKV);
      }
      if (!ok) break;
      const int s = i % V_STAGES, use = i / V_STAGES;
      if (use > 0) ok = wait_all(v_empty + s, (use - 1) & 1);
      if (ok) fetch(&vmap, sm + V_OFF + s * TILE, v_full + s, k_begin + i * BKV);
    }
  } else if (warp == 1) {
    // ---- MMA issue: S_0, S_1; then for every block: O += P V of block i, S of block i + 2
    if (nblk > 0) {
      bool ok = mbar_wait_warp(q_full, 0, err);
      const uint32_t tmem_o = tmem_base + 256;
      // (descriptors differ in their start address only, the low 14 bits in units of 16 bytes, which never carry here)
      const uint64_t dq = desc_k_major(smem_u32(sm + Q_OFF)), dk = desc_k_major(smem_u32(sm + K_OFF)), dv = desc_mn_major(smem_u32(sm + V_OFF));
      auto issue_s = [&](int i) {
        const int s = i % K_STAGES;
        if (!mbar_wait_warp(k_full + s, (i / K_STAGES) & 1, err)) return false;
        tc_fence_after();
        const uint64_t k0 = dk + static_cast<uint32_t>(s * (TILE >> 4));
        const uint32_t tmem_s = tmem_base + (i & 1) * 128;
        if (elect_one()) {
#pragma unroll
          for (int j = 0; j < D / 16; ++j) {
            const uint32_t off = ((j >> 2) * HALF + (j & 3) * 32) >> 4;
            umma(tmem_s, dq + off, k0 + off, kDescQK, j > 0 ? 1u : 0u);
          }
          umma_commit(s_full + (i & 1));
          umma_commit(k_empty + s);
        }
        __syncwarp();
        return true;
      };
      if (ok) ok = issue_s(0);
      if (ok && nblk > 1) ok = issue_s(1);
      for (int i = 0; i < nblk && ok; ++i) {
        const int s = i % V_STAGES;
        ok = mbar_wait_warp(p_full + (i & 1), (i >> 1) & 1, err);      // P of block i lies where S of block i lay
        if (ok) ok = mbar_wait_warp(v_full + s, (i / V_STAGES) & 1, err);
        if (!ok) break;
        tc_fence_after();
        const uint64_t v0 = dv + static_cast<uint32_t>(s * (TILE >> 4));
        const uint32_t tmem_p = tmem_base + (i & 1) * 128, more = i > 0 ? 1u : 0u;
        if (elect_one()) {
#pragma unroll
          for (int j = 0; j < BKV / 16; ++j) umma_a_tmem(tmem_o, tmem_p + j * 8, v0 + j * 128, kDescPV, j > 0 ? 1u : more);
          if (SHAPED && shape.split) {                             // the weights' second terms
#pragma unroll
            for (int j = 0; j < BKV / 16; ++j) umma_a_tmem(tmem_o, tmem_p + 64 + j * 8, v0 + j * 128, kDescPV, 1u);
          }
          umma_commit(pv_done);
          umma_commit(v_empty + s);
        }
        __syncwarp();
        if (i + 2 < nblk) ok = issue_s(i + 2);
      }
    }
  } else {
    // ---- softmax warps: thread r owns query row r of the tile (tensor-memory lane r)
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const int tok = r / group, head = head0 + r % group;
    const bool used = tok < ntok;
    const int qpos = used ? p_lo + tok : -1;
    const int c = SHAPED ? (warp - 2) >> 2 : 0;      // which half of the row's columns (two threads a row)
    constexpr int CHUNKS = SHAPED ? 8 : 16;
    if (nblk > 0) {
      write_q_row<CHUNKS>(sm + Q_OFF, q + (static_cast<size_t>(q_begin + tok0 + tok) * nh + head) * D, r, used, 8 * c);
      __syncwarp();
      if (lane == 0) mbar_arrive(q_full);
    }
    int lo_key = window > 0 ? qpos - window + 1 : 0;
    if (SHAPED && shape.chunk > 0) lo_key = max(lo_key, qpos - qpos % shape.chunk);
    const int hi_key = min(qpos, kv_end - 1);
    // the first key that the tile's last query sees
    int all_see = window > 0 ? p_lo + ntok - window : 0;
    if (SHAPED && shape.chunk > 0) all_see = max(all_see, (p_lo + ntok - 1) - (p_lo + ntok - 1) % shape.chunk);
    RowState st;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    const HalfRows halves = {reinterpret_cast<float*>(sm + XCH_OFF) + 8, reinterpret_cast<volatile int*>(sm + XCH_OFF) + 2 * quarter, c, r, quarter};
    bool ok = true, left = false;
    for (int i = 0; i < nblk; ++i) {
      const int first_key = k_begin + i * BKV;
      if (ok) ok = mbar_wait_warp(s_full + (i & 1), (i >> 1) & 1, err);
      const bool masked = first_key + BKV - 1 > p_lo || first_key + BKV > kv_end || first_key < all_see;
      const uint32_t s_base = lane_base + (i & 1) * 128;
      if (SHAPED)
        ok = softmax_half(ok, s_base, lane_base + 256, first_key, lo_key, hi_key, masked, scale_log2, shape, i, pv_done, halves, st, left, err);
      else if (ok)
        ok = softmax_block(s_base, lane_base + 256, first_key, lo_key, hi_key, masked, scale_log2, i, pv_done, st, err);
      // value rows beyond what the tile may see must not reach P V, whatever the page or the stage held
      if (ok && first_key + BKV > kv_end) {
        const int s = i % V_STAGES;
        ok = mbar_wait_warp(v_full + s, (i / V_STAGES) & 1, err);      // the copies have landed
        if (ok && first_key + r >= kv_end) zero_value_row<CHUNKS>(sm + V_OFF + s * TILE, r, 8 * c);
        proxy_fence();                                                 // the zeroed rows are visible to the tensor cores
      }
      if (!ok) {
        if (!SHAPED || left) break;                                    // (two threads a row leave together, behind a barrier)
        continue;
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full + (i & 1));
    }
    if (ok && nblk > 0) ok = mbar_wait_warp(pv_done, (nblk - 1) & 1, err);
    if constexpr (SHAPED) {
      if (nblk > 0 && !left) {
        st.l_run += halves.meet(st.l_run, nblk & 1, ok, left);         // the row's other half
        if (!left) {
          if (shape.sinks != nullptr && st.l_run > 0.0f) st.l_run += exp2f(shape.sinks[head] * 1.4426950408889634f - st.m_ref);
          if (DIFF)
            store_difference(lane_base + 256, out + (static_cast<size_t>(q_begin + tok0 + tok) * (nh / 2) + head / 2) * D, st.l_run,
                             used, shape, halves, (nblk + 1) & 1);
          else
            store_output(lane_base + 256, out + (static_cast<size_t>(q_begin + tok0 + tok) * nh + head) * D, st.l_run, used, 2 * c, 2 * c + 2);
        }
      }
    } else if (ok && nblk > 0) {
      store_output(lane_base + 256, out + (static_cast<size_t>(q_begin + tok0 + tok) * nh + head) * D, st.l_run, used, 0, 4);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Two query tiles per CTA.  What the kernel above reads per block of keys (K and V, 64 KB from L2) limits it on long
// prompts: the tensor pipe and the softmax wait for the copies.  Here a CTA serves 256 query vectors, two tiles
// A and B of consecutive tokens, and every K and V block is fetched once for both.  Tensor memory holds one score
// buffer and one output accumulator per tile (4 x 128 columns); the MMA thread alternates between the tiles
// (P V of tile A, the next S of tile A, P V of tile B, the next S of tile B), so one tile's products run under the
// other tile's softmax.  Warps 2-5 are tile A's softmax (one thread per query row), warps 6-9 tile B's.
// (Blocks of 64 keys, which leave room for two score buffers per tile, were tried and were slower: twice the
// hand-overs per key.)  A tile's softmax of block b + 1 needs S of block b + 1, which is issued behind P V of block b:
// no barrier of a tile can complete two phases while someone still waits for the first.
constexpr int PAIR_K_STAGES = 2, PAIR_V_STAGES = 2;      // (deeper rings were slower: more copies in flight, same traffic)
constexpr int PAIR_V_OFF = 0, PAIR_K_OFF = PAIR_V_STAGES * TILE, PAIR_Q_OFF = PAIR_K_OFF + PAIR_K_STAGES * TILE;
constexpr int PAIR_BAR_OFF = PAIR_Q_OFF + 2 * TILE;
constexpr int PAIR_N_BARS = 2 * PAIR_K_STAGES + 2 * PAIR_V_STAGES + 2 + 2 + 2 + 2 + 1;
constexpr int PAIR_TBL_OFF = PAIR_BAR_OFF + (PAIR_N_BARS + 1) * 8;
constexpr int PAIR_SMEM_BYTES = PAIR_TBL_OFF + TBL_ENTRIES * 4;

__global__ void __launch_bounds__(PAIR_THREADS, 1)
prefill_tcgen05_pair_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                            const bf16* __restrict__ q, bf16* __restrict__ out, const int* __restrict__ block_table,
                            int table_stride, const int* __restrict__ cu_q, const int* __restrict__ kv_len,
                            const int* __restrict__ prefix_len, const int* __restrict__ rows, int nh, int nkv,
                            int page_size, int box_rows, int window, float scale_log2, int* err) {
  constexpr int KS = PAIR_K_STAGES, VS = PAIR_V_STAGES;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* k_full = reinterpret_cast<uint64_t*>(sm + PAIR_BAR_OFF);
  uint64_t* k_empty = k_full + KS;
  uint64_t* v_full = k_empty + KS;
  uint64_t* v_empty = v_full + VS;
  uint64_t* s_full = v_empty + VS;                                   // [2]: one per tile
  uint64_t* p_full = s_full + 2;                                     // [2]
  uint64_t* p_half = p_full + 2;                                     // [2]: the weights of a block's first 64 keys
  uint64_t* pv_done = p_half + 2;                                    // [2]
  uint64_t* q_full = pv_done + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(q_full + 1);

  const int warp = same_in_warp(threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < KS; ++s) { mbar_init(k_full + s, 1); mbar_init(k_empty + s, 1); }
    for (int s = 0; s < VS; ++s) { mbar_init(v_full + s, 1); mbar_init(v_empty + s, 1); }
    for (int t = 0; t < 2; ++t) { mbar_init(s_full + t, 1); mbar_init(p_full + t, 4); mbar_init(p_half + t, 4); mbar_init(pv_done + t, 1); }
    mbar_init(q_full, 8);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = same_in_warp(*tmem_slot);        // columns: S of tile A 0..127, S of tile B 128..255, O of A 256..383, O of B 384..511
  pdl_launch_dependents();
  pdl_wait();

  // Grid as above, with pairs of tiles in z.
  const int row = rows[blockIdx.y];
  const int kvh = blockIdx.x;
  const int group = nh / nkv, head0 = kvh * group;
  const int tile_tokens = BQ / group, pair_tokens = 2 * tile_tokens;
  const int q_begin = cu_q[row], q_len = cu_q[row + 1] - q_begin;
  const int pair = (q_len + pair_tokens - 1) / pair_tokens - 1 - static_cast<int>(blockIdx.z);
  const bool active = pair >= 0;               // (an idle CTA still walks to the end, where tensor memory is freed)
  const int prefix = prefix_len[row];
  int tok0[2], ntok[2], p_lo[2], kv_end[2], nblk[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    tok0[t] = active ? pair * pair_tokens + t * tile_tokens : 0;
    ntok[t] = active ? max(0, min(tile_tokens, q_len - tok0[t])) : 0;
    p_lo[t] = prefix + tok0[t];
    kv_end[t] = ntok[t] > 0 ? min(kv_len[row], p_lo[t] + ntok[t]) : 0;
  }
  // Both tiles walk the same blocks, from where tile A's window begins; tile B ends at or after tile A.
  int k_begin = window > 0 ? max(0, p_lo[0] - window + 1) : 0;
  k_begin -= k_begin % BKV;
#pragma unroll
  for (int t = 0; t < 2; ++t) nblk[t] = same_in_warp(ntok[t] > 0 ? (kv_end[t] - k_begin + BKV - 1) / BKV : 0);
  const int nblk_all = max(nblk[0], nblk[1]);
  const int kv_end_all = max(kv_end[0], kv_end[1]);
  const int* table = block_table + static_cast<size_t>(row) * table_stride;

  if (warp == 0 || warp >= 10) {
    // ---- copies, as in the kernel above
    const int cw = warp == 0 ? 0 : warp - 9;
    bool ok = true;
    int* tbl = reinterpret_cast<int*>(sm + PAIR_TBL_OFF);
    const int first_page = k_begin / page_size;
    const int n_pages = min(TBL_ENTRIES, (kv_end_all + page_size - 1) / page_size - first_page);
    for (int t = cw * 32 + lane; t < n_pages; t += 32 * PAIR_COPY_WARPS) tbl[t] = table[first_page + t];
    asm volatile("bar.sync 1, %0;\n" ::"n"(32 * PAIR_COPY_WARPS) : "memory");      // (the copy warps only)
    auto fetch = [&](const CUtensorMap* map, unsigned char* dst, uint64_t* bar, int first_key) {
      const int n_sub = (min(BKV, kv_end_all - first_key) + box_rows - 1) / box_rows;
      proxy_fence();
      if (cw == 0 && lane == 0) mbar_expect_tx(bar, static_cast<uint32_t>(n_sub) * 2u * box_rows * 128u);
      __syncwarp();
      for (int j = cw + PAIR_COPY_WARPS * lane; j < n_sub; j += 32 * PAIR_COPY_WARPS) {
        const int key0 = first_key + j * box_rows;
        const int pi = key0 / page_size - first_page;
        const int page = pi < TBL_ENTRIES ? tbl[pi] : table[first_page + pi];
        const int y = (page * nkv + kvh) * page_size + key0 % page_size;
        tma_load_2d(dst + j * box_rows * 128, map, 0, y, bar);
        tma_load_2d(dst + HALF + j * box_rows * 128, map, 64, y, bar);
      }
    };
    int ik = 0;
    for (int i = 0; i < nblk_all && ok; ++i) {
      for (; ik < nblk_all && ik <= i + KS - 1 && ok; ++ik) {
        const int s = ik % KS, use = ik / KS;
        if (use > 0) ok = mbar_wait_warp(k_empty + s, (use - 1) & 1, err);
        if (ok) fetch(&kmap, sm + PAIR_K_OFF + s * TILE, k_full + s, k_begin + ik * BKV);
      }
      if (!ok) break;
      const int s = i % VS, use = i / VS;
      if (use > 0) ok = mbar_wait_warp(v_empty + s, (use - 1) & 1, err);
      if (ok) fetch(&vmap, sm + PAIR_V_OFF + s * TILE, v_full + s, k_begin + i * BKV);
    }
  } else if (warp == 1) {
    // ---- MMA issue
    if (nblk_all > 0) {
      bool ok = mbar_wait_warp(q_full, 0, err);
      // (descriptors differ in their start address only, the low 14 bits in units of 16 bytes, which never carry here)
      const uint64_t dq = desc_k_major(smem_u32(sm + PAIR_Q_OFF)), dk = desc_k_major(smem_u32(sm + PAIR_K_OFF)), dv = desc_mn_major(smem_u32(sm + PAIR_V_OFF));
      // S of tile t over key block b; the block's last user gives the stage back
      auto issue_s = [&](int t, int b) {                         // (t is a constant at every call)
        const int s = b % KS;
        if (!mbar_wait_warp(k_full + s, (b / KS) & 1, err)) return false;
        tc_fence_after();
        const uint64_t q0 = dq + static_cast<uint32_t>(t * (TILE >> 4)), k0 = dk + static_cast<uint32_t>(s * (TILE >> 4));
        const bool last = t == 1 || b >= nblk[1];
        if (elect_one()) {
#pragma unroll
          for (int j = 0; j < D / 16; ++j) {
            const uint32_t off = ((j >> 2) * HALF + (j & 3) * 32) >> 4;
            umma(tmem_base + t * 128, q0 + off, k0 + off, kDescQK, j > 0 ? 1u : 0u);
          }
          umma_commit(s_full + t);
          if (last) umma_commit(k_empty + s);
        }
        __syncwarp();
        return true;
      };
      if (ok && nblk[0] > 0) ok = issue_s(0, 0);
      if (ok && nblk[1] > 0) ok = issue_s(1, 0);
      for (int b = 0; b < nblk_all && ok; ++b) {
        const int s = b % VS;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (!ok || b >= nblk[t]) continue;
          ok = mbar_wait_warp(p_half + t, b & 1, err);            // P of block b lies where S of block b lay
          if (ok) ok = mbar_wait_warp(v_full + s, (b / VS) & 1, err);
          if (!ok) continue;
          tc_fence_after();
          const uint64_t v0 = dv + static_cast<uint32_t>(s * (TILE >> 4));
          const uint32_t tmem_o = tmem_base + 256 + t * 128, tmem_p = tmem_base + t * 128, more = b > 0 ? 1u : 0u;
          const bool last = t == 1 || b >= nblk[1];
          if (elect_one()) {
#pragma unroll
            for (int j = 0; j < BKV / 32; ++j) umma_a_tmem(tmem_o, tmem_p + j * 8, v0 + j * 128, kDescPV, j > 0 ? 1u : more);
          }
          __syncwarp();
          ok = mbar_wait_warp(p_full + t, b & 1, err);            // the weights of the other 64 keys
          if (!ok) continue;
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (int j = BKV / 32; j < BKV / 16; ++j) umma_a_tmem(tmem_o, tmem_p + j * 8, v0 + j * 128, kDescPV, 1u);
            umma_commit(pv_done + t);
            if (last) umma_commit(v_empty + s);
          }
          __syncwarp();
          if (b + 1 < nblk[t]) ok = issue_s(t, b + 1);
        }
      }
    }
  } else {
    // ---- softmax warps: thread (tile t, row r) owns one query row (tensor-memory lane r of the tile's columns)
    const int t = (warp - 2) >> 2, quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const int tok = r / group, head = head0 + r % group;
    const int my_tok0 = t ? tok0[1] : tok0[0], my_ntok = t ? ntok[1] : ntok[0], my_p_lo = t ? p_lo[1] : p_lo[0];
    const int my_kv_end = t ? kv_end[1] : kv_end[0], my_blocks = t ? nblk[1] : nblk[0];
    const bool used = tok < my_ntok;
    const int qpos = used ? my_p_lo + tok : -1;
    if (nblk_all > 0) {
      // (zeros for an unused row, and for all rows of a tile without tokens)
      write_q_row<16>(sm + PAIR_Q_OFF + t * TILE, q + (static_cast<size_t>(q_begin + my_tok0 + tok) * nh + head) * D, r, used, 0);
      __syncwarp();
      if (lane == 0) mbar_arrive(q_full);
    }
    const int lo_key = window > 0 ? qpos - window + 1 : 0, hi_key = min(qpos, my_kv_end - 1);
    RowState st;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t s_base = lane_base + t * 128, o_base = lane_base + 256 + t * 128;
    bool ok = true;
    for (int b = 0; b < my_blocks && ok; ++b) {
      const int first_key = k_begin + b * BKV;
      if (!mbar_wait_warp(s_full + t, b & 1, err)) { ok = false; break; }
      const bool masked = first_key + BKV - 1 > my_p_lo || first_key + BKV > my_kv_end ||
                          (window > 0 && first_key <= my_p_lo + my_ntok - 1 - window);
      // Value rows beyond what the CTA may see must not reach P V, whatever the page or the stage held.  Both tiles
      // write the same zeros, each before its own product.
      if (first_key + BKV > kv_end_all) {
        const int s = b % VS;
        ok = mbar_wait_warp(v_full + s, (b / VS) & 1, err);
        if (!ok) break;
        if (first_key + r >= kv_end_all) zero_value_row<16>(sm + PAIR_V_OFF + s * TILE, r, 0);
        proxy_fence();
      }
      softmax_row(s_base, o_base, first_key, lo_key, hi_key, masked, scale_log2, b, st, [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_half + t);
      });
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full + t);
    }
    // (S of the last block was issued behind P V of the one before it: only this phase can be the one that runs)
    if (ok && my_blocks > 0) ok = mbar_wait_warp(pv_done + t, (my_blocks - 1) & 1, err);
    if (ok && my_blocks > 0)
      store_output(o_base, out + (static_cast<size_t>(q_begin + my_tok0 + tok) * nh + head) * D, st.l_run, used, 0, 4);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

B200_EXPORT int b200_attention_tcgen05_head_dim() { return D; }

// How many launches took the one-tile kernel (plain), the two-tile kernel and the one-tile kernel's further forms so far
// (tests ask which path a model reached).
static long long g_launches[3] = {0, 0, 0};
B200_EXPORT long long b200_attention_tcgen05_launches(int kind) { return g_launches[kind < 0 || kind > 2 ? 0 : kind]; }

// Portions of prompts over a bfloat16 cache, head size 128; the number of query heads per KV head must divide 128
// and the page size must be a power of two.  `k_map`, `v_map`: descriptors of b200_kv_tensor_map (attention_mma.cu)
// with box_rows = min(page_size, 32).  Other arguments as b200_prefill_attention of attention.cu.
// `variant`: 1 = one tile of 128 query vectors per CTA, 2 = two tiles per CTA, 0 = two tiles when the longest
// row then still gives every SM a CTA (pairs halve the traffic per query but also the number of CTAs).
// `softcap` > 0, `split_p`, `chunk` > 0, `sinks` and `diff` (lambda, gain, eps; group even, no sinks): see ScoreShape; any of
// them takes the one-tile kernel's further forms.  `scale` > 0; q and out on 16-byte boundaries.
B200_EXPORT int b200_prefill_attention_tcgen05(const void* q, const void* k_map, const void* v_map, void* out,
                                               const int* block_table, int table_stride, const int* cu_q,
                                               const int* kv_len, const int* prefix_len, const int* rows, int n_rows,
                                               int max_q_len, int nh, int nkv, int page_size, int window, float scale,
                                               int variant, float softcap, int split_p, int chunk, const float* sinks,
                                               const float* diff, int* err, cudaStream_t stream) {
  if (n_rows <= 0 || max_q_len <= 0) return 0;
  if (nh <= 0 || nkv <= 0 || nh % nkv != 0 || page_size <= 0 || (page_size & (page_size - 1)) != 0) return B200_BAD_SIZE;
  if (variant < 0 || variant > 2) return B200_BAD_SIZE;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out)) % 16 != 0) return B200_BAD_ALIGN;
  const int group = nh / nkv;
  if (group > BQ || BQ % group != 0) return B200_BAD_SIZE;
  const int box_rows = page_size < 32 ? page_size : 32;
  const int tile_tokens = BQ / group;
  static int sm_count = 0;
  if (sm_count == 0) {
    int dev = 0, n = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return static_cast<int>(e);
    sm_count = n;
  }
  const bool shaped = softcap > 0.0f || split_p != 0 || chunk > 0 || sinks != nullptr || diff != nullptr;
  if (!(scale > 0.0f)) return B200_BAD_SIZE;                         // maxima and masks are taken of the unscaled scores
  if (shaped && (variant == 2 || (diff != nullptr && (group % 2 != 0 || sinks != nullptr)))) return B200_BAD_SIZE;
  const int n_pairs = (max_q_len + 2 * tile_tokens - 1) / (2 * tile_tokens);
  const bool pairs = variant == 2 || (variant == 0 && !shaped && static_cast<long long>(n_pairs) * nkv * n_rows >= sm_count);
  const size_t smem = 1024 + (pairs ? PAIR_SMEM_BYTES : shaped ? SHAPED_SMEM_BYTES : SMEM_BYTES);
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaSuccess;
    for (auto one : {prefill_tcgen05_kernel<false, false>, prefill_tcgen05_kernel<true, false>, prefill_tcgen05_kernel<true, true>})
      if (e == cudaSuccess) e = cudaFuncSetAttribute(one, cudaFuncAttributeMaxDynamicSharedMemorySize, 1024 + SHAPED_SMEM_BYTES);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(prefill_tcgen05_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 1024 + PAIR_SMEM_BYTES);
    if (e != cudaSuccess) return static_cast<int>(e);
    configured = true;
  }
  CUtensorMap kmap, vmap;
  memcpy(&kmap, k_map, sizeof(kmap));
  memcpy(&vmap, v_map, sizeof(vmap));
  const int n_tiles = pairs ? n_pairs : (max_q_len + tile_tokens - 1) / tile_tokens;
  if (n_rows > 65535 || n_tiles > 65535) return B200_BAD_SIZE;      // the grid's y and z extents
  dim3 grid(nkv, n_rows, n_tiles);
  ++g_launches[shaped ? 2 : pairs ? 1 : 0];
  const float scale_log2 = scale * 1.4426950408889634f;
  if (pairs)
    return b200_launch(prefill_tcgen05_pair_kernel, grid, dim3(PAIR_THREADS), smem, stream, 0, kmap, vmap, static_cast<const bf16*>(q),
                       static_cast<bf16*>(out), block_table, table_stride, cu_q, kv_len, prefix_len, rows, nh, nkv, page_size,
                       box_rows, window, scale_log2, err);
  ScoreShape shape = {};
  if (softcap > 0.0f) { shape.cap_log2 = softcap * 1.4426950408889634f; shape.tanh_in = scale / softcap; }
  shape.split = split_p;
  shape.chunk = chunk;
  shape.sinks = sinks;
  if (diff != nullptr) { shape.diff_lambda = diff[0]; shape.diff_gain = diff[1]; shape.diff_eps = diff[2]; }
  auto kernel = diff != nullptr ? prefill_tcgen05_kernel<true, true> : shaped ? prefill_tcgen05_kernel<true, false> : prefill_tcgen05_kernel<false, false>;
  return b200_launch(kernel, grid, dim3(shaped ? SHAPED_THREADS : THREADS), smem, stream, 0, kmap, vmap, static_cast<const bf16*>(q),
                     static_cast<bf16*>(out), block_table, table_stride, cu_q, kv_len, prefix_len, rows, nh, nkv, page_size,
                     box_rows, window, scale_log2, shape, err);
}
