// C[M, N] = A[M, K] . W[N, K]^T in true 32-bit: no reduced-precision mode.  This is the matrix product of the
// float32 engine (the reference's float path goes through libtorch matmul: src/layers/linear.rs:5-7).
//
// Products whose rows are whole 16-byte pieces run on the tensor cores in terms: a float is the exact sum of three bfloat16
// numbers (8 + 8 + 8 bits), the product of two floats the sum of nine products of terms, each exact in float, and the six that
// reach 2^-24 of it are taken.  32 k are summed by the tensor cores from zero, small products first (what an addition there cuts off
// below a sum's last place stays that of 32 terms); those sums are added in float, an eighth of K (a span) in order, then the eight
// spans in order.  That order depends on k alone and the kernels keep to it, split_kernel (tcgen05: many rows), few_split_kernel and
// pair_split_kernel (mma.sync, which gives the same bits: the tests compare them), so a token's result is bit-identical however the
// batch around it is cut.  Error against 64 bits 0.9e-7 of a product's norm (K = 1,024; FFMA in short sums 2.1e-7, in one chain 2.1e-6 for a model's
// logits).  An element whose terms give no finite sum (an infinity has no second term) is summed again by FFMA, and so is one
// below 2^-80: numbers below 2^-110 lose bits of their third term, for which bfloat16 ends at 2^-133.  (What is left: such numbers
// times others above 2^30, and products that vanish as a whole, below 2^-133.)
// Measured, us with FFMA tiles / in terms, layers of Qwen3-0.6B: QKV at 4, 32 and 300 rows 9.9 / 5.5, 41.7 / 11.0, 119 / 39 (65 of an
// ideal 274 TFLOP/s: the terms are taken apart and the sums added up by CUDA cores), O 6.4 / 5.0, 40.8 / 9.7, 63 / 35, gate and up 11.0 / 7.3,
// 43.2 / 15.6, 127 / 40, down 7.4 / 6.5, 40.8 / 13.6, 65 / 43.
//
// Other products (K or a distance between rows no multiple of four, unaligned pointers) and batched ones keep to FFMA on CUDA cores,
// in an order of their own that depends on k alone as well: K is cut into chunks of 128 and spans of four chunks; a chunk is summed
// over k in order, a span over its chunks in order, an element over its spans in order.
//
// few_rows_kernel (few rows): bound by reading W.  A warp takes 8 rows of W and one span: lane = (row of W, chunk), so
//   the span's chunks are summed side by side and a product of 1,024 x 2,048 still has 512 warps at work.  W comes
//   through a ring of four cp.async stages that only its own warp reads (no block-wide barrier on the way); the rows of x
//   wait in shared memory.
// tiled_kernel (many rows): bound by the FFMA units.  64 x 64 tiles by two warps, 8 x 8 elements a thread: four 16-byte
//   loads of shared memory for 64 FFMA (4 x 8 elements a thread as packed f32x2 pairs, with one operand stored twice, took
//   half again as many loads: 25 against 32 TFLOP/s at 1,000 rows).  The blocks of a cluster take different spans of one tile and add
//   them up in order through distributed shared memory.
// Measured on what is left to them, sixteen products a launch: 4 rows of 128 x 256 5.8 us, 300 rows 22.1 (14 TFLOP/s), 300 of 512 x 128
// 33.1 (19); eight of 1,500 rows of 320 x 320 79.1 (31 TFLOP/s).
//
// The batched form multiplies `batch` independent pairs whose rows may lie apart (leading dimensions lda, ldw, ldc
// and a distance between consecutive matrices of each operand): per-head products of a mixer, where head h's rows are
// column ranges of wider matrices.
#include <cooperative_groups.h>
#include <cuda.h>

#include <initializer_list>
#include <type_traits>

#include "common.cuh"

namespace cg = cooperative_groups;

constexpr int CHUNK = 128, SPAN = 512;          // k a partial sum, k a sum of partial sums

struct Product {
  const float* a;
  const float* w;
  float* c;
  int m, n, k, lda, ldw, ldc;
  long long step_a, step_w, step_c;
};

// ------------------------------------------------------------------ few rows
constexpr int FEW_WN = 8;                       // rows of W a warp
constexpr int FEW_KS = 32;                      // k of every chunk a stage
constexpr int FEW_STAGES = SPAN / CHUNK == 4 ? CHUNK / FEW_KS : 0;
constexpr int FEW_ROW = (SPAN / CHUNK) * FEW_KS + 4;      // floats of a row of W in a stage: 8 rows lie in different banks
constexpr int FEW_STAGE = FEW_WN * FEW_ROW;
constexpr int FEW_XCHUNK = CHUNK + 4;           // the four chunks of a span lie in different banks
static_assert(FEW_STAGES == 4, "a span is four chunks, one stage of the ring holds a quarter of each");

// Asks for the part of W that stage `st` of a warp's span takes: rows n0 .. n0 + 7, of every chunk 32 k.
template <bool VEC>
__device__ __forceinline__ void few_fetch(float* dst, const float* __restrict__ w, int n, int k, int ldw, int n0, int k0, int lane) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int piece = lane + 32 * j, quad = piece & 7, chunk = (piece >> 3) & 3, row = piece >> 5;
    const int kk = k0 + chunk * CHUNK + quad * 4;
    float* to = dst + row * FEW_ROW + chunk * FEW_KS + quad * 4;
    if (VEC) {
      const bool valid = n0 + row < n && kk < k;
      cp_async16(to, valid ? w + static_cast<size_t>(n0 + row) * ldw + kk : w, valid);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        to[e] = n0 + row < n && kk + e < k ? w[static_cast<size_t>(n0 + row) * ldw + kk + e] : 0.0f;
    }
  }
}

// grid (blocks, groups of MR rows, batch); SW warps share a tile of 8 columns (one span each), a block holds NT tiles.
template <int MR, bool VEC>
__global__ void __launch_bounds__(256)
few_rows_kernel(const Product p, int sw, int nt) {
  extern __shared__ __align__(16) float few_smem[];
  const int warps = sw * nt, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* xs = few_smem;                                             // [MR][4 sw chunks][132]
  const int x_row = 4 * sw * FEW_XCHUNK;
  float* red = xs + MR * x_row;                                     // [2][warps][8][MR]
  float* ring = red + 2 * warps * FEW_WN * MR + warp * FEW_STAGES * FEW_STAGE;
  const float* a = p.a + blockIdx.z * p.step_a;
  const float* w = p.w + blockIdx.z * p.step_w;
  float* c = p.c + blockIdx.z * p.step_c;
  const int m0 = blockIdx.y * MR;
  const int spans = (p.k + SPAN - 1) / SPAN, rounds = (spans + sw - 1) / sw;
  const int groups = (p.n + FEW_WN * nt - 1) / (FEW_WN * nt);
  const int my_span = warp % sw, my_tile = warp / sw;
  const int row = lane & 7, chunk = lane >> 3;
  const int mine = blockIdx.x < groups ? (groups - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  const int steps = mine * rounds * FEW_STAGES;                     // of this warp: tiles, then rounds, then stages

  auto fetch = [&](int step) {
    if (step < steps) {
      const int stage = step % FEW_STAGES, unit = step / FEW_STAGES, round = unit % rounds, g = blockIdx.x + unit / rounds * gridDim.x;
      few_fetch<VEC>(ring + stage * FEW_STAGE, w, p.n, p.k, p.ldw, (g * nt + my_tile) * FEW_WN,
                     (round * sw + my_span) * SPAN + stage * FEW_KS, lane);
    }
    cp_async_commit();
  };
  auto fetch_rows = [&](int round) {                                // the rows of x for a round's spans
    const int k0 = round * sw * SPAN, quads = sw * (SPAN / 4);
    for (int i = threadIdx.x; i < MR * quads; i += blockDim.x) {
      const int r = i / quads, kk = (i - r * quads) * 4;
      float* to = xs + r * x_row + (kk / CHUNK) * FEW_XCHUNK + kk % CHUNK;
      const float* src = a + static_cast<size_t>(m0 + r) * p.lda + k0 + kk;
      if (VEC) {
        const bool valid = m0 + r < p.m && k0 + kk < p.k;
        cp_async16(to, valid ? src : a, valid);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) to[e] = m0 + r < p.m && k0 + kk + e < p.k ? src[e] : 0.0f;
      }
    }
  };
  fetch_rows(0);                                                    // (part of the first stage's group of copies)
#pragma unroll
  for (int s = 0; s < FEW_STAGES; ++s) fetch(s);
  cp_async_wait<FEW_STAGES - 1>();
  __syncthreads();

  int step = 0, parity = 0;
  for (int g = blockIdx.x; g < groups; g += gridDim.x) {
    float total = 0.0f;                                             // with several rounds a thread has one element at most
    for (int round = 0; round < rounds; ++round, parity ^= 1) {
      if (rounds > 1 && step > 0) {
        __syncthreads();                                            // the last round's rows have been read
        fetch_rows(round);
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
      }
      float acc[MR];
#pragma unroll
      for (int r = 0; r < MR; ++r) acc[r] = 0.0f;
      const float* xc = xs + (my_span * 4 + chunk) * FEW_XCHUNK;
#pragma unroll
      for (int s = 0; s < FEW_STAGES; ++s, ++step) {
        cp_async_wait<FEW_STAGES - 1>();
        __syncwarp();
        const float* ws = ring + s * FEW_STAGE + row * FEW_ROW + chunk * FEW_KS;
#pragma unroll
        for (int q = 0; q < FEW_KS; q += 4) {
          const float4 wv = *reinterpret_cast<const float4*>(ws + q);
#pragma unroll
          for (int r = 0; r < MR; ++r) {
            const float4 xv = *reinterpret_cast<const float4*>(xc + r * x_row + s * FEW_KS + q);
            acc[r] = fmaf(xv.x, wv.x, acc[r]);
            acc[r] = fmaf(xv.y, wv.y, acc[r]);
            acc[r] = fmaf(xv.z, wv.z, acc[r]);
            acc[r] = fmaf(xv.w, wv.w, acc[r]);
          }
        }
        __syncwarp();                                               // the stage has been read
        fetch(step + FEW_STAGES);
      }
      float* mine_red = red + (parity * warps + warp) * FEW_WN * MR;
#pragma unroll
      for (int r = 0; r < MR; ++r) {                                // the span: its chunks in order
        float t = __shfl_sync(0xffffffffu, acc[r], row);
#pragma unroll
        for (int q = 1; q < 4; ++q) t += __shfl_sync(0xffffffffu, acc[r], row + 8 * q);
        if (chunk == r % 4) mine_red[row * MR + r] = t;
      }
      __syncthreads();
      const int here = min(sw, spans - round * sw);
      for (int i = threadIdx.x; i < nt * FEW_WN * MR; i += blockDim.x) {      // the element: its spans in order
        const int tile = i / (FEW_WN * MR), at = i - tile * FEW_WN * MR;
        const float* src = red + (parity * warps + tile * sw) * FEW_WN * MR + at;
        float t = rounds > 1 ? total : 0.0f;
        for (int s = 0; s < here; ++s) t += src[s * FEW_WN * MR];
        if (rounds > 1) total = t;
        if (round == rounds - 1) {
          const int col = at / MR, r = m0 + at % MR, n = (g * nt + tile) * FEW_WN + col;
          if (r < p.m && n < p.n) c[static_cast<size_t>(r) * p.ldc + n] = t;
        }
      }
    }
  }
  cp_async_wait<0>();
}

// ------------------------------------------------------------------ many rows
constexpr int BM = 64, BN = 64, BK = 16, TILED_THREADS = 64;

// grid (column tiles x cluster, row tiles, batch).
template <bool VEC>
__global__ void __launch_bounds__(TILED_THREADS, 4)
tiled_kernel(const Product p, int ksplit) {
  // Both operands lie k-major ([buffer][A or W][k][row]).  Groups of four rows are exchanged by k (group ^ 2 x quad of k), so
  // that the transposing stores of a warp (8 rows x 4 quads) meet no bank twice; the loads keep their one pass.
  __shared__ __align__(16) float operands[2][2][BK][BM];
  static_assert(BM == BN && sizeof(operands) == BM * BN * sizeof(float), "a span's sums are handed over where the operands were");
  const float* a = p.a + blockIdx.z * p.step_a;
  const float* w = p.w + blockIdx.z * p.step_w;
  float* c = p.c + blockIdx.z * p.step_c;
  const int rank = blockIdx.x % ksplit;
  const int n0 = blockIdx.x / ksplit * BN, m0 = blockIdx.y * BM;
  const int tid = threadIdx.x, tx = tid & 7, ty = (tid >> 3) & 3, half = tid >> 5;      // warp: 32 rows x 64 columns
  const int quad = tid & 3, line = tid >> 2;                         // this thread fetches rows line, + 16, + 32, + 48
  const int spans = (p.k + SPAN - 1) / SPAN, rounds = (spans + ksplit - 1) / ksplit;
  // the thread's elements: rows row_of(0 .. 7), columns col_of(0 .. 7)
  auto row_of = [&](int i) { return half * 32 + (i >> 2) * 16 + ty * 4 + (i & 3); };
  auto col_of = [&](int j) { return (j >> 2) * 32 + tx * 4 + (j & 3); };

  float4 fa[4], fw[4];
  auto fetch_one = [&](float4& f, const float* src, bool row_ok, int kk) {
    f = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!row_ok) return;
    if (VEC) {
      if (kk < p.k) f = *reinterpret_cast<const float4*>(src);
    } else {
      if (kk < p.k) f.x = src[0];
      if (kk + 1 < p.k) f.y = src[1];
      if (kk + 2 < p.k) f.z = src[2];
      if (kk + 3 < p.k) f.w = src[3];
    }
  };
  auto fetch = [&](int k0) {
    const int kk = k0 + quad * 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int m = m0 + line + 16 * i, n = n0 + line + 16 * i;
      fetch_one(fa[i], a + static_cast<size_t>(m) * p.lda + kk, m < p.m, kk);
      fetch_one(fw[i], w + static_cast<size_t>(n) * p.ldw + kk, n < p.n, kk);
    }
  };
  auto stage = [&](int buf) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = line + 16 * i, at = (((r >> 2) ^ (2 * quad)) << 2) | (r & 3);
      const float va[4] = {fa[i].x, fa[i].y, fa[i].z, fa[i].w}, vw[4] = {fw[i].x, fw[i].y, fw[i].z, fw[i].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        operands[buf][0][quad * 4 + e][at] = va[e];
        operands[buf][1][quad * 4 + e][at] = vw[e];
      }
    }
  };

  for (int round = 0; round < rounds; ++round) {
    const int span = round * ksplit + rank;
    const int k_lo = span * SPAN, k_hi = min(p.k, k_lo + SPAN);      // no k at all: this block has no span in this round
    float acc[8][8], sum[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = sum[i][j] = 0.0f;
    if (k_lo < k_hi) {
      fetch(k_lo);
      stage(0);
      __syncthreads();
      int buf = 0;
      for (int k0 = k_lo; k0 < k_hi; k0 += BK, buf ^= 1) {
        if (k0 + BK < k_hi) fetch(k0 + BK);
#pragma unroll
        for (int k = 0; k < BK; ++k) {
          const int swap = 2 * (k >> 2);
          const float* pa = operands[buf][0][k];
          const float* pw = operands[buf][1][k];
          const float4 a0 = *reinterpret_cast<const float4*>(pa + ((half * 8 + ty) ^ swap) * 4);
          const float4 a1 = *reinterpret_cast<const float4*>(pa + ((half * 8 + 4 + ty) ^ swap) * 4);
          const float4 w0 = *reinterpret_cast<const float4*>(pw + (tx ^ swap) * 4);
          const float4 w1 = *reinterpret_cast<const float4*>(pw + ((8 + tx) ^ swap) * 4);
          const float ar[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
          const float wr[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(ar[i], wr[j], acc[i][j]);
        }
        if ((k0 + BK - k_lo) % CHUNK == 0 || k0 + BK >= k_hi) {      // a chunk is complete
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) { sum[i][j] += acc[i][j]; acc[i][j] = 0.0f; }
        }
        if (k0 + BK < k_hi) stage(buf ^ 1);
        __syncthreads();
      }
    }
    if (ksplit == 1) {
      // the spans one after the other, the sum so far in C (every element has one thread)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int m = m0 + row_of(i);
        if (m >= p.m) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int n = n0 + col_of(j);
          float* dst = c + static_cast<size_t>(m) * p.ldc + n;
          if (n < p.n) *dst = round > 0 ? *dst + sum[i][j] : sum[i][j];
        }
      }
      continue;
    }
    // One span a block: every block adds up its share of the tile's elements over the blocks, in order.
    cg::cluster_group cluster = cg::this_cluster();
    float* tile = &operands[0][0][0][0];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; j += 4)
        *reinterpret_cast<float4*>(tile + row_of(i) * BN + col_of(j)) = make_float4(sum[i][j], sum[i][j + 1], sum[i][j + 2], sum[i][j + 3]);
    cluster.sync();
    const int here = min(ksplit, spans - round * ksplit);
    for (int i = rank * TILED_THREADS + tid; i < BM * BN / 4; i += ksplit * TILED_THREADS) {
      const int m = m0 + i / (BN / 4), n = n0 + i % (BN / 4) * 4;
      float4 parts[8];
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s < here) parts[s] = reinterpret_cast<const float4*>(cluster.map_shared_rank(tile, s))[i];
      float t[4] = {0.f, 0.f, 0.f, 0.f};
      if (m >= p.m) continue;
      float* dst = c + static_cast<size_t>(m) * p.ldc + n;
      if (round > 0)
#pragma unroll
        for (int e = 0; e < 4; ++e) t[e] = n + e < p.n ? dst[e] : 0.0f;
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s < here) { t[0] += parts[s].x; t[1] += parts[s].y; t[2] += parts[s].z; t[3] += parts[s].w; }
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (n + e < p.n) dst[e] = t[e];
    }
    cluster.sync();                                                  // the tile is read: it may be filled again, or the block end
  }
}

// ------------------------------------------------------------------ many rows, in terms
constexpr int SP_BN = 128, SP_KS = 32, SP_SPANS = 8;                // rows of W a tile, k a stage, spans an element at most
constexpr int SP_W_BYTES = SP_BN * SP_KS * 4;

__device__ __forceinline__ void sp_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void sp_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void sp_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void sp_load(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n"
               ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y) : "memory");
}
template <bool ADDS>
__device__ __forceinline__ void sp_mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
               ::"r"(d), "r"(a), "l"(b), "r"(idesc), "n"(ADDS ? 1 : 0) : "memory");
}
__device__ __forceinline__ bool elect_one() {                       // true in one lane of a whole warp
  uint32_t is;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.b32 %0, 1, 0, p;\n}\n" : "=r"(is));
  return is != 0;
}
__device__ __forceinline__ void sp_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void sp_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void sp_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void sp_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void sp_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void sp_st(uint32_t at, const uint32_t (&v)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(at), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ void sp_st(uint32_t at, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n"
               ::"r"(at), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
__device__ __forceinline__ void sp_ld8(uint32_t at, uint32_t* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(at) : "memory");
}
__device__ __forceinline__ void sp_ld16(uint32_t at, uint32_t* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
               "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                 "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
               : "r"(at) : "memory");
}

// Two floats as three bfloat16 terms each, packed (the first float in the low half): x = high + mid + low exactly, each term
// the rest rounded to eight bits.  (Rounded, not cut off: the products that are left out then have no common sign.  A value
// that rounds to infinity gives no finite sum.)
__device__ __forceinline__ void sp_split(float x, float y, uint32_t& high, uint32_t& mid, uint32_t& low) {
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(high) : "f"(y), "f"(x));
  x -= __uint_as_float(high << 16);
  y -= __uint_as_float(high & 0xffff0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(mid) : "f"(y), "f"(x));
  x -= __uint_as_float(mid << 16);
  y -= __uint_as_float(mid & 0xffff0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(low) : "f"(y), "f"(x));
}

// Elements for which the terms give no number (an infinity has no second term), or a very small one, are summed again in FFMA, by whole warps: a lane
// takes every 32nd piece of four k, the 32 sums meet by halves.  Lane `l` of the warp that calls this has element (m, n) of C and
// its sum t; it gets t back, or the new sum where `again`.  A row of x that holds a NaN has NaN everywhere and is found in one pass over it: behind
// the first NaN of a prompt's rows every element of theirs comes here.  (One thread an element, down its row of W alone, would
// hold a tile of 128 x 128 up for tens of milliseconds at K = 12,288, by estimate.)
__device__ __forceinline__ bool sp_settled(float t) {
  const float size = fabsf(t);
  return size <= 3.402823466e38f && (size >= 8.2718061e-25f || size == 0.0f);      // (2^-80; a NaN compares false)
}
__device__ __noinline__ float sp_again(const float* __restrict__ a, int lda, const float* __restrict__ w, int ldw, int k, int m, int n, float t, bool again) {
  const int lane = threadIdx.x & 31;
  unsigned todo = __ballot_sync(0xffffffffu, again);
  int looked_at = -1;
  while (todo != 0) {
    const int j = __ffs(todo) - 1, jm = __shfl_sync(0xffffffffu, m, j), jn = __shfl_sync(0xffffffffu, n, j);
    const float4* x = reinterpret_cast<const float4*>(a + static_cast<size_t>(jm) * lda);
    if (jm != looked_at) {
      looked_at = jm;
      bool nan = false;
#pragma unroll 4
      for (int i = lane; i < k / 4; i += 32) {
        const float4 v = x[i];
        nan = nan || v.x != v.x || v.y != v.y || v.z != v.z || v.w != v.w;
      }
      if (__any_sync(0xffffffffu, nan)) {
        if (again && m == jm) t = __int_as_float(0x7fffffff);
        todo &= ~__ballot_sync(0xffffffffu, m == jm);
        continue;
      }
    }
    const float4* y = reinterpret_cast<const float4*>(w + static_cast<size_t>(jn) * ldw);
    float sum = 0.0f;
#pragma unroll 4
    for (int i = lane; i < k / 4; i += 32) {
      const float4 u = x[i], v = y[i];
      sum = fmaf(u.w, v.w, fmaf(u.z, v.z, fmaf(u.y, v.y, fmaf(u.x, v.x, sum))));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == j) t = sum;
    todo &= todo - 1;
  }
  return t;
}
// The same of what this warp has stored as row m of C, columns n0 to n0 + 31 (and on, in steps of 32, up to `columns`).
__device__ __forceinline__ void sp_stored_again(const Product& p, int m, int n0, int columns) {
  for (int n = n0 + (threadIdx.x & 31); n < n0 + columns; n += 32) {
    float* at = p.c + static_cast<size_t>(m) * p.ldc + n;
    const float v = n < p.n ? *at : 0.0f;
    const bool again = !sp_settled(v);
    const float t = sp_again(p.a, p.lda, p.w, p.ldw, p.k, m, n, v, again);
    if (again) *at = t;
  }
}

template <int NT> struct SplitShape {
  static constexpr int WARPS = 16;                                  // that take terms apart and add sums up
  static constexpr int THREADS = (WARPS + 2) * 32;
  static constexpr int GROUPS = WARPS / 4;                          // warps that share 32 rows of W
  static constexpr int COLS = NT / GROUPS;                          // columns of the sums a thread
  static constexpr int SLOTS = NT == 128 ? 2 : 4;                   // stages between their terms and their sums
  static constexpr int TERMS = 3 * NT * SP_KS * 2;                  // bytes of a stage's terms of x
  static constexpr int STAGE = SP_W_BYTES + NT * SP_KS * 4;
  static constexpr int RING = NT == 128 ? 5 : 6;
  static constexpr bool KEEPS = NT == 128;                          // (18 warps leave 96 registers a thread)
  static constexpr int TMEM = 512;
  static constexpr int W_TERMS = SLOTS * NT;                        // first column of the terms of W: 48 a slot
  static constexpr int KEPT = W_TERMS + SLOTS * 48;
  static_assert(KEPT + (KEEPS ? NT : 0) <= TMEM, "columns of tensor memory");
  static constexpr int BYTES = 1024 + RING * STAGE + SLOTS * TERMS + (2 * RING + 2 * SLOTS) * 8 + 16;
};

struct SplitWork {
  Product p;
  int tokens;              // rows of x a tile: a multiple of 16 up to NT
  int m_tiles, tiles, ksplit, spans_a_rank, span_stages, stages;
  int* err;
};

// grid: tiles x ranks of a cluster, or (one rank) at most a block an SM, which walks over tiles.  Warp 16 issues the products, warp 17
// the copies, the other sixteen take stages apart and add their sums up.  Bound by those: of a stage's 2,000 cycles (300 rows of 6,144 x
// 1,024, three tiles of 112 rows of x) the schedulers issue in 69 % and the tensor cores work in 32 %.
template <int NT>
__global__ void __launch_bounds__(SplitShape<NT>::THREADS, 1)
split_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap, const SplitWork job) {
  using S = SplitShape<NT>;
  constexpr int SLOTS = S::SLOTS, LAG = SLOTS - 1;
  extern __shared__ unsigned char split_smem[];
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(split_smem) + 1023) & ~uintptr_t(1023));
  unsigned char* terms = ring + S::RING * S::STAGE;
  uint64_t* raw_full = reinterpret_cast<uint64_t*>(terms + SLOTS * S::TERMS);
  uint64_t* raw_free = raw_full + S::RING;
  uint64_t* terms_full = raw_free + S::RING;
  uint64_t* done = terms_full + SLOTS;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + SLOTS);
  const Product& p = job.p;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int rank = job.ksplit > 1 ? blockIdx.x % job.ksplit : 0;
  const int first_tile = blockIdx.x / job.ksplit, tile_step = gridDim.x / job.ksplit;
  const int k_lo = rank * job.spans_a_rank * job.span_stages;
  const int k_hi = min(job.stages, k_lo + job.spans_a_rank * job.span_stages);
  bool again = false;                                               // this thread has stored a sum that is no number

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::RING; ++s) { sp_init(raw_full + s, 1); sp_init(raw_free + s, S::WARPS); }
    for (int s = 0; s < SLOTS; ++s) { sp_init(terms_full + s, S::WARPS); sp_init(done + s, 1); }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == S::WARPS) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(S::TMEM) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  sp_fence_before();
  __syncthreads();
  sp_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  if (warp == S::WARPS + 1) {
    if (lane == 0) {                                                // copies
      pdl_wait();                                                   // (x, and where it was widened just now W, come from the kernel before)
      const uint32_t bytes = SP_W_BYTES + job.tokens * SP_KS * 4;
      int it = 0;
      bool ok = true;
      for (int tile = first_tile; tile < job.tiles && ok; tile += tile_step) {
        const int n0 = tile / job.m_tiles * SP_BN, m0 = tile % job.m_tiles * job.tokens;
        for (int kst = k_lo; kst < k_hi; ++kst, ++it) {
          const int s = it % S::RING;
          unsigned char* st = ring + s * S::STAGE;
          if (it >= S::RING && !mbar_wait(raw_free + s, (it / S::RING - 1) & 1, job.err)) { ok = false; break; }
          sp_expect(raw_full + s, bytes);
          sp_load(st, &wmap, kst * SP_KS, n0, raw_full + s);
          sp_load(st + SP_W_BYTES, &xmap, kst * SP_KS, m0, raw_full + s);
        }
      }
      for (int j = it > S::RING ? it - S::RING : 0; j < it; ++j)    // no copy is left behind, whatever ran out
        mbar_wait(raw_full + j % S::RING, (j / S::RING) & 1, job.err);
    }
    __syncwarp();
  } else if (warp == S::WARPS) {
    // products: the whole warp walks along, so that descriptors are made once a warp (in uniform registers); one lane issues
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(job.tokens >> 3) << 17) | ((SP_BN >> 4) << 24);
    // terms of x: 8 rows x 16 bytes are contiguous, the next 8 rows follow, the next 8 k come NT x 16 bytes further on
    const uint64_t layout = (static_cast<uint64_t>(NT * 16 >> 4) << 16) | (static_cast<uint64_t>(128 >> 4) << 32) | (1ull << 46);
    const uint64_t first_b = layout | ((smem_u32(terms) >> 4) & 0x3FFFu);          // (the addresses' low bits never carry)
    int it = 0;
    bool ok = true;
    for (int tile = first_tile; tile < job.tiles && ok; tile += tile_step)
      for (int kst = k_lo; kst < k_hi; ++kst, ++it) {
        const int s = it % SLOTS;
        const bool mine = mbar_wait(terms_full + s, (it / SLOTS) & 1, job.err);
        ok = __all_sync(0xffffffffu, mine ? 1 : 0) != 0;
        if (!ok) break;
        sp_fence_after();
        const uint32_t d = tmem + s * NT, a = tmem + S::W_TERMS + s * 48;
        const uint64_t b = first_b + static_cast<uint32_t>(s * (S::TERMS >> 4));
        if (elect_one()) {
          // small products first: what they add is then not cut off below a large sum's last place
          constexpr int WI[6] = {2, 0, 1, 1, 0, 0}, XI[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
          for (int q = 0; q < 12; ++q) {
            const int half = q & 1, t = q >> 1;
            if (q == 0) sp_mma<false>(d, a + WI[t] * 16 + half * 8, b + ((XI[t] * (NT * SP_KS * 2) + half * (2 * NT * 16)) >> 4), idesc);
            else sp_mma<true>(d, a + WI[t] * 16 + half * 8, b + ((XI[t] * (NT * SP_KS * 2) + half * (2 * NT * 16)) >> 4), idesc);
          }
          sp_commit(done + s);
        }
        __syncwarp();
      }
    __syncwarp();
  } else {
    const int row = (warp & 3) * 32 + lane, group = warp >> 2;
    const uint32_t lane_at = static_cast<uint32_t>((warp & 3) * 32) << 16;
    // a span's sums, and the element's so far: in registers, or (128 columns) beside the terms in tensor memory
    float sum[S::COLS], held[S::KEEPS ? 1 : S::COLS];
    const uint32_t kept = tmem + lane_at + S::KEPT + group * S::COLS;
    constexpr int CHUNKS = 8 / S::GROUPS;                           // 16-byte pieces of a row's 32 k
    int it = 0;
    bool ok = true;

    // the sums of stage `of` go to the span's
    auto add_up = [&](int of, bool first) {
      const int s = of % SLOTS;
      const bool mine = mbar_wait(done + s, (of / SLOTS) & 1, job.err);
      if (!__all_sync(0xffffffffu, mine ? 1 : 0)) return false;
      sp_fence_after();
      const uint32_t at = tmem + lane_at + s * NT + group * S::COLS;
      constexpr int STEP = S::COLS < 16 ? S::COLS : 16;
#pragma unroll
      for (int c = 0; c < S::COLS; c += STEP) {
        uint32_t v[STEP];
        if constexpr (STEP == 8) sp_ld8(at + c, v); else sp_ld16(at + c, v);
        sp_wait_ld();
#pragma unroll
        for (int e = 0; e < STEP; ++e) sum[c + e] = first ? __uint_as_float(v[e]) : sum[c + e] + __uint_as_float(v[e]);
      }
      sp_fence_before();
      return true;
    };
    auto span_ends = [&](int kst) {                                 // after stage kst of the rank's
      const int at = kst - k_lo;
      if (kst + 1 != k_hi && (at + 1) % job.span_stages != 0) return;
      if (job.ksplit > 1 && kst + 1 == k_hi && at >= job.span_stages) return;      // (two spans a rank: the second stays in sum)
      const bool first = at < job.span_stages;
      if constexpr (S::KEEPS) {
#pragma unroll
        for (int c = 0; c < S::COLS; c += 8) {
          uint32_t v[8];
          if (!first) {
            sp_ld8(kept + c, v);
            sp_wait_ld();
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = __float_as_uint(first ? sum[c + e] : __uint_as_float(v[e]) + sum[c + e]);
          sp_st(kept + c, v);
        }
        sp_wait_st();
      } else {
#pragma unroll
        for (int c = 0; c < S::COLS; ++c) held[c] = first ? sum[c] : held[c] + sum[c];
      }
    };
    // calls f(column, its total) for the thread's columns
    auto totals = [&](auto f) {
      if constexpr (S::KEEPS) {
#pragma unroll
        for (int c = 0; c < S::COLS; c += 8) {
          uint32_t v[8];
          sp_ld8(kept + c, v);
          sp_wait_ld();
#pragma unroll
          for (int e = 0; e < 8; ++e) f(c + e, __uint_as_float(v[e]));
        }
      } else {
#pragma unroll
        for (int c = 0; c < S::COLS; ++c) f(c, held[c]);
      }
    };

    pdl_wait();
    for (int tile = first_tile; tile < job.tiles && ok; tile += tile_step) {
      const int n0 = tile / job.m_tiles * SP_BN, m0 = tile % job.m_tiles * job.tokens;
      const int it0 = it - k_lo;
      for (int kst = k_lo; kst < k_hi + LAG; ++kst) {
        if (kst < k_hi) {
          const int slot = it % S::RING, s = it % SLOTS;
          const bool mine = mbar_wait(raw_full + slot, (it / S::RING) & 1, job.err);
          ok = __all_sync(0xffffffffu, mine ? 1 : 0) != 0;
          if (!ok) break;
          const unsigned char* w_raw = ring + slot * S::STAGE + row * 128;
          const unsigned char* x_raw = w_raw + SP_W_BYTES;
          uint32_t high[2 * CHUNKS], mid[2 * CHUNKS], low[2 * CHUNKS];
#pragma unroll
          for (int c = 0; c < CHUNKS; ++c) {
            const float4 v = *reinterpret_cast<const float4*>(w_raw + (((group * CHUNKS + c) ^ (row & 7)) << 4));
            sp_split(v.x, v.y, high[2 * c], mid[2 * c], low[2 * c]);
            sp_split(v.z, v.w, high[2 * c + 1], mid[2 * c + 1], low[2 * c + 1]);
          }
          const uint32_t at = tmem + lane_at + S::W_TERMS + s * 48 + group * 2 * CHUNKS;
          sp_st(at, high);
          sp_st(at + 16, mid);
          sp_st(at + 32, low);
          if (row < job.tokens) {
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) {
              const float4 v = *reinterpret_cast<const float4*>(x_raw + (((group * CHUNKS + c) ^ (row & 7)) << 4));
              sp_split(v.x, v.y, high[2 * c], mid[2 * c], low[2 * c]);
              sp_split(v.z, v.w, high[2 * c + 1], mid[2 * c + 1], low[2 * c + 1]);
            }
            unsigned char* to = terms + s * S::TERMS + (row >> 3) * 128 + (row & 7) * 16;
#pragma unroll
            for (int c = 0; c < CHUNKS; c += 2) {
              unsigned char* q = to + (group * CHUNKS + c) / 2 * (NT * 16);
              *reinterpret_cast<uint4*>(q) = make_uint4(high[2 * c], high[2 * c + 1], high[2 * c + 2], high[2 * c + 3]);
              *reinterpret_cast<uint4*>(q + NT * SP_KS * 2) = make_uint4(mid[2 * c], mid[2 * c + 1], mid[2 * c + 2], mid[2 * c + 3]);
              *reinterpret_cast<uint4*>(q + 2 * NT * SP_KS * 2) = make_uint4(low[2 * c], low[2 * c + 1], low[2 * c + 2], low[2 * c + 3]);
            }
          }
          asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
          sp_wait_st();
          sp_fence_before();
          __syncwarp();
          if (lane == 0) { sp_arrive(raw_free + slot); sp_arrive(terms_full + s); }
          ++it;
        }
        const int past = kst - LAG;                                 // the stage whose sums are added up meanwhile
        if (past >= k_lo) {
          ok = add_up(it0 + past, (past - k_lo) % job.span_stages == 0);
          if (!ok) break;
          span_ends(past);
        }
      }
      if (!ok || job.ksplit > 1) break;
      const int n = n0 + row;
      totals([&](int c, float v) {
        const int t = group * S::COLS + c, m = m0 + t;
        if (t < job.tokens && m < p.m && n < p.n) {
          again = again || !sp_settled(v);
          p.c[static_cast<size_t>(m) * p.ldc + n] = v;
        }
      });
    }
    if (job.ksplit > 1) {
      // (every copy has landed and every product has ended: the ring holds the spans' sums from here on)
      float* parts = reinterpret_cast<float*>(ring);                // [spans a rank][NT][128]
      asm volatile("bar.sync 1, %0;\n" ::"n"(S::WARPS * 32) : "memory");
      totals([&](int c, float v) { parts[(group * S::COLS + c) * SP_BN + row] = v; });
      if (job.spans_a_rank > 1)
#pragma unroll
        for (int c = 0; c < S::COLS; ++c) parts[(NT + group * S::COLS + c) * SP_BN + row] = sum[c];
    }
    __syncwarp();
  }
  if (job.ksplit > 1) {
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const int n0 = first_tile / job.m_tiles * SP_BN, m0 = first_tile % job.m_tiles * job.tokens;
    const int spans = (job.stages + job.span_stages - 1) / job.span_stages;
    const float* parts = reinterpret_cast<const float*>(ring);
    // Four rows of W a turn: the other ranks' memory is far, and its requests, not its bytes, take the time (300 rows of 1,024 x
    // 2,048 one float a turn 34.6 us, four 28.0; 1,024 x 3,072 42.5 -> 35.7).
    for (int i = rank * S::THREADS + threadIdx.x; i < job.tokens * SP_BN / 4; i += job.ksplit * S::THREADS) {
      const int m = m0 + i / (SP_BN / 4), n = n0 + i % (SP_BN / 4) * 4;
      float4 v[SP_SPANS];
#pragma unroll
      for (int s = 0; s < SP_SPANS; ++s)
        if (s < spans)
          v[s] = reinterpret_cast<const float4*>(cluster.map_shared_rank(parts, s / job.spans_a_rank) + s % job.spans_a_rank * NT * SP_BN)[i];
      float t[4] = {v[0].x, v[0].y, v[0].z, v[0].w};
#pragma unroll
      for (int s = 1; s < SP_SPANS; ++s)
        if (s < spans) { t[0] += v[s].x; t[1] += v[s].y; t[2] += v[s].z; t[3] += v[s].w; }
      if (m >= p.m) continue;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (n + e < p.n) {
          again = again || !sp_settled(t[e]);
          p.c[static_cast<size_t>(m) * p.ldc + n + e] = t[e];
        }
    }
    cluster.sync();                                                 // the sums are read: the block may end
  }
  sp_fence_before();
  __syncthreads();
  if (warp == S::WARPS) {
    sp_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(S::TMEM) : "memory");
  }
  // Last of all, where the loops' registers are free and no warp waits for another (a call among the stores: 300 rows of 1,024 x
  // 2,048 28 -> 46 us), each warp the elements that it has stored itself.
  if (__any_sync(0xffffffffu, again)) {
    if (job.ksplit > 1) {                                           // (32 threads have one row of the tile, 128 columns of C)
      const int n0 = first_tile / job.m_tiles * SP_BN, m0 = first_tile % job.m_tiles * job.tokens;
      for (int i = rank * S::THREADS + warp * 32; i < job.tokens * SP_BN / 4; i += job.ksplit * S::THREADS)
        if (m0 + i / (SP_BN / 4) < p.m) sp_stored_again(p, m0 + i / (SP_BN / 4), n0, SP_BN);
    } else {
      for (int tile = first_tile; tile < job.tiles; tile += tile_step) {
        const int n0 = tile / job.m_tiles * SP_BN, m0 = tile % job.m_tiles * job.tokens, first = (warp >> 2) * S::COLS;
        for (int t = first; t < first + S::COLS && t < job.tokens && m0 + t < p.m; ++t) sp_stored_again(p, m0 + t, n0 + (warp & 3) * 32, 32);
      }
    }
  }
}

// ------------------------------------------------------------------ few rows, in the same terms
// The same products in the same order through mma.sync, whose sums have the bits of tcgen05's (the tests compare them): what a
// warp needs of W (16 rows, one span) comes through a ring of cp.async stages that only this warp reads, is taken apart in
// registers and multiplied there, without the way through tensor memory and its barriers.  The eight warps of a block take the
// eight spans of a tile and their sums meet in shared memory.
template <int MR, int WN> struct FewSplit {                         // rows of x a block, rows of W a tile
  static constexpr int WARPS = SP_SPANS;
  static constexpr int RING = WN == 16 ? (MR == 8 ? 4 : 3) : (MR == 8 ? 10 : 6);
  static constexpr int STAGE = (WN + MR) * SP_KS;                   // floats
  static constexpr int RED = WARPS * WN * MR;                       // floats of a tile's spans
  static constexpr int BYTES = (WARPS * RING * STAGE + 2 * RED) * 4;
};

__device__ __forceinline__ void sp_mma_sync(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// grid (blocks, groups of MR rows of x).  WN = 8 leaves half of an instruction's rows empty: for products whose tiles of 16 would
// not reach every SM.
template <int MR, int WN>
__global__ void __launch_bounds__(256, MR == 8 && WN == 16 ? 2 : 1)
few_split_kernel(const Product p, int tiles, int stages, int span_stages) {
  using F = FewSplit<MR, WN>;
  extern __shared__ __align__(128) float few_split_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, c4 = lane & 3;
  const int m0 = blockIdx.y * MR;
  float* ring = few_split_smem + warp * F::RING * F::STAGE;
  float* red = few_split_smem + F::WARPS * F::RING * F::STAGE;      // [2][8 spans][16][MR]
  const int k_lo = min(stages, warp * span_stages), mine = min(stages, k_lo + span_stages) - k_lo;      // this warp's stages of a tile
  const int spans = (stages + span_stages - 1) / span_stages;
  const int my_tiles = static_cast<int>(blockIdx.x) < tiles ? (tiles - 1 - blockIdx.x) / gridDim.x + 1 : 0, steps = my_tiles * mine;

  // Stage `step` of this warp: 16 rows of W and the rows of x, 32 k each; a row's 16-byte pieces are exchanged by twice its number
  // mod 4, so that the four rows of a half warp's reads lie in different banks.
  int f_tile = blockIdx.x, f_at = 0;
  auto fetch = [&](int step) {
    if (step < steps) {
      float* st = ring + step % F::RING * F::STAGE;
      const int k0 = (k_lo + f_at) * SP_KS;
#pragma unroll
      for (int j = 0; j < (WN + MR) / 4; ++j) {
        const int line = j * 4 + (lane >> 3), piece = lane & 7, kk = k0 + piece * 4;
        const bool of_w = line < WN;
        const int row = of_w ? f_tile * WN + line : m0 + line - WN;
        const bool valid = row < (of_w ? p.n : p.m) && kk < p.k;
        const float* src = of_w ? p.w + static_cast<size_t>(row) * p.ldw + kk : p.a + static_cast<size_t>(row) * p.lda + kk;
        cp_async16(st + line * SP_KS + ((piece ^ (2 * (line & 3))) << 2), valid ? src : p.w, valid);
      }
      if (++f_at == mine) { f_at = 0; f_tile += gridDim.x; }
    }
    cp_async_commit();
  };
  pdl_wait();
#pragma unroll
  for (int s = 0; s < F::RING - 1; ++s) fetch(s);

  int step = 0, parity = 0;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, parity ^= 1) {
    float sum[MR / 8][4];
    for (int at = 0; at < mine; ++at, ++step) {
      fetch(step + F::RING - 1);
      cp_async_wait<F::RING - 1>();
      __syncwarp();
      const float* st = ring + step % F::RING * F::STAGE;
      float t[MR / 8][4] = {};
      uint32_t a[2][3][4], b[MR / 8][2][3][2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {                                 // sixteen k each
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (WN == 8 && (e & 1)) {
            a[h][0][e] = a[h][1][e] = a[h][2][e] = 0;
            continue;
          }
          const int line = r + (e & 1) * 8, piece = h * 4 + (e >> 1) * 2 + (c4 >> 1);
          const float2 v = *reinterpret_cast<const float2*>(st + line * SP_KS + ((piece ^ (2 * (line & 3))) << 2) + (c4 & 1) * 2);
          sp_split(v.x, v.y, a[h][0][e], a[h][1][e], a[h][2][e]);
        }
#pragma unroll
        for (int x = 0; x < MR / 8; ++x)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int line = WN + x * 8 + r, piece = h * 4 + e * 2 + (c4 >> 1);
            const float2 v = *reinterpret_cast<const float2*>(st + line * SP_KS + ((piece ^ (2 * (line & 3))) << 2) + (c4 & 1) * 2);
            sp_split(v.x, v.y, b[x][h][0][e], b[x][h][1][e], b[x][h][2][e]);
          }
      }
      constexpr int WI[6] = {2, 0, 1, 1, 0, 0}, XI[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
      for (int q = 0; q < 12; ++q)
#pragma unroll
        for (int x = 0; x < MR / 8; ++x) sp_mma_sync(t[x], a[q & 1][WI[q >> 1]], b[x][q & 1][XI[q >> 1]]);
#pragma unroll
      for (int x = 0; x < MR / 8; ++x)
#pragma unroll
        for (int i = 0; i < 4; ++i) sum[x][i] = at == 0 ? t[x][i] : sum[x][i] + t[x][i];
      __syncwarp();                                                 // the stage is read
    }
    float* to = red + (parity * F::WARPS + warp) * WN * MR;
    if (mine > 0)
#pragma unroll
      for (int x = 0; x < MR / 8; ++x)
#pragma unroll
        for (int i = 0; i < WN / 4; ++i) to[(x * 8 + 2 * c4 + (i & 1)) * WN + r + (i >> 1) * 8] = sum[x][i];
    __syncthreads();
    static_assert(WN * MR % 32 == 0, "whole warps");
    for (int i = threadIdx.x; i < WN * MR; i += 256) {           // the element: its spans in order
      const int m = m0 + i / WN, n = tile * WN + i % WN;
      const bool mine_here = m < p.m && n < p.n;
      const float* from = red + parity * F::WARPS * WN * MR + i;
      float v = from[0];
      for (int s = 1; s < spans; ++s) v += from[s * WN * MR];
      const bool again = mine_here && !sp_settled(v);
      if (__any_sync(0xffffffffu, again)) v = sp_again(p.a, p.lda, p.w, p.ldw, p.k, m, n, v, again);
      if (mine_here) p.c[static_cast<size_t>(m) * p.ldc + n] = v;
    }
  }
  cp_async_wait<0>();
}

// ------------------------------------------------------------------ up to four rows, in the same terms
// The same products in the same order once more.  A block takes x apart once, for all the tiles that it walks over (few_split_kernel
// with every 16 rows of W again).  The instruction's sixteen rows are eight rows of W at one stage and the same eight at the next, its
// eight columns four rows of x at the one and at the other: two of its four quarters are the two stages' sums, so that tiles have
// eight rows of W and chains of products half the length.  A chain of twelve takes 255 cycles for 98 of the tensor cores' time, so
// a step has U pairs of stages side by side.  Which of a 16's k lie in which place of the instruction is the same for both operands, and
// of no account for a sum's bits.
// G groups of eight warps (a warp a span, as in few_split_kernel) share x and take every G-th tile; x is asked for before W, which
// otherwise holds it up (deeper rings of W were slower for that: 1,024 x 3,072 5.9 us with two steps, 6.4 with four).
// Shared memory: x as [stage][row][c4][half][term][2] words (48 bytes a lane), [G][2][8 spans][rows][8] sums, the rings.
// Bound by W's bytes where it is large.  One row, us: FFMA / few_split_kernel / this: 24,576 x 4,096 62 / 77 / 63 (6.4 TB/s), 151,936 x 1,024
// 105 / 118 / 106, 6,144 x 4,096 20.5 / 23.1 / 20.3, 4,096 x 12,288 48 / 44 / 38, 1,024 x 3,072 5.4 / 7.1 / 5.5, 2,048 x 8,192 17.6 / 28.1 / 14.3
// (FFMA stays ahead at 1,024 x 4,096, 5.8 / 8.8 / 6.5, and with two rows of 151,936 x 1,024, 98.9 / 118 / 106);
// four rows: 24,576 x 4,096 (x does not fit) 90 / 77, 151,936 x 1,024 134 / 118 / 106, 1,024 x 3,072 7.8 / 7.1 / 6.0.
constexpr int PAIR_ROWS = 4, PAIR_WN = 8;
static size_t pair_split_bytes(int m, int stages, int ring, int pairs, int groups) {
  return (static_cast<size_t>(stages + 2 * pairs) * m * 48 + groups * (2 * SP_SPANS * m * PAIR_WN + SP_SPANS * ring * pairs * 512)) * sizeof(float);
}

template <int RING, int U, int G>
__global__ void __launch_bounds__(256 * G, 1)
pair_split_kernel(const Product p, int tiles, int stages, int span_stages) {
  extern __shared__ __align__(128) float few_split_smem[];
  uint32_t* xt = reinterpret_cast<uint32_t*>(few_split_smem);
  float* red = few_split_smem + (stages + 2 * U) * p.m * 48;
  const int group = threadIdx.x >> 8, warp = (threadIdx.x >> 5) & 7, lane = threadIdx.x & 31, r = lane >> 2, c4 = lane & 3;
  float4* ring = reinterpret_cast<float4*>(red + G * 2 * SP_SPANS * p.m * PAIR_WN) + (group * 8 + warp) * RING * U * 128;
  red += group * 2 * SP_SPANS * p.m * PAIR_WN;
  const int first_tile = blockIdx.x + group * gridDim.x, tile_step = G * gridDim.x;
  const int k_lo = min(stages, warp * span_stages), mine = min(stages, k_lo + span_stages) - k_lo;      // this warp's stages of a tile
  const int spans = (stages + span_stages - 1) / span_stages, units = (mine + 2 * U - 1) / (2 * U);
  const int k_end = min(p.k, (k_lo + mine) * SP_KS);

  // 2 U stages of the tile's eight rows, whole lines of 128 bytes; an odd row's pieces are exchanged by four, so that the two rows of
  // a quarter warp's reads lie in different banks.
  int f_tile = first_tile, f_unit = 0, f_slot = 0;
  auto fetch = [&]() {
    if (f_tile < tiles && units > 0) {
      const int line = lane >> 3, piece = lane & 7, row = f_tile * PAIR_WN + line, kk = (k_lo + 2 * U * f_unit) * SP_KS + 4 * piece;
      const float* src = p.w + static_cast<size_t>(row) * p.ldw + kk;
      float4* to = ring + f_slot * U * 128 + line * 8 + (piece ^ (4 * (line & 1)));
#pragma unroll
      for (int e = 0; e < 4 * U; ++e) {                             // [stage][four rows]
        const bool valid = row + 4 * (e & 1) < p.n && kk + SP_KS * (e >> 1) < k_end;
        cp_async16(to + (e >> 1) * 64 + (e & 1) * 32, valid ? src + (e & 1) * 4 * static_cast<size_t>(p.ldw) + SP_KS * (e >> 1) : p.w, valid);
      }
      if (++f_unit == units) { f_unit = 0; f_tile += tile_step; }
    }
    if (++f_slot == RING) f_slot = 0;
    cp_async_commit();
  };
  pdl_wait();
  // x of this span: its warps (one a group) take every G-th 32 pieces each, four at a time
  const int pieces = mine * 8;                                      // of a row
  auto take_apart = [&](int i0, bool begin) {
    float4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = i0 + 32 * G * j, row = i / max(pieces, 1), kk = k_lo * SP_KS + (i - row * pieces) * 4;
      v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (i < p.m * pieces && kk < p.k) v[j] = *reinterpret_cast<const float4*>(p.a + static_cast<size_t>(row) * p.lda + kk);
    }
    if (begin) {
      __syncthreads();                                              // W is asked for behind all of x's first pieces, which everything waits for
#pragma unroll
      for (int s = 0; s < RING - 1; ++s) fetch();
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = i0 + 32 * G * j, row = i / max(pieces, 1), at = i - row * pieces, stage = k_lo + (at >> 3), piece = at & 7;
      if (i >= p.m * pieces) break;
      uint2 high, mid, low;
      sp_split(v[j].x, v[j].y, high.x, mid.x, low.x);
      sp_split(v[j].z, v[j].w, high.y, mid.y, low.y);
      uint2* to = reinterpret_cast<uint2*>(xt + ((stage * p.m + row) * 4 + (piece & 3)) * 12 + (piece >> 2) * 6);
      to[0] = high; to[1] = mid; to[2] = low;
    }
  };
  take_apart(group * 32 + lane, true);
  for (int i = group * 32 + lane + 128 * G; i < p.m * pieces; i += 128 * G) take_apart(i, false);
  if (G > 1) asm volatile("bar.sync %0, %1;\n" ::"r"(G + 1 + warp), "r"(32 * G) : "memory"); else __syncwarp();

  const bool has_x = (r & 3) < p.m;
  const uint4* my_x = reinterpret_cast<const uint4*>(xt + (((k_lo + (r >> 2)) * p.m + (r & 3)) * 4 + c4) * 12);
  static_assert(U <= 2, "a step of fewer pairs than U has one");
  // `pairs` pairs of stages from pair `at` of this warp on: their sums to those of the tile
  auto multiply = [&](auto pairs, int at, int slot, float (&sum)[2]) {
    constexpr int N = decltype(pairs)::value;
    uint32_t a[N][2][3][4], b[N][2][3][2];                          // [pair][half][term]
#pragma unroll
    for (int x = 0; x < N; ++x) {
      uint4 terms_of_x[3] = {};
      if (has_x) {
        const uint4* from = my_x + (at + x) * 2 * p.m * 12;
#pragma unroll
        for (int i = 0; i < 3; ++i) terms_of_x[i] = from[i];
      }
      memcpy(b[x], terms_of_x, sizeof(b[x]));
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int s = 0; s < 2; ++s) {                               // (stage s: the instruction's rows 8 s to 8 s + 7)
          const float4 v = ring[(slot * 2 * U + 2 * x + s) * 64 + r * 8 + ((h * 4 + c4) ^ (4 * (r & 1)))];
          sp_split(v.x, v.y, a[x][h][0][s], a[x][h][1][s], a[x][h][2][s]);
          sp_split(v.z, v.w, a[x][h][0][2 + s], a[x][h][1][2 + s], a[x][h][2][2 + s]);
        }
    }
    constexpr int WI[6] = {2, 0, 1, 1, 0, 0}, XI[6] = {0, 2, 1, 0, 1, 0};
    float t[N][4] = {};
#pragma unroll
    for (int q = 0; q < 12; ++q)
#pragma unroll
      for (int x = 0; x < N; ++x) sp_mma_sync(t[x], a[x][q & 1][WI[q >> 1]], b[x][q & 1][XI[q >> 1]]);
    // rows 0 to 7 x columns 0 to 3: the first stage; rows 8 to 15 x columns 4 to 7: the second, in the lane two further on
#pragma unroll
    for (int x = 0; x < N; ++x)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float second = __shfl_down_sync(0xffffffffu, t[x][2 + i], 2);
        sum[i] = at + x == 0 ? t[x][i] : sum[i] + t[x][i];
        if (2 * (at + x) + 1 < mine) sum[i] += second;
      }
  };
  int parity = 0, slot = 0, turn = 0;
  for (int tile = first_tile; tile < tiles; tile += tile_step, parity ^= 1) {
    float sum[2] = {};
    for (int u = 0; u < units; ++u) {
      __syncwarp();                                                 // (the slot that is filled has been read)
      fetch();
      cp_async_wait<RING - 1>();
      __syncwarp();
      if (2 * (U * u + U - 1) < mine) multiply(std::integral_constant<int, U>(), U * u, slot, sum);
      else multiply(std::integral_constant<int, 1>(), U * u, slot, sum);
      if (++slot == RING) slot = 0;
    }
    float* to = red + (parity * SP_SPANS + warp) * PAIR_WN * p.m;
    if (mine > 0)
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (2 * c4 + i < p.m) to[(2 * c4 + i) * PAIR_WN + r] = sum[i];
    asm volatile("bar.sync %0, 256;\n" ::"r"(group + 1) : "memory");
    if (warp == turn) {                                             // the elements: their spans in order (at most 4 x 8 of them)
      const int m = lane / PAIR_WN, n = tile * PAIR_WN + lane % PAIR_WN;
      const bool mine_here = m < p.m && n < p.n;
      float v = 0.0f;
      if (mine_here) {
        const float* from = red + parity * SP_SPANS * PAIR_WN * p.m + lane;
        v = from[0];
        for (int s = 1; s < spans; ++s) v += from[s * PAIR_WN * p.m];
      }
      const bool again = mine_here && !sp_settled(v);
      if (__any_sync(0xffffffffu, again)) v = sp_again(p.a, p.lda, p.w, p.ldw, p.k, m, n, v, again);
      if (mine_here) p.c[static_cast<size_t>(m) * p.ldc + n] = v;
    }
    turn = (turn + 1) & 7;
  }
  cp_async_wait<0>();
}

// ------------------------------------------------------------------ launchers
constexpr size_t FEW_SMEM_LIMIT = 225 * 1024;
constexpr int DEVICES = 16;                     // whose launch limits are remembered

static size_t few_bytes(int mr, int sw, int nt) {
  return (static_cast<size_t>(mr) * 4 * sw * FEW_XCHUNK + 2 * sw * nt * FEW_WN * mr + sw * nt * FEW_STAGES * FEW_STAGE) * sizeof(float);
}

template <int MR, bool VEC>
static int launch_few(const Product& p, int batch, int sw, int nt, int device, int sms, cudaStream_t stream) {
  const int warps = sw * nt;
  const size_t smem = few_bytes(MR, sw, nt);
  // Once a device, and the same size whoever comes first: a size that grew with the launches could be taken back by a thread
  // whose smaller launch met a larger one.
  static bool configured[DEVICES];
  if (device >= DEVICES || !configured[device]) {
    cudaError_t e = cudaFuncSetAttribute(few_rows_kernel<MR, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(FEW_SMEM_LIMIT));
    if (e != cudaSuccess) return static_cast<int>(e);
    if (device < DEVICES) configured[device] = true;
  }
  const int groups = (p.n + FEW_WN * nt - 1) / (FEW_WN * nt);
  const int resident = static_cast<int>((227 * 1024) / (smem + 1024));
  const int blocks = sms * (resident < 1 ? 1 : resident > 8 ? 8 : resident);
  dim3 grid(groups < blocks ? groups : blocks, (p.m + MR - 1) / MR, batch);
  few_rows_kernel<MR, VEC><<<grid, warps * 32, smem, stream>>>(p, sw, nt);
  return b200_check_launch();
}

// How many blocks (of one cluster) share a tile's spans: as many as give the fullest SM the least time (of equal times the
// fewest rounds, then the fewest blocks).  An SM holds four blocks, and a block's two warps keep half of its schedulers busy, so a second block
// costs nothing beside the first, a third and a fourth half as much again (one span, 1 to 4 blocks on an SM: 41, 43, 63, 66 us;
// more come in waves of four).  Counted as if two blocks took an SM twice the time, 128 tiles of two spans stayed one block each:
// N x K = 4,096 x 1,024 at 65 to 128 rows 84 us for 44, 6,144 x 1,024 at 17 to 64 rows 83 for 43, 1,024 x 2,048 at 500 176 for
// 65 (the single chain of 64 x 64 tiles that came before: 69, 70, 124).
static int blocks_a_tile(long long tiles, int spans, int sms) {
  int best = 1;
  long long best_cost = 0, best_rounds = 0;
  for (int s = 1; s <= 8 && s <= spans; ++s) {
    const long long blocks = (tiles * s + sms - 1) / sms, rounds = (spans + s - 1) / s;
    const long long cost = rounds * (3 * (blocks / 4) + (blocks % 4 == 0 ? 0 : blocks % 4 <= 2 ? 2 : 3));
    if (s == 1 || cost < best_cost || (cost == best_cost && rounds < best_rounds)) { best = s; best_cost = cost; best_rounds = rounds; }
  }
  return best;
}
B200_EXPORT int b200_gemm_f32_blocks_a_tile(long long tiles, int spans, int sms) { return blocks_a_tile(tiles, spans, sms); }

// How many clusters of `ranks` of split_kernel's blocks (one an SM) a device holds at once; device < 0: a B200 as measured.
static int clusters_at_once(int ranks, int sms, int device) {
  static int known[DEVICES][SP_SPANS + 1];
  constexpr int MEASURED[SP_SPANS + 1] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
  if (device < 0) return MEASURED[ranks];
  if (device < DEVICES && known[device][ranks] > 0) return known[device][ranks];
  using S = SplitShape<64>;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(ranks);
  config.blockDim = dim3(S::THREADS);
  config.dynamicSmemBytes = S::BYTES;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = ranks;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  config.attrs = &attr;
  config.numAttrs = 1;
  int n = 0;
  cudaError_t e = cudaFuncSetAttribute(split_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::BYTES);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, split_kernel<64>, &config);
  if (e != cudaSuccess || n <= 0) {
    cudaGetLastError();
    n = sms / ranks > 0 ? sms / ranks : 1;
  }
  if (device < DEVICES) known[device][ranks] = n;
  return n;
}

// What a product costs split_kernel, in stages of one block: rounds of blocks over the SMs, each its stages and what begins and ends a
// block (a cluster's placement and its exchange of sums take as long as nine to eleven stages).  `ranks`: how many blocks share a
// tile's k, one or two spans each.  How many clusters the SMs hold at once is less than their blocks: a cluster stays within one of the
// chip's parts, 15 of eight blocks and not 18 (by blocks, 200 rows of 1,024 x 2,048 took eight, 32.3 us; four: 27.2).  Measured with
// one, four and eight: 4,096 x 1,024 at 64 rows 31.5 / 16.8 / 32.6 us, 6,144 x 1,024 at 64 31.9 / 31.1 / 43.5, 2,048 x 2,048 at 64 56.9 / 22.5 /
// 28.4, 1,024 x 3,072 at 300 95 / 34.7 / 40.8, at 600 97 / 68 / 62, 6,144 x 4,096 at 64 111 / 70 / 82.
static long long split_cost(int tiles, int spans, int stages, int sms, int device, int& ranks) {
  ranks = 1;
  long long least = static_cast<long long>((tiles + sms - 1) / sms) * (stages + 3);
  for (int r : {(spans + 1) / 2, spans}) {
    const int at_once = clusters_at_once(r, sms, device);
    const long long cost = static_cast<long long>((tiles + at_once - 1) / at_once) * ((stages + r - 1) / r + 11);
    if (spans >= 3 && cost < least) { ranks = r; least = cost; }
  }
  return least;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// Boxes of `box_rows` rows x 32 floats, 128-byte swizzle; what lies outside reads as zeros.
static int encode_rows(CUtensorMap* map, const float* base, int rows, int cols, int ld, int box_rows) {
  static EncodeTiledFn encode = nullptr;
  if (encode == nullptr) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (fn == nullptr || found != cudaDriverEntryPointSuccess) return static_cast<int>(cudaErrorNotSupported);
    encode = reinterpret_cast<EncodeTiledFn>(fn);
  }
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * sizeof(float)};
  const cuuint32_t box[2] = {SP_KS, static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t elem_strides[2] = {1u, 1u};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, elem_strides,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : 1000 + static_cast<int>(r);
}

static SplitWork split_work(const Product& p, int nt, int sms, int device, int* err, long long& cost) {
  SplitWork job = {};
  job.p = p;
  job.err = err;
  job.m_tiles = (p.m + nt - 1) / nt;
  job.tokens = ((p.m + job.m_tiles - 1) / job.m_tiles + 15) / 16 * 16;
  job.m_tiles = (p.m + job.tokens - 1) / job.tokens;
  const long long tiles = static_cast<long long>((p.n + SP_BN - 1) / SP_BN) * job.m_tiles;
  job.tiles = tiles > (1 << 28) ? 0 : static_cast<int>(tiles);
  job.stages = (p.k + SP_KS - 1) / SP_KS;
  job.span_stages = (job.stages + SP_SPANS - 1) / SP_SPANS;
  const int spans = (job.stages + job.span_stages - 1) / job.span_stages;
  cost = split_cost(job.tiles, spans, job.stages, sms, device, job.ksplit);
  job.spans_a_rank = job.ksplit > 1 ? (spans + job.ksplit - 1) / job.ksplit : spans;
  return job;
}

template <int NT>
static int launch_split(const SplitWork& job, int device, int sms, cudaStream_t stream) {
  using S = SplitShape<NT>;
  static bool configured[DEVICES];
  if (device >= DEVICES || !configured[device]) {
    cudaError_t e = cudaFuncSetAttribute(split_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::BYTES);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (device < DEVICES) configured[device] = true;
  }
  const Product& p = job.p;
  if (job.tiles <= 0) return B200_BAD_SIZE;
  CUtensorMap wmap, xmap;
  int rc = encode_rows(&wmap, p.w, p.n, p.k, p.ldw, SP_BN);
  if (rc == 0) rc = encode_rows(&xmap, p.a, p.m, p.k, p.lda, job.tokens);
  if (rc != 0) return rc;
  const int grid = job.ksplit > 1 ? job.tiles * job.ksplit : job.tiles < sms ? job.tiles : sms;
  return b200_launch(split_kernel<NT>, dim3(grid), dim3(S::THREADS), S::BYTES, stream, job.ksplit > 1 ? job.ksplit : 0, wmap, xmap, job);
}

template <int MR, int WN>
static int launch_few_split(const Product& p, int device, int sms, cudaStream_t stream) {
  using F = FewSplit<MR, WN>;
  static bool configured[DEVICES];
  if (device >= DEVICES || !configured[device]) {
    cudaError_t e = cudaFuncSetAttribute(few_split_kernel<MR, WN>, cudaFuncAttributeMaxDynamicSharedMemorySize, F::BYTES);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (device < DEVICES) configured[device] = true;
  }
  const int tiles = (p.n + WN - 1) / WN, stages = (p.k + SP_KS - 1) / SP_KS, span_stages = (stages + SP_SPANS - 1) / SP_SPANS;
  const int places = sms * (MR == 8 && WN == 16 ? 2 : 1);
  const dim3 grid(tiles < places ? tiles : places, (p.m + MR - 1) / MR);
  return b200_launch(few_split_kernel<MR, WN>, grid, dim3(256), F::BYTES, stream, 0, p, tiles, stages, span_stages);
}

template <int RING, int U, int G>
static int launch_pair_split(const Product& p, int device, int sms, cudaStream_t stream) {
  static bool configured[DEVICES];
  if (device >= DEVICES || !configured[device]) {
    cudaError_t e = cudaFuncSetAttribute(pair_split_kernel<RING, U, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(FEW_SMEM_LIMIT));
    if (e != cudaSuccess) return static_cast<int>(e);
    if (device < DEVICES) configured[device] = true;
  }
  const int tiles = (p.n + PAIR_WN - 1) / PAIR_WN, stages = (p.k + SP_KS - 1) / SP_KS, span_stages = (stages + SP_SPANS - 1) / SP_SPANS;
  return b200_launch(pair_split_kernel<RING, U, G>, dim3(tiles < sms ? tiles : sms), dim3(256 * G), pair_split_bytes(p.m, stages, RING, U, G), stream, 0,
                     p, tiles, stages, span_stages);
}
// How many groups pair_split_kernel takes a product with, 0: few_split_kernel takes it.  Measured in hundredths of a microsecond on 148
// SMs, one to four rows of 128 to 8,192 columns and 256 to 16,384 rows of W; ss: stages a span.  few_split_kernel costs 245 and, a round of
// tiles over the SMs, 84 ss (40 ss with tiles of eight rows of W); this kernel 290 + 20 ss with one group and one round, 335 and a round of
// 33 (1 + ss) with two, 300 and 20 + 24 ss with one group where shared memory holds no two (two rounds at most: 2,048 x 8,192, two
// rows, 28.1 / 18.0, but 6,144 x 4,096, four rows, 23.3 / 26.4).  So short rows stay
// with few_split_kernel (16,384 x 512 9.9 / 11.0, 4,096 x 1,024 5.9 / 6.5; 16,384 x 1,024 16.5 / 14.6, 2,048 x 1,024 5.9 / 5.0).
static int pair_groups(int m, int n, int k, int sms) {
  if (m > PAIR_ROWS) return 0;
  auto rounds = [](long long tiles, long long places) { return (tiles + places - 1) / places; };
  const int stages = (k + SP_KS - 1) / SP_KS;
  const long long ss = (stages + SP_SPANS - 1) / SP_SPANS, tiles = (n + 7) / 8, wide = (n + 15) / 16;
  const long long few = 245 + ss * (wide < sms ? 40 * rounds(tiles, sms) : 84 * rounds(wide, 2 * sms));
  const bool one = pair_split_bytes(m, stages, 2, 2, 1) <= FEW_SMEM_LIMIT, two = pair_split_bytes(m, stages, 2, 2, 2) <= FEW_SMEM_LIMIT;
  if (tiles <= sms) return one && 290 + 20 * ss <= few ? 1 : 0;
  if (two) return 335 + rounds(tiles, 2 * sms) * 33 * (1 + ss) <= few ? 2 : 0;
  return one && rounds(tiles, sms) <= 2 && 300 + rounds(tiles, sms) * (20 + 24 * ss) <= few ? 1 : 0;
}
B200_EXPORT int b200_gemm_f32_pair_groups(int m, int n, int k, int sms) { return pair_groups(m, n, k, sms); }

// Which kernel takes a product in terms: few_split_kernel up to 16 rows, and up to 128 in groups of 32 where that is the shorter way.
// Its groups cost a tile of 16 rows of W 0.135 us a stage, a block an SM at a time (and 2.7 us to begin), split_kernel's stage costs 0.88
// us with up to 64 rows of x and 1.1 with 128.  (us on few_split / split, 32 rows: 4,096 x 1,024 11.3 / 15.9, 16,384 x 1,024 34.5 / 32.2; 64
// rows: 1,024 x 2,048 10.1 / 14.8, 2,048 x 2,048 19.2 / 22.5, 4,096 x 4,096 67 / 36.5, 151,936 x 1,024 593 / 252; 96: 1,024 x 3,072 26.6 / 20.5, and on
// the line 1,024 x 2,048 18.9 / 16.8, 6,144 x 1,024 40.1 / 37.7.)
// Tiles of eight rows of W where those of sixteen leave SMs without a block (1,024 x 2,048, one row: 5.6 -> 4.9 us).
static bool few_split_takes(const Product& p, int sms, long long split_stages, int nt) {
  if (p.m <= 16) return true;
  if (p.m > 128) return false;
  const long long tiles = static_cast<long long>((p.n + 15) / 16) * ((p.m + 31) / 32), stages = (p.k + SP_KS - 1) / SP_KS;
  return 20 + (tiles + sms - 1) / sms * stages <= split_stages * (nt == 64 ? 13 : 16) / 2;
}

static int launch_terms(const Product& p, int* err, int device, int sms, cudaStream_t stream) {
  const int nt = p.m <= 64 ? 64 : 128;
  long long cost = 0;
  const SplitWork job = split_work(p, nt, sms, device, err, cost);
  if (few_split_takes(p, sms, cost, nt)) {
    const bool narrow = (p.n + 15) / 16 < sms;
    const int groups = pair_groups(p.m, p.n, p.k, sms);
    if (groups != 0) return groups == 1 ? launch_pair_split<2, 2, 1>(p, device, sms, stream) : launch_pair_split<2, 2, 2>(p, device, sms, stream);
    if (p.m <= 8) return narrow ? launch_few_split<8, 8>(p, device, sms, stream) : launch_few_split<8, 16>(p, device, sms, stream);
    if (p.m <= 16) return narrow ? launch_few_split<16, 8>(p, device, sms, stream) : launch_few_split<16, 16>(p, device, sms, stream);
    return launch_few_split<32, 16>(p, device, sms, stream);
  }
  return nt == 64 ? launch_split<64>(job, device, sms, stream) : launch_split<128>(job, device, sms, stream);
}
// (0: few_split_kernel, 1: split_kernel)
B200_EXPORT int b200_gemm_f32_route(int m, int n, int k, int sms) {
  Product p = {};
  p.m = m; p.n = n; p.k = k;
  long long cost = 0;
  split_work(p, m <= 64 ? 64 : 128, sms, -1, nullptr, cost);
  return few_split_takes(p, sms, cost, m <= 64 ? 64 : 128) ? 0 : 1;
}

static int launch(const Product& p, int batch, bool vec, int* err, cudaStream_t stream) {
  int device = 0, sms = 148;
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (vec && batch == 1) return launch_terms(p, err, device, sms, stream);
  const int spans = (p.k + SPAN - 1) / SPAN;
  // (What is left here are batched and unaligned products; the figures are of single, aligned ones, which these kernels took as well.)
  // Up to 16 rows the weights are streamed, in passes of `mr` rows: as many as fit shared memory beside the rings, 16 to K = 1,536
  // (2,048 where N leaves a block one tile), 8 to 3,072, 4 beyond.  One pass is 2 to 9 times as fast as a tile of 64 that is
  // mostly padding, and three passes or four still are where a span has a warp (16 rows of N x K = 4,096 x 1,024 / 1,024 x 3,072 /
  // 8,192 x 3,072 / 24,576 x 4,096: 18 / 18 / 79 / 348 us against 42 / 41 / 122 / 363; four passes of 4,096 x 4,096 67 against 65).
  // From nine spans on the warps go round, and three passes over many columns lose to tiles (9 rows of 4,096 x 5,120 / 8,192 x 8,192 /
  // 4,096 x 12,288: 128 / 256 / 201 us against 124 / 245 / 185; 16 rows 164 / 341 / 259; 16 of 1,024 x 12,288 still 74 against 124).
  // 17 to 32 rows are two passes or more everywhere (the first two sizes: 44 to 52 / 54 to 73 us) and stay on tiles.
  if (p.m <= 16) {
    const int sw = spans < 8 ? spans : 8, tiles = (p.n + FEW_WN - 1) / FEW_WN;
    int nt = 8 / sw;
    while (nt > 1 && (tiles + nt - 1) / nt < sms) --nt;              // small products: a block an SM before warps a block
    int mr = p.m > 8 ? 16 : p.m > 4 ? 8 : p.m > 2 ? 4 : p.m;
    while (mr > 1 && few_bytes(mr, sw, nt) > FEW_SMEM_LIMIT) mr /= 2;
    const bool streams = spans <= 8 || (p.m + mr - 1) / mr <= 2 || p.n < 4096;
    if (streams) switch (mr) {
      case 16: return vec ? launch_few<16, true>(p, batch, sw, nt, device, sms, stream) : launch_few<16, false>(p, batch, sw, nt, device, sms, stream);
      case 8: return vec ? launch_few<8, true>(p, batch, sw, nt, device, sms, stream) : launch_few<8, false>(p, batch, sw, nt, device, sms, stream);
      case 4: return vec ? launch_few<4, true>(p, batch, sw, nt, device, sms, stream) : launch_few<4, false>(p, batch, sw, nt, device, sms, stream);
      case 2: return vec ? launch_few<2, true>(p, batch, sw, nt, device, sms, stream) : launch_few<2, false>(p, batch, sw, nt, device, sms, stream);
      default: return vec ? launch_few<1, true>(p, batch, sw, nt, device, sms, stream) : launch_few<1, false>(p, batch, sw, nt, device, sms, stream);
    }
  }
  const int n_tiles = (p.n + BN - 1) / BN, m_tiles = (p.m + BM - 1) / BM;
  const long long tiles = static_cast<long long>(n_tiles) * m_tiles * batch;
  const int ksplit = blocks_a_tile(tiles, spans, sms);
  if (m_tiles > 65535) return B200_BAD_SIZE;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(n_tiles * ksplit, m_tiles, batch);
  config.blockDim = dim3(TILED_THREADS);
  config.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = ksplit;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  config.attrs = &attr;
  config.numAttrs = ksplit > 1 ? 1 : 0;
  e = vec ? cudaLaunchKernelEx(&config, tiled_kernel<true>, p, ksplit) : cudaLaunchKernelEx(&config, tiled_kernel<false>, p, ksplit);
  return e == cudaSuccess ? b200_check_launch() : static_cast<int>(e);
}

static bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

B200_EXPORT int b200_gemm_f32(const float* a, const float* w, float* c, int m, int n, int k, int* err, cudaStream_t stream) {
  if (m <= 0 || n <= 0) return 0;
  if (k <= 0) return B200_BAD_SIZE;
  const Product p = {a, w, c, m, n, k, k, k, n, 0, 0, 0};
  return launch(p, 1, k % 4 == 0 && aligned16(a) && aligned16(w), err, stream);
}

// c[b] (m x n, rows ldc apart) = a[b] (m x k, rows lda apart) . w[b] (n x k, rows ldw apart)^T for b < batch; matrix b
// of an operand starts step_* floats behind matrix b - 1.
B200_EXPORT int b200_gemm_f32_batched(const float* a, const float* w, float* c, int m, int n, int k, int batch, int lda,
                                      int ldw, int ldc, long long step_a, long long step_w, long long step_c,
                                      int* err, cudaStream_t stream) {
  if (m <= 0 || n <= 0 || batch <= 0) return 0;
  if (k <= 0 || lda < k || ldw < k || ldc < n || batch > 65535) return B200_BAD_SIZE;
  const Product p = {a, w, c, m, n, k, lda, ldw, ldc, step_a, step_w, step_c};
  return launch(p, batch, k % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && step_a % 4 == 0 && step_w % 4 == 0 && aligned16(a) && aligned16(w), err, stream);
}
