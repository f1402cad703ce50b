// C[M, N] = A[M, K] . W[N, K]^T in true 32-bit: FFMA on CUDA cores only, no
// tensor cores and no reduced-precision mode.  This is the matrix product of the
// float32 engine (the reference's float path goes through libtorch matmul:
// src/layers/linear.rs:5-7).
//
// The order of the additions depends on k alone: K is cut into chunks of 128 and spans of four chunks; a chunk is summed
// over k in order, a span over its chunks in order, an element over its spans in order.  Both kernels below keep to it,
// whatever M and N are, however many blocks share an element and wherever it sits in a tile, so a token's result is
// bit-identical however the batch around it is cut.  (Short sums of short sums also round less than one long one.)
//
// few_rows_kernel (few rows): bound by reading W.  A warp takes 8 rows of W and one span: lane = (row of W, chunk), so
//   the span's chunks are summed side by side and a product of 1,024 x 2,048 still has 512 warps at work.  W comes
//   through a ring of four cp.async stages that only its own warp reads (no block-wide barrier on the way); the rows of x
//   wait in shared memory.
// tiled_kernel (many rows): bound by the FFMA units.  64 x 64 tiles by two warps, 8 x 8 elements a thread: four 16-byte
//   loads of shared memory for 64 FFMA (4 x 8 elements a thread as packed f32x2 pairs, with one operand stored twice, took
//   half again as many loads: 25 against 32 TFLOP/s at 1,000 rows).  The blocks of a cluster take different spans of one tile and add
//   them up in order through distributed shared memory.
// Measured in a step at the Qwen3-0.6B sizes, mean of a layer's four products, beside one 64 x 64 kernel that summed k in
// one chain for both: 4 rows 122 -> 9.1 us (1.7 TB/s; the head alone 5 TB/s), 300 rows 145 -> 93 us (25 TFLOP/s).
//
// The batched form multiplies `batch` independent pairs whose rows may lie apart (leading dimensions lda, ldw, ldc
// and a distance between consecutive matrices of each operand): per-head products of a mixer, where head h's rows are
// column ranges of wider matrices.
#include <cooperative_groups.h>

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

static int launch(const Product& p, int batch, bool vec, cudaStream_t stream) {
  int device = 0, sms = 148;
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return static_cast<int>(e);
  const int spans = (p.k + SPAN - 1) / SPAN;
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

B200_EXPORT int b200_gemm_f32(const float* a, const float* w, float* c, int m, int n, int k, cudaStream_t stream) {
  if (m <= 0 || n <= 0) return 0;
  if (k <= 0) return B200_BAD_SIZE;
  const Product p = {a, w, c, m, n, k, k, k, n, 0, 0, 0};
  return launch(p, 1, k % 4 == 0 && aligned16(a) && aligned16(w), stream);
}

// c[b] (m x n, rows ldc apart) = a[b] (m x k, rows lda apart) . w[b] (n x k, rows ldw apart)^T for b < batch; matrix b
// of an operand starts step_* floats behind matrix b - 1.
B200_EXPORT int b200_gemm_f32_batched(const float* a, const float* w, float* c, int m, int n, int k, int batch, int lda,
                                      int ldw, int ldc, long long step_a, long long step_w, long long step_c,
                                      cudaStream_t stream) {
  if (m <= 0 || n <= 0 || batch <= 0) return 0;
  if (k <= 0 || lda < k || ldw < k || ldc < n || batch > 65535) return B200_BAD_SIZE;
  const Product p = {a, w, c, m, n, k, lda, ldw, ldc, step_a, step_w, step_c};
  return launch(p, batch, k % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && step_a % 4 == 0 && step_w % 4 == 0 && aligned16(a) && aligned16(w), stream);
}
