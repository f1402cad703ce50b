// Causal grouped-query attention over the paged cache, for head sizes up to
// HEAD_DIM (compile with -DHEAD_DIM=<multiple of 16>): a kernel for portions of
// prompts (many query positions per row) and a split-KV kernel for single decoded
// tokens, both for float and bfloat16 caches.  These are the all-sizes CUDA-core
// kernels: they serve the float32 engine and are the reference point of the
// tensor-core kernels.  The real head size `hd` (any even number up to HEAD_DIM; the
// reference's configuration allows every even head size: src/models/qwen3/config.rs:160-162)
// is a run-time argument: rows of q, the cache and the output are `hd` wide, the tiles
// in shared memory HEAD_DIM wide with zeros beyond `hd`.  Values may have a width of their own (`hd_v`, rows of
// the value cache and of the output; HEAD_DIM covers the wider of the two), and a score may be soft-capped:
// s <- cap * tanh(s / cap) after the scale and before the mask (cap <= 0: no cap).
// Two more masks and a term of the denominator, each off unless asked for: `chunk` C > 0 lets the query at position p
// see key j only if j >= p - p % C (keys of the query's own block of C positions, blocks counted from position 0 of
// the sequence); `sinks` (one float per query head) adds exp(sink_h) to the softmax's denominator: a term without a
// key and without a value, not scaled.
//
// Semantics (reference: src/models/attention/backend.rs:1455-1498): query head h
// reads KV head h / (nh / nkv); score = q.k / sqrt(d) (the scale is a
// parameter); key j is visible to the query at absolute position p iff j <= p,
// and with a window W iff also p - W < j; softmax over the visible keys in
// float; output = P.V.  Keys and values are always read from the cache: the
// step writes them before it attends (src/models/qwen3/model.rs:495-513), so a
// position's result does not depend on how the tokens were cut into steps.
//
// Work split.  A warp owns up to 4 query vectors (a query vector is one
// (token, query head)); it walks blocks of 32 keys: lane j scores key j for the
// warp's vectors (q in shared memory, K rows padded against bank conflicts),
// an online softmax keeps (max, sum) per vector, then every lane accumulates
// its own output dimensions over the 32 keys.  Rows of a key block that lie
// beyond the sequence are zero-filled, never read: a page that is used again may
// hold anything.
//
// Bound by instructions, not by bytes: a key's row is therefore looked up once a block (a lane a key) and handed to the
// copying lanes by shuffles; a division and a table read for each 16 bytes took longer than the arithmetic (float32, 4 rows
// of up to 900 keys in one split: 100 us, in four: 18 us; a prompt of 300 tokens with the next block's copies under the
// arithmetic as well: 78.6 -> 60.9 us; float32 prompts of heads up to 128 have a kernel on the tensor cores now, see below).
#include <math.h>

#include "common.cuh"

#ifndef HEAD_DIM
#error "compile with -DHEAD_DIM=<head size, a multiple of 16>"
#endif
static_assert(HEAD_DIM % 16 == 0 && HEAD_DIM >= 16 && HEAD_DIM <= 512, "head size must be a multiple of 16 in [16, 512]");

constexpr int D = HEAD_DIM;
constexpr int NV = 4;                    // query vectors per warp
constexpr int KB = 32;                   // keys per block (one per lane)
constexpr int PAIRS = (D + 63) / 64;     // output dimension pairs per lane: dims 2*lane + 64*k, +1

template <typename T> struct RowGeom {
  static constexpr int CHUNK = 16 / sizeof(T);     // elements per 16 bytes
  static constexpr int CHUNKS = D / CHUNK;         // 16-byte chunks per row
  static constexpr int STRIDE = D + CHUNK;         // padded row: conflict-free 16-byte reads per lane
};

__device__ __forceinline__ void load_pair(const float* p, float& a, float& b) {
  float2 v = *reinterpret_cast<const float2*>(p); a = v.x; b = v.y;
}
__device__ __forceinline__ void load_pair(const __nv_bfloat16* p, float& a, float& b) {
  uint32_t v = *reinterpret_cast<const uint32_t*>(p);
  a = __uint_as_float(v << 16); b = __uint_as_float(v & 0xffff0000u);
}

struct VecState {
  float m[NV], l[NV], acc[NV][2 * PAIRS];
  __device__ __forceinline__ void init() {
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      m[v] = -INFINITY; l[v] = 0.0f;
#pragma unroll
      for (int i = 0; i < 2 * PAIRS; ++i) acc[v][i] = 0.0f;
    }
  }
};

// One block of 32 keys for the warp's NV query vectors.
//  ks, vs : shared memory, 32 rows of RowGeom<T>::STRIDE elements
//  qs     : shared memory, NV rows of D floats, already multiplied by the softmax scale
//  qpos   : absolute position of each vector's query, -1 for an unused vector
//  ps     : shared memory, 32 * NV floats private to the warp
template <typename T>
__device__ __forceinline__ void warp_key_block(const T* ks, const T* vs, const float* qs, const int* qpos,
                                               int first_key, int kv_end, int window, int chunk, VecState& st,
                                               float* ps, float softcap) {
  using G = RowGeom<T>;
  const int lane = threadIdx.x & 31;
  float s[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) s[v] = 0.0f;
  const T* krow = ks + lane * G::STRIDE;
#pragma unroll 4
  for (int c = 0; c < G::CHUNKS; ++c) {
    float kf[G::CHUNK];
    Vec16<T>::load(krow + c * G::CHUNK, kf);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const float* qv = qs + v * D + c * G::CHUNK;
#pragma unroll
      for (int e = 0; e < G::CHUNK; e += 4) {
        const float4 q4 = *reinterpret_cast<const float4*>(qv + e);
        s[v] = fmaf(kf[e], q4.x, s[v]);
        s[v] = fmaf(kf[e + 1], q4.y, s[v]);
        s[v] = fmaf(kf[e + 2], q4.z, s[v]);
        s[v] = fmaf(kf[e + 3], q4.w, s[v]);
      }
    }
  }
  const int key = first_key + lane;
  if (softcap > 0.0f) {
    const float inv_cap = 1.0f / softcap;
#pragma unroll
    for (int v = 0; v < NV; ++v) s[v] = softcap * tanhf(s[v] * inv_cap);
  }
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int p = qpos[v];
    const bool visible = p >= 0 && key <= p && key < kv_end && (window <= 0 || key > p - window) &&
                         (chunk <= 0 || key >= p - p % chunk);
    const float sv = visible ? s[v] : -INFINITY;
    const float m_new = fmaxf(st.m[v], warp_max(sv));
    float prob = 0.0f, corr = 1.0f;
    if (m_new != -INFINITY) {
      prob = visible ? expf(sv - m_new) : 0.0f;
      corr = expf(st.m[v] - m_new);          // exp(-inf) = 0 on the first visible block
    }
    st.l[v] = st.l[v] * corr + warp_sum(prob);
    st.m[v] = m_new;
#pragma unroll
    for (int i = 0; i < 2 * PAIRS; ++i) st.acc[v][i] *= corr;
    ps[lane * NV + v] = prob;
  }
  __syncwarp();
#pragma unroll 4
  for (int j = 0; j < KB; ++j) {
    const float4 pj = *reinterpret_cast<const float4*>(ps + j * NV);
    const T* vrow = vs + j * G::STRIDE;
#pragma unroll
    for (int k = 0; k < PAIRS; ++k) {
      const int dim = 2 * lane + 64 * k;
      if (dim < D) {
        float a, b;
        load_pair(vrow + dim, a, b);
        st.acc[0][2 * k] = fmaf(pj.x, a, st.acc[0][2 * k]); st.acc[0][2 * k + 1] = fmaf(pj.x, b, st.acc[0][2 * k + 1]);
        st.acc[1][2 * k] = fmaf(pj.y, a, st.acc[1][2 * k]); st.acc[1][2 * k + 1] = fmaf(pj.y, b, st.acc[1][2 * k + 1]);
        st.acc[2][2 * k] = fmaf(pj.z, a, st.acc[2][2 * k]); st.acc[2][2 * k + 1] = fmaf(pj.z, b, st.acc[2][2 * k + 1]);
        st.acc[3][2 * k] = fmaf(pj.w, a, st.acc[3][2 * k]); st.acc[3][2 * k + 1] = fmaf(pj.w, b, st.acc[3][2 * k + 1]);
      }
    }
  }
  __syncwarp();
}

// Where key `first_key + lane` lies: its row of the cache (cache[page][kv head][offset in page] are the rows), -1 beyond the
// sequence.  One lookup and one division a key and block of keys; a thread that copies looks its rows up in the other lanes.
__device__ __forceinline__ long long lane_row(const int* __restrict__ table, int page_size, int nkv, int kvh, int first_key,
                                              int kv_end) {
  const int key = first_key + (threadIdx.x & 31);
  if (key >= kv_end) return -1;
  const int page = key / page_size;
  return (static_cast<long long>(table[page]) * nkv + kvh) * page_size + (key - page * page_size);
}

// Copies the 32 key rows of a block into shared memory with `nthreads` threads (whole warps; thread index `tid`): `mine` is
// the calling lane's row (lane_row); rows beyond the sequence become zeros.  A row's first `hd` elements are copied; rows lie
// `stride` elements apart (values that are the leading columns of wider key rows: stride > hd).
template <typename T>
__device__ __forceinline__ void load_key_block(T* dst, const T* __restrict__ cache, long long mine, int hd, int stride, int tid,
                                               int nthreads) {
  using G = RowGeom<T>;
  if (hd % G::CHUNK == 0 && stride % G::CHUNK == 0) {
    // rows start on 16-byte boundaries: asynchronous 16-byte copies, zeros beyond the row and beyond the sequence
    // (KB * CHUNKS is a multiple of 32 and so is every step: a warp stays together)
    const int row_chunks = hd / G::CHUNK;
#pragma unroll 8
    for (int c = tid; c < KB * G::CHUNKS; c += nthreads) {
      const int r = c / G::CHUNKS, part = c - r * G::CHUNKS;
      const long long row = __shfl_sync(0xffffffffu, mine, r);
      const bool valid = row >= 0 && part < row_chunks;
      cp_async16(dst + r * G::STRIDE + part * G::CHUNK, valid ? cache + row * stride + part * G::CHUNK : cache, valid);
    }
  } else {
    // an even head size whose rows are not 16-byte aligned: pairs of elements with plain loads
    for (int c = tid; c < KB * (D / 2); c += nthreads) {
      const int r = c / (D / 2), pair = c - r * (D / 2);
      const long long row = __shfl_sync(0xffffffffu, mine, r);
      T a = from_f32<T>(0.0f), b = a;
      if (row >= 0 && 2 * pair < hd) {
        a = cache[row * stride + 2 * pair];
        b = cache[row * stride + 2 * pair + 1];
      }
      dst[r * G::STRIDE + 2 * pair] = a;
      dst[r * G::STRIDE + 2 * pair + 1] = b;
    }
  }
}

// ------------------------------------------------------------------ prompt portions
// grid (query tiles, nkv * head chunks, prefill rows); 8 warps; a tile holds `tile_tokens` consecutive query
// positions of one row and up to 32 of the `group` query heads of one KV head (head chunk hc holds heads
// 32 hc ..): tile_tokens * heads <= 32 vectors.
constexpr int PF_WARPS = 8;

// One tile of a portion, by CUDA cores (shared memory: PrefillShape<T>::SMEM); of its vectors those in `which` are stored.
template <typename T>
__device__ __forceinline__ void prefill_tile(const T* __restrict__ q, const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                         T* __restrict__ out, const int* __restrict__ block_table, int table_stride,
                         const int* __restrict__ cu_q, const int* __restrict__ kv_len,
                         const int* __restrict__ prefix_len, const int* __restrict__ rows, int nh, int nkv,
                         int page_size, int window, float scale, int tile_tokens, int head_chunks, int hd,
                         int hd_v, float softcap, int chunk, const float* __restrict__ sinks, int v_stride, int stages,
                         uint32_t which) {
  using G = RowGeom<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* qs = reinterpret_cast<float*>(smem_raw);                        // [32][D]
  float* ps = qs + 32 * D;                                               // [PF_WARPS][32 * NV]
  T* tiles = reinterpret_cast<T*>(ps + PF_WARPS * KB * NV);              // [stages][K, V][32][STRIDE]

  const int row = rows[blockIdx.z];
  const int kvh = blockIdx.y / head_chunks, hc = blockIdx.y - kvh * head_chunks;
  const int head_base = kvh * (nh / nkv) + hc * 32;                      // first query head of this CTA
  const int group = min(32, nh / nkv - hc * 32);                         // query heads of this CTA
  const int q_begin = cu_q[row], q_len = cu_q[row + 1] - q_begin;
  const int tok0 = (gridDim.x - 1 - blockIdx.x) * tile_tokens;           // the tiles that see the most keys start first
  if (tok0 >= q_len) return;
  const int ntok = min(tile_tokens, q_len - tok0);
  const int nvec = ntok * group;
  const int prefix = prefix_len[row];
  const int kv_end = min(kv_len[row], prefix + tok0 + ntok);            // causal: nothing later is visible
  const int p_lo = prefix + tok0;
  int k_begin = window > 0 ? max(0, p_lo - window + 1) : 0;
  if (chunk > 0) k_begin = max(k_begin, p_lo - p_lo % chunk);      // the tile's first query sees the earliest block
  k_begin -= k_begin % KB;
  const int* table = block_table + static_cast<size_t>(row) * table_stride;

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < 32 * D; i += blockDim.x) {
    const int v = i / D, dim = i - v * D;
    float val = 0.0f;
    if (v < nvec && dim < hd) {
      const int tok = v / group, head = head_base + v % group;
      val = to_f32<T>(q[(static_cast<size_t>(q_begin + tok0 + tok) * nh + head) * hd + dim]) * scale;
    }
    qs[i] = val;
  }
  int qpos[NV];
  int warp_p_max = -1, warp_p_min = 0x7fffffff;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int vec = warp * NV + v;
    qpos[v] = vec < nvec ? p_lo + vec / group : -1;
    if (qpos[v] >= 0) { warp_p_max = max(warp_p_max, qpos[v]); warp_p_min = min(warp_p_min, qpos[v]); }
  }
  VecState st;
  st.init();
  // The next block's copies run under this one's arithmetic where two blocks fit (`stages`).
  auto fetch = [&](int kb, int stage) {
    T* ks = tiles + stage * 2 * KB * G::STRIDE;
    const long long mine = lane_row(table, page_size, nkv, kvh, kb, kv_end);
    load_key_block<T>(ks, k_cache, mine, hd, hd, threadIdx.x, blockDim.x);
    load_key_block<T>(ks + KB * G::STRIDE, v_cache, mine, hd_v, v_stride, threadIdx.x, blockDim.x);
  };
  if (stages > 1) fetch(k_begin, 0);
  cp_async_commit();
  int stage = 0;
  for (int kb = k_begin; kb < kv_end; kb += KB) {
    __syncthreads();                                   // the block before is no longer read
    if (stages == 1) fetch(kb, 0);
    else if (kb + KB < kv_end) fetch(kb + KB, stage ^ 1);
    cp_async_commit();
    if (stages == 1) cp_async_wait<0>(); else cp_async_wait<1>();
    __syncthreads();
    const T* ks = tiles + stage * 2 * KB * G::STRIDE;
    const bool touches = warp_p_max >= kb && (window <= 0 || kb + KB - 1 > warp_p_min - window) &&
                         (chunk <= 0 || kb + KB - 1 >= warp_p_min - warp_p_min % chunk);
    if (touches)
      warp_key_block<T>(ks, ks + KB * G::STRIDE, qs + warp * NV * D, qpos, kb, kv_end, window, chunk, st, ps + warp * KB * NV, softcap);
    if (stages > 1) stage ^= 1;
  }
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int vec = warp * NV + v;
    if (vec >= nvec || (which >> vec & 1) == 0) continue;
    const int tok = vec / group, head = head_base + vec % group;
    T* dst = out + (static_cast<size_t>(q_begin + tok0 + tok) * nh + head) * hd_v;
    float l = st.l[v];
    if (sinks != nullptr && l > 0.0f) l += expf(sinks[head] - st.m[v]);
    const float inv = l > 0.0f ? 1.0f / l : 0.0f;
#pragma unroll
    for (int k = 0; k < PAIRS; ++k) {
      const int dim = 2 * lane + 64 * k;
      if (dim < hd_v) {
        dst[dim] = from_f32<T>(st.acc[v][2 * k] * inv);
        dst[dim + 1] = from_f32<T>(st.acc[v][2 * k + 1] * inv);
      }
    }
  }
}

// (Reached by bfloat16, and in float by heads above 128, of no multiple of 16, or of another width than their values; others have
// prefill_split_kernel below.  Builds for heads of 16 are held to three CTAs an SM: with 88 registers instead of 80 they had two, and 2,000
// float32 tokens behind 1,000, 40 query heads, took 2,949 us for 2,383.  0 leaves the others to the compiler, which stays at 80 or at what shared memory allows;
// told that one CTA is enough it took all registers, and heads of 32 6,336 us for 2,546.)
template <typename T>
__global__ void __launch_bounds__(PF_WARPS * 32, D <= 16 ? 3 : 0)
prefill_attention_kernel(const T* __restrict__ q, const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                         T* __restrict__ out, const int* __restrict__ block_table, int table_stride,
                         const int* __restrict__ cu_q, const int* __restrict__ kv_len,
                         const int* __restrict__ prefix_len, const int* __restrict__ rows, int nh, int nkv,
                         int page_size, int window, float scale, int tile_tokens, int head_chunks, int hd,
                         int hd_v, float softcap, int chunk, const float* __restrict__ sinks, int v_stride, int stages) {
  prefill_tile<T>(q, k_cache, v_cache, out, block_table, table_stride, cu_q, kv_len, prefix_len, rows, nh, nkv, page_size, window,
                  scale, tile_tokens, head_chunks, hd, hd_v, softcap, chunk, sinks, v_stride, stages, 0xffffffffu);
}

#if HEAD_DIM <= 128
// ------------------------------------------------------------------ prompt portions in float, on the tensor cores
// The same tiles (up to 32 query vectors of one KV head) with both products on mma.sync: a float is the exact sum of three
// bfloat16 terms, and of the nine products of two such floats the six that reach 2^-24 are taken, the small ones first.
// Every 16 columns (or keys) are summed from zero by the tensor cores and added to the rest in float by the thread, so that
// what they cut off below a sum's last place stays that of sixteen terms.
// Eight warps: two halves of the vectors (16 each) x four quarters of every block of 64 keys (16 keys each); each warp runs a
// softmax of its own over its keys and the four parts of a vector are added up at the end in order.  Which keys a warp takes
// depends on their positions alone, so a position's result has the same bits however the prompt was cut.
// The query's terms stay in registers; keys and values are taken apart as they are read, since a block serves two warps only.
// A vector whose result holds an infinity or a NaN is done again by prefill_tile (an infinity has no second term), and so is one with
// sums of weighted values below 2^-80: values below 2^-110 lose bits of their third term, for which bfloat16 ends at 2^-133.  The
// tile's other vectors keep what they have: which they share a tile with follows from how the prompt was cut.
// Bound by the latencies of two warps a scheduler (they issue in 34 % of its cycles), most of them those of taking keys and values apart
// (22 instructions for a thread's four numbers, six products).  us,
// CUDA cores / this: 16 heads of 128, 8 KV heads, 300 tokens 59.3 / 30.7, 17 tokens 13.5 / 10.5, 2,000 tokens 991 / 598, 64 behind 2,000
// cached 343 / 170, 16 rows of 5 behind 100 21.6 / 13.8; heads of 64, 300 tokens 42.3 / 18.7, of 16 37.6 / 11.5.  Error against 64 bits
// 7.2e-7 -> 2.5e-7 (300 tokens).  Heads beyond 128 or of another width than their values stay with prefill_tile.
constexpr int SPLIT_KEYS = 64;

struct SplitPrefill {
  static constexpr int K_ROW = D % 32 == 16 ? D : D + 16;      // floats of a row: 16-byte reads of two rows meet no bank twice
  static constexpr int V_ROW = D + 4;                          // four rows, two apart, of a column each
  static constexpr int STAGE = SPLIT_KEYS * (K_ROW + V_ROW);   // floats
  static constexpr int MERGE = 4 * 32 * (D + 4);               // floats: the four parts of 32 vectors
  static constexpr size_t TILES = sizeof(float) * (2 * STAGE > MERGE ? 2 * STAGE : MERGE);
  static constexpr size_t AGAIN = TILES + sizeof(float) * 4 * 32 * 2;      // a word: the vectors that are done again
  static constexpr size_t SMEM = AGAIN + 16;
};
__device__ __forceinline__ uint32_t* split_again() {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  return reinterpret_cast<uint32_t*>(smem_raw + SplitPrefill::AGAIN);
}

// Two floats as three bfloat16 terms each, packed (the first float in the low half): x = high + mid + low, each term the rest
// rounded to eight bits; exactly from 2^-110 on.
__device__ __forceinline__ void terms_of(float x, float y, uint32_t& high, uint32_t& mid, uint32_t& low) {
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(high) : "f"(y), "f"(x));
  x -= __uint_as_float(high << 16);
  y -= __uint_as_float(high & 0xffff0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(mid) : "f"(y), "f"(x));
  x -= __uint_as_float(mid << 16);
  y -= __uint_as_float(mid & 0xffff0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(low) : "f"(y), "f"(x));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// sum[n] += a . b[n] over 16 columns, a and b in three terms; the tiles' chains of products side by side.
template <int TILES>
__device__ __forceinline__ void add_products(float (*sum)[4], const uint32_t (&a)[3][4], const uint32_t (&b0)[TILES][3], const uint32_t (&b1)[TILES][3]) {
  constexpr int AI[6] = {2, 0, 1, 1, 0, 0}, BI[6] = {0, 2, 1, 0, 1, 0};
  float t[TILES][4] = {};
#pragma unroll
  for (int i = 0; i < 6; ++i)
#pragma unroll
    for (int n = 0; n < TILES; ++n) mma_bf16(t[n], a[AI[i]], b0[n][BI[i]], b1[n][BI[i]]);
#pragma unroll
  for (int n = 0; n < TILES; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) sum[n][i] += t[n][i];
}

__device__ __noinline__ void prefill_tile_again(const float* q, const float* k_cache, const float* v_cache, float* out,
                                                const int* block_table, int table_stride, const int* cu_q, const int* kv_len,
                                                const int* prefix_len, const int* rows, int nh, int nkv, int page_size, int window,
                                                float scale, int tile_tokens, int head_chunks, float softcap, int chunk,
                                                const float* sinks) {
  prefill_tile<float>(q, k_cache, v_cache, out, block_table, table_stride, cu_q, kv_len, prefix_len, rows, nh, nkv, page_size,
                      window, scale, tile_tokens, head_chunks, D, D, softcap, chunk, sinks, D, 1, *split_again());
}

__global__ void __launch_bounds__(PF_WARPS * 32, 1)
prefill_split_kernel(const float* __restrict__ q, const float* __restrict__ k_cache, const float* __restrict__ v_cache,
                     float* __restrict__ out, const int* __restrict__ block_table, int table_stride,
                     const int* __restrict__ cu_q, const int* __restrict__ kv_len, const int* __restrict__ prefix_len,
                     const int* __restrict__ rows, int nh, int nkv, int page_size, int window, float scale, int tile_tokens,
                     int head_chunks, float softcap, int chunk, const float* __restrict__ sinks) {
  using S = SplitPrefill;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* tiles = reinterpret_cast<float*>(smem_raw);                     // [2][K rows, V rows]
  float* parts_ml = reinterpret_cast<float*>(smem_raw + S::TILES);       // [4][32][2]
  const int row = rows[blockIdx.z];
  const int kvh = blockIdx.y / head_chunks, hc = blockIdx.y - kvh * head_chunks;
  const int head_base = kvh * (nh / nkv) + hc * 32;
  const int group = min(32, nh / nkv - hc * 32);
  const int q_begin = cu_q[row], q_len = cu_q[row + 1] - q_begin;
  const int tok0 = (gridDim.x - 1 - blockIdx.x) * tile_tokens;           // the tiles that see the most keys start first
  if (tok0 >= q_len) return;
  const int ntok = min(tile_tokens, q_len - tok0);
  const int nvec = ntok * group;
  const int p_lo = prefix_len[row] + tok0;
  const int kv_end = min(kv_len[row], p_lo + ntok);
  int k_begin = window > 0 ? max(0, p_lo - window + 1) : 0;
  if (chunk > 0) k_begin = max(k_begin, p_lo - p_lo % chunk);
  k_begin -= k_begin % SPLIT_KEYS;
  const int* table = block_table + static_cast<size_t>(row) * table_stride;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int half = warp >> 2, quarter = warp & 3;
  const int r = lane >> 2, c4 = lane & 3;                                // of a fragment: row (or column of B), place among four

  auto fetch = [&](int first, int stage) {
    float* ks = tiles + stage * S::STAGE;
    float* vs = ks + SPLIT_KEYS * S::K_ROW;
    const long long low = lane_row(table, page_size, nkv, kvh, first, kv_end), up = lane_row(table, page_size, nkv, kvh, first + 32, kv_end);
    constexpr int PIECES = D / 4;
#pragma unroll 4
    for (int i = threadIdx.x; i < SPLIT_KEYS * PIECES; i += PF_WARPS * 32) {
      const int key = i / PIECES, part = i - key * PIECES;
      const long long a = __shfl_sync(0xffffffffu, low, key & 31), b = __shfl_sync(0xffffffffu, up, key & 31);
      const long long at = key < 32 ? a : b;
      cp_async16(ks + key * S::K_ROW + part * 4, at >= 0 ? k_cache + at * D + part * 4 : k_cache, at >= 0);
      cp_async16(vs + key * S::V_ROW + part * 4, at >= 0 ? v_cache + at * D + part * 4 : v_cache, at >= 0);
    }
  };
  fetch(k_begin, 0);
  cp_async_commit();

  // The warp's 16 vectors, rows r and r + 8 of a fragment: their positions, and their terms (four columns 16 s + 4 c4 .. + 3 of
  // a k-step s: the tensor cores sum over k, in whatever order both operands hold it).
  int pos[2];
  uint32_t qt[D / 16][3][4];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int vec = half * 16 + r + 8 * e;
    const bool used = vec < nvec;
    pos[e] = used ? p_lo + vec / group : -1;
    const float* src = q + (static_cast<size_t>(q_begin + tok0 + (used ? vec / group : 0)) * nh + head_base + (used ? vec % group : 0)) * D;
#pragma unroll
    for (int s = 0; s < D / 16; ++s) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (used) v = *reinterpret_cast<const float4*>(src + 16 * s + 4 * c4);
      terms_of(v.x * scale, v.y * scale, qt[s][0][e], qt[s][1][e], qt[s][2][e]);
      terms_of(v.z * scale, v.w * scale, qt[s][0][2 + e], qt[s][1][2 + e], qt[s][2][2 + e]);
    }
  }
  int p_max = max(pos[0], pos[1]), p_min = min(pos[0] < 0 ? 0x7fffffff : pos[0], pos[1] < 0 ? 0x7fffffff : pos[1]);
  p_max = __reduce_max_sync(0xffffffffu, p_max);
  p_min = __reduce_min_sync(0xffffffffu, p_min);
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.0f, 0.0f}, o[D / 8][4];
#pragma unroll
  for (int n = 0; n < D / 8; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) o[n][i] = 0.0f;

  int stage = 0;
  for (int kb = k_begin; kb < kv_end; kb += SPLIT_KEYS, stage ^= 1) {
    if (kb + SPLIT_KEYS < kv_end) fetch(kb + SPLIT_KEYS, stage ^ 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    const int first = kb + 16 * quarter;
    if (p_max >= first && first < kv_end && (window <= 0 || first + 15 > p_min - window) && (chunk <= 0 || first + 15 >= p_min - p_min % chunk)) {
      const float* ks = tiles + stage * S::STAGE + 16 * quarter * S::K_ROW;
      const float* vs = tiles + stage * S::STAGE + SPLIT_KEYS * S::K_ROW + 16 * quarter * S::V_ROW;
      float s[2][4] = {};                                                // scores: keys 8 t + 2 c4, + 1 of rows r and r + 8
#pragma unroll
      for (int step = 0; step < D / 16; ++step) {
        uint32_t b0[2][3], b1[2][3];
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const float4 kv = *reinterpret_cast<const float4*>(ks + (8 * t + r) * S::K_ROW + 16 * step + 4 * c4);
          terms_of(kv.x, kv.y, b0[t][0], b0[t][1], b0[t][2]);
          terms_of(kv.z, kv.w, b1[t][0], b1[t][1], b1[t][2]);
        }
        add_products<2>(s, qt[step], b0, b1);
      }
      uint32_t pt[3][4];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float v[4], mx = -INFINITY;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int key = first + 8 * (i >> 1) + 2 * c4 + (i & 1), p = pos[e];
          float x = s[i >> 1][2 * e + (i & 1)];
          if (softcap > 0.0f) x = softcap * tanhf(x * (1.0f / softcap));
          const bool visible = p >= 0 && key <= p && key < kv_end && (window <= 0 || key > p - window) && (chunk <= 0 || key >= p - p % chunk);
          v[i] = visible ? x : -INFINITY;
          mx = fmaxf(mx, v[i]);
        }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float top = fmaxf(m[e], mx);
        float sum = 0.0f, corr = 1.0f;
        if (top != -INFINITY) {
          corr = expf(m[e] - top);
#pragma unroll
          for (int i = 0; i < 4; ++i) { v[i] = expf(v[i] - top); sum += v[i]; }
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) v[i] = v[i] != v[i] ? v[i] : 0.0f;   // (a NaN stays one: the tile is done again)
        }
        l[e] = l[e] * corr + sum;                                        // (this lane's keys; the four lanes are added up at the end)
        m[e] = top;
        terms_of(v[0], v[1], pt[0][e], pt[1][e], pt[2][e]);
        terms_of(v[2], v[3], pt[0][2 + e], pt[1][2 + e], pt[2][2 + e]);
        if (__any_sync(0xffffffffu, corr != 1.0f ? 1 : 0))
#pragma unroll
          for (int n = 0; n < D / 8; ++n) { o[n][2 * e] *= corr; o[n][2 * e + 1] *= corr; }
      }
#pragma unroll
      for (int n = 0; n < D / 8; n += 2) {
        uint32_t b0[2][3], b1[2][3];
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const float* col = vs + 8 * (n + t) + r + 2 * c4 * S::V_ROW;
          terms_of(col[0], col[S::V_ROW], b0[t][0], b0[t][1], b0[t][2]);
          terms_of(col[8 * S::V_ROW], col[9 * S::V_ROW], b1[t][0], b1[t][1], b1[t][2]);
        }
        add_products<2>(o + n, pt, b0, b1);
      }
    }
    __syncthreads();                                                     // this block is read: the next copies may overwrite it
  }
  // The four parts of a vector.
  if (threadIdx.x == 0) *split_again() = 0;
  float* parts = tiles;                                                  // [4][32][D + 4]
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int vec = half * 16 + r + 8 * e;
    float sum = l[e] + __shfl_xor_sync(0xffffffffu, l[e], 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if (c4 == 0) {
      parts_ml[(quarter * 32 + vec) * 2] = m[e];
      parts_ml[(quarter * 32 + vec) * 2 + 1] = sum;
    }
#pragma unroll
    for (int n = 0; n < D / 8; ++n)
      *reinterpret_cast<float2*>(parts + (quarter * 32 + vec) * (D + 4) + 8 * n + 2 * c4) = make_float2(o[n][2 * e], o[n][2 * e + 1]);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nvec * (D / 4); i += PF_WARPS * 32) {
    const int vec = i / (D / 4), at = i - vec * (D / 4);
    float top = -INFINITY;
#pragma unroll
    for (int w = 0; w < 4; ++w) top = fmaxf(top, parts_ml[(w * 32 + vec) * 2]);
    float sum = 0.0f, acc[4] = {};
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float pm = parts_ml[(w * 32 + vec) * 2], f = top == -INFINITY ? 0.0f : expf(pm - top);
      const float4 v = *reinterpret_cast<const float4*>(parts + (w * 32 + vec) * (D + 4) + 4 * at);
      sum += parts_ml[(w * 32 + vec) * 2 + 1] * f;
      acc[0] += v.x * f; acc[1] += v.y * f; acc[2] += v.z * f; acc[3] += v.w * f;
    }
    const int tok = vec / group, head = head_base + vec % group;
    if (sinks != nullptr && sum > 0.0f) sum += expf(sinks[head] - top);
    const float inv = sum > 0.0f ? 1.0f / sum : 0.0f;
    const float4 v = make_float4(acc[0] * inv, acc[1] * inv, acc[2] * inv, acc[3] * inv);
    bool settled = fabsf(sum) < INFINITY;
#pragma unroll
    for (int e = 0; e < 4; ++e) settled = settled && fabsf(acc[e]) < INFINITY && (fabsf(acc[e]) >= 8.2718061e-25f || acc[e] == 0.0f);
    if (!settled) atomicOr(split_again(), 1u << vec);
    *reinterpret_cast<float4*>(out + (static_cast<size_t>(q_begin + tok0 + tok) * nh + head) * D + 4 * at) = v;
  }
  __syncthreads();
  if (*split_again() != 0)
    prefill_tile_again(q, k_cache, v_cache, out, block_table, table_stride, cu_q, kv_len, prefix_len, rows, nh, nkv, page_size, window,
                       scale, tile_tokens, head_chunks, softcap, chunk, sinks);
}
#endif

// ------------------------------------------------------------------ decoded tokens, split over the keys
// grid (splits, nkv * vector groups, decode rows); DEC_WARPS warps, each walking its own key blocks
// through a private two-stage cp.async pipeline.  A CTA serves up to 4 query heads of one KV head
// (vector group vg holds heads kvh * group + 4 * vg ..).  Split s of a row covers an equal share of
// the row's key blocks; it writes (max, sum, unnormalised output) per head to scratch, or the
// final output when there is one split.
// DEC_WARPS is 4 where the tiles of four warps fit shared memory, else 2 or 1 (large heads in float).
template <typename T, int DEC_WARPS>
__global__ void __launch_bounds__(DEC_WARPS * 32)
decode_attention_kernel(const T* __restrict__ q, const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                        T* __restrict__ out, float* __restrict__ part_acc, float* __restrict__ part_ml,
                        const int* __restrict__ block_table, int table_stride, const int* __restrict__ cu_q,
                        const int* __restrict__ kv_len, const int* __restrict__ rows, int nh, int nkv,
                        int page_size, int window, float scale, int vec_groups, int stages, int hd, int hd_v,
                        float softcap, int chunk, const float* __restrict__ sinks, int v_stride) {
  using G = RowGeom<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* qs = reinterpret_cast<float*>(smem_raw);                        // [NV][D]
  float* ps = qs + NV * D;                                               // [DEC_WARPS][32 * NV]
  T* tiles = reinterpret_cast<T*>(ps + DEC_WARPS * KB * NV);             // [DEC_WARPS][stages][2][32][STRIDE]

  const int splits = gridDim.x, split = blockIdx.x;
  const int kvh = blockIdx.y / vec_groups, vg = blockIdx.y - kvh * vec_groups;
  const int row = rows[blockIdx.z];
  const int group = nh / nkv;
  const int head0 = kvh * group + vg * NV;
  const int nvec = min(NV, group - vg * NV);
  const int tok = cu_q[row];
  const int kv_end = kv_len[row];
  const int qp = kv_end - 1;                                             // the decoded token's position
  int k_begin = window > 0 ? max(0, qp - window + 1) : 0;
  if (chunk > 0) k_begin = max(k_begin, qp - qp % chunk);
  k_begin -= k_begin % KB;
  const int blocks_total = (kv_end - k_begin + KB - 1) / KB;
  const int per_split = (blocks_total + splits - 1) / splits;
  const int blk_lo = split * per_split, blk_hi = min(blocks_total, blk_lo + per_split);
  const int* table = block_table + static_cast<size_t>(row) * table_stride;

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < NV * D; i += blockDim.x) {
    const int v = i / D, dim = i - v * D;
    qs[i] = (v < nvec && dim < hd) ? to_f32<T>(q[(static_cast<size_t>(tok) * nh + head0 + v) * hd + dim]) * scale : 0.0f;
  }
  __syncthreads();
  int qpos[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) qpos[v] = v < nvec ? qp : -1;

  const int tile_elems = 2 * KB * G::STRIDE;
  T* my_tiles = tiles + static_cast<size_t>(warp) * stages * tile_elems;
  VecState st;
  st.init();
  // Prologue: issue the first `stages - 1` blocks of this warp.
  int issue = blk_lo + warp;
  for (int s = 0; s < stages - 1; ++s) {
    if (issue < blk_hi) {
      T* t = my_tiles + s * tile_elems;
      const long long mine = lane_row(table, page_size, nkv, kvh, k_begin + issue * KB, kv_end);
      load_key_block<T>(t, k_cache, mine, hd, hd, lane, 32);
      load_key_block<T>(t + KB * G::STRIDE, v_cache, mine, hd_v, v_stride, lane, 32);
    }
    cp_async_commit();
    issue += DEC_WARPS;
  }
  int stage = 0;
  for (int blk = blk_lo + warp; blk < blk_hi; blk += DEC_WARPS) {
    if (stages > 1) {
      const int s_issue = (stage + stages - 1) % stages;
      if (issue < blk_hi) {
        T* t = my_tiles + s_issue * tile_elems;
        const long long mine = lane_row(table, page_size, nkv, kvh, k_begin + issue * KB, kv_end);
        load_key_block<T>(t, k_cache, mine, hd, hd, lane, 32);
        load_key_block<T>(t + KB * G::STRIDE, v_cache, mine, hd_v, v_stride, lane, 32);
      }
      cp_async_commit();
      issue += DEC_WARPS;
      cp_async_wait<1>();          // stages is 1 or 2: all but the newest group have landed
    } else {
      T* t = my_tiles;
      const long long mine = lane_row(table, page_size, nkv, kvh, k_begin + blk * KB, kv_end);
      load_key_block<T>(t, k_cache, mine, hd, hd, lane, 32);
      load_key_block<T>(t + KB * G::STRIDE, v_cache, mine, hd_v, v_stride, lane, 32);
      cp_async_commit();
      cp_async_wait<0>();
    }
    __syncwarp();
    const T* t = my_tiles + stage * tile_elems;
    warp_key_block<T>(t, t + KB * G::STRIDE, qs, qpos, k_begin + blk * KB, kv_end, window, chunk, st,
                      ps + warp * KB * NV, softcap);
    stage = (stage + 1) % stages;
  }
  cp_async_wait<0>();
  __syncthreads();
  // Merge the warps: shared memory is reused as [DEC_WARPS][NV][D + 2] floats.
  float* merge = reinterpret_cast<float*>(tiles);
  constexpr int MS = D + 2;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    float* dst = merge + (warp * NV + v) * MS;
#pragma unroll
    for (int k = 0; k < PAIRS; ++k) {
      const int dim = 2 * lane + 64 * k;
      if (dim < D) { dst[dim] = st.acc[v][2 * k]; dst[dim + 1] = st.acc[v][2 * k + 1]; }
    }
    if (lane == 0) { dst[D] = st.m[v]; dst[D + 1] = st.l[v]; }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nvec * D; i += blockDim.x) {
    const int v = i / D, dim = i - v * D;
    float m = -INFINITY;
#pragma unroll
    for (int w = 0; w < DEC_WARPS; ++w) m = fmaxf(m, merge[(w * NV + v) * MS + D]);
    float l = 0.0f, o = 0.0f;
    if (m != -INFINITY) {
#pragma unroll
      for (int w = 0; w < DEC_WARPS; ++w) {
        const float* src = merge + (w * NV + v) * MS;
        const float f = expf(src[D] - m);
        l += src[D + 1] * f;
        o += src[dim] * f;
      }
    }
    const int head = head0 + v;
    if (splits == 1) {
      if (sinks != nullptr && l > 0.0f) l += expf(sinks[head] - m);
      if (dim < hd_v) out[(static_cast<size_t>(tok) * nh + head) * hd_v + dim] = from_f32<T>(l > 0.0f ? o / l : 0.0f);
    } else {
      const size_t slot = (static_cast<size_t>(blockIdx.z) * nh + head) * splits + split;
      part_acc[slot * D + dim] = o;
      if (dim == 0) { part_ml[slot * 2] = m; part_ml[slot * 2 + 1] = l; }
    }
  }
}

// grid (decode rows, nh): combines the splits of one head.
template <typename T>
__global__ void decode_merge_kernel(T* __restrict__ out, const float* __restrict__ part_acc,
                                    const float* __restrict__ part_ml, const int* __restrict__ cu_q,
                                    const int* __restrict__ rows, int nh, int splits, int hd,
                                    const float* __restrict__ sinks) {
  const int head = blockIdx.y;
  const int tok = cu_q[rows[blockIdx.x]];
  const size_t base = (static_cast<size_t>(blockIdx.x) * nh + head) * splits;
  float m = -INFINITY;
  for (int s = 0; s < splits; ++s) m = fmaxf(m, part_ml[(base + s) * 2]);
  for (int dim = threadIdx.x; dim < hd; dim += blockDim.x) {
    float l = 0.0f, o = 0.0f;
    if (m != -INFINITY) {
      for (int s = 0; s < splits; ++s) {
        const float f = expf(part_ml[(base + s) * 2] - m);
        l += part_ml[(base + s) * 2 + 1] * f;
        o += part_acc[(base + s) * D + dim] * f;
      }
      if (sinks != nullptr && l > 0.0f) l += expf(sinks[head] - m);
    }
    out[(static_cast<size_t>(tok) * nh + head) * hd + dim] = from_f32<T>(l > 0.0f ? o / l : 0.0f);
  }
}

// ------------------------------------------------------------------ launchers
// A prefill CTA: two blocks of keys and values where two CTAs of that size still share an SM, else one.
template <typename T>
struct PrefillShape {
  static constexpr size_t FIXED = (32 * D + PF_WARPS * KB * NV) * sizeof(float), BLOCK = 2 * KB * RowGeom<T>::STRIDE * sizeof(T);
  static constexpr int STAGES = FIXED + 2 * BLOCK <= 110 * 1024 ? 2 : 1;
  static constexpr size_t SMEM = FIXED + STAGES * BLOCK;
};
// How many prefill CTAs an SM of the current device holds (tests: their registers decide how fast long prompts are).
template <typename T>
static int prefill_ctas_per_sm() {
  int n = 0;
  cudaError_t e = cudaFuncSetAttribute(prefill_attention_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(PrefillShape<T>::SMEM));
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, prefill_attention_kernel<T>, PF_WARPS * 32, PrefillShape<T>::SMEM);
  return e == cudaSuccess ? n : -static_cast<int>(e);
}
B200_EXPORT int b200_prefill_attention_ctas_per_sm(int dtype) {
  return dtype == B200_F32 ? prefill_ctas_per_sm<float>() : prefill_ctas_per_sm<__nv_bfloat16>();
}

#if HEAD_DIM <= 128
// Local memory of prefill_split_kernel, whose terms of the query and accumulators take up to all of a thread's registers (one CTA an SM
// at every head size): anything above zero are spills.
B200_EXPORT int b200_prefill_split_local_bytes(void) {
  cudaFuncAttributes a;
  const cudaError_t e = cudaFuncGetAttributes(&a, prefill_split_kernel);
  return e == cudaSuccess ? static_cast<int>(a.localSizeBytes) : -static_cast<int>(e);
}
#endif

template <typename T>
static int launch_prefill(const void* q, const void* kc, const void* vc, void* out, const int* block_table,
                          int table_stride, const int* cu_q, const int* kv_len, const int* prefix_len,
                          const int* rows, int n_rows, int max_q_len, int nh, int nkv, int page_size, int window,
                          float scale, int hd, int hd_v, float softcap, int chunk, const float* sinks,
                          int v_stride, cudaStream_t stream) {
  using G = RowGeom<T>;
  const int group = nh / nkv;
  const int head_chunks = (group + 31) / 32;                  // more than 32 query heads per KV head: several CTAs
  const int tile_tokens = group >= 32 ? 1 : 32 / group;
  constexpr int stages = PrefillShape<T>::STAGES;
  constexpr size_t smem = PrefillShape<T>::SMEM;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(prefill_attention_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    configured = true;
  }
  if (static_cast<long long>(nkv) * head_chunks > 65535 || n_rows > 65535) return B200_BAD_SIZE;
  dim3 grid((max_q_len + tile_tokens - 1) / tile_tokens, nkv * head_chunks, n_rows);
#if HEAD_DIM <= 128
  if constexpr (sizeof(T) == 4) {
    const auto aligned = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
    if (hd == D && hd_v == D && (v_stride <= 0 || v_stride == D) && aligned(q) && aligned(kc) && aligned(vc) && aligned(out)) {
      static_assert(SplitPrefill::AGAIN >= PrefillShape<float>::FIXED + PrefillShape<float>::BLOCK, "a tile may be done again");
      constexpr int DEVICES = 16;                              // whose launch limit is remembered
      static bool split_configured[DEVICES];
      int device = 0;
      cudaError_t e = cudaGetDevice(&device);
      if (e == cudaSuccess && (device >= DEVICES || !split_configured[device])) {
        e = cudaFuncSetAttribute(prefill_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SplitPrefill::SMEM));
        if (e == cudaSuccess && device < DEVICES) split_configured[device] = true;
      }
      if (e != cudaSuccess) return static_cast<int>(e);
      prefill_split_kernel<<<grid, PF_WARPS * 32, SplitPrefill::SMEM, stream>>>(
          static_cast<const float*>(q), static_cast<const float*>(kc), static_cast<const float*>(vc), static_cast<float*>(out), block_table,
          table_stride, cu_q, kv_len, prefix_len, rows, nh, nkv, page_size, window, scale, tile_tokens, head_chunks, softcap, chunk, sinks);
      return b200_check_launch();
    }
  }
#endif
  prefill_attention_kernel<T><<<grid, PF_WARPS * 32, smem, stream>>>(
      static_cast<const T*>(q), static_cast<const T*>(kc), static_cast<const T*>(vc), static_cast<T*>(out),
      block_table, table_stride, cu_q, kv_len, prefix_len, rows, nh, nkv, page_size, window, scale, tile_tokens,
      head_chunks, hd, hd_v, softcap, chunk, sinks, v_stride > 0 ? v_stride : hd_v, stages);
  return b200_check_launch();
}

// A decode CTA: four warps with two stages of keys and values each where that fits, else one stage, else fewer warps.
template <typename T>
struct DecodeShape {
  static constexpr size_t TILE = 2 * KB * RowGeom<T>::STRIDE * sizeof(T), LIMIT = 200 * 1024;
  static constexpr size_t FIXED4 = (NV * D + 4 * KB * NV) * sizeof(float);
  static constexpr int WARPS = FIXED4 + 4 * TILE <= LIMIT ? 4 : (FIXED4 + 2 * TILE <= LIMIT ? 2 : 1);
  static constexpr size_t FIXED = (NV * D + WARPS * KB * NV) * sizeof(float);
  static_assert(FIXED + WARPS * TILE <= 220 * 1024, "one key block per warp must fit shared memory");
  static constexpr int STAGES = FIXED + WARPS * 2 * TILE <= LIMIT ? 2 : 1;
  static constexpr size_t MERGE = WARPS * NV * (D + 2) * sizeof(float);
  static constexpr size_t SMEM = FIXED + (MERGE > WARPS * STAGES * TILE ? MERGE : WARPS * STAGES * TILE);
};
// Shared memory of a decode CTA in bytes: how many of them an SM holds.
B200_EXPORT int b200_decode_attention_smem(int dtype) {
  return static_cast<int>(dtype == B200_F32 ? DecodeShape<float>::SMEM : DecodeShape<__nv_bfloat16>::SMEM);
}

template <typename T>
static int launch_decode(const void* q, const void* kc, const void* vc, void* out, float* part_acc, float* part_ml,
                         const int* block_table, int table_stride, const int* cu_q, const int* kv_len,
                         const int* rows, int n_rows, int nh, int nkv, int page_size, int window, float scale,
                         int splits, int hd, int hd_v, float softcap, int chunk, const float* sinks,
                         int v_stride, cudaStream_t stream) {
  using G = RowGeom<T>;
  const int group = nh / nkv;
  const int vec_groups = (group + NV - 1) / NV;
  constexpr int DEC_WARPS = DecodeShape<T>::WARPS, stages = DecodeShape<T>::STAGES;
  constexpr size_t smem = DecodeShape<T>::SMEM;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(decode_attention_kernel<T, DEC_WARPS>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    configured = true;
  }
  dim3 grid(splits, nkv * vec_groups, n_rows);
  decode_attention_kernel<T, DEC_WARPS><<<grid, DEC_WARPS * 32, smem, stream>>>(
      static_cast<const T*>(q), static_cast<const T*>(kc), static_cast<const T*>(vc), static_cast<T*>(out),
      part_acc, part_ml, block_table, table_stride, cu_q, kv_len, rows, nh, nkv, page_size, window, scale,
      vec_groups, stages, hd, hd_v, softcap, chunk, sinks, v_stride > 0 ? v_stride : hd_v);
  int rc = b200_check_launch();
  if (rc != 0 || splits == 1) return rc;
  dim3 mgrid(n_rows, nh);
  decode_merge_kernel<T><<<mgrid, D >= 128 ? 128 : 64, 0, stream>>>(static_cast<T*>(out), part_acc, part_ml, cu_q,
                                                                   rows, nh, splits, hd_v, sinks);
  return b200_check_launch();
}

B200_EXPORT int b200_attention_head_dim() { return D; }

// Portions of prompts.  `rows` lists the batch rows to serve (n_rows of them); max_q_len bounds their length.
B200_EXPORT int b200_prefill_attention(const void* q, const void* k_cache, const void* v_cache, void* out,
                                       const int* block_table, int table_stride, const int* cu_q,
                                       const int* kv_len, const int* prefix_len, const int* rows, int n_rows,
                                       int max_q_len, int nh, int nkv, int page_size, int window, float scale,
                                       int dtype, int head_dim, int v_head_dim, float softcap, int chunk,
                                       const float* sinks, int v_stride, cudaStream_t stream) {
  if (n_rows <= 0 || max_q_len <= 0) return 0;
  if (nh <= 0 || nkv <= 0 || nh % nkv != 0 || page_size <= 0) return B200_BAD_SIZE;
  if (head_dim <= 0 || head_dim > D || (head_dim & 1)) return B200_BAD_SIZE;
  if (v_head_dim <= 0 || v_head_dim > D || (v_head_dim & 1)) return B200_BAD_SIZE;
  if (dtype == B200_F32)
    return launch_prefill<float>(q, k_cache, v_cache, out, block_table, table_stride, cu_q, kv_len, prefix_len,
                                 rows, n_rows, max_q_len, nh, nkv, page_size, window, scale, head_dim, v_head_dim,
                                 softcap, chunk, sinks, v_stride, stream);
  if (dtype == B200_BF16)
    return launch_prefill<__nv_bfloat16>(q, k_cache, v_cache, out, block_table, table_stride, cu_q, kv_len,
                                         prefix_len, rows, n_rows, max_q_len, nh, nkv, page_size, window, scale,
                                         head_dim, v_head_dim, softcap, chunk, sinks, v_stride, stream);
  return B200_BAD_DTYPE;
}

// Scratch floats that b200_decode_attention needs for (n_rows, nh, splits): acc then (max, sum); rows of HEAD_DIM
// floats whatever the real head size.
B200_EXPORT long long b200_decode_scratch_floats(int n_rows, int nh, int splits) {
  return splits <= 1 ? 0 : static_cast<long long>(n_rows) * nh * splits * (D + 2);
}

// Single decoded tokens.  `scratch` holds b200_decode_scratch_floats(...) floats (unused when splits == 1).
B200_EXPORT int b200_decode_attention(const void* q, const void* k_cache, const void* v_cache, void* out,
                                      float* scratch, const int* block_table, int table_stride,
                                      const int* cu_q, const int* kv_len, const int* rows, int n_rows, int nh,
                                      int nkv, int page_size, int window, float scale, int splits, int dtype,
                                      int head_dim, int v_head_dim, float softcap, int chunk, const float* sinks,
                                      int v_stride, cudaStream_t stream) {
  if (n_rows <= 0) return 0;
  if (nh <= 0 || nkv <= 0 || nh % nkv != 0 || page_size <= 0 || splits <= 0) return B200_BAD_SIZE;
  if (head_dim <= 0 || head_dim > D || (head_dim & 1)) return B200_BAD_SIZE;
  if (v_head_dim <= 0 || v_head_dim > D || (v_head_dim & 1)) return B200_BAD_SIZE;
  float* part_acc = scratch;
  float* part_ml = scratch + static_cast<size_t>(n_rows) * nh * splits * D;
  if (dtype == B200_F32)
    return launch_decode<float>(q, k_cache, v_cache, out, part_acc, part_ml, block_table, table_stride, cu_q,
                                kv_len, rows, n_rows, nh, nkv, page_size, window, scale, splits, head_dim, v_head_dim,
                                softcap, chunk, sinks, v_stride, stream);
  if (dtype == B200_BF16)
    return launch_decode<__nv_bfloat16>(q, k_cache, v_cache, out, part_acc, part_ml, block_table, table_stride,
                                        cu_q, kv_len, rows, n_rows, nh, nkv, page_size, window, scale, splits,
                                        head_dim, v_head_dim, softcap, chunk, sinks, v_stride, stream);
  return B200_BAD_DTYPE;
}
