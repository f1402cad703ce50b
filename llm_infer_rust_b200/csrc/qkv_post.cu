// What stands between the QKV projection and attention, in one kernel:
// per-head RMSNorm of q and k, half-split rotary position encoding of q and k,
// and the store of k and v into the paged cache.  One warp owns one
// (token, head); the head's values are read once and written once.
//
// Reference semantics: src/layers/fused_ops.cu:69-87 (per-head norm, float sum
// of squares, rsqrt(mean + eps) * weight), :108-133 (rotation in float from a
// float cos/sin table, pairs (i, i + rot/2)), src/models/attention/kv_store.cu:7-33
// (copy to the row of cache slot = page * page_size + offset; slot 0 is skipped).  The reference runs three kernels
// and rounds after the norm and again after the rotation; here both happen in
// float and the value is rounded once.  A position beyond the table or a slot
// outside the pool sets an error bit and the access is skipped (the reference
// skips the first silently and asserts on the second).
#include "common.cuh"

constexpr int MAX_HEAD_DIM = 512;
constexpr int WARPS = 4;

template <typename TA, typename TW>
__global__ void qkv_post_kernel(const TA* __restrict__ qkv, TA* __restrict__ q_out,
                                TA* __restrict__ k_cache, TA* __restrict__ v_cache,
                                const TW* __restrict__ q_w, const TW* __restrict__ k_w, float eps,
                                const float* __restrict__ cos_table, const float* __restrict__ sin_table,
                                int rot_dim, int max_pos, const int* __restrict__ positions,
                                const int* __restrict__ slots, int tokens, int nh, int nkv, int d,
                                int page_size, long long cache_slots, int* err) {
  __shared__ float buf[WARPS][MAX_HEAD_DIM];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int heads = nh + 2 * nkv;
  const long long work = static_cast<long long>(blockIdx.x) * WARPS + warp;
  if (work >= static_cast<long long>(tokens) * heads) return;
  const int t = static_cast<int>(work / heads);
  const int h = static_cast<int>(work - static_cast<long long>(t) * heads);
  const TA* src = qkv + (static_cast<size_t>(t) * heads + h) * d;
  const bool is_q = h < nh, is_k = !is_q && h < nh + nkv;

  TA* dst;
  if (is_q) {
    dst = q_out + (static_cast<size_t>(t) * nh + h) * d;
  } else {
    if (slots == nullptr) return;                 // this execution reads another entry's cache
    const int slot = slots[t];
    if (slot == 0) return;                        // the sink: padding rows write nothing
    if (slot < 0 || slot >= cache_slots) {
      if (lane == 0) atomicOr(err, B200_ERR_SLOT_RANGE);
      return;
    }
    const int kvh = is_k ? h - nh : h - nh - nkv;
    // cache[page][kv head][offset in page][d]: a page's rows of one KV head are contiguous
    const int page = slot / page_size, offset = slot - page * page_size;
    dst = (is_k ? k_cache : v_cache) + ((static_cast<size_t>(page) * nkv + kvh) * page_size + offset) * d;
  }
  if (!is_q && !is_k) {                           // v: a plain copy
    for (int i = lane; i < d; i += 32) dst[i] = src[i];
    return;
  }

  float* row = buf[warp];
  float ss = 0.0f;
  for (int i = lane; i < d; i += 32) {
    const float v = to_f32<TA>(src[i]);
    row[i] = v;
    ss += v * v;
  }
  const TW* w = is_q ? q_w : k_w;
  if (w != nullptr) {
    ss = warp_sum(ss);
    const float scale = rsqrtf(ss / static_cast<float>(d) + eps);
    for (int i = lane; i < d; i += 32) row[i] = row[i] * scale * to_f32<TW>(w[i]);
  }
  __syncwarp();
  const int half = rot_dim / 2;
  bool rotate = cos_table != nullptr && half > 0;
  int pos = 0;
  if (rotate) {
    pos = positions[t];
    if (pos < 0 || pos >= max_pos) {
      if (lane == 0) atomicOr(err, B200_ERR_POSITION_RANGE);
      rotate = false;
    }
  }
  if (rotate) {
    const float* c = cos_table + static_cast<size_t>(pos) * half;
    const float* s = sin_table + static_cast<size_t>(pos) * half;
    for (int i = lane; i < half; i += 32) {
      const float a = row[i], b = row[i + half];
      dst[i] = from_f32<TA>(a * c[i] - b * s[i]);
      dst[i + half] = from_f32<TA>(b * c[i] + a * s[i]);
    }
    for (int i = rot_dim + lane; i < d; i += 32) dst[i] = from_f32<TA>(row[i]);
  } else {
    for (int i = lane; i < d; i += 32) dst[i] = from_f32<TA>(row[i]);
  }
}

// The same work for heads whose size is 16 bytes times a power of two of at most 32 (64, 128 or 256 elements in bfloat16)
// and a rotation over the whole head: `lanes` = head_dim / (elements of 16 bytes) lanes share HG heads of one
// token.  A lane holds 8 bytes of a head's first half and the 8 bytes that they are rotated with, so the rotation needs no
// other lane; its angles and the token's position and slot are fetched once for the HG heads (a head's angles are twice its
// bytes), and all heads' loads are in flight together.  Bound by memory at many tokens, where HG = 4 saves most (one head a
// lane group with its halves in different lanes, bfloat16, 32 + 2 x 8 heads of 128: 22.7 -> 16.7 us at 2,048 tokens, 84.6 -> 75.9
// at 8,192; float32, 16 + 2 x 8 heads: 23.3 -> 16.5 and 82.6 -> 58.9 us), and by the latency of a lane's chain at few, where one
// head after the other is that chain (see heads_a_group).
template <typename TA> struct Half16;                           // 8 bytes of a row as floats, and back
template <> struct Half16<float> {
  static constexpr int N = 2;
  __device__ __forceinline__ static void load(const float* p, float (&v)[2]) {
    const float2 a = *reinterpret_cast<const float2*>(p);
    v[0] = a.x; v[1] = a.y;
  }
  __device__ __forceinline__ static void store(float* p, const float (&v)[2]) { *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]); }
};
template <> struct Half16<__nv_bfloat16> {
  static constexpr int N = 4;
  __device__ __forceinline__ static void load(const __nv_bfloat16* p, float (&v)[4]) { load_floats<__nv_bfloat16, 4>(p, v); }
  __device__ __forceinline__ static void store(__nv_bfloat16* p, const float (&v)[4]) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
  }
};
// N consecutive floats or bfloat16 numbers, N = 2 or 4, aligned to what they occupy.
template <typename T, int N>
__device__ __forceinline__ void load_few(const T* p, float (&v)[N]) {
  if constexpr (sizeof(T) == 4 && N == 4) load_floats<float, 4>(p, v);
  else if constexpr (sizeof(T) == 2 && N == 4) load_floats<__nv_bfloat16, 4>(p, v);
  else {
#pragma unroll
    for (int e = 0; e < N; ++e) v[e] = to_f32<T>(p[e]);
  }
}

template <typename TA, typename TW, int HG>
__global__ void __launch_bounds__(256)
qkv_post_vec_kernel(const TA* __restrict__ qkv, TA* __restrict__ q_out, TA* __restrict__ k_cache,
                    TA* __restrict__ v_cache, const TW* __restrict__ q_w, const TW* __restrict__ k_w, float eps,
                    const float* __restrict__ cos_table, const float* __restrict__ sin_table, int max_pos,
                    const int* __restrict__ positions, const int* __restrict__ slots, int tokens, int nh, int nkv,
                    int d, int page_size, long long cache_slots, int lanes, int* err) {
  constexpr int N = Half16<TA>::N;
  const int heads = nh + 2 * nkv, head_groups = (heads + HG - 1) / HG;
  const int sub = threadIdx.x % lanes;                          // this lane's place inside its heads
  const long long work = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) / lanes;
  const bool live = work < static_cast<long long>(tokens) * head_groups;
  const int t = live ? static_cast<int>(work / head_groups) : 0;
  const int h0 = live ? static_cast<int>(work - static_cast<long long>(t) * head_groups) * HG : 0;
  const int here = live ? min(HG, heads - h0) : 0;
  const bool turns = cos_table != nullptr && h0 < nh + nkv && here > 0;
  const bool stores = slots != nullptr && h0 + here > nh;
  // The token's position and slot first, and the angles as soon as the position is known: they depend on nothing else.
  const int pos = turns ? positions[t] : 0;
  const int slot = stores ? slots[t] : 0;
  float a[HG][N], b[HG][N];
#pragma unroll
  for (int i = 0; i < HG; ++i) {
#pragma unroll
    for (int e = 0; e < N; ++e) a[i][e] = b[i][e] = 0.0f;
    if (i < here) {
      const TA* src = qkv + (static_cast<size_t>(t) * heads + h0 + i) * d + sub * N;
      Half16<TA>::load(src, a[i]);
      Half16<TA>::load(src + d / 2, b[i]);
    }
  }
  const bool in_table = turns && pos >= 0 && pos < max_pos;
  float c[N], sn[N];
  if (in_table) {
    load_few<float, N>(cos_table + static_cast<size_t>(pos) * (d / 2) + sub * N, c);
    load_few<float, N>(sin_table + static_cast<size_t>(pos) * (d / 2) + sub * N, sn);
  }
  bool slot_ok = stores && slot != 0;                           // slot 0 is the sink: padding rows write nothing
  if (stores && (slot < 0 || slot >= cache_slots)) {
    slot_ok = false;
    if (sub == 0) atomicOr(err, B200_ERR_SLOT_RANGE);
  }
  if (turns && !in_table && sub == 0) atomicOr(err, B200_ERR_POSITION_RANGE);
  const int page = slot_ok ? slot / page_size : 0, offset = slot_ok ? slot - page * page_size : 0;
  // Every lane of the warp executes the shuffles (a warp may hold other heads beside these).
  float ss[HG];
#pragma unroll
  for (int i = 0; i < HG; ++i) {
    ss[i] = 0.0f;
#pragma unroll
    for (int e = 0; e < N; ++e) ss[i] += a[i][e] * a[i][e] + b[i][e] * b[i][e];
  }
  if (q_w != nullptr)
    for (int o = lanes >> 1; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < HG; ++i) ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], o, lanes);
#pragma unroll
  for (int i = 0; i < HG; ++i) {
    if (i >= here) break;
    const int h = h0 + i;
    const bool is_q = h < nh, is_k = !is_q && h < nh + nkv;
    if ((is_q || is_k) && q_w != nullptr) {
      const TW* w = (is_q ? q_w : k_w) + sub * N;
      const float scale = rsqrtf(ss[i] / static_cast<float>(d) + eps);
      float wa[N], wb[N];
      load_few<TW, N>(w, wa);
      load_few<TW, N>(w + d / 2, wb);
#pragma unroll
      for (int e = 0; e < N; ++e) {
        a[i][e] = a[i][e] * scale * wa[e];
        b[i][e] = b[i][e] * scale * wb[e];
      }
    }
    if ((is_q || is_k) && in_table) {
#pragma unroll
      for (int e = 0; e < N; ++e) {
        const float x = a[i][e], y = b[i][e];
        a[i][e] = x * c[e] - y * sn[e];
        b[i][e] = y * c[e] + x * sn[e];
      }
    }
    TA* dst;
    if (is_q) {
      dst = q_out + (static_cast<size_t>(t) * nh + h) * d;
    } else {
      if (!slot_ok) continue;
      const int kvh = is_k ? h - nh : h - nh - nkv;
      dst = (is_k ? k_cache : v_cache) + ((static_cast<size_t>(page) * nkv + kvh) * page_size + offset) * d;
    }
    Half16<TA>::store(dst + sub * N, a[i]);
    Half16<TA>::store(dst + d / 2 + sub * N, b[i]);
  }
}

// Many tokens: the same lane groups (HG heads of one token a step) walk over the step's work, and what the next step reads
// (its heads, its token's position and slot) is on its way while this one is normed, turned and stored.  A thread that comes
// and goes with one group of heads has loads in flight for a part of its life only, and its index cost a 64-bit division.
// Eight blocks an SM, four at a time by registers; bound by issue (76 % of cycles) more than by bytes (31 % of DRAM).  bfloat16, 16 + 2 x 8 heads of 128, us in a graph before / now: 8,192
// tokens 51.8 / 35.0 (134 MB: 3.8 TB/s), 2,919 20.2 / 14.1, 1,020 8.7 / 6.5; 32 + 2 x 8 heads, 2,048 tokens 20.3 / 14.6.  One head a
// lane group: 44.0, 17.6, 7.2, 17.8.
template <typename TA, typename TW, int HG>
__global__ void __launch_bounds__(256, 4)
qkv_post_walk_kernel(const TA* __restrict__ qkv, TA* __restrict__ q_out, TA* __restrict__ k_cache,
                     TA* __restrict__ v_cache, const TW* __restrict__ q_w, const TW* __restrict__ k_w, float eps,
                     const float* __restrict__ cos_table, const float* __restrict__ sin_table, int max_pos,
                     const int* __restrict__ positions, const int* __restrict__ slots, int tokens, int nh, int nkv,
                     int d, int page_size, long long cache_slots, int lanes, int* err) {
  constexpr int N = Half16<TA>::N;
  const int heads = nh + 2 * nkv, head_groups = (heads + HG - 1) / HG;
  const int sub = threadIdx.x % lanes;
  const int groups = gridDim.x * (blockDim.x / lanes), step_t = groups / head_groups, step_g = groups - step_t * head_groups;
  const int first = blockIdx.x * (blockDim.x / lanes) + threadIdx.x / lanes;
  int t = first / head_groups, g = first - t * head_groups;
  const bool rotates = cos_table != nullptr, stores_any = slots != nullptr;
  uint2 next_a[HG], next_b[HG];                                 // 8 bytes of a head's first half, and what they are rotated with
  int next_pos = 0, next_slot = 0;
  auto fetch = [&](int ft, int fg) {
    if (ft >= tokens) return;
    const int h0 = fg * HG;
    const TA* src = qkv + (static_cast<size_t>(ft) * heads + h0) * d + sub * N;
#pragma unroll
    for (int i = 0; i < HG; ++i)
      if (h0 + i < heads) {
        next_a[i] = *reinterpret_cast<const uint2*>(src + i * d);
        next_b[i] = *reinterpret_cast<const uint2*>(src + i * d + d / 2);
      }
    if (rotates) next_pos = positions[ft];
    if (stores_any) next_slot = slots[ft];
  };
  fetch(t, g);
  // (the lane groups of a warp leave together: those without work go on with the shuffles)
  while (__any_sync(0xffffffffu, t < tokens)) {
    const bool live = t < tokens;
    const int h0 = g * HG, here = live ? min(HG, heads - h0) : 0;
    float a[HG][N], b[HG][N];
#pragma unroll
    for (int i = 0; i < HG; ++i) {
      Half16<TA>::load(reinterpret_cast<const TA*>(&next_a[i]), a[i]);
      Half16<TA>::load(reinterpret_cast<const TA*>(&next_b[i]), b[i]);
    }
    const int pos = next_pos, slot = next_slot, now = t;
    t += step_t;
    g += step_g;
    if (g >= head_groups) { g -= head_groups; ++t; }
    fetch(t, g);
    const bool turns = rotates && h0 < nh + nkv && here > 0, stores = stores_any && h0 + here > nh && here > 0;
    const bool in_table = turns && pos >= 0 && pos < max_pos;
    float c[N], sn[N];
    if (in_table) {
      load_few<float, N>(cos_table + static_cast<size_t>(pos) * (d / 2) + sub * N, c);
      load_few<float, N>(sin_table + static_cast<size_t>(pos) * (d / 2) + sub * N, sn);
    }
    bool slot_ok = stores && slot != 0;
    if (stores && (slot < 0 || slot >= cache_slots)) {
      slot_ok = false;
      if (sub == 0) atomicOr(err, B200_ERR_SLOT_RANGE);
    }
    if (turns && !in_table && sub == 0) atomicOr(err, B200_ERR_POSITION_RANGE);
    float ss[HG];
#pragma unroll
    for (int i = 0; i < HG; ++i) {
      ss[i] = 0.0f;
#pragma unroll
      for (int e = 0; e < N; ++e) ss[i] += a[i][e] * a[i][e] + b[i][e] * b[i][e];
    }
    if (q_w != nullptr)
      for (int o = lanes >> 1; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < HG; ++i) ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], o, lanes);
    const int page = slot_ok ? slot / page_size : 0, offset = slot_ok ? slot - page * page_size : 0;
#pragma unroll
    for (int i = 0; i < HG; ++i) {
      if (i >= here) break;
      const int h = h0 + i;
      const bool is_q = h < nh, is_k = !is_q && h < nh + nkv;
      if ((is_q || is_k) && q_w != nullptr) {
        const TW* w = (is_q ? q_w : k_w) + sub * N;
        const float scale = rsqrtf(ss[i] / static_cast<float>(d) + eps);
        float wa[N], wb[N];
        load_few<TW, N>(w, wa);
        load_few<TW, N>(w + d / 2, wb);
#pragma unroll
        for (int e = 0; e < N; ++e) {
          a[i][e] = a[i][e] * scale * wa[e];
          b[i][e] = b[i][e] * scale * wb[e];
        }
      }
      if ((is_q || is_k) && in_table) {
#pragma unroll
        for (int e = 0; e < N; ++e) {
          const float x = a[i][e], y = b[i][e];
          a[i][e] = x * c[e] - y * sn[e];
          b[i][e] = y * c[e] + x * sn[e];
        }
      }
      TA* dst;
      if (is_q) {
        dst = q_out + (static_cast<size_t>(now) * nh + h) * d;
      } else {
        if (!slot_ok) continue;
        const int kvh = is_k ? h - nh : h - nh - nkv;
        dst = (is_k ? k_cache : v_cache) + ((static_cast<size_t>(page) * nkv + kvh) * page_size + offset) * d;
      }
      Half16<TA>::store(dst + sub * N, a[i]);
      Half16<TA>::store(dst + d / 2 + sub * N, b[i]);
    }
  }
}

// How many heads a lane group takes, by the blocks of 256 threads that one head each would be: few blocks are all resident and
// the shortest chain is fastest, many share the SMs and the fetches saved count.  Measured, us with 1 / 2 / 4 (bfloat16, 16 + 2 x 8
// heads of 128): 64 tokens (128 blocks) 3.4 / 3.7 / 4.9, 200 (400) 3.5 / 4.1 / 4.9, 300 (600) 4.8 / 4.5 / 5.5, 500 (1,000) 5.5 / 5.1 /
// 5.4, 777 (1,554) 7.4 / 6.4 / 6.0; float32: 64 (256) 3.6 / 3.6 / 4.1, 200 (800) 5.1 / 4.4 / 4.4, 300 (1,200) 6.0 / 5.1 / 5.0.
static int heads_a_group(long long work, int lanes) {
  const long long blocks = (work * lanes + 255) / 256;
  return blocks <= 3 * 148 ? 1 : blocks <= 8 * 148 ? 2 : 4;
}
B200_EXPORT int b200_qkv_post_heads_a_group(long long work, int lanes) { return heads_a_group(work, lanes); }

// The walking kernel takes bfloat16 steps of more than six blocks of 256 threads an SM: below, all of a step's threads are
// resident at once (777 tokens x 32 heads 5.2 / 5.2, 500 4.1 / 4.3), and float32's two elements of 8 bytes leave a lane group of
// 32 too little to have on its way (2,000 tokens 15.0 / 16.4).
constexpr int WALK_HEADS = 2, WALK_BLOCKS = 8 * 148;
static bool walk_takes(int act_dtype, long long threads) { return act_dtype == B200_BF16 && threads > 6ll * 148 * 256; }
B200_EXPORT int b200_qkv_post_walks(int act_dtype, long long threads) { return walk_takes(act_dtype, threads); }

B200_EXPORT int b200_qkv_post(const void* qkv, void* q_out, void* k_cache, void* v_cache, const void* q_w,
                              const void* k_w, float eps, const float* cos_table, const float* sin_table,
                              int rot_dim, int max_pos, const int* positions, const int* slots, int tokens,
                              int nh, int nkv, int d, int page_size, long long cache_slots, int act_dtype, int w_dtype,
                              int* err, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (d <= 0 || d > MAX_HEAD_DIM || nh <= 0 || nkv <= 0 || page_size <= 0) return B200_BAD_SIZE;
  if (rot_dim < 0 || rot_dim > d || (rot_dim & 1)) return B200_BAD_SIZE;
  const long long work = static_cast<long long>(tokens) * (nh + 2 * nkv);
  {
    const int vec = act_dtype == B200_F32 ? 4 : 8;
    const int lanes = d % vec == 0 ? d / vec : 0;
    const bool aligned = reinterpret_cast<uintptr_t>(qkv) % 16 == 0 && reinterpret_cast<uintptr_t>(q_out) % 16 == 0 &&
                         reinterpret_cast<uintptr_t>(k_cache) % 16 == 0 && reinterpret_cast<uintptr_t>(v_cache) % 16 == 0 &&
                         reinterpret_cast<uintptr_t>(q_w) % 16 == 0 && reinterpret_cast<uintptr_t>(k_w) % 16 == 0 &&
                         reinterpret_cast<uintptr_t>(cos_table) % 16 == 0 && reinterpret_cast<uintptr_t>(sin_table) % 16 == 0;
    const bool whole_rotation = cos_table == nullptr || rot_dim == d;
    if (lanes >= 2 && lanes <= 32 && (lanes & (lanes - 1)) == 0 && aligned && whole_rotation) {
      const int hg = heads_a_group(work, lanes);
      const long long threads = static_cast<long long>(tokens) * ((nh + 2 * nkv + hg - 1) / hg) * lanes;
      const long long steps = static_cast<long long>(tokens) * ((nh + 2 * nkv + WALK_HEADS - 1) / WALK_HEADS);
      const bool walks = walk_takes(act_dtype, steps * lanes);
      const unsigned vblocks = static_cast<unsigned>((threads + 255) / 256);
#define CALLW(TA, TW)                                                                                          \
      qkv_post_walk_kernel<TA, TW, WALK_HEADS><<<WALK_BLOCKS, 256, 0, stream>>>(                                          \
          static_cast<const TA*>(qkv), static_cast<TA*>(q_out), static_cast<TA*>(k_cache), static_cast<TA*>(v_cache), \
          static_cast<const TW*>(q_w), static_cast<const TW*>(k_w), eps, cos_table, sin_table, max_pos, positions, \
          slots, tokens, nh, nkv, d, page_size, cache_slots, lanes, err)
#define CALLG(TA, TW, HG)                                                                                      \
      qkv_post_vec_kernel<TA, TW, HG><<<vblocks, 256, 0, stream>>>(                                             \
          static_cast<const TA*>(qkv), static_cast<TA*>(q_out), static_cast<TA*>(k_cache), static_cast<TA*>(v_cache), \
          static_cast<const TW*>(q_w), static_cast<const TW*>(k_w), eps, cos_table, sin_table, max_pos, positions, \
          slots, tokens, nh, nkv, d, page_size, cache_slots, lanes, err)
#define CALLV(TA, TW)                                                                                          \
      if (walks) { if constexpr (sizeof(TA) == 2) { CALLW(TA, TW); } } else if (hg == 1) { CALLG(TA, TW, 1); } else if (hg == 2) { CALLG(TA, TW, 2); } else { CALLG(TA, TW, 4); }
      if (act_dtype == B200_F32 && w_dtype == B200_F32) { CALLV(float, float); }
      else if (act_dtype == B200_BF16 && w_dtype == B200_BF16) { CALLV(__nv_bfloat16, __nv_bfloat16); }
      else if (act_dtype == B200_BF16 && w_dtype == B200_F32) { CALLV(__nv_bfloat16, float); }
      else if (act_dtype == B200_F32 && w_dtype == B200_BF16) { CALLV(float, __nv_bfloat16); }
      else return B200_BAD_DTYPE;
#undef CALLV
#undef CALLG
#undef CALLW
      return b200_check_launch();
    }
  }
  const unsigned blocks = static_cast<unsigned>((work + WARPS - 1) / WARPS);
#define CALL(TA, TW)                                                                                   \
  qkv_post_kernel<TA, TW><<<blocks, WARPS * 32, 0, stream>>>(                                          \
      static_cast<const TA*>(qkv), static_cast<TA*>(q_out), static_cast<TA*>(k_cache),                 \
      static_cast<TA*>(v_cache), static_cast<const TW*>(q_w), static_cast<const TW*>(k_w), eps,        \
      cos_table, sin_table, rot_dim, max_pos, positions, slots, tokens, nh, nkv, d, page_size, cache_slots, err)
  if (act_dtype == B200_F32 && w_dtype == B200_F32) { CALL(float, float); }
  else if (act_dtype == B200_BF16 && w_dtype == B200_BF16) { CALL(__nv_bfloat16, __nv_bfloat16); }
  else if (act_dtype == B200_BF16 && w_dtype == B200_F32) { CALL(__nv_bfloat16, float); }
  else if (act_dtype == B200_F32 && w_dtype == B200_BF16) { CALL(float, __nv_bfloat16); }
  else return B200_BAD_DTYPE;
#undef CALL
  return b200_check_launch();
}
