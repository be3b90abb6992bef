// Causal grouped-query attention over the paged cache, any sizes, float32 arithmetic.
//
// One warp owns one (token, query head); up to 64 channels four do while there are few of them.  Keys are visited in tiles of 32 that start
// at absolute positions 0, 32, 64, ...: lane j scores key tile+j, the warp keeps a
// running maximum and sum (online softmax), then all lanes add p_j * v_j in key order.
// The order of every sum is a function of the token's own position alone, so a
// token's output does not depend on how the prompt was cut or what shares the batch.
// Visible keys: max(0, pos-window+1) <= j <= pos (window 0 = all), as in the reference
// (kernel/attention/attention_NH_32_NKV_4_HS_64.h:169-172,228-232); scores are scaled
// by the given factor instead of the reference's constant for head size 64 (:197).
// This is the attention of the 32-bit path and of bfloat16 shapes that the tensor-core
// kernels refuse.  Options, all off at zero: values of another size than the keys (vdim); a soft cap
// on the scaled scores, s <- cap * tanh(s / cap); a sink, a key with score 0 and no value that only
// adds 1 to the softmax's denominator; and, with a window, the first keep_first keys of the request,
// which stay visible (at their true positions) after the window has passed them.  Further: the sink's score may be a
// learned number per head (sink_values; it is not scaled); the mask may be by chunks instead of a window (chunk > 0: a
// query sees the keys at or before it whose position has the same floor(position / chunk)); and the weights may be
// sigmoid(score + bias[head]) without a softmax (sigmoid_bias given: no maximum, no normalisation, no sink).
// Two more: a bias that grows with the distance, r1[head] * ln(1 + r2[head] * (position - key position)), taken off the capped
// score; and key heads that share value heads (v_share neighbouring key heads read one value head: several attention maps,
// each with keys of its own, over one set of values).
#include "common.cuh"

namespace {

constexpr int WARPS = 4;
// The kernel is built for head sizes up to 64, 128, 256, 512 and 1024: a lane walks over MAXD / 32 channels of every key, whether the head has
// them or not, and with one warp on a scheduler each of these instructions costs its latency.  (Head size 32, up to 113 keys, float32, inside
// steps of four requests: 29.0 us a launch when the smallest build was 256 and a key's values were loaded one key after the other; 18.3 us
// this way, with the rows asked for ahead.)
constexpr int MAX_HEAD_DIM = 1024;
constexpr int PREFETCH_TILES = 4;      // tiles of keys and values that a warp asks into L1 ahead of their turn
// Small heads: a head's tiles are dealt to four parts in turn (to which one follows from a tile's position alone, so the order of a token's
// sums still does) and the parts' sums are put together at the end.  The block's four warps take a part each: 18.2 -> 5.8 us a launch of few
// requests.  In a launch of many (token, head) pairs (prompts of many short requests) a block's other warps have nothing to take, and a warp
// takes the four parts after one another instead, the same numbers in the same order.  Where the line lies, in pairs an SM: us a launch in
// float32, head size 32, one warp a head without parts / four warps / one warp with parts: 4,096 pairs of 8 keys 6.8 / 18.1 / 6.0, of 32 keys
// 15.5 / 22.3 / 10.9, of 113 keys 47 / 36 / 34, of 1,000 keys 557 / 226 / 238; 2,048 pairs of 8 keys 6.0 / 10.1 / 5.0, of 32 keys 13.2 / 12.2 /
// 8.0, of 113 keys 42 / 20 / 24, of 1,000 keys 353 / 126 / 171: up to 16 an SM what long contexts gain is more than what the shortest lose.
// Beyond it one long prompt is what pays: 2,048 tokens, 4 heads of 32: 1,038 / 458 / 508 (551 before its last tokens, which have the most keys, came
// first), 16 heads 3,356 / 1,667 / 1,727.
constexpr int SERIAL_FROM = 16;
__host__ __device__ constexpr int split_of(int max_dim) { return max_dim <= 64 ? WARPS : 1; }

template <typename T>
__device__ __forceinline__ float dot_row(const float* __restrict__ q, const T* __restrict__ k, int head_dim);

template <>
__device__ __forceinline__ float dot_row<float>(const float* __restrict__ q, const float* __restrict__ k,
                                                int head_dim) {
  float s = 0.f;
#pragma unroll 8
  for (int d = 0; d < head_dim; d += 4) {
    const float4 kv = *reinterpret_cast<const float4*>(k + d);
    s = fmaf(q[d], kv.x, s);
    s = fmaf(q[d + 1], kv.y, s);
    s = fmaf(q[d + 2], kv.z, s);
    s = fmaf(q[d + 3], kv.w, s);
  }
  return s;
}

template <>
__device__ __forceinline__ float dot_row<__nv_bfloat16>(const float* __restrict__ q,
                                                        const __nv_bfloat16* __restrict__ k, int head_dim) {
  float s = 0.f;
  for (int d = 0; d < head_dim; d += 8) {
    const uint4 u = *reinterpret_cast<const uint4*>(k + d);
    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      s = fmaf(q[d + 2 * i], __low2float(p[i]), s);
      s = fmaf(q[d + 2 * i + 1], __high2float(p[i]), s);
    }
  }
  return s;
}

// a row that does not start on a 16-byte boundary, or is no whole number of 16-byte pieces
// (head sizes off the 8-grid in bfloat16, off the 4-grid in float32): element by element
template <typename T>
__device__ __forceinline__ float dot_row_scalar(const float* __restrict__ q, const T* __restrict__ k, int head_dim) {
  float s = 0.f;
  for (int d = 0; d < head_dim; ++d) s = fmaf(q[d], to_f32(k[d]), s);
  return s;
}

template <typename T, int MAXD, bool SERIAL>
__global__ void __launch_bounds__(WARPS * 32)
paged_attention_generic_kernel(T* __restrict__ out, long long out_stride, const T* __restrict__ q,
                               long long q_stride, const T* __restrict__ k_pages,
                               const T* __restrict__ v_pages, const int* __restrict__ block_table,
                               int table_width, const int* __restrict__ token_entry,
                               const int* __restrict__ positions, int n_tokens, int n_heads, int n_kv,
                               int head_dim, int vdim, int page_size, int window, int keep_first, float scale,
                               float softcap, int sink, bool vec, const float* __restrict__ sink_values, int chunk,
                               const float* __restrict__ sigmoid_bias, const float* __restrict__ dist_r1,
                               const float* __restrict__ dist_r2, int v_share) {
  constexpr int AHEAD = MAXD <= 256 ? 8 : MAXD <= 512 ? 4 : 2;
  constexpr int SPLIT = split_of(MAXD);            // parts of a (token, head)
  constexpr int SHARE = SERIAL ? 1 : SPLIT;        // warps that share them
  __shared__ float q_s[WARPS][MAXD];
  __shared__ __align__(16) float p_s[WARPS][32];
  __shared__ __align__(16) long long row_s[WARPS][32];
  pdl_launch_dependents();      // let the next kernel start its own prologue now
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long items = (long long)n_tokens * n_heads, place = ((long long)blockIdx.x * WARPS + warp) / SHARE;
  if (place >= items) return;
  const long long item = SERIAL ? items - 1 - place : place;      // the tokens with the most keys first, so that none of them ends alone
  const int t = (int)(item / n_heads), h = (int)(item % n_heads);
  const int g = h / (n_heads / n_kv);
  const int pos = positions[t];
  const int* table = block_table + (size_t)token_entry[t] * table_width;
  const int lo = chunk > 0 ? (pos / chunk) * chunk : (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
  const int keep_end = min(keep_first, lo);      // keys [0, keep_end) lie before the window and are seen all the same
  const int lo_tile = (lo / 32) * 32;
  const int used = SERIAL ? max(1, min(SPLIT, (pos >> 5) + 1)) : SPLIT;      // a short context leaves parts without a tile: nothing to merge
  const float inv_cap = softcap > 0.f ? 1.f / softcap : 0.f;
  const float r1 = dist_r1 ? dist_r1[h] : 0.f, r2 = dist_r1 ? dist_r2[h] : 0.f;
  const int n_v = n_kv / v_share, gv = g / v_share;      // v_share neighbouring key heads read one value head

  const T* q_row = q + (size_t)t * q_stride + (size_t)h * head_dim;
  for (int d = lane; d < head_dim; d += 32) q_s[warp][d] = to_f32(q_row[d]);
  __syncwarp();

  // a tile's page number, keys and values follow from one another, three trips to L2: short rows are asked for some tiles ahead
  auto prefetch_tile = [&](int tile) {
    const int kp = tile + lane;
    if (kp > pos || kp < lo) return;
    const int page = table[kp / page_size], at = kp % page_size;
    const char* k = reinterpret_cast<const char*>(k_pages + (((long long)page * n_kv + g) * page_size + at) * head_dim);
    const char* v = reinterpret_cast<const char*>(v_pages + (((long long)page * n_v + gv) * page_size + at) * vdim);
    for (int b = 0; b < head_dim * (int)sizeof(T); b += 128) asm volatile("prefetch.global.L1 [%0];" ::"l"(k + b));
    for (int b = 0; b < vdim * (int)sizeof(T); b += 128) asm volatile("prefetch.global.L1 [%0];" ::"l"(v + b));
  };
  const bool ahead = MAXD <= 64 && keep_end == 0;
  if (ahead)
    for (int i = 0, tile = lo_tile; i < PREFETCH_TILES * SHARE; ++i, tile += 32)
      if ((tile >> 5) % SHARE == warp % SHARE) prefetch_tile(tile);

  const bool gated = sigmoid_bias != nullptr;
  const float bias = gated ? sigmoid_bias[h] : 0.f;
  float acc[MAXD / 32], m, l;
  __shared__ float m_s[WARPS / SHARE][SPLIT], l_s[WARPS / SHARE][SPLIT], acc_s[SPLIT > 1 ? WARPS / SHARE : 1][SPLIT][SPLIT > 1 ? MAXD : 1];
  const int owner = warp / SHARE;                  // of the (token, head) among the block's
  int part = warp % SHARE;
#pragma unroll 1
  do {
#pragma unroll
    for (int i = 0; i < MAXD / 32; ++i) acc[i] = 0.f;
    // the sink is the first term of the softmax: score 0, weight exp(0 - m), no value
    const bool with_sink = sink && part == 0;
    m = with_sink ? (sink_values ? sink_values[h] : 0.f) : -INFINITY;
    l = with_sink ? 1.f : 0.f;

    for (int tile = keep_end > 0 ? 0 : lo_tile; tile <= pos; tile += 32) {
      if (tile >= keep_end && tile < lo_tile) {      // between the kept keys and the window: nothing to see
        tile = lo_tile - 32;
        continue;
      }
      if (SPLIT > 1 && (tile >> 5) % SPLIT != part) continue;      // by absolute position, whatever the window's start
      if (ahead) prefetch_tile(tile + 32 * PREFETCH_TILES * SPLIT);
      const int kp = tile + lane;
      const bool valid = kp <= pos && (kp >= lo || kp < keep_end);
      long long row = 0;                             // the value's place in units of rows of vdim
      float s = -INFINITY;
      if (valid) {
        const int page = table[kp / page_size];
        row = ((long long)page * n_v + gv) * page_size + kp % page_size;
        const T* k_row = k_pages + (((long long)page * n_kv + g) * page_size + kp % page_size) * head_dim;
        s = (vec ? dot_row<T>(q_s[warp], k_row, head_dim) : dot_row_scalar<T>(q_s[warp], k_row, head_dim)) * scale;
        if (softcap > 0.f) s = softcap * tanhf(s * inv_cap);
        if (dist_r1) s -= r1 * log1pf(r2 * (float)(pos - kp));      // a bias that grows with the distance to the key
      }
      float p;
      if (gated) {
        p = valid ? 1.f / (1.f + expf(-(s + bias))) : 0.f;
      } else {
        const float m_new = fmaxf(m, warp_max(s));
        // a score of -inf weighs nothing, also in a first tile that holds no other (a warp's first, where four share a head): -inf - -inf is NaN
        const float alpha = m_new == -INFINITY ? 1.f : expf(m - m_new);
        p = valid && s != -INFINITY ? expf(s - m_new) : 0.f;
        l = l * alpha + warp_sum(p);
        m = m_new;
#pragma unroll
        for (int i = 0; i < MAXD / 32; ++i) acc[i] *= alpha;
      }
      // the values of several keys asked for together (a key after the other waits for memory 32 times a tile), added in the keys' order
      __syncwarp();                                  // the tile before has been read
      p_s[warp][lane] = p;
      row_s[warp][lane] = row;
      __syncwarp();
      const int n_valid = min(32, pos - tile + 1);
#pragma unroll 1
      for (int j = 0; j < n_valid; j += AHEAD) {
        float v[AHEAD][MAXD / 32], pj[AHEAD];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
          pj[u] = p_s[warp][j + u];                    // 0 for a key past the last (AHEAD divides 32)
          const T* at = v_pages + row_s[warp][j + u] * vdim;
#pragma unroll
          for (int i = 0; i < MAXD / 32; ++i) v[u][i] = pj[u] != 0.f && lane + 32 * i < vdim ? to_f32(at[lane + 32 * i]) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < AHEAD; ++u)
          if (pj[u] != 0.f)
#pragma unroll
            for (int i = 0; i < MAXD / 32; ++i) acc[i] = fmaf(pj[u], v[u][i], acc[i]);
      }
    }
    if (SPLIT > 1) {
      if (lane == 0) { m_s[owner][part] = m; l_s[owner][part] = l; }
#pragma unroll
      for (int i = 0; i < MAXD / 32; ++i) acc_s[owner][part][lane + 32 * i] = acc[i];
    }
  } while (SERIAL && ++part < used);
  if (SPLIT > 1) {
    // the parts' sums in their order, against the largest of their maxima (a part without a tile, or with scores of -inf alone: -inf, weight
    // 0).  The values of a part of weight 0 are left out, as those of a key of weight 0 are: an infinite one would make a NaN.
    if (SHARE > 1) __syncthreads();
    else __syncwarp();
    if (warp % SHARE) return;
    float all = m_s[owner][0];
#pragma unroll
    for (int w = 1; w < SPLIT; ++w)
      if (w < used) all = fmaxf(all, m_s[owner][w]);
    l = 0.f;
#pragma unroll
    for (int i = 0; i < MAXD / 32; ++i) acc[i] = 0.f;
#pragma unroll
    for (int w = 0; w < SPLIT; ++w) {
      if (w >= used) break;
      const float f = gated ? 1.f : expf(m_s[owner][w] - all);
      l += l_s[owner][w] * f;
      if (f != 0.f)
#pragma unroll
        for (int i = 0; i < MAXD / 32; ++i) acc[i] += acc_s[owner][w][lane + 32 * i] * f;
    }
  }
  const float inv = gated ? 1.f : 1.f / l;
  T* o = out + (size_t)t * out_stride + (size_t)h * vdim;
#pragma unroll
  for (int i = 0; i < MAXD / 32; ++i) {
    const int d = lane + 32 * i;
    if (d < vdim) o[d] = from_f32<T>(acc[i] * inv);
  }
}

}  // namespace

// q [n_tokens, q_stride] with head h at column h*head_dim; out [n_tokens, out_stride] with head h at column
// h*vdim.  k_pages [pages, n_kv, page_size, head_dim], v_pages [pages, n_kv, page_size, vdim]; block_table [entries, table_width] holds,
// for batch entry e, the page of positions [i*page_size, (i+1)*page_size) at column i.
// Further options: dist_r1, dist_r2 (float32 [heads], both or neither): r1[h] * ln(1 + r2[h] * (query position - key
// position)) is taken off every score after the cap; v_share > 1: v_pages has n_kv / v_share heads and the key heads
// v_share * i .. v_share * i + v_share - 1 read value head i (several attention maps over one set of values).
LLMK_API int llmk_paged_attention_generic_ex(void* out, long long out_stride, const void* q, long long q_stride,
                                             const void* k_pages, const void* v_pages, const int* block_table,
                                             int table_width, const int* token_entry, const int* positions,
                                             int n_tokens, int n_heads, int n_kv, int head_dim, int vdim, int page_size,
                                             int window, int keep_first, float scale, float softcap, int sink, int dtype,
                                             cudaStream_t stream, const float* sink_values, int chunk, const float* sigmoid_bias,
                                             const float* dist_r1, const float* dist_r2, int v_share) {
  if (n_tokens == 0) return 0;
  LLMK_REQUIRE(v_share >= 1 && n_kv % v_share == 0, "paged_attention: %d key heads do not share values in runs of %d", n_kv, v_share);
  LLMK_REQUIRE((dist_r1 != nullptr) == (dist_r2 != nullptr), "paged_attention: the distance bias takes both of its numbers");
  LLMK_REQUIRE(head_dim > 0 && head_dim <= MAX_HEAD_DIM, "paged_attention: head_dim %d must be 1 to %d", head_dim, MAX_HEAD_DIM);
  LLMK_REQUIRE(n_kv > 0 && n_heads % n_kv == 0, "paged_attention: %d query heads do not divide into %d kv heads",
               n_heads, n_kv);
  LLMK_REQUIRE(vdim > 0 && vdim <= MAX_HEAD_DIM, "paged_attention: value size %d must be 1 to %d", vdim, MAX_HEAD_DIM);
  LLMK_REQUIRE(page_size > 0 && window >= 0, "paged_attention: bad page_size %d or window %d", page_size, window);
  LLMK_REQUIRE(keep_first >= 0 && softcap >= 0.f, "paged_attention: bad keep_first %d or soft cap %f", keep_first, (double)softcap);
  LLMK_REQUIRE(chunk >= 0 && !(chunk > 0 && keep_first > 0), "paged_attention: bad chunk %d", chunk);
  if (sigmoid_bias) sink = 0;
  if (window == 0) keep_first = 0;
  const int widest = head_dim > vdim ? head_dim : vdim;
  const long long items = (long long)n_tokens * n_heads;
  const bool serial = split_of(widest) > 1 && items > (long long)SERIAL_FROM * llmk_sm_count();
  const int per_block = serial ? WARPS : WARPS / split_of(widest);
  const long long blocks = (items + per_block - 1) / per_block;
  LLMK_REQUIRE(blocks < (1ll << 31), "paged_attention: too many (token, head) items");
  return dispatch_dtype(dtype, [&](auto* tag) {
    using T = LLMK_ELEM(tag);
    const bool vec = head_dim % (16 / (int)sizeof(T)) == 0 && (uintptr_t)k_pages % 16 == 0;      // whole 16-byte pieces per key row
    auto kern = serial ? paged_attention_generic_kernel<T, 64, true> : widest <= 64 ? paged_attention_generic_kernel<T, 64, false>
                : widest <= 128 ? paged_attention_generic_kernel<T, 128, false> : widest <= 256 ? paged_attention_generic_kernel<T, 256, false>
                : widest <= 512 ? paged_attention_generic_kernel<T, 512, false>      // the wide head of a latent attention (its rank)
                : paged_attention_generic_kernel<T, MAX_HEAD_DIM, false>;
    launch_kernel(kern, dim3((unsigned)blocks), dim3(WARPS * 32), 0, stream,
        (T*)out, out_stride, (const T*)q, q_stride, (const T*)k_pages, (const T*)v_pages, block_table,
        table_width, token_entry, positions, n_tokens, n_heads, n_kv, head_dim, vdim, page_size, window, keep_first, scale,
        softcap, sink, vec, sink_values, chunk, sigmoid_bias, dist_r1, dist_r2, v_share);
    LLMK_LAUNCH_CHECK("paged_attention_generic");
  });
}

LLMK_API int llmk_paged_attention_generic(void* out, long long out_stride, const void* q, long long q_stride,
                                          const void* k_pages, const void* v_pages, const int* block_table,
                                          int table_width, const int* token_entry, const int* positions,
                                          int n_tokens, int n_heads, int n_kv, int head_dim, int vdim, int page_size,
                                          int window, int keep_first, float scale, float softcap, int sink, int dtype,
                                          cudaStream_t stream, const float* sink_values, int chunk, const float* sigmoid_bias) {
  return llmk_paged_attention_generic_ex(out, out_stride, q, q_stride, k_pages, v_pages, block_table, table_width, token_entry,
                                         positions, n_tokens, n_heads, n_kv, head_dim, vdim, page_size, window, keep_first, scale,
                                         softcap, sink, dtype, stream, sink_values, chunk, sigmoid_bias, nullptr, nullptr, 1);
}
