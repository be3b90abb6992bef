// Decode attention on the warp-level tensor cores (bfloat16, head size 64 or 128).
//
// The same split of the keys into ranges, one CTA per (range, kv head, request), as the CUDA-core
// kernel in attention_decode.cu, merged by the last CTA to arrive as there or, few short ranges, by a
// cluster's CTAs a part each; what differs most is the inside of a range.  The query heads of the kv group are the rows of an m16n8k16 MMA (up to 16
// per pass): one instruction scores 8 keys for all of them, so the arithmetic per key no longer
// grows with the group size.  Each of the four warps works alone on tiles of 32 keys, without
// block-wide barriers: keys and values are staged per warp through one to three stages of shared
// memory with cp.async (with several, the next tiles are in flight while one is computed) and read back with ldmatrix
// (values transposed); scores, maxima, sums and the output are float32, P is rounded to
// bfloat16 for the second MMA as in the prompt kernel.  A single decoded token has no use for
// the 128-row tcgen05 MMA; this is the tensor path that fits 8 to 16 rows.
#pragma once

#include "common.cuh"
#include "tcgen05.cuh"
#include "warp_mma.cuh"

namespace decode_mma {

constexpr int THREADS = 128;
constexpr int ROWS = 16;         // query heads per pass
constexpr int TILE = 32;         // keys per warp tile
constexpr int COUNTER_WORDS = 4096;

__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t smem_addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_addr));
}
__device__ __forceinline__ void cp_async_16(uint32_t smem_addr, const void* src, bool valid) {
  const int bytes = valid ? 16 : 0;                      // 0: the 16 bytes are filled with zeros
  // .cg: the keys and values stream through once; they need no place in L1
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t smem_addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_addr));
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Wait until at most n of the most recent groups are still in flight (n = 0..3).
__device__ __forceinline__ void cp_async_wait_pending(int n) {
  if (n <= 0) asm volatile("cp.async.wait_all;" ::: "memory");
  else if (n == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
  else if (n == 2) asm volatile("cp.async.wait_group 2;" ::: "memory");
  else asm volatile("cp.async.wait_group 3;" ::: "memory");
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// The sigmoid in float32 without the branch of the library's division, which keeps a tile's 16 scores a lane from running side by side:
// 1 + e^-x by a step of Newton's iteration for the reciprocal on the hardware's approximation (which stands where the step would
// overflow).  Every float32 number against 64 bits: the same largest error as 1 / (1 + expf(-x)) in every range down to -87 (3.43 units in the last
// place of the smallest, 8.9e-8 absolute); below that the result is less than 1.2e-38 and may be 0.
__device__ __forceinline__ float sigmoid_flat(float x) {
  const float y = 1.f + expf(-x);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  return y < 1e37f ? fmaf(r, fmaf(-y, r, 1.f), r) : r;
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// Two adjacent values (idx even): of a tensor, or the sums in split order of split-K partial
// results, with the loads of up to eight splits in flight (a split past the last adds zero).
__device__ __forceinline__ float2 sum2(const MaybePartial<__nv_bfloat16>& s, size_t idx) {
  if (s.parts) {
    float2 acc = make_float2(0.f, 0.f);
    for (int sp = 0; sp < s.splits; sp += 8) {
      float2 t[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        t[u] = sp + u < s.splits ? *reinterpret_cast<const float2*>(s.parts + (size_t)(sp + u) * s.split_stride + idx)
                                 : make_float2(0.f, 0.f);
#pragma unroll
      for (int u = 0; u < 8; ++u) { acc.x += t[u].x; acc.y += t[u].y; }
    }
    return acc;
  }
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(s.direct + idx));
}

// Scratch layout as in attention_decode.cu: counters, then ml [entries, heads, splits, 2] (the
// maximum here in the base-2 domain of the pre-scaled scores, with EXT of the scores), then o [entries, heads, splits, HS].
//
// CLUSTER: the CTAs of the ranges of one (request, kv head) form a thread-block cluster (2 to 8
// along blockIdx.x).  They exchange their results through distributed shared memory (into the receivers' dynamic
// shared memory, about heads of a pass x HS floats) and each merges its part of the outputs: no scratch in global
// memory, no fence, no counter.  Every CTA arrives at a first cluster barrier when it starts and waits for it only
// before it writes to the others, which must be running by then; a second barrier publishes the writes.
//
// BALANCE: long contexts, whose ranges are handed out by the requests' lengths (ranges_of).  A variant of its own, because the code alone,
// never run, cost short contexts 0.7 us a launch (64 requests of 600 keys inside a decode step).
//
// FUSED: the kernel takes the row of the QKV product itself (a tensor or unsummed split-K
// partial results) instead of rotated queries.  Every CTA sums and rotates its group's queries
// into shared memory; the CTA whose range holds the newest position also sums and rotates that
// token's key, stores key and value in the pages (unless the layer reads another layer's
// pages) and keeps a copy in shared memory for its own use.  This replaces the separate
// rotate-and-store kernel of a decode step.
struct FusedQkv {
  MaybePartial<__nv_bfloat16> src;     // [entries, src_stride]: q heads, then k heads, then v heads
  long long src_stride;
  const float* cos_table;              // [max_position, HS/2], or null: nothing is rotated
  const float* sin_table;
  int write_kv;
};

// EXT: the options of the CUDA-core kernel (attention_decode.cu) and the sigmoid weights of the general one.  The visible keys
// are walked as a list: the kept first keys, then the window's (or the chunk's); index u of the list is key u or u + skip.  Scores and
// weights are float32 numbers from the library's functions, as in those kernels, and P enters the second product as three bfloat16
// numbers whose sum it is.  Against 64 bits the outputs that are not the correctly rounded ones are as many as theirs (0.02 to 0.03 %; with
// two bfloat16 numbers and functions of hardware approximations 0.1 to 0.2 %, 1.4 % under a cap of 500).  Microseconds a launch, the CUDA-core
// kernel or (sigmoid weights) two bfloat16 numbers and approximations -> this one: window, cap and sink, 3 requests of 1,900 keys, 43.9 -> 10.9;
// cap, distance bias and shared values, 5 requests of 1,100, 52.7 -> 14.2; latents with a learned sink, 8 requests of 700, 68.1 -> 7.9;
// chunks of 256 with sigmoid weights, head size 64, 4.15 -> 4.8 (a decode step with two of the general kernel's launches 1,402 us, with these 831).
struct Options {
  float softcap;                 // > 0: scores pass cap * tanh(score / cap)
  int sink;                      // one more term in the denominator, of score sink_values[head] or 0
  int keep_first;                // with a window: the first keys that stay visible
  int chunk;                     // > 0: instead of a window, the keys with the same floor(position / chunk)
  int v_share;                   // neighbouring key heads that read one value head
  const float* sink_values;
  const float* dist_r1;          // r1[head] ln(1 + r2[head] distance) is taken off the capped score
  const float* dist_r2;
  const float* sigmoid_bias;     // weights sigmoid(score + bias[head]), nothing is normalised
};

// Which of a request's keys its newest token sees: a window's (0: all) or a chunk's, and the first ones that a window keeps.
struct Mask {
  int window, chunk, keep_first;
  __host__ __device__ int begin(int held) const {
    const int pos = held - 1;
    return chunk > 0 ? pos / chunk * chunk : (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
  }
  __host__ __device__ int kept(int begin) const { return keep_first < begin ? keep_first : begin; }
  __host__ __device__ int visible(int held) const { return held > 0 ? held - begin(held) + kept(begin(held)) : 0; }
};

// How long contexts are cut: `balance` ranges for all requests together and kv head, as many as run at once, handed out by length, so that
// one long request among short ones is not walked by as few CTAs as each of them (one of 6,000 keys beside seven of 400, 8 kv heads of
// 128: four ranges a request 33 us a launch, by length 14.6 us).  A request gets its share of the `total` of all visible keys, rounded down, so that
// the ranges run in one wave: rounded to the nearest, equal requests got a piece more than fits (8 of 8,192 keys, 37 places taken as 5 each, 320
// CTAs for 296 places, 69 us; 4 each 47 us; 8 of 3,000 33.9 -> 23.1; at head size 64, 4 kv heads, 8 of 8,192 24.0 -> 19.8, 20 of 4,096 25.2 -> 21.9;
// slower: 12 of 300 to 3,600 keys 24.2 -> 25.3).  At least one, of at least 256 keys, at most `splits`.  The sum is at most `balance` and one for
// each request whose share is less than one.  (Lengths found by halving, the shortest with which all ranges run at once, keep ragged requests
// as even, but eight passes over the lengths before the first key is asked for took more than that gave: 8 of 8,000 keys inside decode steps of
// 32 layers 4.59 ms a step, this way 4.46.)
__host__ __device__ inline int ranges_of(int keys, int total, int balance, int splits) {
  const int share = total > 0 ? (int)((float)keys * (float)balance / (float)total) : 0, most = (keys + 255) / 256 < splits ? (keys + 255) / 256 : splits;
  return share < 1 || most < 1 ? 1 : share < most ? share : most;      // (an entry without keys: zeros are written)
}

template <int HS, bool CLUSTER, bool FUSED, bool LIGHT = false, bool EXT = false, bool BALANCE = false>
__global__ void __launch_bounds__(THREADS, (LIGHT && HS == 64) ? 4 : 1)
decode_attention_mma_kernel(__nv_bfloat16* __restrict__ out, long long out_stride, float* __restrict__ scratch,
                            const __nv_bfloat16* __restrict__ q, long long q_stride,
                            __nv_bfloat16* __restrict__ k_pages, __nv_bfloat16* __restrict__ v_pages,
                            const int* __restrict__ block_table, int table_width, const int* __restrict__ kv_lens,
                            int n_entries, int n_heads, int n_kv, int page_size, int window, float scale_log2e, int splits,
                            FusedQkv fused, int kv_share, Options opt, int balance) {
  static_assert(!(FUSED && EXT), "the fused kernel has no options");
  // weights from scores: base 2 of scores that carry the factor already, or (EXT) the float32 exponential of the scores as they are
  auto weight = [](float x) { return EXT ? expf(x) : ex2(x); };
  constexpr int KS = HS / 16;                  // k-steps of Q K^T
  constexpr int DT = HS / 8;                   // 8-wide tiles of the output row
  constexpr int CH = HS / 8;                   // 16-byte chunks of a row
  constexpr int V_BYTES = TILE * HS * 2;       // one tile of keys, or of values
  // Stages of (keys, values) per warp.  Several let the next tiles fly while one is computed,
  // which pays for long ranges (three where two CTAs then still fit on an SM).  A cluster is only
  // formed for short ranges on a small grid; there one stage keeps the CTA small enough to become
  // resident beside the CTAs of the kernel before it, which is what lets its early requests
  // overlap that kernel.  LIGHT: one stage without a cluster, for grids of more CTAs than fit on
  // the SMs at once with deep stages: more CTAs per SM then keep as many bytes in flight, and
  // the grid runs as one wave instead of two.
  constexpr int NST = (CLUSTER || LIGHT) ? 1 : (HS == 64 ? 3 : 2);
  constexpr int WARP_BYTES = NST * 2 * V_BYTES;
  constexpr int RANGES = CLUSTER ? 8 : 64;     // most ranges that a merge in shared memory takes
  static_assert(4 * WARP_BYTES >= 4 * ROWS * HS * 4, "the warps' results are merged in the stage buffers");
  extern __shared__ __align__(128) uint8_t vbuf[];            // 4 warps x WARP_BYTES, then (CLUSTER) the receive buffer
  __shared__ float wm_s[4][ROWS], wl_s[4][ROWS], hm_s[ROWS], hl_s[ROWS];      // per warp and head; per head over the warps
  __shared__ float w_s[ROWS][RANGES], l_in[ROWS][RANGES];    // merge: per (head, range)
  __shared__ int last_s;
  __shared__ __align__(16) __nv_bfloat16 q_s[FUSED ? ROWS * HS : 8];
  __shared__ __align__(16) __nv_bfloat16 kv_new_s[FUSED ? 2 * HS : 8];    // the newest key, then the newest value

  float* recv_s = reinterpret_cast<float*>(vbuf + 4 * WARP_BYTES);   // CLUSTER: what the ranges send to this CTA
  pdl_launch_dependents();
  if (CLUSTER) tc::cluster_arrive();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = blockIdx.y;
  const Mask mask{window, EXT ? opt.chunk : 0, EXT ? opt.keep_first : 0};
  // The entry, its range and how many it has: the grid's, or (BALANCE) by the requests' lengths, the ranges of all entries one after
  // the other along blockIdx.x.  Every CTA finds that from the lengths, warp by warp, before it waits for anybody.  (Grids of `splits` places
  // an entry, of which the unneeded ones leave at once, leave the SMs unevenly filled: 8 requests of 8,192 keys, 8 kv heads of 128, 4 of 16
  // places each in use, 57 us, and packed 49 us.)
  int e = blockIdx.z, split = blockIdx.x, n_ranges = splits;
  int running = (int)(gridDim.x * gridDim.z);                 // ranges of all entries, per kv head
  if constexpr (BALANCE) {
    auto seen_by = [&](int i) { return mask.visible(min(kv_lens[i], table_width * page_size)); };
    int total = 0;
#pragma unroll 1
    for (int i = lane; i < n_entries; i += 32) total += seen_by(i);
    total = __reduce_add_sync(0xffffffffu, total);
    running = max(balance, n_entries);
    e = -1;
#pragma unroll 1
    for (int i0 = 0, before = 0; i0 < n_entries && e < 0; i0 += 32) {
      const int own = i0 + lane < n_entries ? ranges_of(seen_by(i0 + lane), total, balance, splits) : 0;
      int upto = own;
#pragma unroll
      for (int o = 1; o < 32; o *= 2) {
        const int below = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += below;
      }
      const uint32_t behind = __ballot_sync(0xffffffffu, (int)blockIdx.x < before + upto);
      const int at = behind ? __ffs(behind) - 1 : 31;
      const int first = before + __shfl_sync(0xffffffffu, upto - own, at);
      n_ranges = __shfl_sync(0xffffffffu, own, at);
      if (behind) { e = i0 + at; split = (int)blockIdx.x - first; }
      before = first + n_ranges;
    }
    if (e < 0) return;                                        // the grid holds the most ranges that there can be
  }
  const int group = n_heads / n_kv;
  // kv_share > 1: that many neighbouring groups of query heads read one key/value head (a group of many heads split over
  // several CTAs, each with its own pass over the keys): the pages hold n_kv / kv_share heads
  // (not with FUSED, which stores a key per group: nothing is divided there)
  const int kv_heads = FUSED ? n_kv : n_kv / kv_share, g_kv = FUSED ? g : g / kv_share;
  // a length beyond the entry's table row is cut to what the row can hold; an entry without keys
  // gets zeros (every range of it sees the same length and leaves here, so nobody waits for anybody)
  const int n_held = min(kv_lens[e], table_width * page_size);
  if (n_held <= 0) {
    pdl_wait();
    if (split == 0)
      for (int i = tid; i < group * HS; i += THREADS)
        out[(size_t)e * out_stride + (size_t)g * group * HS + i] = __float2bfloat16_rn(0.f);
    return;
  }
  const int pos = n_held - 1;
  const int lo = mask.begin(n_held);
  // EXT: the visible keys as a list, [0, keep_end) and then [lo, pos]; below, a key's number is its place in that list and
  // `last` the newest key's.  Otherwise a key's number is its position.
  const int keep_end = mask.kept(lo), skip = EXT ? lo - keep_end : 0;
  const int first = EXT ? 0 : lo, last = pos - skip;
  const int n_keys = last - first + 1;
  auto position_of = [&](int k) { return EXT && k >= keep_end ? k + skip : k; };
  int chunk = (n_keys + n_ranges - 1) / n_ranges;
  chunk = (chunk + TILE - 1) / TILE * TILE;
  const int n_active = min(splits, (n_keys + chunk - 1) / chunk);      // ranges that hold keys
  if (!CLUSTER && split >= n_active) return;
  const int k_begin = first + split * chunk;
  const int k_end = min(last + 1, k_begin + chunk);
  const int* table = block_table + (size_t)e * table_width;
  // One vector per token that is key and value at once (the latents of a latent attention, whose pages are
  // given as both): the tile of keys is also the tile of values, so only one of the two is requested.
  const bool same_kv = !FUSED && k_pages == v_pages;
  const int qrow = lane >> 2, qcol = (lane & 3) * 2;
  // the row of key k of this request and kv head in the pages.  The page size is a power of two
  // (the host sends other sizes to the CUDA-core kernel): a division per row of every tile would
  // cost more than the tile's arithmetic
  const int page_shift = __ffs(page_size) - 1;
  // (counted in rows: a cache holds fewer than 2^32 of them)
  auto row_of = [&](int k) -> uint32_t {
    const int p = position_of(k);
    return (((uint32_t)table[p >> page_shift] * kv_heads + g_kv) << page_shift) + (p & (page_size - 1));
  };
  // the same of its value, where key heads share value heads
  auto v_row_of = [&](int k, uint32_t key_row) -> uint32_t {
    if (!EXT || opt.v_share <= 1) return key_row;
    const int p = position_of(k);
    return (((uint32_t)table[p >> page_shift] * (kv_heads / opt.v_share) + g_kv / opt.v_share) << page_shift) + (p & (page_size - 1));
  };
  uint8_t* w_buf = vbuf + warp * WARP_BYTES;                 // stage st: keys at st * 2 * V_BYTES, values V_BYTES further
  const uint32_t w_addr = (uint32_t)__cvta_generic_to_shared(w_buf);
  const int t_first = k_begin + warp * TILE;                // this warp's first tile
  const int n_tiles = t_first < k_end ? (k_end - t_first + 4 * TILE - 1) / (4 * TILE) : 0;

  // request a tile's keys and values: 32 rows of CH chunks each, swizzled by the row; rows past
  // the range are filled with zeros.  A lane finds one key's row; the loops here and below are left rolled where they are not
  // the tile's arithmetic: a launch of a decode step runs through this code once or twice, so that fetching it is what it waits for
  // (ncu: 4.7 of 12 cycles an instruction stalled on instructions with everything unrolled; 8 requests of 512 keys, 8 kv heads of 64, rolled: 6.3 to 4.3 us a launch).
  auto stage_tile = [&](int j) {
    const int t = t_first + j * 4 * TILE;
    const uint32_t dst = w_addr + (j % NST) * 2 * V_BYTES;
    const int own = t + lane < k_end ? t + lane : k_begin;
    const uint32_t own_row = row_of(own), own_v = v_row_of(own, own_row);
#pragma unroll 4
    for (int i = 0; i < CH; ++i) {
      const int idx = i * 32 + lane;
      const int kl = idx / CH, c = idx % CH;
      const bool valid = t + kl < k_end;
      const int cs = (c & ~7) | ((c ^ kl) & 7);
      const size_t row = (size_t)__shfl_sync(0xffffffffu, own_row, kl) * HS;
      const size_t v_row = EXT ? (size_t)__shfl_sync(0xffffffffu, own_v, kl) * HS : row;
      cp_async_16(dst + kl * (HS * 2) + cs * 16, k_pages + row + c * 8, valid);
      if (!same_kv) cp_async_16(dst + V_BYTES + kl * (HS * 2) + cs * 16, v_pages + v_row + c * 8, valid);
    }
    cp_async_commit();
  };

  // Lengths and block tables were copied before the step's first kernel, and every key but the
  // newest was stored by an earlier step.  So each warp requests its first tiles, and the
  // CTA asks the rest of its range into L2, while the kernels before this one still run; only
  // the queries and the newest key and value (stored by a kernel of this step, or by this one)
  // have to wait.  The newest row of a tile is replaced after it has landed, see below.
#pragma unroll
  for (int j = 0; j < NST; ++j)
    if (j < n_tiles) stage_tile(j);
  {
    // at most 32 MB over all ranges that run: asking for more than L2 keeps evicts the lines before
    // they are used and fetches them from memory twice (long ranges stream through the stages)
    constexpr int LINES = HS * 2 / 128;                    // 128-byte lines per row
    const int ask_limit = (32 << 20) / (running * (int)gridDim.y) / (HS * 4);
    const int n_rows = min(ask_limit, max(0, k_end - k_begin - NST * 4 * TILE));
    for (int i = tid; i < n_rows * LINES * 2; i += THREADS) {
      const int which = i & 1, line = (i >> 1) % LINES, kp = k_begin + NST * 4 * TILE + (i >> 1) / LINES;
      if (which && same_kv) continue;
      const uint32_t row = row_of(kp);
      const __nv_bfloat16* src = (which ? v_pages + (size_t)v_row_of(kp, row) * HS : k_pages + (size_t)row * HS) + line * 64;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(src));
    }
  }
  pdl_wait();

  // the newest key and value are read, once they are valid, from the pages, or from this CTA's
  // shared copy when it computes them itself
  const uint32_t last_row = row_of(last);
  const size_t new_row = (size_t)last_row * HS, new_v_row = (size_t)v_row_of(last, last_row) * HS;
  const bool owner = FUSED && fused.write_kv && k_begin <= pos && pos < k_end;
  // FUSED, owner: the last threads sum the newest token's key (two pairs each) and value (two
  // elements each); their loads are issued here and used after the queries' loads below
  const int kv_item = THREADS - 1 - tid;
  const bool does_k = owner && kv_item < HS / 4, does_v = owner && !does_k && kv_item < HS / 4 + HS / 2;
  float2 nk_a = make_float2(0.f, 0.f), nk_b = nk_a, nv = nk_a;
  if constexpr (FUSED) {
    const size_t src_row = (size_t)e * fused.src_stride;
    if (does_k) {
      const size_t h = src_row + (size_t)(n_heads + g) * HS + kv_item * 2;
      nk_a = sum2(fused.src, h);
      nk_b = sum2(fused.src, h + HS / 2);
    } else if (does_v) {
      nv = sum2(fused.src, src_row + (size_t)(n_heads + n_kv + g) * HS + (kv_item - HS / 4) * 2);
    }
  }

  // the sum of weighted values over the sum of the weights: with a sink, whose weight joins the sum; sigmoid weights are not
  // normalised
  auto finish = [&](int head, float m, float l, float acc) -> float {
    if (EXT && opt.sigmoid_bias) return acc;
    if (EXT && opt.sink) {
      const float sv = opt.sink_values ? opt.sink_values[head] : 0.f, top = fmaxf(m, sv), f = weight(m - top);
      return acc * f / (l * f + weight(sv - top));
    }
    return acc / l;
  };

  int* counters = reinterpret_cast<int*>(scratch);
  float* partial_ml = scratch + COUNTER_WORDS;
  float* partial_o = partial_ml + (size_t)n_entries * n_heads * splits * 2;

  // (in a cluster a range without keys still has to meet the others at the barriers)
  for (int h0 = 0; h0 < group && (CLUSTER || k_begin < k_end); h0 += ROWS) {
    const int nh = min(ROWS, group - h0);
    const int head0 = g * group + h0;
    // Q fragments: rows = heads, straight from global memory (4 bytes = 2 bf16 per load)
    uint32_t qf[KS][4];
    const __nv_bfloat16* q0;
    if constexpr (FUSED) {
      // the pass's queries: summed, rotated, rounded to bfloat16 into shared memory; two pairs
      // (i, i+1 and their partners half a head further) per item, all loads issued before any use
      constexpr int ITEMS = ROWS * (HS / 4) / THREADS;
      float2 qa[ITEMS], qb[ITEMS], qc[ITEMS], qs[ITEMS];
#pragma unroll
      for (int it = 0; it < ITEMS; ++it) {
        const int idx = tid + it * THREADS;
        if (idx < nh * (HS / 4)) {
          const int h = idx / (HS / 4), i = (idx % (HS / 4)) * 2;
          const size_t src = (size_t)e * fused.src_stride + (size_t)(head0 + h) * HS + i;
          qa[it] = sum2(fused.src, src);
          qb[it] = sum2(fused.src, src + HS / 2);
          qc[it] = fused.cos_table ? *reinterpret_cast<const float2*>(fused.cos_table + (size_t)pos * (HS / 2) + i) : make_float2(1.f, 1.f);
          qs[it] = fused.cos_table ? *reinterpret_cast<const float2*>(fused.sin_table + (size_t)pos * (HS / 2) + i) : make_float2(0.f, 0.f);
        }
      }
      if (h0 == 0 && (does_k || does_v)) {
        if (does_k) {
          const int i = kv_item * 2;
          const float2 c = fused.cos_table ? *reinterpret_cast<const float2*>(fused.cos_table + (size_t)pos * (HS / 2) + i) : make_float2(1.f, 1.f);
          const float2 sn = fused.cos_table ? *reinterpret_cast<const float2*>(fused.sin_table + (size_t)pos * (HS / 2) + i) : make_float2(0.f, 0.f);
          const __nv_bfloat162 ya = __floats2bfloat162_rn(nk_a.x * c.x - nk_b.x * sn.x, nk_a.y * c.y - nk_b.y * sn.y);
          const __nv_bfloat162 yb = __floats2bfloat162_rn(nk_a.x * sn.x + nk_b.x * c.x, nk_a.y * sn.y + nk_b.y * c.y);
          *reinterpret_cast<__nv_bfloat162*>(k_pages + new_row + i) = ya;
          *reinterpret_cast<__nv_bfloat162*>(k_pages + new_row + i + HS / 2) = yb;
          *reinterpret_cast<__nv_bfloat162*>(kv_new_s + i) = ya;
          *reinterpret_cast<__nv_bfloat162*>(kv_new_s + i + HS / 2) = yb;
        } else {
          const int d = (kv_item - HS / 4) * 2;
          const __nv_bfloat162 x = __floats2bfloat162_rn(nv.x, nv.y);
          *reinterpret_cast<__nv_bfloat162*>(v_pages + new_row + d) = x;
          *reinterpret_cast<__nv_bfloat162*>(kv_new_s + HS + d) = x;
        }
      }
#pragma unroll
      for (int it = 0; it < ITEMS; ++it) {
        const int idx = tid + it * THREADS;
        if (idx < nh * (HS / 4)) {
          const int h = idx / (HS / 4), i = (idx % (HS / 4)) * 2;
          const float2 a = qa[it], b = qb[it], c = qc[it], sn = qs[it];
          *reinterpret_cast<__nv_bfloat162*>(q_s + h * HS + i) = __floats2bfloat162_rn(a.x * c.x - b.x * sn.x, a.y * c.y - b.y * sn.y);
          *reinterpret_cast<__nv_bfloat162*>(q_s + h * HS + i + HS / 2) = __floats2bfloat162_rn(a.x * sn.x + b.x * c.x, a.y * sn.y + b.y * c.y);
        }
      }
      __syncthreads();                  // queries, and the owner's newest key and value, in shared memory
      q0 = q_s + qrow * HS;
    } else {
      q0 = q + (size_t)e * q_stride + (size_t)(head0 + qrow) * HS;
    }
    {
      // Q fragments: rows = heads (4 bytes = 2 bf16 per load)
      const __nv_bfloat16* q1 = q0 + 8 * HS;
      const bool r0 = qrow < nh, r1 = qrow + 8 < nh;
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) {
        qf[ks][0] = r0 ? *reinterpret_cast<const uint32_t*>(q0 + ks * 16 + qcol) : 0u;
        qf[ks][1] = r1 ? *reinterpret_cast<const uint32_t*>(q1 + ks * 16 + qcol) : 0u;
        qf[ks][2] = r0 ? *reinterpret_cast<const uint32_t*>(q0 + ks * 16 + 8 + qcol) : 0u;
        qf[ks][3] = r1 ? *reinterpret_cast<const uint32_t*>(q1 + ks * 16 + 8 + qcol) : 0u;
      }
    }
    float o[DT][4];
#pragma unroll
    for (int d = 0; d < DT; ++d) o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.f;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;        // rows qrow and qrow + 8 (l: this lane's share)
    // EXT: numbers per head of those rows: the distance bias, or the sigmoid's bias
    const bool r0 = qrow < nh, r1 = qrow + 8 < nh, dist = EXT && opt.dist_r1 != nullptr, gated = EXT && opt.sigmoid_bias != nullptr;
    float ra0 = 0.f, ra1 = 0.f, rb0 = 0.f, rb1 = 0.f;
    if (dist) {
      ra0 = r0 ? opt.dist_r1[head0 + qrow] : 0.f;
      ra1 = r1 ? opt.dist_r1[head0 + qrow + 8] : 0.f;
      rb0 = r0 ? opt.dist_r2[head0 + qrow] : 0.f;
      rb1 = r1 ? opt.dist_r2[head0 + qrow + 8] : 0.f;
    } else if (gated) {
      ra0 = r0 ? opt.sigmoid_bias[head0 + qrow] : 0.f;
      ra1 = r1 ? opt.sigmoid_bias[head0 + qrow + 8] : 0.f;
    }
    const float inv_cap = EXT && opt.softcap > 0.f ? 1.f / opt.softcap : 0.f;

    if (h0 > 0) {                                                 // a later pass requests its tiles again
#pragma unroll
      for (int j = 0; j < NST; ++j)
        if (j < n_tiles) stage_tile(j);
    }
    for (int j = 0; j < n_tiles; ++j) {
      const int t = t_first + j * 4 * TILE;
      const uint32_t k_addr = w_addr + (j % NST) * 2 * V_BYTES, v_addr = same_kv ? k_addr : k_addr + V_BYTES;
      cp_async_wait_pending(min(n_tiles - 1 - j, NST - 1));          // tile j has landed; later ones may still fly
      __syncwarp();
      if (last < t + TILE) {                                      // last >= t: the range ends at the newest key
        // The newest row: not valid when the tile was requested early (before the wait for the
        // kernels of this step).  It is taken from the CTA's own copy, or from L2.
        if (lane < 2 * CH) {
          const int c = lane % CH, kl = last - t;
          const bool is_v = lane >= CH;
          const uint4 row = owner ? *reinterpret_cast<const uint4*>(kv_new_s + (is_v ? HS : 0) + c * 8)
                                  : __ldcg(reinterpret_cast<const uint4*>((is_v ? v_pages + new_v_row : k_pages + new_row) + c * 8));
          const int cs = (c & ~7) | ((c ^ kl) & 7);
          *reinterpret_cast<uint4*>(w_buf + (j % NST) * 2 * V_BYTES + (is_v ? V_BYTES : 0) + kl * (HS * 2) + cs * 16) = row;
        }
        __syncwarp();
      }
      // ---- S = Q K^T: K fragments with ldmatrix, two k-steps per instruction ----
      float s[4][4];
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.f;
        const int kl = nt * 8 + (lane & 7);
#pragma unroll
        for (int k2 = 0; k2 < KS / 2; ++k2) {
          const int c = k2 * 4 + (lane >> 3);
          const int cs = (c & ~7) | ((c ^ kl) & 7);
          uint32_t kb[4];
          ldmatrix_x4(kb, k_addr + kl * (HS * 2) + cs * 16);
          mma_16816(s[nt], qf[2 * k2], kb[0], kb[1]);
          mma_16816(s[nt], qf[2 * k2 + 1], kb[2], kb[3]);
        }
      }
      // ---- scale, mask the keys past the range, running maximum and sum ----
      float t0 = -INFINITY, t1 = -INFINITY;
      // EXT: what the options make of the scores.  Rolled over the tile's four parts, a part of which goes to the end of the array when it is made:
      // inside a decode step the code is fetched once a launch (3 requests of 1,900 keys, cap and sink: a step of four launches 725 us unrolled,
      // 715 rolled; 8 requests with sigmoid weights 620 and 615)
      if constexpr (EXT) {                                         // scale_log2e is the plain scale here
#pragma unroll 1
        for (int nt = 0; nt < 4; ++nt) {
          float x[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            x[i] = s[0][i] * scale_log2e;
            if (opt.softcap > 0.f) x[i] = opt.softcap * tanhf(x[i] * inv_cap);
            if (dist) {
              const float away = (float)(pos - position_of(t + nt * 8 + qcol + (i & 1)));
              x[i] -= (i < 2 ? ra0 : ra1) * log1pf((i < 2 ? rb0 : rb1) * away);
            }
            if (gated) x[i] = sigmoid_flat(x[i] + (i < 2 ? ra0 : ra1));
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) { s[0][i] = s[1][i]; s[1][i] = s[2][i]; s[2][i] = s[3][i]; s[3][i] = x[i]; }
        }
      }
      const float factor = EXT ? 1.f : scale_log2e, none = gated ? 0.f : -INFINITY;
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const int kp = t + nt * 8 + qcol;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const bool valid = kp + j < k_end;
          s[nt][j] = valid ? s[nt][j] * factor : none;
          s[nt][2 + j] = valid ? s[nt][2 + j] * factor : none;
          t0 = fmaxf(t0, s[nt][j]);
          t1 = fmaxf(t1, s[nt][2 + j]);
        }
      }
      t0 = fmaxf(t0, __shfl_xor_sync(0xffffffffu, t0, 1));
      t0 = fmaxf(t0, __shfl_xor_sync(0xffffffffu, t0, 2));
      t1 = fmaxf(t1, __shfl_xor_sync(0xffffffffu, t1, 1));
      t1 = fmaxf(t1, __shfl_xor_sync(0xffffffffu, t1, 2));
      // finite: the tile holds at least one key.  Sigmoid weights have no maximum: 0, and factors of 1
      const float n0 = gated ? 0.f : fmaxf(m0, t0), n1 = gated ? 0.f : fmaxf(m1, t1);
      const float a0 = gated ? 1.f : weight(m0 - n0), a1 = gated ? 1.f : weight(m1 - n1);
      m0 = n0; m1 = n1;
      l0 *= a0; l1 *= a1;
#pragma unroll
      for (int d = 0; d < DT; ++d) { o[d][0] *= a0; o[d][1] *= a0; o[d][2] *= a1; o[d][3] *= a1; }
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        if (!gated) {
          s[nt][0] = weight(s[nt][0] - n0); s[nt][1] = weight(s[nt][1] - n0);
          s[nt][2] = weight(s[nt][2] - n1); s[nt][3] = weight(s[nt][3] - n1);
        }
        l0 += s[nt][0] + s[nt][1];
        l1 += s[nt][2] + s[nt][3];
      }
      // ---- O += P V ----
      // EXT: P as three bfloat16 numbers, whose sum it is, and GV 16-column parts of the output at a time, so that the three products of an
      // accumulator, each waiting for the one before, run among those of others (5 requests of 1,100 keys: unrolled, one part at a time 14.2 us, this way 13.7)
      constexpr int PN = EXT ? 3 : 1, GV = EXT ? 4 : 1;
      const int mid = lane >> 3, r8 = lane & 7;
#pragma unroll
      for (int kk = 0; kk < 2; ++kk) {
        uint32_t pf[PN][4];                                        // P as the A operand of a k-step of 16 keys
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float x = s[kk * 2 + (r >> 1)][(r & 1) * 2], y = s[kk * 2 + (r >> 1)][(r & 1) * 2 + 1];
          if constexpr (EXT) {
            uint32_t parts[3];
            split3(x, y, parts);
#pragma unroll
            for (int i = 0; i < 3; ++i) pf[i][r] = parts[i];
          } else {
            pf[0][r] = pack2(x, y);
          }
        }
        const int kl = kk * 16 + (mid & 1) * 8 + r8;               // the key whose row this lane points at
#pragma unroll
        for (int dp = 0; dp < DT / 2; dp += GV) {
          uint32_t vb[GV][4];
#pragma unroll
          for (int u = 0; u < GV; ++u) {
            const int c = (dp + u) * 2 + (mid >> 1);
            const int cs = (c & ~7) | ((c ^ kl) & 7);
            ldmatrix_x4_trans(vb[u], v_addr + kl * (HS * 2) + cs * 16);
          }
#pragma unroll
          for (int i = PN - 1; i >= 0; --i) {                      // the small parts first
#pragma unroll
            for (int u = 0; u < GV; ++u) {
              mma_16816(o[(dp + u) * 2], pf[i], vb[u][0], vb[u][1]);
              mma_16816(o[(dp + u) * 2 + 1], pf[i], vb[u][2], vb[u][3]);
            }
          }
        }
      }
      __syncwarp();                                               // the stage is consumed before it is requested again
      if (j + NST < n_tiles) stage_tile(j + NST);
    }
    l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
    l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 2);

    // ---- the four warps' results, merged in their order ----
    __syncthreads();                                              // every warp is done with its staged values
    float* wo = reinterpret_cast<float*>(vbuf) + (size_t)warp * ROWS * HS;
    if ((lane & 3) == 0) {
      wm_s[warp][qrow] = m0; wm_s[warp][qrow + 8] = m1;
      wl_s[warp][qrow] = l0; wl_s[warp][qrow + 8] = l1;
    }
#pragma unroll
    for (int d = 0; d < DT; ++d) {
      *reinterpret_cast<float2*>(wo + qrow * HS + d * 8 + qcol) = make_float2(o[d][0], o[d][1]);
      *reinterpret_cast<float2*>(wo + (qrow + 8) * HS + d * 8 + qcol) = make_float2(o[d][2], o[d][3]);
    }
    __syncthreads();
    if (tid < ROWS) {                                             // per head: maximum and sum, and each warp's factor (0: no keys)
      float m = -INFINITY, l = 0.f;
#pragma unroll
      for (int w = 0; w < 4; ++w) m = fmaxf(m, wm_s[w][tid]);
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const float f = wm_s[w][tid] > -INFINITY ? weight(wm_s[w][tid] - m) : 0.f;
        l += f * wl_s[w][tid];
        wm_s[w][tid] = f;
      }
      hm_s[tid] = m;
      hl_s[tid] = l;
    }
    __syncthreads();
    // CLUSTER: every CTA merges the ranges for an equal part of the outputs: each sends an element to the CTA whose part it is in, and
    // its maxima and sums to all.  (With the first CTA merging all of them, four elements of six ranges a thread, the merge and
    // its stores were 2.2 of a launch's 8.3 us.)  The others run once the barrier of the kernel's start has completed (a later
    // pass: once they have merged the pass before).
    const uint32_t rank = CLUSTER ? tc::cluster_ctarank() : 0u;
    const int part = CLUSTER ? (nh * HS + splits - 1) / splits : 0;      // outputs of a CTA
    const uint32_t slots = (uint32_t)__cvta_generic_to_shared(recv_s);
    if (CLUSTER) {
      if (h0 == 0) tc::cluster_wait(); else tc::cluster_sync();
    }
#pragma unroll 2
    for (int i = tid; i < nh * HS; i += THREADS) {
      const int h = i / HS, d = i % HS;
      float acc = 0.f;
#pragma unroll
      for (int w = 0; w < 4; ++w) acc += wm_s[w][h] * reinterpret_cast<const float*>(vbuf)[((size_t)w * ROWS + h) * HS + d];
      if (CLUSTER) {
        const int to = i / part;
        tc::st_cluster_f32(tc::map_to_cta(slots + ((int)rank * part + i - to * part) * 4u, to), acc);
        if (d < splits) {                                           // a thread a CTA: at most eight of the head's
          tc::st_cluster_f32(tc::map_to_cta((uint32_t)__cvta_generic_to_shared(&w_s[h][rank]), d), hm_s[h]);
          tc::st_cluster_f32(tc::map_to_cta((uint32_t)__cvta_generic_to_shared(&l_in[h][rank]), d), hl_s[h]);
        }
      } else if (n_active == 1) {
        out[(size_t)e * out_stride + (size_t)(head0 + h) * HS + d] = __float2bfloat16_rn(finish(head0 + h, hm_s[h], hl_s[h], acc));
      } else {
        partial_o[(((size_t)e * n_heads + head0 + h) * splits + split) * HS + d] = acc;
        if (d == 0) {
          float* ml = partial_ml + (((size_t)e * n_heads + head0 + h) * splits + split) * 2;
          ml[0] = hm_s[h];
          ml[1] = hl_s[h];
        }
      }
    }
    if (CLUSTER) {
      tc::cluster_sync();
      for (int j = tid; j < part; j += THREADS) {
        const int i = (int)rank * part + j;
        if (i >= nh * HS) break;
        const int h = i / HS, d = i % HS;
        float m = -INFINITY;
        for (int r = 0; r < splits; ++r) m = fmaxf(m, w_s[h][r]);
        float l = 0.f, acc = 0.f;
        for (int r = 0; r < splits; ++r) {                          // in the order of the ranges
          const float mr = w_s[h][r];
          if (mr > -INFINITY) {
            const float f = weight(mr - m);
            l += f * l_in[h][r];
            acc += f * recv_s[r * part + j];
          }
        }
        out[(size_t)e * out_stride + (size_t)(head0 + h) * HS + d] = __float2bfloat16_rn(finish(head0 + h, m, l, acc));
      }
    }
    __syncthreads();                                              // vbuf is reused by the next pass
  }
  if (n_active == 1 || CLUSTER) return;

  // ---- the last range to arrive merges all of them ----
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    const int arrived = atomicAdd(&counters[e * n_kv + g], 1);
    last_s = arrived == n_active - 1;
  }
  __syncthreads();
  if (!last_s) return;
  __threadfence();
  for (int h0 = 0; h0 < group; h0 += ROWS) {
    const int nh = min(ROWS, group - h0);
    const size_t base0 = ((size_t)e * n_heads + g * group + h0) * splits;
    __syncthreads();
    for (int i = tid; i < nh * n_active; i += THREADS) {
      const int h = i / n_active, sp = i % n_active;
      const float2 ml = __ldcg(reinterpret_cast<const float2*>(partial_ml + (base0 + (size_t)h * splits + sp) * 2));
      w_s[h][sp] = ml.x;
      l_in[h][sp] = ml.y;
    }
    __syncthreads();
    if (tid < nh) {
      const float sv = !EXT || !opt.sink ? -INFINITY : (opt.sink_values ? opt.sink_values[g * group + h0 + tid] : 0.f);
      float m = sv;                                               // the sink is one more range: maximum its score, sum 1, no values
      for (int sp = 0; sp < n_active; ++sp) m = fmaxf(m, w_s[tid][sp]);
      float l = EXT && opt.sink ? weight(sv - m) : 0.f;
      for (int sp = 0; sp < n_active; ++sp) {
        const float f = weight(w_s[tid][sp] - m);
        l += f * l_in[tid][sp];
        w_s[tid][sp] = f;
      }
      const float inv = EXT && opt.sigmoid_bias ? 1.f : 1.f / l;
      for (int sp = 0; sp < n_active; ++sp) w_s[tid][sp] *= inv;
    }
    __syncthreads();
    for (int i = tid; i < nh * HS; i += THREADS) {
      const int h = i / HS, d = i % HS;
      const float* po = partial_o + (base0 + (size_t)h * splits) * HS + d;
      float acc = 0.f;
      int sp = 0;
      for (; sp + 8 <= n_active; sp += 8) {
        float ov[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) ov[u] = __ldcg(po + (size_t)(sp + u) * HS);
#pragma unroll
        for (int u = 0; u < 8; ++u) acc = fmaf(w_s[h][sp + u], ov[u], acc);
      }
      for (; sp < n_active; ++sp) acc = fmaf(w_s[h][sp], __ldcg(po + (size_t)sp * HS), acc);
      out[(size_t)e * out_stride + (size_t)(g * group + h0 + h) * HS + d] = __float2bfloat16_rn(acc);
    }
  }
  if (tid == 0) counters[e * n_kv + g] = 0;
}

}  // namespace decode_mma
