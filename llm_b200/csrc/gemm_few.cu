// Products of a few rows (up to 8): a stream of weights past warp-level MMAs, every output whole in one CTA.
//
// out[m][n] = sum_k a[m][k] w[n][k], bfloat16 operands, float32 accumulation.  Such a product is bound by the weights' bytes and, in a
// chain of dependent kernels, by what it does between the end of the kernel before it and its own end.  A tile is up to 16 weight rows
// over the whole of K.  One warp brings it by TMA (boxes of 64 k x the tile's rows x 8, 128-byte swizzle; two or four boxes a step) into a
// ring; eight warps share a box, 64 k each, hold the weights as the A operand of m16n8k16 and the rows as its B, and their accumulators
// are summed once in shared memory, in the order of the warps.  So there are no partial results in memory, and the epilogue has complete
// sums: it can apply a gated activation, or add to the residual stream.
//
// k runs in another order inside a block of 64, the same for both operands: lane `quad` of a row holds k = 16 quad .. 16 quad + 15, two
// 16-byte loads of each (which the swizzle spreads over the banks).  The rows are staged behind the wait by the warp that uses them (no
// barrier of the block): either bfloat16 rows, or float32 rows of the residual stream under an RMS norm; then x * gain is rounded and the factor
// 1 / rms(x), which is a row's, multiplies the sums (a rounding of x * gain has the same relative size as one of x * gain / rms).
//
// Tiles hold as many rows as divide the weight rows evenly over the SMs (14 of the 16 for 2,048 rows on 148 SMs); a CTA walks over its
// tiles with the stream running across them.
#include <atomic>
#include <mutex>

#include "tcgen05.cuh"
#include "warp_mma.cuh"

namespace {

constexpr int FEW_WARPS = 8;                      // that multiply; one more brings the weights
constexpr int FEW_BLOCK = 64;                     // k of a warp in a step
constexpr int FEW_BOX = FEW_WARPS * FEW_BLOCK;
constexpr int FEW_RED = 160;                      // floats of a warp's 16 x 8 accumulators in shared memory: 8 rows with a pitch of 20

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_addr(dst)),
               "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_addr(bar)), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)), "l"(src),
               "r"(bytes), "r"(smem_addr(bar)) : "memory");
}
// Shared memory by its own instructions and 32-bit addresses: through generic pointers (which is what the compiler makes of these kernels'
// computed places) a step of the loop below took 550 cycles instead of 200.
__device__ __forceinline__ uint4 lds16(uint32_t at) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at));
  return v;
}
__device__ __forceinline__ float4 lds4f(uint32_t at) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at));
  return v;
}
__device__ __forceinline__ float lds(uint32_t at) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at));
  return v;
}
__device__ __forceinline__ void sts16(uint32_t at, const uint4& v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void sts8(uint32_t at, uint32_t x, uint32_t y) { asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(at), "r"(x), "r"(y) : "memory"); }
__device__ __forceinline__ void sts(uint32_t at, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory"); }

constexpr int FEW_MAX_STAGES = 16;

enum : int { FEW_OUT_F32 = 0, FEW_OUT_BF16 = 1, FEW_OUT_ADD = 2, FEW_OUT_SILU = 3, FEW_OUT_RELU = 4, FEW_OUT_CLAMPED = 5 };

struct FewArgs {
  const __nv_bfloat16* a;      // rows, or
  const float* x;              // rows of the residual stream with
  const float* gain;           // the norm's gain and
  float eps, inv_k;            // its epsilon; 1 / K
  long long lda;               // of a or x
  void* out;
  long long ldo;
  int M, N, K;                 // N: outputs (gated: half the weight rows)
  int tile;                    // weight rows of a tile (gated: gate rows, as many up rows), up to 16 (8)
  int tiles, stages, boxes;    // boxes: of a step
  const float* bias;           // of the weight rows, or null
  float limit, alpha;          // of the clamped unit
  int early;                   // steps that are asked for before the rows, at most the stages
  int* error;
};

// Shared memory: [stages][stage] [rows: (block, half, row, quad) of 16 bytes] [gain, under a norm] [sums] [squares] [barriers]
inline int few_rest(int M, int K, bool normed) {
  return K * M * 2 + (normed ? K * 4 : 0) + 2 * FEW_WARPS * FEW_RED * 4 + FEW_WARPS * 32 + (2 * FEW_MAX_STAGES + 2) * 8;
}

// OUT: what becomes of the sums.  KEEP: K of up to four boxes; a step is a tile then, and a lane keeps its part of the rows in registers over its
// tiles (the products are bound by what they read from shared memory once the weights are there: 16 KB a box, and 8 more for the rows).
template <int OUT, bool KEEP>
__global__ void __launch_bounds__(FEW_WARPS * 32 + 32)
few_rows_kernel(const __grid_constant__ CUtensorMap weights, const __grid_constant__ CUtensorMap weights_tail, const FewArgs p) {
  constexpr bool GATED = OUT >= FEW_OUT_SILU;
  pdl_launch_dependents();
  extern __shared__ __align__(1024) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = lane >> 2, quad = lane & 3;
  const int blocks = p.K / FEW_BLOCK, all_boxes = (blocks + FEW_WARPS - 1) / FEW_WARPS;
  const int half_box = p.tile * 1024, box_bytes = GATED ? 2 * half_box : half_box, stage_bytes = p.boxes * box_bytes;
  const uint32_t ring = smem_addr(smem), acts = ring + p.stages * stage_bytes, gain = acts + p.K * p.M * 2;
  const uint32_t red = gain + (p.x ? p.K * 4 : 0), squares = red + 2 * FEW_WARPS * FEW_RED * 4;      // [2][warp][FEW_RED], [warp][8]
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + (squares + FEW_WARPS * 8 * 4 - ring));         // [stages]
  uint64_t* empty = full + p.stages;                                                         // [stages]
  uint64_t* gain_bar = empty + p.stages;
  uint64_t* asked = gain_bar + 1;                  // the rows are on their way
  if (threadIdx.x == 0) {
    tc::prefetch_tensormap(&weights);
    for (int s = 0; s < p.stages; ++s) { tc::mbar_init(full + s, 1); tc::mbar_init(empty + s, FEW_WARPS); }
    tc::mbar_init(gain_bar, 1);
    tc::mbar_init(asked, FEW_WARPS);
    tc::fence_mbar_init();
  }
  __syncthreads();

  if (warp == FEW_WARPS) {
    if (lane) return;
    // the weights, as far ahead as there are stages; they depend on no kernel
    bool ok = true;
    int s = 0, issued = 0;
    uint32_t phase = 1;                                // a fresh barrier's preceding phase counts as complete
    if (p.x) { tc::mbar_arrive_expect_tx(gain_bar, p.K * 4); bulk_copy(smem + (gain - ring), p.gain, p.K * 4, gain_bar); }
    for (int tile = blockIdx.x; ok && tile < p.tiles; tile += gridDim.x) {
      const int n = min(tile * p.tile, p.N - p.tile);  // the last tile ends with the weights, and repeats rows of the one before
      for (int b = 0; b < all_boxes;) {
        // what a load waits for is what was asked for before it: the rows come before all but the first steps
        // (and the bounded waits, from this one on, begin when the kernels before this one have ended, however long they take)
        if (issued == p.early) { pdl_wait(); ok = tc::mbar_wait(asked, 0); }
        ok = ok && tc::mbar_wait(empty + s, phase);
        if (!ok) break;
        const int end = min(b + p.boxes, all_boxes);
        const int missing = max(0, end * FEW_WARPS - blocks);      // a ragged last box has a map of its own: none reaches past K
        tc::mbar_arrive_expect_tx(full + s, (end - b) * box_bytes - missing * (box_bytes / FEW_WARPS));
        for (unsigned char* dst = smem + s * stage_bytes; b < end; ++b, dst += box_bytes) {
          const CUtensorMap* map = (b + 1) * FEW_WARPS <= blocks ? &weights : &weights_tail;
          tma_load_3d(dst, map, 0, n, b * FEW_WARPS, full + s);
          if (GATED) tma_load_3d(dst + half_box, map, 0, p.N + n, b * FEW_WARPS, full + s);
        }
        ++issued;
        if (++s == p.stages) { s = 0; phase ^= 1; }
      }
    }
    if (!ok) {
      atomicExch(p.error, 10);
      for (int i = max(0, issued - p.stages); i < issued; ++i) tc::mbar_wait(full + i % p.stages, (i / p.stages) & 1);      // its copies in flight
    }
    return;
  }

  pdl_wait();
  if (warp >= blocks && lane == 0) tc::mbar_arrive(asked);      // none of its own
  // the rows, the warp's blocks warp, warp + 8, ...: [block][half of a lane's 16 k][row][quad] of 16 bytes, all lanes along k
  bool ok = true;
  if (p.x) {
    // four blocks at a time, a lane four k of the first or second and four of the third or fourth, the same for every row
    const int place = ((lane >> 1) & 1) * p.M * 64 + ((lane >> 2) & 3) * 16 + (lane & 1) * 8;      // of 4 k in a block
    ok = tc::mbar_wait(gain_bar, 0);
    for (int b0 = warp; b0 < blocks; b0 += 4 * FEW_WARPS) {
      const int block[2] = {b0 + (lane >> 4) * FEW_WARPS, b0 + (2 + (lane >> 4)) * FEW_WARPS};
      float4 g[2];
#pragma unroll
      for (int i = 0; i < 2; ++i)
        g[i] = block[i] < blocks ? lds4f(gain + (block[i] * FEW_BLOCK + (lane & 15) * 4) * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
      float4 v[8][2];
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          v[r][i] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (r < p.M && block[i] < blocks)
            v[r][i] = *reinterpret_cast<const float4*>(p.x + (size_t)r * p.lda + block[i] * FEW_BLOCK + (lane & 15) * 4);
        }
      if (b0 == warp && lane == 0) tc::mbar_arrive(asked);
      float q[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        q[r] = 0.f;
        if (r >= p.M) continue;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float4 y = v[r][i];
          q[r] += fmaf(y.x, y.x, y.y * y.y) + fmaf(y.z, y.z, y.w * y.w);
          const __nv_bfloat162 h[2] = {__floats2bfloat162_rn(y.x * g[i].x, y.y * g[i].y), __floats2bfloat162_rn(y.z * g[i].z, y.w * g[i].w)};
          if (block[i] < blocks)
            sts8(acts + (block[i] * 2 * p.M + r) * 64 + place, *reinterpret_cast<const uint32_t*>(&h[0]), *reinterpret_cast<const uint32_t*>(&h[1]));
        }
      }
      // eight sums over the warp: lanes exchange halves of the rows, then the four lanes of a row add theirs
#pragma unroll
      for (int w = 16, n = 4; n; w >>= 1, n >>= 1)
#pragma unroll
        for (int r = 0; r < n; ++r) {
          const bool up = lane & w;
          const float keep = up ? q[r + n] : q[r], give = up ? q[r] : q[r + n];
          q[r] = keep + __shfl_xor_sync(~0u, give, w);
        }
      q[0] += __shfl_xor_sync(~0u, q[0], 2);
      q[0] += __shfl_xor_sync(~0u, q[0], 1);
      if ((lane & 3) == 0) {                         // of row (bits 4, 3, 2 of the lane)
        const uint32_t at = squares + (warp * 8 + (lane >> 2)) * 4;
        sts(at, b0 == warp ? q[0] : lds(at) + q[0]);
      }
    }
    if (warp >= blocks && lane < 8) sts(squares + (warp * 8 + lane) * 4, 0.f);
  } else {
    const int place = (lane & 1) * p.M * 64 + ((lane >> 1) & 3) * 16;      // of 8 k in a block
#pragma unroll 1
    for (int b0 = warp; b0 < blocks; b0 += 8 * FEW_WARPS) {
      const int block[2] = {b0 + (lane >> 3) * FEW_WARPS, b0 + (4 + (lane >> 3)) * FEW_WARPS};
      uint4 v[8][2];
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (r < p.M && block[i] < blocks) v[r][i] = *reinterpret_cast<const uint4*>(p.a + (size_t)r * p.lda + block[i] * FEW_BLOCK + (lane & 7) * 8);
      if (b0 == warp && lane == 0) tc::mbar_arrive(asked);
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (r < p.M && block[i] < blocks) sts16(acts + (block[i] * 2 * p.M + r) * 64 + place, v[r][i]);
    }
  }
  __syncwarp();

  // Lanes of weight rows past the tile's, and of rows past M, read the last one's again: they make sums that nobody stores.
  const int lo_row = warp * p.tile + min(row, p.tile - 1);
  const int hi_row = warp * p.tile + min(GATED ? row : row + 8, p.tile - 1);
  uint32_t lo_at[2], hi_at[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    lo_at[j] = ring + lo_row * 128 + (((2 * quad + j) ^ (lo_row & 7)) << 4);
    hi_at[j] = ring + (GATED ? half_box : 0) + hi_row * 128 + (((2 * quad + j) ^ (hi_row & 7)) << 4);
  }
  const uint32_t act_at = acts + (warp * 2 * p.M + min(row, p.M - 1)) * 64 + quad * 16;
  const int act_box = FEW_WARPS * 2 * p.M * 64, act_half = p.M * 64;
  struct Weights { uint4 lo[2], hi[2]; };
  struct Rows { uint4 b[2]; };
  auto load = [&](Weights& o, int weight) {
#pragma unroll
    for (int j = 0; j < 2; ++j) { o.lo[j] = lds16(lo_at[j] + weight); o.hi[j] = lds16(hi_at[j] + weight); }
  };
  auto load_rows = [&](Rows& o, int box) {
#pragma unroll
    for (int j = 0; j < 2; ++j) o.b[j] = lds16(act_at + box * act_box + j * act_half);
  };
  auto multiply = [&](float (&c)[2][4], const Weights& o, const Rows& r) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint32_t a0[4] = {o.lo[j].x, o.hi[j].x, o.lo[j].y, o.hi[j].y}, a1[4] = {o.lo[j].z, o.hi[j].z, o.lo[j].w, o.hi[j].w};
      mma(c[0], a0, r.b[j].x, r.b[j].y);
      mma(c[1], a1, r.b[j].z, r.b[j].w);
    }
  };
  Rows kept[4];
  if (KEEP) {
#pragma unroll
    for (int b = 0; b < 4; ++b)
      if (b * FEW_WARPS + warp < blocks) load_rows(kept[b], b);
  }
  const int out_row = threadIdx.x & 15, out_token = threadIdx.x >> 4;
  int s = 0, buffer = 0;
  uint32_t phase = 0;
  float scale = 1.f;
#pragma unroll 1
  for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
    const int n0 = min(tile * p.tile, p.N - p.tile), n = n0 + out_row;
    const bool mine = out_token < p.M && n >= tile * p.tile && out_row < p.tile;
    float before = 0.f;
    float bias = 0.f, bias_up = 0.f;
    if (p.bias && mine) { bias = p.bias[n]; if (GATED) bias_up = p.bias[p.N + n]; }
    if (OUT == FEW_OUT_ADD && mine) before = reinterpret_cast<float*>(p.out)[(size_t)out_token * p.ldo + n];
    float c[2][4] = {};
    auto release = [&]() {
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(empty + s);
      if (++s == p.stages) { s = 0; phase ^= 1; }
    };
    if (KEEP) {
      ok = ok && tc::mbar_wait(full + s, phase);
      const int weight = s * stage_bytes;
#pragma unroll
      for (int b = 0; b < 4; b += 2) {                          // a pair of boxes: all of their loads, then the products
        Weights one, two;
        const bool first = b * FEW_WARPS + warp < blocks, second = (b + 1) * FEW_WARPS + warp < blocks;
        if (first) load(one, weight + b * box_bytes);
        if (second) load(two, weight + (b + 1) * box_bytes);
        if (first) multiply(c, one, kept[b]);
        if (second) multiply(c, two, kept[b + 1]);
      }
      release();
    } else {
#pragma unroll 1
      for (int b = 0; b < all_boxes;) {
        ok = ok && tc::mbar_wait(full + s, phase);
        const int end = min(b + p.boxes, all_boxes);
        int weight = s * stage_bytes;
#pragma unroll 1
        for (; b < end; b += 2, weight += 2 * box_bytes) {
          Weights one, two;
          Rows x, y;
          const bool first = b * FEW_WARPS + warp < blocks, second = b + 1 < end && (b + 1) * FEW_WARPS + warp < blocks;
          if (first) { load(one, weight); load_rows(x, b); }
          if (second) { load(two, weight + box_bytes); load_rows(y, b + 1); }
          if (first) multiply(c, one, x);
          if (second) multiply(c, two, y);
        }
        b = end;
        release();
      }
    }
    const uint32_t put = red + ((buffer * FEW_WARPS + warp) * FEW_RED + 2 * quad * 20 + row) * 4;
    sts(put, c[0][0] + c[1][0]);
    sts(put + 20 * 4, c[0][1] + c[1][1]);
    sts(put + 8 * 4, c[0][2] + c[1][2]);
    sts(put + 28 * 4, c[0][3] + c[1][3]);
    asm volatile("bar.sync 1, %0;" ::"n"(FEW_WARPS * 32) : "memory");
    if (mine) {
      if (tile == blockIdx.x && p.x) {                 // the row's factor, once
        float q = 0.f;
#pragma unroll
        for (int i = 0; i < FEW_WARPS; ++i) q += lds(squares + (i * 8 + out_token) * 4);
        scale = rsqrtf(q * p.inv_k + p.eps);
      }
      const uint32_t get = red + (buffer * FEW_WARPS * FEW_RED + out_token * 20 + out_row) * 4;
      float z = 0.f, u = 0.f;
#pragma unroll
      for (int i = 0; i < FEW_WARPS; ++i) {
        z += lds(get + i * FEW_RED * 4);
        if (GATED) u += lds(get + (i * FEW_RED + 8) * 4);
      }
      z = fmaf(z, scale, bias); u = fmaf(u, scale, bias_up);
      const size_t at = (size_t)out_token * p.ldo + n;
      if (OUT == FEW_OUT_ADD) z += before;
      if (OUT == FEW_OUT_SILU) z = z / (1.f + expf(-z)) * u;
      if (OUT == FEW_OUT_RELU) z = fmaxf(z, 0.f) * u;
      if (OUT == FEW_OUT_CLAMPED) {
        z = fminf(z, p.limit);
        z = z / (1.f + expf(-p.alpha * z)) * (fminf(fmaxf(u, -p.limit), p.limit) + 1.f);
      }
      if (OUT == FEW_OUT_F32 || OUT == FEW_OUT_ADD) reinterpret_cast<float*>(p.out)[at] = z;
      else reinterpret_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16_rn(z);
    }
    buffer ^= 1;
  }
  if (!ok && lane == 0) atomicExch(p.error, 12);
}

typedef CUresult (*EncodeFewFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeFewFn encode_few_fn() {
  static EncodeFewFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeFewFn>(f);
  });
  return fn;
}

// w [rows, K] as [K / 64][rows][64]; a box holds `blocks` blocks of `tile` rows.
int encode_weights(CUtensorMap* out, const void* w, long long rows, int K, long long ldw, int tile, int blocks) {
  EncodeFewFn fn = encode_few_fn();
  if (!fn) return llmk_fail(-2, "cuTensorMapEncodeTiled is not available from the driver");
  cuuint64_t dims[3] = {(cuuint64_t)FEW_BLOCK, (cuuint64_t)rows, (cuuint64_t)(K / FEW_BLOCK)}, strides[2] = {(cuuint64_t)ldw * 2, FEW_BLOCK * 2};
  cuuint32_t box[3] = {FEW_BLOCK, (cuuint32_t)tile, (cuuint32_t)blocks}, step[3] = {1, 1, 1};
  auto encode = [&] {
    return fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(w), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult r = encode();
  // a thread whose first call into CUDA this is: the runtime binds the device's context at its own calls, the driver's function does not
  int device = 0;
  if (r == CUDA_ERROR_INVALID_CONTEXT && cudaGetDevice(&device) == cudaSuccess && cudaSetDevice(device) == cudaSuccess) r = encode();
  return r == CUDA_SUCCESS ? 0 : llmk_fail(-2, "cuTensorMapEncodeTiled failed with %d", (int)r);
}

// What must be left beside the rows, in boxes of 16 KB; a gain of K numbers is counted with the rows whether they are normed or not, so that one limit
// holds for all forms.  Beyond it the tcgen05 kernel's swapped mode is ahead.  Replayed decode steps, that kernel / this one: 8 rows of 8,448 (3.2
// boxes left) 581 / 590 us, 5 rows of 14,336 (1.3) 2,930 / 2,995, 4 rows (3.03) 2,913 / 2,917, 2 rows (6.5) 2,894 / 2,846.
constexpr int FEW_SMEM = 227 * 1024, FEW_LEAST_STAGES = 4;
// The most that is in flight, and how much of it is asked for before the rows, which wait behind that.  Decode steps of 1.1 B (1, 4, 8 rows), all of the
// ring first: 64 KB 771, 795, 828 us; 100 KB 695, 712, 746; 140 KB 666, 690, 750; 200 KB 677, 719, 755 (649, 675, 738 with 140 KB once the rows
// were kept in registers); of 140 KB first 96 KB: 634, 665, 717; 72 KB: 629, 667, 716; 57 KB: 638, 668, 727.
constexpr int FEW_RING = 140 * 1000, FEW_EARLY = 72 * 1000;

template <bool KEEP>
int launch_few(const CUtensorMap& map, const CUtensorMap& tail, const FewArgs& p, int out_kind, int grid, size_t smem, cudaStream_t stream) {
  void (*kern)(CUtensorMap, CUtensorMap, FewArgs) =
      out_kind == FEW_OUT_F32 ? few_rows_kernel<FEW_OUT_F32, KEEP> : out_kind == FEW_OUT_BF16 ? few_rows_kernel<FEW_OUT_BF16, KEEP>
      : out_kind == FEW_OUT_ADD ? few_rows_kernel<FEW_OUT_ADD, KEEP> : out_kind == FEW_OUT_SILU ? few_rows_kernel<FEW_OUT_SILU, KEEP>
      : out_kind == FEW_OUT_RELU ? few_rows_kernel<FEW_OUT_RELU, KEEP> : few_rows_kernel<FEW_OUT_CLAMPED, KEEP>;
  // once per build and device, the most that any launch asks for: the size belongs to the kernel and not to the launch, and another thread's
  // smaller one, set between this thread's setting and its launch, would make the launch fail
  static std::atomic<bool> ready[FEW_OUT_CLAMPED + 1][64];
  int device = -1;
  const bool known = cudaGetDevice(&device) == cudaSuccess && device >= 0 && device < 64;
  if (!known || !ready[out_kind][device].load(std::memory_order_acquire)) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FEW_SMEM);
    if (e != cudaSuccess) return llmk_fail((int)e, "gemm_few: %s", cudaGetErrorString(e));
    if (known) ready[out_kind][device].store(true, std::memory_order_release);
  }
  launch_kernel(kern, dim3(grid), dim3(FEW_WARPS * 32 + 32), smem, stream, map, tail, p);
  LLMK_LAUNCH_CHECK("gemm_few");
}

}  // namespace

// Whether llmk_gemm_few takes M rows of K: up to 8 rows, K a multiple of 64, rows that fit in shared memory beside the least stages.
LLMK_API int llmk_gemm_few_supported(int M, int K) {
  return M > 0 && M <= 8 && K > 0 && K % FEW_BLOCK == 0 && K < (1 << 20) && few_rest(M, K, true) + FEW_LEAST_STAGES * 16384 <= FEW_SMEM;
}

// out = rows @ w^T.  rows: a (bfloat16) or, with a null, the float32 rows x under an RMS norm with `gain` and `eps`.  out_kind: 0 float32,
// 1 bfloat16, 2 added to float32 out, 3 / 4 silu / relu of the first N weight rows' product times that of the N behind them, bfloat16;
// 5 the clamped unit of the two, g = min(., limit), g sigmoid(alpha g) (clamp(., -limit, limit) + 1).  bias: float32, one per weight row, or null.
LLMK_API int llmk_gemm_few(const void* a, const float* x, const float* gain, float eps, long long lda, const void* w, long long ldw, void* out,
                           long long ldo, int M, int N, int K, int out_kind, const float* bias, float limit, float alpha, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  LLMK_REQUIRE(M > 0 && N > 0 && llmk_gemm_few_supported(M, K), "gemm_few: M=%d N=%d K=%d", M, N, K);
  LLMK_REQUIRE(lda >= K && ldw >= K && ldo >= N && ldw % 8 == 0 && (uintptr_t)w % 16 == 0, "gemm_few: strides %lld %lld %lld", lda, ldw, ldo);
  LLMK_REQUIRE((a != nullptr) != (x != nullptr) && (!a || (lda % 8 == 0 && (uintptr_t)a % 16 == 0)) &&
               (!x || (lda % 4 == 0 && (uintptr_t)x % 16 == 0 && gain && (uintptr_t)gain % 16 == 0)), "gemm_few: rows of one kind, 16-byte aligned");
  LLMK_REQUIRE(out_kind >= 0 && out_kind <= 5, "gemm_few: unknown output kind %d", out_kind);
  const bool gated = out_kind >= FEW_OUT_SILU;
  FewArgs p = {(const __nv_bfloat16*)a, x, gain, eps, 1.f / K, lda, out, ldo, M, N, K};
  p.bias = bias; p.limit = limit; p.alpha = alpha;
  p.error = llmk_error_word(1);
  LLMK_REQUIRE(p.error, "gemm_few: no error word");
  const int sms = llmk_sm_count(), most = gated ? 8 : 16;
  const int rounds = (N + most * sms - 1) / (most * sms);
  p.tile = (N + rounds * sms - 1) / (rounds * sms);
  p.tiles = (N + p.tile - 1) / p.tile;
  const int grid = p.tiles < sms ? p.tiles : sms;
  const int box_bytes = (gated ? 2 : 1) * p.tile * 1024, all_boxes = (K + FEW_BOX - 1) / FEW_BOX;
  const int rest = few_rest(M, K, x != nullptr), room = FEW_SMEM - rest < FEW_RING ? FEW_SMEM - rest : FEW_RING;
  const bool keep = all_boxes <= 4 && room >= 2 * all_boxes * box_bytes;
  // four boxes a step (a step costs a wait) while three steps fit, or all there are; else two, else one
  for (p.boxes = 4;; p.boxes /= 2) {
    if (p.boxes > all_boxes) p.boxes = all_boxes;
    const int all = ((p.tiles + sms - 1) / sms) * ((all_boxes + p.boxes - 1) / p.boxes), fit = room / (p.boxes * box_bytes);
    p.stages = all < fit ? all : fit;
    if (keep || p.boxes == 1 || p.stages >= 3 || p.stages >= all) break;
  }
  if (p.stages > FEW_MAX_STAGES) p.stages = FEW_MAX_STAGES;
  p.early = FEW_EARLY / (p.boxes * box_bytes);
  if (p.early < 1) p.early = 1;
  if (p.early > p.stages) p.early = p.stages;      // no stage is waited for before the rows
  // at least half of the shared memory: a CTA that shared its SM with another of the same launch would end long after the rest (a kernel that
  // starts while the one before it leaves SMs finds room for two on some: a decode step of 1.1 B then took 880 us instead of 720)
  const size_t need = rest + (size_t)p.stages * p.boxes * box_bytes, smem = need < FEW_SMEM / 2 + 1024 ? FEW_SMEM / 2 + 1024 : need;
  CUtensorMap map, tail;
  const int last = K / FEW_BLOCK % FEW_WARPS, w_rows = gated ? 2 * N : N;
  if (int rc = encode_weights(&map, w, w_rows, K, ldw, p.tile, all_boxes == 1 && last ? last : FEW_WARPS)) return rc;
  tail = map;
  if (last)
    if (int rc = encode_weights(&tail, w, w_rows, K, ldw, p.tile, last)) return rc;
  return keep ? launch_few<true>(map, tail, p, out_kind, grid, smem, stream) : launch_few<false>(map, tail, p, out_kind, grid, smem, stream);
}
