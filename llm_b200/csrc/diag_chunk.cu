// Recurrences with a diagonal decay over prompts, sixteen tokens at a time on warp-level MMAs (bfloat16 projections):
//
//   S_t = diag(a_t) S_(t-1) + k_t v_t^T,     o_t = S_t^T q_t      (bonus form: o_t = (S_(t-1) + diag(u) k_t v_t^T)^T q_t)
//
// over a chunk of C = 16 tokens that starts from S, with P_t = a_1 .. a_t and R_s = a_(s+1) .. a_C (products per key channel):
//
//   o_t = S^T (q_t P_t) + sum_(s <= t) A_ts v_s,      A_ts = sum_d q_td k_sd a_(s+1)d .. a_td
//   S  <- diag(P_C) S + sum_s (k_s R_s) v_s^T
//
// (bonus form: P_(t-1), products up to a_(t-1), and A_tt = sum_d q_td u_d k_td).  Every product of decays runs forward from one
// token to a later one, so that nothing is divided and a decay of zero is as good as any other; A is made by plain float32
// multiply-adds, a running product per (s, d).  The three contractions run as bfloat16 MMAs on operands split into three
// bfloat16 numbers each (v is bfloat16 to begin with): S^T q takes the six products above 2^-24, the others three, summed in
// float32; S itself stays in float32 registers as MMA accumulators of S^T, which are in the layout of the next product's operand,
// and the decay and sum of the update are float32 multiply-adds.
//
// What is not finite reaches its own token and the later ones of its request, as token by token: queries, keys and decays do by the
// form of the sums (a weight of a later token is set to 0, not multiplied), but a value that is infinite or no number would meet the
// zeros of the earlier tokens' rows of A in the MMA.  From a chunk on that holds one in the CTA's columns, the segment is walked token by
// token (walk_rest), which a healthy model never sees; looking for one costs nothing that shows (a piece of 16 bytes a thread and chunk).
//
// Work split: a CTA owns (segment of an entry, head, 16 value columns a warp).  Segments run side by side in two passes as in
// scan.cu: pass 1 leaves the end state from zero and the product of the decays of every segment but an entry's last, a chain
// kernel turns those into start states, pass 2 writes the outputs and the request's new state.
//
// What bounds it: latency at 16 (eight-warp form) or 8 to 16 warps an SM: half of the issue slots and a fifth of the tensor pipe are in use
// (what the warps wait for is shared memory and the barriers between a chunk's three parts).  2,048 tokens, the three launches against
// the token-by-token passes that they took the place of: power form, 8 heads of 128 x 256: 261 -> 132 us; bonus form, 32 heads of
// 64 x 64: 214 -> 103; scalar form, 32 heads of 128 x 64: 245 -> 76; gate form, 16 heads of 128 x 128: 350 -> 123.  Seven entries of 1
// to 150 tokens, 8 heads of 32 x 32: 54 -> 39; heads of 8 x 8: 149 -> 39 (the tiles are then mostly padding, and still ahead).
// Errors against 64 bits (relative, outputs / states): power form 7.8e-7 / 8.7e-7 -> 7.4e-7 / 8.4e-7, bonus form 1.1e-7 / 8.4e-8 ->
// 9.4e-8 / 6.8e-8, scalar form 1.7e-7 / 1.4e-7 -> 1.5e-7 / 1.3e-7, gate form 1.7e-7 / 3.2e-7 -> 1.5e-7 / 2.8e-7.
#include "diag_chunk.cuh"
#include "warp_mma.cuh"

namespace diag_chunk {
namespace {

using bf16 = __nv_bfloat16;
constexpr int C = 16;                    // tokens of a chunk: the MMAs' M (read-out) and K (update)
constexpr int AP = C + 8;                // pitch of A in shared memory, conflict-free for 16-byte rows
constexpr int MAX_SEG = 256;             // tokens of a segment (the scalar form keeps sixteen numbers a token)

__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float log_sigmoid_f(float z) { return fminf(z, 0.f) - log1pf(expf(-fabsf(z))); }

// c += A B, the product in accumulators of its own and the sum a float32 addition.  An MMA that accumulates cuts off what does not fit below
// its largest term; over the eight steps of 128 channels that was most of the outputs' error (relative to the token-by-token kernel, seven
// entries of 1 to 150 tokens, eight sets of inputs: gate form of 128 x 128 1.11 with accumulating MMAs, 0.88 this way; bonus form 1.02 and 0.85).
__device__ __forceinline__ void add_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  float part[4] = {};
  mma(part, a, b0, b1);
#pragma unroll
  for (int i = 0; i < 4; ++i) c[i] += part[i];
}

// Whether one of eight bfloat16 numbers is infinite or no number.
__device__ __forceinline__ bool not_finite8(const bf16* p) {
  const uint4 w = *reinterpret_cast<const uint4*>(p);
  auto two = [](uint32_t x) { return (x & 0x7f80u) == 0x7f80u || (x & 0x7f800000u) == 0x7f800000u; };
  return two(w.x) || two(w.y) || two(w.z) || two(w.w);
}

// Segment `index` of the step: its entry and tokens [t0, t1).  False behind the last one.
__device__ __forceinline__ bool segment_of(const int* cu, int n_entries, int seg_len, int index, int& entry, int& t0, int& t1, int& end) {
  int b = cu[0];
  for (int e = 0; e < n_entries; ++e) {
    const int n = cu[e + 1], segs = (n - b + seg_len - 1) / seg_len;
    if (index < segs) {
      entry = e; end = n;
      t0 = b + index * seg_len;
      t1 = min(n, t0 + seg_len);
      return true;
    }
    index -= segs;
    b = n;
  }
  return false;
}

// The tokens [from, t1) of a segment one after the other, a thread per value column: the state starts and stays in the segment's place,
// from where it goes to the request's if the segment is its entry's last.  rows: shared memory for 3 * dim numbers; decays: thread d's
// product of pass 1 so far.
template <int FORM, bool STATE_ONLY>
__device__ void walk_rest(const Args& a, float* rows, int entry, int from, int t1, bool last, int colb, int vt, float decays) {
  const int tid = threadIdx.x, head = blockIdx.y, qk_head = head / (a.heads / a.qk_heads), dim = a.dim, vdim = a.vdim;
  const size_t unit = (size_t)blockIdx.z * a.heads + head;
  float *a_s = rows, *q_s = rows + dim, *k_s = rows + 2 * dim;
  const int col = colb + tid;
  const bool live = tid < vt && col < vdim;
  float* S = a.seg_state + unit * dim * vdim + col;
  for (int t = from; t < t1; ++t) {
    __syncthreads();
    for (int d = tid; d < dim; d += blockDim.x) {
      const size_t at = (size_t)t * a.qk_stride + (size_t)qk_head * dim + d;
      float av, qv = __bfloat162float(a.q[at]), kv = FORM == GATE ? 0.f : __bfloat162float(a.k[at]);
      if (FORM == SCALAR) {
        const float dt = softplus_f(__bfloat162float(a.dt[(size_t)t * a.dt_stride + head]) + a.dt_bias[head]);
        av = expf(-expf(a.a_log[head]) * dt);
        kv *= dt;
      } else {
        const float z = a.z[(size_t)t * a.z_stride + (size_t)head * dim + d] + (a.z_bias ? a.z_bias[head * dim + d] : 0.f);
        if (FORM == BONUS) {
          av = expf(-expf(z));
        } else if (FORM == POWER) {
          av = expf(log_sigmoid_f(z) * a.inv_tau);
        } else {
          const float low = a.bonus[head * dim + d];
          qv = qv / (1.f + expf(-qv));
          av = low + (1.f - low) / (1.f + expf(-z));
          kv = 1.f - av;
        }
      }
      a_s[d] = av; q_s[d] = qv; k_s[d] = kv;
      decays *= av;                                                    // dim <= blockDim.x: one channel a thread
    }
    __syncthreads();
    if (!live) continue;
    const float v = __bfloat162float(a.v[(size_t)t * a.v_stride + (size_t)head * vdim + col]);
    float o = 0.f;
    for (int d = 0; d < dim; ++d) {
      const float old = S[(size_t)d * vdim], kv = k_s[d] * v, now = fmaf(a_s[d], old, kv);
      o = fmaf(q_s[d], FORM == BONUS ? fmaf(a.bonus[head * dim + d], kv, old) : now, o);
      S[(size_t)d * vdim] = now;
    }
    if (FORM == POWER) o *= a.q_scale;
    if (FORM == SCALAR) o = fmaf(a.skip[head], v, o);
    if (!STATE_ONLY) a.out[(size_t)t * a.out_stride + (size_t)head * vdim + col] = o;
  }
  if (STATE_ONLY) {
    if (blockIdx.x == 0 && tid < dim) a.seg_decay[unit * dim + tid] = decays;
  } else if (last && live) {
    float* to = a.state + (size_t)a.state_slots[entry] * a.slot_stride + (size_t)head * dim * vdim + col;
    for (int d = 0; d < dim; ++d) to[(size_t)d * vdim] = S[(size_t)d * vdim];
  }
}

// ---- scalar form ----------------------------------------------------------------------------------------------
// One decay per head and token: it comes out of every contraction.  q and k enter as they are (bfloat16), A = (q . k) times the product
// of the decays between, which is one number per pair of tokens, and the update's scale stands on v:
//   o_t = P_t S^T q_t + sum_(s <= t) (q_t . k_s) D_ts v_s,   D_ts = dt_s a_(s+1) .. a_t,     S <- P_C S + sum_s k_s (D_Cs v_s)^T
// The numbers of a segment (P, D) are made at its start; the scores pass from one MMA's result to the next one's operand in registers.
// 2,048 tokens, 32 heads of 128 x 64: 155 us for the three launches on the general chunk kernel below, 76 us here.
template <int DP>
struct ScalarShape {
  static constexpr int VT = 64, VP = VT + 8, SP = DP + 8, NT = 128;
  static constexpr int STAGE = (2 * C * SP + C * VP) * 2;              // q, k, v
};

template <int DP, bool STATE_ONLY>
__global__ void __launch_bounds__(128, 4)
scalar_chunk_kernel(const __grid_constant__ Args a) {
  using Sh = ScalarShape<DP>;
  constexpr int NT = Sh::NT, VT = Sh::VT, VP = Sh::VP, SP = Sh::SP;
  extern __shared__ __align__(16) unsigned char smem[];
  float* a_s = reinterpret_cast<float*>(smem + 2 * Sh::STAGE);         // decays of the segment, padded to whole chunks with 1
  float* p_s = a_s + a.seg_len + C;                                    // P of every token
  float* d_s = p_s + a.seg_len + C;                                    // [chunk][t][s]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int head = blockIdx.y, group = head / (a.heads / a.qk_heads), dim = a.dim, vdim = a.vdim, colb = blockIdx.x * VT;
  pdl_launch_dependents();
  const float neg_a = -expf(a.a_log[head]), bias = a.dt_bias[head], skip = a.skip[head];
  int entry = 0, t0 = 0, t1 = 0, end = 0;
  const bool there = segment_of(a.cu_tokens, a.n_entries, a.seg_len, blockIdx.z, entry, t0, t1, end);
  pdl_wait();
  if (!there) return;
  const bool last = t1 == end;
  if (STATE_ONLY && last) return;
  const size_t unit = (size_t)blockIdx.z * a.heads + head;
  float* S_seg = a.seg_state + unit * dim * vdim;
  const int chunks = (t1 - t0 + C - 1) / C;

  auto bring = [&](int c0, int stage) {
    const int n = min(C, t1 - c0);
    bf16* q_r = reinterpret_cast<bf16*>(smem + stage * Sh::STAGE);
    const size_t at = (size_t)c0 * a.qk_stride + (size_t)group * dim;
    if (!STATE_ONLY) bring_rows<C, NT>(q_r, SP, a.q + at, a.qk_stride, n, dim, DP);
    bring_rows<C, NT>(q_r + C * SP, SP, a.k + at, a.qk_stride, n, dim, DP);
    bring_rows<C, NT>(q_r + 2 * C * SP, VP, a.v + (size_t)c0 * a.v_stride + (size_t)head * vdim + colb, a.v_stride, n, min(VT, vdim - colb), VT);
  };
  bring(t0, 0);
  // steps and decays, then a running product per token s of a chunk
  for (int i = tid; i < chunks * C; i += NT) {
    const float dt = i < t1 - t0 ? softplus_f(__bfloat162float(a.dt[(size_t)(t0 + i) * a.dt_stride + head]) + bias) : 0.f;
    p_s[i] = dt;
    a_s[i] = expf(neg_a * dt);                                         // 1 behind the end
  }
  __syncthreads();
  for (int i = tid; i < chunks * C; i += NT) {
    const int c = i / C, s = i % C;
    const float dt = p_s[i];
    float f = 1.f, lack = 0.f;
    for (int t = 0; t < C; ++t) {
      if (t > s) {
        const float av = a_s[c * C + t];
        lack = fmaf(1.f - av, f, lack);
        f = lack < 0.5f ? 1.f - lack : f * av;
      }
      d_s[(c * C + t) * C + s] = t < s ? 0.f : f * dt;
    }
  }
  __syncthreads();
  for (int c = tid; c < chunks; c += NT) {
    float f = 1.f, lack = 0.f;
    for (int t = 0; t < C; ++t) {
      const float av = a_s[c * C + t];
      lack = fmaf(1.f - av, f, lack);
      f = lack < 0.5f ? 1.f - lack : f * av;
      p_s[c * C + t] = f;
    }
  }

  const int wcol = warp * 16, vr = colb + wcol + (lane >> 2), dc = 2 * (lane & 3);
  float st[DP / 8][4];                                                 // S^T as in the general kernel
#pragma unroll
  for (int i = 0; i < DP / 8; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int dd = i * 8 + dc + (j & 1), vv = vr + (j >> 1) * 8;
      st[i][j] = (!STATE_ONLY && dd < dim && vv < vdim) ? S_seg[(size_t)dd * vdim + vv] : 0.f;
    }
  }
  float decays = 1.f;
  const int tr = (lane & 7) + ((lane >> 3) & 1) * 8, th = (lane >> 4) * 8;      // ldmatrix: rows by lane bit 3, halves by bit 4
  const int hr = (lane & 7) + (lane >> 4) * 8, hh = ((lane >> 3) & 1) * 8;      // the other way round
  static_assert(C * VT / 8 == NT, "a thread looks at what it brought itself: one piece of the values");
  int ch = 0;
  for (; ch < chunks; ++ch) {
    const int c0 = t0 + ch * C, n = min(C, t1 - c0);
    const bf16* q_r = reinterpret_cast<const bf16*>(smem + (ch & 1) * Sh::STAGE);
    const bf16 *k_r = q_r + C * SP, *v_r = k_r + C * SP;
    cp_async_wait_all();
    if (__syncthreads_or(not_finite8(v_r + tid / (VT / 8) * VP + tid % (VT / 8) * 8))) break;
    if (ch + 1 < chunks) bring(c0 + C, (ch + 1) & 1);
    const float *P = p_s + ch * C, *D = d_s + ch * C * C;
    uint32_t va[4];
    ldsm4_t(va, v_r + hr * VP + wcol + hh);
    if (!STATE_ONLY) {
      float sc[2][4] = {}, hi[2][4] = {}, lo[2][4] = {}, own[2][4] = {};
#pragma unroll
      for (int ks = 0; ks < DP / 16; ++ks) {
        uint32_t qf[4], kf[4];
        ldsm4(qf, q_r + tr * SP + ks * 16 + th);
        ldsm4(kf, k_r + hr * SP + ks * 16 + hh);
        add_mma(sc[0], qf, kf[0], kf[1]);
        add_mma(sc[1], qf, kf[2], kf[3]);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          uint32_t b0[3], b1[3];
          split3(st[2 * ks][2 * nt], st[2 * ks][2 * nt + 1], b0);
          split3(st[2 * ks + 1][2 * nt], st[2 * ks + 1][2 * nt + 1], b1);
          add_mma(hi[nt], qf, b0[0], b1[0]);
          mma(lo[nt], qf, b0[1], b1[1]);
          mma(lo[nt], qf, b0[2], b1[2]);
        }
      }
      uint32_t af[3][4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {                                    // (t, s) quarters: t + 8 (r & 1), s + 8 (r >> 1)
        const int t = (lane >> 2) + (r & 1) * 8, s = dc + (r >> 1) * 8;
        const float2 w = *reinterpret_cast<const float2*>(D + t * C + s);
        const float x = s <= t ? sc[r >> 1][2 * (r & 1)] * w.x : 0.f, y = s + 1 <= t ? sc[r >> 1][2 * (r & 1) + 1] * w.y : 0.f;
        uint32_t p[3];
        split3(x, y, p);
#pragma unroll
        for (int i = 0; i < 3; ++i) af[i][r] = p[i];
      }
#pragma unroll
      for (int i = 0; i < 3; ++i) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) mma(i ? lo[nt] : own[nt], af[i], va[nt], va[2 + nt]);
        if (i == 0) {
          // P_t times what the state gave, before the chunk's own small products join the sum
#pragma unroll
          for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float pt = P[(lane >> 2) + (e >> 1) * 8];
              hi[nt][e] *= pt;
              lo[nt][e] *= pt;
            }
        }
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int t = (lane >> 2) + r * 8, vc = wcol + nt * 8 + dc;
          if (t >= n || colb + vc >= vdim) continue;
          float x[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            x[e] = hi[nt][2 * r + e] + (own[nt][2 * r + e] + lo[nt][2 * r + e]);
            x[e] = fmaf(skip, __bfloat162float(v_r[t * VP + vc + e]), x[e]);
          }
          *reinterpret_cast<float2*>(a.out + (size_t)(c0 + t) * a.out_stride + (size_t)head * vdim + colb + vc) = make_float2(x[0], x[1]);
        }
      }
    }
    // the update's first operand: V^T times the last row of D, split
    uint32_t vp[3][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float2 w = *reinterpret_cast<const float2*>(D + (C - 1) * C + dc + (r >> 1) * 8);
      const __nv_bfloat162 v2 = *reinterpret_cast<const __nv_bfloat162*>(&va[r]);
      uint32_t p[3];
      split3(__low2float(v2) * w.x, __high2float(v2) * w.y, p);
#pragma unroll
      for (int i = 0; i < 3; ++i) vp[i][r] = p[i];
    }
    const float pc = P[C - 1];
    decays *= pc;
#pragma unroll
    for (int i = 0; i < DP / 16; ++i) {
      float u[2][4] = {};
      uint32_t kf[4];
      ldsm4_t(kf, k_r + hr * SP + i * 16 + hh);
#pragma unroll
      for (int p = 2; p >= 0; --p) {
        mma(u[0], vp[p], kf[0], kf[2]);
        mma(u[1], vp[p], kf[1], kf[3]);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) st[2 * i + j][e] = fmaf(st[2 * i + j][e], pc, u[j][e]);
    }
  }
  const bool rest = ch < chunks;                                       // a chunk that is not finite
  if (!STATE_ONLY && !last && !rest) return;
  float* S_out = STATE_ONLY || rest ? S_seg : a.state + (size_t)a.state_slots[entry] * a.slot_stride + (size_t)head * dim * vdim;
#pragma unroll
  for (int i = 0; i < DP / 8; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int dd = i * 8 + dc + (j & 1), vv = vr + (j >> 1) * 8;
      if (dd < dim && vv < vdim) S_out[(size_t)dd * vdim + vv] = st[i][j];
    }
  }
  if (rest) {
    __syncthreads();
    walk_rest<SCALAR, STATE_ONLY>(a, reinterpret_cast<float*>(smem), entry, t0 + ch * C, t1, last, colb, VT, decays);
    return;
  }
  if (STATE_ONLY && blockIdx.x == 0) {
    for (int d = tid; d < dim; d += NT) a.seg_decay[unit * dim + d] = decays;
  }
}

// ---- a decay per key channel -----------------------------------------------------------------------------------
template <int DP, int WARPS>
struct Shape {
  static constexpr int VT = WARPS * 16, VP = VT + 8, SP = DP + 8, NT = WARPS * 32;
  // bytes of one stage of inputs as they lie in global memory: z, q, k, v
  static constexpr int Z = C * DP * 4, QK = C * DP * 2, V = C * VP * 2, STAGE = Z + 2 * QK + V;
  static constexpr int F32 = C * DP * 4;                      // one of a, q, k in float32
  static constexpr int SPLIT = C * SP * 2;                    // one of the three parts of q P or k R
  static constexpr int BYTES = 2 * STAGE + 3 * F32 + 6 * SPLIT + 3 * C * AP * 2 + 2 * DP * 4;
};

template <int FORM, int DP, int WARPS, bool STATE_ONLY>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 8 ? 2 : DP == 128 ? 2 : 4)
diag_chunk_kernel(const __grid_constant__ Args a) {
  using Sh = Shape<DP, WARPS>;
  constexpr int NT = Sh::NT, VT = Sh::VT, VP = Sh::VP, SP = Sh::SP;
  constexpr bool HAS_K = FORM != GATE;
  extern __shared__ __align__(16) unsigned char smem[];
  float* a_s = reinterpret_cast<float*>(smem + 2 * Sh::STAGE);         // [C][DP]
  float* q_s = a_s + C * DP;
  float* k_s = q_s + C * DP;
  bf16* qp_s = reinterpret_cast<bf16*>(k_s + C * DP);                  // [3][C][SP]
  bf16* kr_s = qp_s + 3 * C * SP;
  bf16* A_s = kr_s + 3 * C * SP;                                       // [3][C][AP]
  float* p_s = reinterpret_cast<float*>(A_s + 3 * C * AP);             // [DP]
  float* u_s = p_s + DP;                                               // bonus form: u [DP]
  float* e_s = u_s + DP;                                               // and the exponents of the decays, a = exp(-e) [C][DP]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int head = blockIdx.y, qk_head = head / (a.heads / a.qk_heads);
  const int dim = a.dim, vdim = a.vdim, colb = blockIdx.x * VT;
  const int d = tid % DP;                                              // this thread's key channel outside the contractions
  static_assert(NT % DP == 0, "a thread keeps its channel");
  pdl_launch_dependents();
  const float zb = (d < dim && a.z_bias) ? a.z_bias[head * dim + d] : 0.f;
  const float low = (FORM == GATE && d < dim) ? a.bonus[head * dim + d] : 0.f;
  int entry = 0, t0 = 0, t1 = 0, end = 0;
  const bool there = segment_of(a.cu_tokens, a.n_entries, a.seg_len, blockIdx.z, entry, t0, t1, end);
  pdl_wait();
  if (!there) return;
  const bool last = t1 == end;
  if (STATE_ONLY && last) return;                                      // nothing follows an entry's last segment
  const size_t unit = (size_t)blockIdx.z * a.heads + head;
  float* S_seg = a.seg_state + unit * dim * vdim;

  if (FORM == BONUS && !STATE_ONLY && a.shift_state && last) {
    const bf16* src = a.shift_src + (size_t)(t1 - 1) * a.shift_stride;
    float* dst = a.shift_state + (size_t)a.state_slots[entry] * a.shift_slot_stride;
    for (int c = (head * gridDim.x + blockIdx.x) * NT + tid; c < a.shift_width; c += gridDim.x * a.heads * NT) dst[c] = __bfloat162float(src[c]);
  }

  auto bring = [&](int c0, int stage) {
    const int n = min(C, t1 - c0);
    unsigned char* base = smem + stage * Sh::STAGE;
    float* z_r = reinterpret_cast<float*>(base);
    bf16 *q_r = reinterpret_cast<bf16*>(base + Sh::Z), *k_r = q_r + C * DP, *v_r = k_r + C * DP;
    for (int i = tid; i < C * (DP / 4); i += NT) {
      const int c = i / (DP / 4), x = i % (DP / 4) * 4;
      if (c < n && x < dim) cp_async16(z_r + c * DP + x, a.z + (size_t)(c0 + c) * a.z_stride + (size_t)head * dim + x);
    }
    for (int i = tid; i < C * (DP / 8); i += NT) {
      const int c = i / (DP / 8), x = i % (DP / 8) * 8;
      if (c >= n || x >= dim) continue;
      const size_t at = (size_t)(c0 + c) * a.qk_stride + (size_t)qk_head * dim + x;
      if (!STATE_ONLY) cp_async16(q_r + c * DP + x, a.q + at);
      if (HAS_K) cp_async16(k_r + c * DP + x, a.k + at);
    }
    for (int i = tid; i < C * (VT / 8); i += NT) {
      const int c = i / (VT / 8), x = i % (VT / 8) * 8;
      bf16* dst = v_r + c * VP + x;
      if (c < n && colb + x < vdim) cp_async16(dst, a.v + (size_t)(c0 + c) * a.v_stride + (size_t)head * vdim + colb + x);
      else *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
    }
  };
  bring(t0, 0);
  if (FORM == BONUS && tid < DP) u_s[tid] = tid < dim ? a.bonus[head * dim + tid] : 0.f;

  // S^T: rows = value columns wcol + lane / 4 (+ 8), columns = channels 8 i + 2 (lane % 4) (+ 1)
  const int wcol = warp * 16, vr = colb + wcol + (lane >> 2), dc = 2 * (lane & 3);
  float st[DP / 8][4];
#pragma unroll
  for (int i = 0; i < DP / 8; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int dd = i * 8 + dc + (j & 1), vv = vr + (j >> 1) * 8;
      st[i][j] = (!STATE_ONLY && dd < dim && vv < vdim) ? S_seg[(size_t)dd * vdim + vv] : 0.f;
    }
  }
  float decays = FORM == BONUS ? 0.f : 1.f;                            // pass 1: the segment's product (bonus: exponent), channel d
  static_assert(C * VT / 8 == NT, "a thread looks at what it brought itself: one piece of the values");
  int stage = 0, c0 = t0;
  for (; c0 < t1; c0 += C, stage ^= 1) {
    const int n = min(C, t1 - c0);
    const unsigned char* base = smem + stage * Sh::STAGE;
    const float* z_r = reinterpret_cast<const float*>(base);
    const bf16 *q_r = reinterpret_cast<const bf16*>(base + Sh::Z), *k_r = q_r + C * DP, *v_r = k_r + C * DP;
    cp_async_wait_all();
    // behind the barrier this chunk is here and the last one's operands are read
    if (__syncthreads_or(not_finite8(v_r + tid / (VT / 8) * VP + tid % (VT / 8) * 8))) break;
    if (c0 + C < t1) bring(c0 + C, stage ^ 1);
    // decays, queries and keys in float32; tokens behind the end and channels behind dim: a = 1, q = k = 0
#pragma unroll 4
    for (int c = tid / DP; c < C; c += NT / DP) {
      float av = 1.f, qv = 0.f, kv = 0.f, ev = 0.f;
      if (c < n && d < dim) {
        if (!STATE_ONLY) qv = __bfloat162float(q_r[c * DP + d]);
        if (HAS_K) kv = __bfloat162float(k_r[c * DP + d]);
        if (FORM == BONUS) {
          ev = expf(z_r[c * DP + d] + zb);
          av = expf(-ev);
        } else if (FORM == POWER) {
          av = expf(log_sigmoid_f(z_r[c * DP + d] + zb) * a.inv_tau);
        } else {
          if (!STATE_ONLY) qv = qv / (1.f + expf(-qv));
          av = low + (1.f - low) / (1.f + expf(-(z_r[c * DP + d] + zb)));
          kv = 1.f - av;
        }
      }
      a_s[c * DP + d] = av;
      if (FORM == BONUS) e_s[c * DP + d] = ev;
      if (!STATE_ONLY) q_s[c * DP + d] = qv;
      k_s[c * DP + d] = kv;
    }
    __syncthreads();
    if (!STATE_ONLY) {
      // A: sixteen lanes per s, DP / 16 channels a lane, NS numbers s a lane (they share the loads of a and q); a lane ends with the
      // sum of t = its number
      constexpr int G = DP / 64, NS = C * 16 / NT;
      const int g = tid & 15;
      float kk[NS][G][4], w[NS][G][4], acc[NS][C];
#pragma unroll
      for (int m = 0; m < NS; ++m) {
#pragma unroll
        for (int i = 0; i < G; ++i) {
          Vec4<float>::load(k_s + ((tid >> 4) + m * (NT / 16)) * DP + i * 64 + g * 4, kk[m][i]);
#pragma unroll
          for (int e = 0; e < 4; ++e) w[m][i][e] = 0.f;
        }
      }
#pragma unroll
      for (int t = 0; t < C; ++t) {
#pragma unroll
        for (int m = 0; m < NS; ++m) acc[m][t] = 0.f;
        if (t < 2 * warp) continue;                                    // before this warp's first s
#pragma unroll
        for (int i = 0; i < G; ++i) {
          float at[4], qt[4];
          Vec4<float>::load(a_s + t * DP + i * 64 + g * 4, at);
          Vec4<float>::load(q_s + t * DP + i * 64 + g * 4, qt);
#pragma unroll
          for (int m = 0; m < NS; ++m) {
            const bool own = t == (tid >> 4) + m * (NT / 16);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              if (FORM == BONUS) {
                acc[m][t] = fmaf(qt[e], own ? u_s[i * 64 + g * 4 + e] * kk[m][i][e] : w[m][i][e], acc[m][t]);
                w[m][i][e] = own ? kk[m][i][e] : w[m][i][e] * at[e];
              } else {
                w[m][i][e] = own ? kk[m][i][e] : w[m][i][e] * at[e];
                acc[m][t] = fmaf(qt[e], w[m][i][e], acc[m][t]);
              }
            }
          }
        }
      }
#pragma unroll
      for (int m = 0; m < NS; ++m) {
        const int s = (tid >> 4) + m * (NT / 16);
#pragma unroll
        for (int t = 0; t < C; ++t) acc[m][t] = t >= s ? acc[m][t] : 0.f;
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) {
#pragma unroll
          for (int i = 0; i < off; ++i) {
            const bool up = g & off;
            const float send = up ? acc[m][i] : acc[m][i + off], keep = up ? acc[m][i + off] : acc[m][i];
            acc[m][i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
          }
        }
        uint32_t p[3];
        split3(acc[m][0], 0.f, p);
#pragma unroll
        for (int i = 0; i < 3; ++i) *reinterpret_cast<unsigned short*>(A_s + (i * C + g) * AP + s) = (unsigned short)(p[i] & 0xffffu);
      }
    }
    // q P (forward) and k R (backward), split.  A product is kept from what it lacks to one while that is less than a half: with
    // decays close to one the plain product's roundings were most of the state's error (gate form, 2,048 tokens, against 64 bits:
    // plain 5.2e-7, token by token 3.2e-7, this way 2.8e-7).  The bonus form has the decays' exponents at hand and sums those: a product
    // is rounded once then, however many tokens it spans (32 heads of 64 x 64: token by token 8.4e-8, products 8.7e-8, this way 6.8e-8; 93
    // us for the three launches with products, 103 this way).
    for (int task = tid; task < (STATE_ONLY ? DP : 2 * DP); task += NT) {
      float f = 1.f, lack = 0.f;
      auto on = [&](int t) {                                           // f <- f a_t
        if (FORM == BONUS) {
          lack += e_s[t * DP + d];
          f = expf(-lack);
          return;
        }
        const float av = a_s[t * DP + d];
        lack = fmaf(1.f - av, f, lack);
        f = lack < 0.5f ? 1.f - lack : f * av;
      };
      if (!STATE_ONLY && task < DP) {
#pragma unroll
        for (int t = 0; t < C; t += 2) {
          float x[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (FORM != BONUS) on(t + i);
            x[i] = q_s[(t + i) * DP + d] * f;
            if (FORM == BONUS) on(t + i);
          }
          uint32_t p[3];
          split3(x[0], x[1], p);
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            *reinterpret_cast<unsigned short*>(qp_s + (i * C + t) * SP + d) = (unsigned short)(p[i] & 0xffffu);
            *reinterpret_cast<unsigned short*>(qp_s + (i * C + t + 1) * SP + d) = (unsigned short)(p[i] >> 16);
          }
        }
      } else {
#pragma unroll
        for (int t = C - 2; t >= 0; t -= 2) {
          float x[2];
#pragma unroll
          for (int i = 1; i >= 0; --i) {
            x[i] = k_s[(t + i) * DP + d] * f;
            on(t + i);
          }
          uint32_t p[3];
          split3(x[0], x[1], p);
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            *reinterpret_cast<unsigned short*>(kr_s + (i * C + t) * SP + d) = (unsigned short)(p[i] & 0xffffu);
            *reinterpret_cast<unsigned short*>(kr_s + (i * C + t + 1) * SP + d) = (unsigned short)(p[i] >> 16);
          }
        }
        p_s[d] = f;
        if (STATE_ONLY) decays = FORM == BONUS ? decays + lack : decays * f;
      }
    }
    __syncthreads();
    // v of the chunk: rows s, columns of this warp; the same registers are V^T as the update's first operand and V as the
    // read-out's second
    uint32_t va[4];
    ldsm4_t(va, v_r + ((lane >> 4) * 8 + (lane & 7)) * VP + wcol + ((lane >> 3) & 1) * 8);
    const int row16 = (lane & 7) + ((lane >> 3) & 1) * 8, half = (lane >> 4) * 8;      // ldmatrix rows of a first operand
    if (!STATE_ONLY) {
      float hi[2][4] = {}, lo[2][4] = {};
#pragma unroll
      for (int ks = 0; ks < DP / 16; ++ks) {
        uint32_t qf[3][4];
#pragma unroll
        for (int i = 0; i < 3; ++i) ldsm4(qf[i], qp_s + (i * C + row16) * SP + ks * 16 + half);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          uint32_t b0[3], b1[3];
          split3(st[2 * ks][2 * nt], st[2 * ks][2 * nt + 1], b0);
          split3(st[2 * ks + 1][2 * nt], st[2 * ks + 1][2 * nt + 1], b1);
          add_mma(hi[nt], qf[0], b0[0], b1[0]);
          mma(lo[nt], qf[0], b0[1], b1[1]);
          mma(lo[nt], qf[1], b0[0], b1[0]);
          mma(lo[nt], qf[0], b0[2], b1[2]);
          mma(lo[nt], qf[2], b0[0], b1[0]);
          mma(lo[nt], qf[1], b0[1], b1[1]);
        }
      }
      float own[2][4] = {};
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        uint32_t af[4];
        ldsm4(af, A_s + (i * C + row16) * AP + half);
        mma(i == 0 ? own[0] : lo[0], af, va[0], va[2]);
        mma(i == 0 ? own[1] : lo[1], af, va[1], va[3]);
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int t = (lane >> 2) + r * 8, vc = wcol + nt * 8 + dc;
          if (t >= n || colb + vc >= vdim) continue;
          float x[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            x[e] = hi[nt][2 * r + e] + (own[nt][2 * r + e] + lo[nt][2 * r + e]);
            if (FORM == POWER) x[e] *= a.q_scale;
          }
          *reinterpret_cast<float2*>(a.out + (size_t)(c0 + t) * a.out_stride + (size_t)head * vdim + colb + vc) = make_float2(x[0], x[1]);
        }
      }
    }
    // S^T <- S^T diag(P_C) + V^T (k R): the product in accumulators of its own, the decay and the sum in float32 multiply-adds
#pragma unroll
    for (int i = 0; i < DP / 16; ++i) {
      float u[2][4] = {};
#pragma unroll
      for (int p = 2; p >= 0; --p) {
        uint32_t kf[4];
        ldsm4_t(kf, kr_s + (p * C + (lane >> 4) * 8 + (lane & 7)) * SP + i * 16 + ((lane >> 3) & 1) * 8);
        mma(u[0], va, kf[0], kf[2]);
        mma(u[1], va, kf[1], kf[3]);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float2 pc = *reinterpret_cast<const float2*>(p_s + i * 16 + j * 8 + dc);
        float(&s)[4] = st[2 * i + j];
        s[0] = fmaf(s[0], pc.x, u[j][0]); s[1] = fmaf(s[1], pc.y, u[j][1]);
        s[2] = fmaf(s[2], pc.x, u[j][2]); s[3] = fmaf(s[3], pc.y, u[j][3]);
      }
    }
  }
  if (FORM == BONUS) decays = expf(-decays);
  const bool rest = c0 < t1;                                           // a chunk that is not finite
  if (!STATE_ONLY && !last && !rest) return;
  float* S_out = STATE_ONLY || rest ? S_seg : a.state + (size_t)a.state_slots[entry] * a.slot_stride + (size_t)head * dim * vdim;
#pragma unroll
  for (int i = 0; i < DP / 8; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int dd = i * 8 + dc + (j & 1), vv = vr + (j >> 1) * 8;
      if (dd < dim && vv < vdim) S_out[(size_t)dd * vdim + vv] = st[i][j];
    }
  }
  if (rest) {
    __syncthreads();
    walk_rest<FORM, STATE_ONLY>(a, a_s, entry, c0, t1, last, colb, VT, decays);
    return;
  }
  if (STATE_ONLY && blockIdx.x == 0 && tid < dim) a.seg_decay[unit * dim + d] = decays;
}

// Every segment's true start state from the end states from zero: start_(s+1) = diag(P_s) start_s + E_s, start_0 the request's
// state.  Four elements a thread, four segments' loads in flight.
__global__ void __launch_bounds__(128)
diag_chain_kernel(const Args a) {
  pdl_launch_dependents();
  const size_t per = (size_t)a.heads * a.dim * a.vdim, el = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  const int entry = blockIdx.y, rows = a.heads * a.dim;
  const size_t row = el / a.vdim;
  size_t seg0 = 0;
  int b = a.cu_tokens[0];
  for (int e = 0; e < entry; ++e) {
    const int n = a.cu_tokens[e + 1];
    seg0 += (n - b + a.seg_len - 1) / a.seg_len;
    b = n;
  }
  const int segs = (a.cu_tokens[entry + 1] - b + a.seg_len - 1) / a.seg_len;
  const float* S_slot = a.state + (size_t)a.state_slots[entry] * a.slot_stride;
  pdl_wait();
  if (el >= per) return;
  float4 S = *reinterpret_cast<const float4*>(S_slot + el);
  for (int s0 = 0; s0 < segs; s0 += 4) {
    float4 E[4];
    float P[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (s0 + i + 1 < segs) {
        E[i] = *reinterpret_cast<const float4*>(a.seg_state + (seg0 + s0 + i) * per + el);
        P[i] = a.seg_decay[(seg0 + s0 + i) * rows + row];
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (s0 + i >= segs) break;
      *reinterpret_cast<float4*>(a.seg_state + (seg0 + s0 + i) * per + el) = S;
      if (s0 + i + 1 < segs) {
        S.x = fmaf(P[i], S.x, E[i].x); S.y = fmaf(P[i], S.y, E[i].y); S.z = fmaf(P[i], S.z, E[i].z); S.w = fmaf(P[i], S.w, E[i].w);
      }
    }
  }
}

// The two passes with the chain between them.
template <typename Kernel>
int launch_passes(Kernel ends, Kernel outs, const Args& a, int vt, int threads, size_t smem, int segs, cudaStream_t stream) {
  cudaFuncSetAttribute(ends, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaFuncSetAttribute(outs, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const dim3 grid((a.vdim + vt - 1) / vt, a.heads, segs), block(threads);
  launch_kernel(ends, grid, block, smem, stream, a);
  const size_t per = (size_t)a.heads * a.dim * a.vdim;
  launch_kernel(diag_chain_kernel, dim3((unsigned)((per / 4 + 127) / 128), a.n_entries), dim3(128), (size_t)0, stream, a);
  launch_kernel(outs, grid, block, smem, stream, a);
  LLMK_LAUNCH_CHECK("diag_chunk");
}

template <int FORM, int DP, int WARPS>
int launch_shape(const Args& a, int segs, cudaStream_t stream) {
  using Sh = Shape<DP, WARPS>;
  return launch_passes(diag_chunk_kernel<FORM, DP, WARPS, true>, diag_chunk_kernel<FORM, DP, WARPS, false>, a, Sh::VT, Sh::NT,
                       Sh::BYTES + (FORM == BONUS ? Sh::F32 : 0), segs, stream);
}

template <int DP>
int launch_scalar(const Args& a, int segs, cudaStream_t stream) {
  using Sh = ScalarShape<DP>;
  const size_t smem = 2 * Sh::STAGE + ((size_t)2 * (a.seg_len + C) + (size_t)(a.seg_len + C) * C) * sizeof(float);
  return launch_passes(scalar_chunk_kernel<DP, true>, scalar_chunk_kernel<DP, false>, a, Sh::VT, Sh::NT, smem, segs, stream);
}

template <int FORM>
int launch_form(const Args& a, int segs, cudaStream_t stream) {
  if (a.dim <= 64) return a.vdim <= 64 ? launch_shape<FORM, 64, 4>(a, segs, stream) : launch_shape<FORM, 64, 8>(a, segs, stream);
  return a.vdim <= 64 ? launch_shape<FORM, 128, 4>(a, segs, stream) : launch_shape<FORM, 128, 8>(a, segs, stream);
}

}  // namespace

bool takes(const Args& a, int seg_len) {
  auto on16 = [](const void* p) { return (uintptr_t)p % 16 == 0; };
  return seg_len > 0 && seg_len <= MAX_SEG && a.dim % 8 == 0 && a.dim <= 128 && a.vdim % 8 == 0 && a.qk_stride % 8 == 0 && a.v_stride % 8 == 0 && a.z_stride % 4 == 0 &&
         a.out_stride % 2 == 0 && a.slot_stride % 4 == 0 && on16(a.q) && on16(a.k) && on16(a.v) && on16(a.z) && on16(a.state) &&
         on16(a.seg_state) && (uintptr_t)a.out % 8 == 0;
}

int launch(Args a, int form, int n_tokens, int seg_len, cudaStream_t stream) {
  // Longer segments than asked for, while the step's CTAs are four fifths of those that the GPU holds at once: less of the state to leave
  // and to chain (2,048 tokens, 8 heads of 128 x 256: segments of 64 146 us for the three launches, of 128 134, of 256 180).
  const bool narrow = a.vdim <= 64 || form == SCALAR;
  const int vt = narrow ? 64 : 128, resident = (narrow && (a.dim <= 64 || form == SCALAR) ? 4 : 2) * llmk_sm_count();
  const long long units = (long long)a.heads * ((a.vdim + vt - 1) / vt);
  while (seg_len * 2 <= MAX_SEG && units * (n_tokens / (seg_len * 2)) * 5 >= 4 * resident) seg_len *= 2;
  a.seg_len = seg_len;
  const int segs = n_tokens / seg_len + a.n_entries;
  LLMK_REQUIRE(segs <= 65535 && a.heads <= 65535, "diag_chunk: too many segments or heads for one launch");
  switch (form) {
    case BONUS: return launch_form<BONUS>(a, segs, stream);
    case SCALAR: return a.dim <= 64 ? launch_scalar<64>(a, segs, stream) : launch_scalar<128>(a, segs, stream);
    case GATE: return launch_form<GATE>(a, segs, stream);
    default: return launch_form<POWER>(a, segs, stream);
  }
}

}  // namespace diag_chunk
