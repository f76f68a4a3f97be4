// Token scans of the gated delta rule with a decay per head (Qwen3-Next) and of the Mamba-2 state-space recurrence, sixteen
// tokens at a time on the tensor cores, in fp32 accuracy. Per head, with a [DK, DV] state S in fp32,
//
//   delta rule:  S <- e^{g_t} S ;  r_t = beta_t (v_t - S^T k_t) ;  S <- S + k_t r_t^T ;  o_t = scale S^T q_t
//   state space: S <- e^{dt_t A} S + B_t (dt_t x_t)^T ;                                  y_t = S^T C_t + D x_t
//
// and for a chunk of sixteen tokens behind a state S_0 (decays are exponentials of sums over (i, j], never of differences):
//
//   y_j = k_j . S_0 ;  r = T (beta v - eb y),  T = (1 + M)^-1,  M_ji = beta_j e^{g_{i+1} + .. + g_j} k_j . k_i   (i < j)
//   o_j = es_j q_j . S_0 + sum_{i<=j} P_ji r_i,                 P_ji = scale e^{g_{i+1} + .. + g_j} q_j . k_i
//   S_16 = e^{g_1 + .. + g_16} S_0 + sum_i e^{g_{i+1} + .. + g_16} k_i r_i^T
//
// (state space: r_i = x_i, without y and T; dt_i and D are folded into P and the tails).
//
// Accuracy. k, q, B, C, x and v are bf16, so they are exact operands. An fp32 operand enters as three bf16 parts that add up
// to its 24 bits; products of two such operands take the six pairs of parts that reach 2^-24. Leading parts have accumulators
// of their own, and the update of the state is summed from zero and then added in fp32, so the state is rounded once per chunk
// instead of once per token.
//
//   * chunk_coef: a warp per (chunk, head) forms the 16 x 16 products (mma.sync on the rows as they lie), the decays, T by
//     forward substitution, and stores the parts of T and P in the order the scan's lanes read them.
//   * chunk_scan: the columns of a state never meet. A warp owns 16 of them: S^T lies in the accumulator layout, which is also
//     the layout of a left operand, so the state never leaves its registers; warps need no exchange. Rows, values and
//     coefficients come by cp.async, two chunks ahead. What bounds it is the rate of the products: 168 of 16 x 8 x 16 per warp
//     and chunk for the delta rule with DK = 128, 102 for the state space, at about 20 clocks each (delta rule below, at most
//     one warp per scheduler: 0.60 ms) and 23 per scheduler (second pass over the segments of the state space below: 0.20 ms),
//     and with one warp per scheduler the chain y -> T -> P behind them.
//
// 5328 + 2864 tokens, 32 heads of 128 x 128: 0.64 ms (eight tokens at a time on the FMA pipe 1.90 ms, one at a time 19.4 ms);
// 6000 tokens in three sequences, 64 state-space heads of 64 x 128: 0.32 ms (0.74 ms, 4.4 ms). Bytes at the copy rate: 43 and
// 18 us. State-space sequences are cut into segments where that fills the GPU (cs_span): 8192 tokens of one sequence, 64 heads
// 0.93 -> 0.38 ms, 8 heads 0.91 -> 0.09 ms. A value that is not finite reaches its column from its token on only, as in
// a walk token by token: a chunk that holds one is summed on the FMA pipe (cs_triangle).
// Compiled without fast-math.
#include "common.cuh"

namespace edl {
namespace {

constexpr int CS_C = 16;                  // tokens per chunk
constexpr int CS_WARPS = 4;
constexpr int CS_THREADS = CS_WARPS * 32;
constexpr int CS_CT = CS_WARPS * 16;      // columns of a CTA
constexpr int CS_STAGES = 3;

enum CsMode { CS_DELTA = 0, CS_SSD = 1 };

// Record of a (chunk, head), in bytes: parts of P [3][32 lanes][16] | es 16 | tail 16 | total, pad (floats), and for the delta
// rule parts of T | beta 16 | eb 16.
constexpr int CS_P = 0, CS_ES = 1536, CS_TAIL = CS_ES + 64, CS_TOTAL = CS_TAIL + 64, CS_T = CS_TOTAL + 16,
              CS_BETA = CS_T + 1536, CS_EB = CS_BETA + 64;
template <int MODE>
constexpr int cs_rec_bytes() { return MODE == CS_SSD ? CS_T : CS_EB + 64; }

struct CsParams {
  const __nv_bfloat16 *q, *k, *v;    // [T, G, DK] x 2, [T, H, DV]
  const float* g;                    // delta: [T, H] log decays, or null
  const __nv_bfloat16* beta;         // delta: [T, H] or null
  const __nv_bfloat16* dt;           // state space: [T, H]
  const float *A, *Dskip, *dt_bias;  // [H]
  int softplus;
  const int* cu;
  int T, B, H, G, DV;
  float scale;
  uint8_t* rec;                      // [slots, H, record]
  float* state;                      // delta [B, H, DK, DV], state space [B, H, DV, DK]; or null
  __nv_bfloat16* o;                  // [T, H, DV]
  bool vec_v;                        // values can be fetched 16 bytes at a time
  int w0, w1;                        // the window of tokens this launch takes
  const float* carry_in;             // without `state`: what the sequence cut by the window's start left in front of it, and
  float* carry_out;                  // where the one cut by its end leaves its own, [H, state]
  int seg;                           // tokens of a segment (a multiple of 16), or 0: sequences are walked from end to end
  float *seg_state, *seg_decay;      // [segments, H, DV, DK], [segments, H]
};

// Segments of long state-space sequences run side by side: the state behind one is its decay times the state in front of it
// plus what its tokens leave in an empty state. A first pass computes the latter (48 of the 102 products of a chunk), one
// thread per element carries states from segment to segment, then every segment runs in full from the state in front of it.
// A segment's place, as a chunk's: unique and increasing, below T / seg + B + 1.
// Long inputs go in windows of tokens, so that the records of one fit a workspace of bounded size: a window's part of every
// sequence is a sequence of its own whose state comes from the one before.
__device__ __forceinline__ int cs_pos(const CsParams& p, int b) { return min(max(p.cu[b], p.w0), p.w1); }

struct CsSpan {
  int b, t0, t1, slot;
};
__device__ __forceinline__ CsSpan cs_span(const CsParams& p, int z) {
  CsSpan s;
  s.slot = z;
  if (p.seg == 0) {
    s.b = z;
    s.t0 = cs_pos(p, z);
    s.t1 = cs_pos(p, z + 1);
    return s;
  }
  int lo = 0, hi = p.B;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if ((cs_pos(p, mid) - p.w0) / p.seg + mid <= z) lo = mid;
    else hi = mid;
  }
  s.b = lo;
  const long long first = cs_pos(p, lo), at = first + (long long)(z - (((int)first - p.w0) / p.seg + lo)) * p.seg;
  const int end = cs_pos(p, lo + 1);
  s.t0 = at < first || at >= end ? end : (int)at;
  s.t1 = min(end, (int)min((long long)end, s.t0 + (long long)p.seg));
  return s;
}

// A chunk's place in the record array: unique and increasing over (sequence, chunk), below (tokens of the window) / 16 + B + 1.
__device__ __forceinline__ int cs_slot(const CsParams& p, int t, int b) { return (t - p.w0) / CS_C + b; }

// States in front of and behind this window's part of sequence b, head h; null: zeros, nobody asks.
__device__ __forceinline__ const float* cs_state_in(const CsParams& p, int b, int h, long long size) {
  if (p.state) return p.state + ((long long)b * p.H + h) * size;
  return p.cu[b] < p.w0 ? p.carry_in + h * size : nullptr;
}
__device__ __forceinline__ float* cs_state_out(const CsParams& p, int b, int h, long long size) {
  if (p.state) return p.state + ((long long)b * p.H + h) * size;
  return p.cu[b + 1] > p.w1 ? p.carry_out + h * size : nullptr;
}

__device__ __forceinline__ float cs_softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }

__device__ __forceinline__ void cs_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cs_ldmatrix(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void cs_ldmatrix_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
// 16 bytes to shared memory, or zeros
__device__ __forceinline__ void cs_copy16(uint32_t dst, const void* src, bool on) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(on ? 16 : 0) : "memory");
}

// Two fp32 values as three bf16 pairs that add up to them (24 bits).
__device__ __forceinline__ void cs_split(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack_bf16x2(x, y);
  x -= __uint_as_float(hi << 16);
  y -= __uint_as_float(hi & 0xffff0000u);
  mid = pack_bf16x2(x, y);
  x -= __uint_as_float(mid << 16);
  y -= __uint_as_float(mid & 0xffff0000u);
  lo = pack_bf16x2(x, y);
}
// A 16 x 16 block in the accumulator layout (two column halves) as the parts of a left operand.
__device__ __forceinline__ void cs_split_block(const float (&c0)[4], const float (&c1)[4], uint32_t (&a)[3][4]) {
  cs_split(c0[0], c0[1], a[0][0], a[1][0], a[2][0]);
  cs_split(c0[2], c0[3], a[0][1], a[1][1], a[2][1]);
  cs_split(c1[0], c1[1], a[0][2], a[1][2], a[2][2]);
  cs_split(c1[2], c1[3], a[0][3], a[1][3], a[2][3]);
}

// Values that a product with zero does not take out: not finite, or so large that a bf16 part is not.
__device__ __forceinline__ bool cs_unsafe(const float (&r)[2][4]) {
  bool x = false;
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) x |= !(fabsf(r[j][e]) < 3.38e38f);
  return __any_sync(0xffffffffu, x);
}

// sum_{i <= j} W_ji r_i for the tokens j of this lane, token by token, so that what is not finite reaches no token before its
// own (the products multiply it with the zeros above W's diagonal). W as stored: parts in the order of a right operand; r: the
// first N parts of a left operand.
template <int N>
__device__ __forceinline__ void cs_triangle(const uint8_t* parts, const uint32_t (&a)[3][4], int lane, float (&out)[2][4]) {
  const int quad = lane & 3;
  float r[2][4];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      auto part = [&](int n) { const uint32_t w = a[n][2 * j + (e >> 1)]; return __uint_as_float(e & 1 ? w & 0xffff0000u : w << 16); };
      r[j][e] = part(0);
      if (N > 1 && isfinite(r[j][e])) r[j][e] += part(1) + part(2);
    }
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) out[j][e] = 0.f;
#pragma unroll 1
  for (int i = 0; i < CS_C; ++i) {
    const int from = (lane & 28) + ((i & 7) >> 1);
    float v[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float x = i & 1 ? r[0][2 * h + 1] : r[0][2 * h], y = i & 1 ? r[1][2 * h + 1] : r[1][2 * h];
      v[h] = __shfl_sync(0xffffffffu, i & 8 ? y : x, from);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int t = 2 * quad + e;
        const uint8_t* at = parts + (t * 4 + ((i & 7) >> 1)) * 16 + (2 * j + (i >> 3)) * 4 + (i & 1) * 2;
        float w = 0.f;
#pragma unroll
        for (int part = 2; part >= 0; --part) w += __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(at + part * 512));
        if (8 * j + t >= i) {
          out[j][e] = fmaf(w, v[0], out[j][e]);
          out[j][e + 2] = fmaf(w, v[1], out[j][e + 2]);
        }
      }
  }
}

// ---- coefficients -----------------------------------------------------------------------------------------------------
template <int MODE, int DK>
__global__ void __launch_bounds__(128) chunk_coef_kernel(const CsParams p, int heads_per_warp) {
  constexpr int REC = cs_rec_bytes<MODE>();
  __shared__ float s_m[4][16][17], s_p[4][16][17], s_g[4][16], s_a[4][16];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, row = lane >> 2, quad = lane & 3;
  const int h0 = (blockIdx.y * 4 + w) * heads_per_warp;
  if (h0 >= p.H) return;
  const int slot = blockIdx.x;
  int lo = 0, hi = p.B;                 // the last sequence whose first chunk is not past this slot
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (cs_slot(p, cs_pos(p, mid), mid) <= slot) lo = mid;
    else hi = mid;
  }
  const int first = cs_pos(p, lo), end = cs_pos(p, lo + 1);
  const int t0 = first + (slot - cs_slot(p, first, lo)) * CS_C;
  if (t0 < first || t0 >= end) return;
  const int n = min(CS_C, end - t0);
  const int rows = h0 / (p.H / p.G);
  // products: a lane takes 16-byte pieces of rows `row` and `row + 8`; which dimension a position of the reduction stands for
  // does not matter as long as both operands agree
  float qk[2][4], kk[2][4];
#pragma unroll
  for (int e = 0; e < 4; ++e) qk[0][e] = qk[1][e] = kk[0][e] = kk[1][e] = 0.f;
  auto piece = [&](const __nv_bfloat16* m, int t, int d) {
    return t < n && d < DK ? *reinterpret_cast<const uint4*>(m + ((long long)(t0 + t) * p.G + rows) * DK + d) : make_uint4(0u, 0u, 0u, 0u);
  };
#pragma unroll
  for (int d = 0; d < DK; d += 32) {
    const uint4 k0 = piece(p.k, row, d + 8 * quad), k1 = piece(p.k, row + 8, d + 8 * quad);
    const uint4 q0 = piece(p.q, row, d + 8 * quad), q1 = piece(p.q, row + 8, d + 8 * quad);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const uint32_t ka[4] = {half ? k0.z : k0.x, half ? k1.z : k1.x, half ? k0.w : k0.y, half ? k1.w : k1.y};
      const uint32_t qa[4] = {half ? q0.z : q0.x, half ? q1.z : q1.x, half ? q0.w : q0.y, half ? q1.w : q1.y};
      cs_mma(qk[0], qa, ka[0], ka[2]);
      cs_mma(qk[1], qa, ka[1], ka[3]);
      if (MODE == CS_DELTA) {
        cs_mma(kk[0], ka, ka[0], ka[2]);
        cs_mma(kk[1], ka, ka[1], ka[3]);
      }
    }
  }
  for (int h = h0; h < min(p.H, h0 + heads_per_warp); ++h) {
    float g = 0.f, a = 0.f;             // log decay; beta or dt
    if (lane < n) {
      const long long at = (long long)(t0 + lane) * p.H + h;
      if (MODE == CS_SSD) {
        a = __bfloat162float(p.dt[at]) + (p.dt_bias ? p.dt_bias[h] : 0.f);
        if (p.softplus) a = cs_softplus(a);
        g = a * p.A[h];
      } else {
        a = p.beta ? __bfloat162float(p.beta[at]) : 1.f;
        if (p.g) g = p.g[at];
      }
    }
    __syncwarp();
    if (lane < 16) {
      s_g[w][lane] = g;
      s_a[w][lane] = a;
    }
    __syncwarp();
    float before = 0.f, after = 0.f;
#pragma unroll
    for (int l = 0; l < 16; ++l) {
      const float x = s_g[w][l];
      if (l <= lane) before += x;
      else after += x;
    }
    uint8_t* dst = p.rec + ((long long)slot * p.H + h) * REC;
    if (lane <= 16) {                   // lane 16: the whole chunk
      const float e = expf(before);
      if (lane == 16) {
        *reinterpret_cast<float*>(dst + CS_TOTAL) = e;
      } else {
        reinterpret_cast<float*>(dst + CS_ES)[lane] = e * p.scale;
        reinterpret_cast<float*>(dst + CS_TAIL)[lane] = expf(after) * (MODE == CS_SSD ? a : 1.f);
        if (MODE == CS_DELTA) {
          reinterpret_cast<float*>(dst + CS_BETA)[lane] = a;
          reinterpret_cast<float*>(dst + CS_EB)[lane] = e * a;
        }
      }
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {      // rows j = row, row + 8
      const int j = row + 8 * half;
      float d[4] = {0.f, 0.f, 0.f, 0.f}, sum = 0.f;   // decays from columns 2 quad, 2 quad + 1, and eight further
#pragma unroll
      for (int l = 15; l >= 0; --l) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (l == 2 * quad + (e & 1) + 8 * (e >> 1)) d[e] = sum;
        if (l <= j) sum += s_g[w][l];
      }
      const float aj = s_a[w][j];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = 2 * quad + (e & 1) + 8 * (e >> 1);
        const float f = i <= j ? expf(d[e]) : 0.f;
        float pv = f * qk[e >> 1][2 * half + (e & 1)];
        if (MODE == CS_SSD) {
          pv *= s_a[w][i];
          if (i == j && p.Dskip) pv += p.Dskip[h];
        } else {
          pv *= p.scale;
          s_m[w][j][i] = i < j ? aj * f * kk[e >> 1][2 * half + (e & 1)] : 0.f;
        }
        s_p[w][j][i] = i <= j ? pv : 0.f;
      }
    }
    __syncwarp();
    float t[16];
    if (MODE == CS_DELTA) {             // lane c: column c of the inverse of 1 + M
#pragma unroll
      for (int j = 0; j < 16; ++j) t[j] = j == (lane & 15) ? 1.f : 0.f;
#pragma unroll
      for (int i = 0; i < 15; ++i)
#pragma unroll
        for (int j = i + 1; j < 16; ++j) t[j] = fmaf(-s_m[w][j][i], t[i], t[j]);
      __syncwarp();
      if (lane < 16)
#pragma unroll
        for (int j = 0; j < 16; ++j) s_m[w][j][lane] = t[j];
      __syncwarp();
    }
    // parts in the order of a right operand: for both halves of columns j, rows i = 2 quad, 2 quad + 1 and eight further
#pragma unroll
    for (int which = 0; which < (MODE == CS_DELTA ? 2 : 1); ++which) {
      uint32_t x[3][4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float* m = which ? &s_m[w][row + 8 * (e >> 1)][2 * quad + 8 * (e & 1)] : &s_p[w][row + 8 * (e >> 1)][2 * quad + 8 * (e & 1)];
        cs_split(m[0], m[1], x[0][e], x[1][e], x[2][e]);
      }
#pragma unroll
      for (int part = 0; part < 3; ++part)
        *reinterpret_cast<uint4*>(dst + (which ? CS_T : CS_P) + part * 512 + lane * 16) =
            make_uint4(x[part][0], x[part][1], x[part][2], x[part][3]);
    }
  }
}

// ---- scan -------------------------------------------------------------------------------------------------------------
template <int MODE, int DK>
struct CsCfg {
  static constexpr int PITCH = DK * 2 + 16;              // bytes of a row of k or q
  static constexpr int VPITCH = CS_CT * 2 + 16;
  static constexpr int REC = cs_rec_bytes<MODE>();
  static constexpr int OFF_Q = CS_C * PITCH, OFF_V = 2 * CS_C * PITCH, OFF_R = OFF_V + CS_C * VPITCH;
  static constexpr int STAGE = OFF_R + REC;
  static_assert(STAGE % 16 == 0 && CS_STAGES * STAGE <= 48 * 1024, "");
};

// LOCAL: only the state that a segment's tokens leave in an empty one, and its decay.
template <int MODE, int DK, bool LOCAL>
__global__ void __launch_bounds__(CS_THREADS) chunk_scan_kernel(const CsParams p) {
  using C = CsCfg<MODE, DK>;
  constexpr int NT = DK / 8, NK = DK / 16;
  __shared__ __align__(128) uint8_t smem[CS_STAGES * C::STAGE];
  const uint32_t base = smem_u32(smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, row = lane >> 2, quad = lane & 3;
  const CsSpan span = cs_span(p, blockIdx.z);
  const int h = blockIdx.y, b = span.b, t0 = span.t0, t1 = span.t1;
  if (t0 >= t1) return;
  const int H = p.H, DV = p.DV, rows = h / (p.H / p.G);
  const int cta_col = blockIdx.x * CS_CT, col = cta_col + warp * 16 + row;    // this lane's columns: col, col + 8

  auto fetch = [&](int tb, int st) {
    const int n = min(CS_C, t1 - tb);
    const uint32_t dst = base + st * C::STAGE;
    for (int i = tid; i < (LOCAL ? 1 : 2) * CS_C * (DK / 8); i += CS_THREADS) {
      const int which = i / (CS_C * (DK / 8)), t = (i / (DK / 8)) % CS_C, c = i % (DK / 8);
      const __nv_bfloat16* src = (which ? p.q : p.k) + ((long long)(tb + (t < n ? t : 0)) * p.G + rows) * DK + c * 8;
      cs_copy16(dst + which * C::OFF_Q + t * C::PITCH + c * 16, src, t < n);
    }
    if (p.vec_v) {
      for (int i = tid; i < CS_C * (CS_CT / 8); i += CS_THREADS) {
        const int t = i / (CS_CT / 8), c = i % (CS_CT / 8);
        const bool on = t < n && cta_col + c * 8 < DV;
        const __nv_bfloat16* src = p.v + ((long long)(tb + (on ? t : 0)) * H + h) * DV + (on ? cta_col + c * 8 : 0);
        cs_copy16(dst + C::OFF_V + t * C::VPITCH + c * 16, src, on);
      }
    } else {
      for (int i = tid; i < CS_C * CS_CT; i += CS_THREADS) {
        const int t = i / CS_CT, c = i % CS_CT;
        const bool on = t < n && cta_col + c < DV;
        *reinterpret_cast<__nv_bfloat16*>(smem + st * C::STAGE + C::OFF_V + t * C::VPITCH + c * 2) =
            on ? p.v[((long long)(tb + t) * H + h) * DV + cta_col + c] : __float2bfloat16(0.f);
      }
    }
    const uint8_t* rec = p.rec + ((long long)cs_slot(p, tb, b) * H + h) * C::REC;
    for (int i = tid; i < C::REC / 16; i += CS_THREADS) cs_copy16(dst + C::OFF_R + i * 16, rec + i * 16, true);
  };
  auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };

  fetch(t0, 0);
  commit();
  if (t0 + CS_C < t1) fetch(t0 + CS_C, 1);
  commit();

  // S^T in the accumulator layout: S[nt][e] is row 8 nt + 2 quad + (e & 1) of the state, column col + 8 (e >> 1)
  float S[NT][4];
  float* const at_seg = p.seg ? p.seg_state + ((long long)span.slot * H + h) * DK * DV : nullptr;
  const float* pool = p.seg ? at_seg : cs_state_in(p, b, h, (long long)DK * DV);
  float decay = 1.f;
  const long long row_step = MODE == CS_SSD ? 1 : DV, col_step = MODE == CS_SSD ? DK : 1;
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int c = col + 8 * (e >> 1);
      S[i][e] = !LOCAL && pool && c < DV ? pool[(8 * i + 2 * quad + (e & 1)) * row_step + c * col_step] : 0.f;
    }

  int st = 0;
  for (int tb = t0; tb < t1; tb += CS_C) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();                    // this chunk has landed, and every warp has left the stage that is filled next
    if (tb + 2 * CS_C < t1) fetch(tb + 2 * CS_C, st == 0 ? 2 : st - 1);
    commit();
    const uint32_t stage = base + st * C::STAGE;
    const uint8_t* rec = smem + st * C::STAGE + C::OFF_R;
    // ---- products with the state: leading parts, and the others
    float yq[2][2][4], yk[2][2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) yq[i][j][e] = yk[i][j][e] = 0.f;
    const uint32_t lrow = (lane & 7) + ((lane >> 4) << 3), lchunk = (lane >> 3) & 1;
#pragma unroll
    for (int ks = 0; ks < (LOCAL ? 0 : NK); ++ks) {
      uint32_t a[3][4], f[4];
      cs_split_block(S[2 * ks], S[2 * ks + 1], a);
      if (MODE == CS_DELTA) {
        cs_ldmatrix(stage + lrow * C::PITCH + (ks * 2 + lchunk) * 16, f);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          cs_mma(yk[0][j], a[0], f[2 * j], f[2 * j + 1]);
          cs_mma(yk[1][j], a[1], f[2 * j], f[2 * j + 1]);
          cs_mma(yk[1][j], a[2], f[2 * j], f[2 * j + 1]);
        }
      }
      cs_ldmatrix(stage + C::OFF_Q + lrow * C::PITCH + (ks * 2 + lchunk) * 16, f);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        cs_mma(yq[0][j], a[0], f[2 * j], f[2 * j + 1]);
        cs_mma(yq[1][j], a[1], f[2 * j], f[2 * j + 1]);
        cs_mma(yq[1][j], a[2], f[2 * j], f[2 * j + 1]);
      }
    }
    // ---- values of this warp's columns, transposed: tokens 8 j + 2 quad + (e & 1), column col + 8 (e >> 1)
    uint32_t vf[4];
    cs_ldmatrix_trans(stage + C::OFF_V + lrow * C::VPITCH + (warp * 2 + lchunk) * 16, vf);
    float r[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float2 x = unpack_bf16x2(vf[2 * j]), y = unpack_bf16x2(vf[2 * j + 1]);
      r[j][0] = x.x; r[j][1] = x.y; r[j][2] = y.x; r[j][3] = y.y;
    }
    uint32_t ra[3][4];
    if (MODE == CS_DELTA) {
      const float *beta = reinterpret_cast<const float*>(rec + CS_BETA), *eb = reinterpret_cast<const float*>(rec + CS_EB);
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int t = 8 * j + 2 * quad + (e & 1);
          r[j][e] = beta[t] * r[j][e] - eb[t] * (yk[0][j][e] + yk[1][j][e]);
        }
      cs_split_block(r[0], r[1], ra);
      const bool unsafe = cs_unsafe(r);
      uint4 tp[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) tp[i] = *reinterpret_cast<const uint4*>(rec + CS_T + i * 512 + lane * 16);
      float lead[2][4], rest[2][4];
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) lead[j][e] = rest[j][e] = 0.f;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
#define EDL_B(part) (j ? tp[part].z : tp[part].x), (j ? tp[part].w : tp[part].y)
        cs_mma(rest[j], ra[2], EDL_B(0));
        cs_mma(rest[j], ra[0], EDL_B(2));
        cs_mma(rest[j], ra[1], EDL_B(1));
        cs_mma(rest[j], ra[1], EDL_B(0));
        cs_mma(rest[j], ra[0], EDL_B(1));
        cs_mma(lead[j], ra[0], EDL_B(0));
#pragma unroll
        for (int e = 0; e < 4; ++e) r[j][e] = lead[j][e] + rest[j][e];
      }
      if (unsafe) cs_triangle<3>(rec + CS_T, ra, lane, r);
      cs_split_block(r[0], r[1], ra);
    } else {                            // the inputs are exact in one part
#pragma unroll
      for (int i = 0; i < 4; ++i) ra[0][i] = vf[i];
    }
    const bool unsafe = !LOCAL && cs_unsafe(r);
    // ---- the state behind the chunk
    {
      const float* tail = reinterpret_cast<const float*>(rec + CS_TAIL);
      const float total = *reinterpret_cast<const float*>(rec + CS_TOTAL);
      if (LOCAL) decay *= total;
      float rs[2][4];
      uint32_t sa[3][4];
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) rs[j][e] = r[j][e] * tail[8 * j + 2 * quad + (e & 1)];
      cs_split_block(rs[0], rs[1], sa);
      const uint32_t trow = lane & 15, tchunk = lane >> 4;
#pragma unroll
      for (int i = 0; i < NK; ++i) {
        uint32_t f[4];
        cs_ldmatrix_trans(stage + trow * C::PITCH + (i * 2 + tchunk) * 16, f);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float d[4] = {0.f, 0.f, 0.f, 0.f};
          cs_mma(d, sa[2], f[2 * j], f[2 * j + 1]);
          cs_mma(d, sa[1], f[2 * j], f[2 * j + 1]);
          cs_mma(d, sa[0], f[2 * j], f[2 * j + 1]);
#pragma unroll
          for (int e = 0; e < 4; ++e) S[2 * i + j][e] = fmaf(total, S[2 * i + j][e], d[e]);
        }
      }
    }
    // ---- outputs
    if constexpr (!LOCAL) {
      const float* es = reinterpret_cast<const float*>(rec + CS_ES);
      uint4 tp[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) tp[i] = *reinterpret_cast<const uint4*>(rec + CS_P + i * 512 + lane * 16);
      const int n = min(CS_C, t1 - tb);
      float x[2][4];                    // what the chunk's own tokens give
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        float lead[4] = {0.f, 0.f, 0.f, 0.f}, rest[4] = {0.f, 0.f, 0.f, 0.f};
        if (MODE == CS_DELTA) {
          cs_mma(rest, ra[2], EDL_B(0));
          cs_mma(rest, ra[0], EDL_B(2));
          cs_mma(rest, ra[1], EDL_B(1));
          cs_mma(rest, ra[1], EDL_B(0));
          cs_mma(rest, ra[0], EDL_B(1));
        } else {
          cs_mma(rest, ra[0], EDL_B(2));
          cs_mma(rest, ra[0], EDL_B(1));
        }
        cs_mma(lead, ra[0], EDL_B(0));
#pragma unroll
        for (int e = 0; e < 4; ++e) x[j][e] = lead[e] + rest[e];
      }
      if (unsafe) cs_triangle<MODE == CS_DELTA ? 3 : 1>(rec + CS_P, ra, lane, x);
#undef EDL_B
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int t = 8 * j + 2 * quad + (e & 1), c = col + 8 * (e >> 1);
          const float o = es[t] * (yq[0][j][e] + yq[1][j][e]) + x[j][e];
          if (t < n && c < DV) p.o[((long long)(tb + t) * H + h) * DV + c] = __float2bfloat16(o);
        }
    }
    st = st == CS_STAGES - 1 ? 0 : st + 1;
  }
  if (LOCAL && blockIdx.x == 0 && tid == 0) p.seg_decay[(long long)span.slot * H + h] = decay;
  float* const left = LOCAL ? at_seg : p.seg ? nullptr : cs_state_out(p, b, h, (long long)DK * DV);
  if (left) {
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int c = col + 8 * (e >> 1);
        if (c < DV) left[(8 * i + 2 * quad + (e & 1)) * row_step + c * col_step] = S[i][e];
      }
  }
}

// Turns what the segments of a sequence leave behind into the states in front of them; the state behind the last one goes out.
__global__ void chunk_carry_kernel(const CsParams p, int n4) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, h = blockIdx.y, b = blockIdx.z;
  if (i >= n4) return;
  const int first = cs_pos(p, b), n = (cs_pos(p, b + 1) - first + p.seg - 1) / p.seg, slot = (first - p.w0) / p.seg + b;
  if (n <= 0) return;
  const float4* in = reinterpret_cast<const float4*>(cs_state_in(p, b, h, 4LL * n4));
  float4* left = reinterpret_cast<float4*>(cs_state_out(p, b, h, 4LL * n4));
  float4* at = reinterpret_cast<float4*>(p.seg_state) + ((long long)slot * p.H + h) * n4 + i;
  const float* decay = p.seg_decay + (long long)slot * p.H + h;
  const long long step = (long long)p.H * n4;
  float4 s = in ? in[i] : make_float4(0.f, 0.f, 0.f, 0.f), next = at[0];
  for (int k = 0; k < n; ++k) {
    const float4 own = next;
    if (k + 1 < n) next = at[(k + 1) * step];
    const float d = decay[(long long)k * p.H];
    at[k * step] = s;
    s = make_float4(fmaf(d, s.x, own.x), fmaf(d, s.y, own.y), fmaf(d, s.z, own.z), fmaf(d, s.w, own.w));
  }
  if (left) left[i] = s;
}

template <int MODE, int DK>
int run_chunk_window(const CsParams& p, cudaStream_t s) {
  int per = 1;                          // heads that share a chunk's products
  if (MODE == CS_SSD)
    while (per < 8 && (p.H / p.G) % (2 * per) == 0) per *= 2;
  const int tokens = p.w1 - p.w0;
  chunk_coef_kernel<MODE, DK><<<dim3(tokens / CS_C + p.B + 1, (p.H / per + 3) / 4), 128, 0, s>>>(p, per);
  if (check_cuda(cudaGetLastError(), "chunk_coef launch")) return -1;
  const int tiles = (p.DV + CS_CT - 1) / CS_CT, spans = p.seg ? tokens / p.seg + p.B + 1 : p.B;
  if constexpr (MODE == CS_SSD) {
    if (p.seg) {
      chunk_scan_kernel<MODE, DK, true><<<dim3(tiles, p.H, spans), CS_THREADS, 0, s>>>(p);
      if (check_cuda(cudaGetLastError(), "chunk_scan (segments) launch")) return -1;
      const int n4 = p.DV * DK / 4;
      chunk_carry_kernel<<<dim3((n4 + 255) / 256, p.H, p.B), 256, 0, s>>>(p, n4);
      if (check_cuda(cudaGetLastError(), "chunk_carry launch")) return -1;
    }
  }
  chunk_scan_kernel<MODE, DK, false><<<dim3(tiles, p.H, spans), CS_THREADS, 0, s>>>(p);
  return check_cuda(cudaGetLastError(), "chunk_scan launch");
}

template <int MODE, int DK>
int run_chunk_scan(CsParams p, int window, float* carry, cudaStream_t s) {
  const long long size = (long long)p.H * DK * p.DV;
  for (long long w = 0, i = 0; w < p.T; w += window, ++i) {
    p.w0 = (int)w;
    p.w1 = (int)(w + window < p.T ? w + window : p.T);
    if (carry) p.carry_in = carry + (i & 1) * size, p.carry_out = carry + ((i + 1) & 1) * size;
    if (run_chunk_window<MODE, DK>(p, s)) return -1;
  }
  return 0;
}

bool cs_aligned(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

int cs_check(const char* who, CsParams& p, int DK, int window, const float* carry) {
  if (window < CS_C || window % CS_C || (window < p.T && !p.state && (!carry || !cs_aligned(carry)))) {
    set_last_error("%s: a window of %d tokens", who, window);
    return -1;
  }
  if (p.H < 1 || p.H > 65535 || p.B > 65535 || p.DV < 1 || p.DV > 256 || !p.rec || !cs_aligned(p.rec) || !cs_aligned(p.q) ||
      !cs_aligned(p.k) || (DK & 15)) {
    set_last_error("%s: sizes (B=%d, H=%d, DK=%d, DV=%d) or unaligned operands", who, p.B, p.H, DK, p.DV);
    return -1;
  }
  p.vec_v = p.DV % 8 == 0 && cs_aligned(p.v);
  return 0;
}

}  // namespace
}  // namespace edl

using namespace edl;

// q, k [T, H, DK], v [T, H, DV], beta [T, H] or null: bf16; g fp32 [T, H] or null; state fp32 [nseq, H, DK, DV] or null; o bf16
// [T, H, DV]. window: tokens taken at a time, a multiple of 16; rec: workspace of (min(window, T) / 16 + nseq + 1) * H * 3344
// bytes; carry: without a state and with more tokens than a window, two states of one sequence. DK 32, 64 or 128, DV up to 256.
EDL_HOST_API int edl_delta_rule_chunks(const void* q, const void* k, const void* v, const float* g, const void* beta,
                                       const int* cu, int T, int nseq, int H, int DK, int DV, float scale, float* state, void* o,
                                       void* rec, int window, float* carry, void* stream) {
  if (nseq <= 0 || H <= 0 || T <= 0) return 0;
  CsParams p{};
  p.q = (const __nv_bfloat16*)q; p.k = (const __nv_bfloat16*)k; p.v = (const __nv_bfloat16*)v; p.g = g;
  p.beta = (const __nv_bfloat16*)beta; p.cu = cu; p.T = T; p.B = nseq; p.H = p.G = H; p.DV = DV; p.scale = scale;
  p.rec = (uint8_t*)rec; p.state = state; p.o = (__nv_bfloat16*)o;
  if (cs_check("edl_delta_rule_chunks", p, DK, window, carry)) return -1;
  cudaStream_t s = (cudaStream_t)stream;
  switch (DK) {
    case 32: return run_chunk_scan<CS_DELTA, 32>(p, window, carry, s);
    case 64: return run_chunk_scan<CS_DELTA, 64>(p, window, carry, s);
    case 128: return run_chunk_scan<CS_DELTA, 128>(p, window, carry, s);
  }
  set_last_error("edl_delta_rule_chunks: key head_dim %d not in {32, 64, 128}", DK);
  return -1;
}

// x [T, H, P], dt [T, H], B, C [T, G, N]: bf16; A, D, dt_bias fp32 [H] (D, dt_bias or null); state fp32 [nseq, H, P, N] or
// null; y bf16 [T, H, P]; window, rec (1680 bytes per place), carry: as above. N 16, 32, 64 or 128, P up to 256.
// seg: tokens of a segment (a multiple of 16) or 0; segments: workspace of (min(window, T) / seg + nseq + 1) * H * (P * N + 1)
// floats, 16-byte aligned, as `state` has to be then.
EDL_HOST_API int edl_ssd_scan_chunks(const void* x, const void* dt, const float* A, const void* B, const void* C,
                                     const float* D, const float* dt_bias, int softplus, const int* cu, int T, int nseq, int H,
                                     int P, int G, int N, float* state, void* y, void* rec, int window, float* carry,
                                     int seg, float* segments, void* stream) {
  if (nseq <= 0 || H <= 0 || T <= 0) return 0;
  const int tokens = window < T ? window : T;            // at a time
  if (seg < 0 || seg % CS_C || (seg && (!segments || !cs_aligned(segments) || !cs_aligned(state) || tokens / seg + nseq + 1 > 65535))) {
    set_last_error("edl_ssd_scan_chunks: segments of %d tokens", seg);
    return -1;
  }
  if (G < 1 || H % G) {
    set_last_error("edl_ssd_scan_chunks: heads %d not a multiple of groups %d", H, G);
    return -1;
  }
  CsParams p{};
  p.q = (const __nv_bfloat16*)C; p.k = (const __nv_bfloat16*)B; p.v = (const __nv_bfloat16*)x; p.dt = (const __nv_bfloat16*)dt;
  p.A = A; p.Dskip = D; p.dt_bias = dt_bias; p.softplus = softplus; p.cu = cu; p.T = T; p.B = nseq; p.H = H; p.G = G; p.DV = P;
  p.scale = 1.f; p.rec = (uint8_t*)rec; p.state = state; p.o = (__nv_bfloat16*)y;
  p.seg = seg;
  p.seg_state = segments;
  if (seg) p.seg_decay = segments + (long long)(tokens / seg + nseq + 1) * H * P * N;
  if (cs_check("edl_ssd_scan_chunks", p, N, window, carry)) return -1;
  cudaStream_t s = (cudaStream_t)stream;
  switch (N) {
    case 16: return run_chunk_scan<CS_SSD, 16>(p, window, carry, s);
    case 32: return run_chunk_scan<CS_SSD, 32>(p, window, carry, s);
    case 64: return run_chunk_scan<CS_SSD, 64>(p, window, carry, s);
    case 128: return run_chunk_scan<CS_SSD, 128>(p, window, carry, s);
  }
  set_last_error("edl_ssd_scan_chunks: state size %d not in {16, 32, 64, 128}", N);
  return -1;
}
