// Token scans of the gated delta rule (Qwen3-Next, Kimi delta attention) and of the Mamba-2 state-space recurrence, eight
// tokens at a time. Per head, with a [DK, DV] state S in fp32,
//
//   delta rule:  S <- e^{g_t} S ;  r_t = beta_t (v_t - S^T k_t) ;  S <- S + k_t r_t^T ;  o_t = scale S^T q_t
//   state space: S <- e^{dt_t A} S + B_t (dt_t x_t)^T ;                                  y_t = S^T C_t + D x_t
//
// (g_t a number per head, or one per key channel). Walking token by token, a step costs the latency of its own chain: two
// products with the state, each summed over lanes, one behind the other. Here a block of eight tokens meets the state once:
//
//   y_j = k_j . S_0 and q_j . S_0 for all eight (independent of one another, summed over lanes together)
//   r_j = beta_j v_j - eb_j y_j - sum_{i<j} M_ji r_i              M_ji = beta_j e^{g_{i+1} + .. + g_j} k_j . k_i
//   o_j = es_j q_j . S_0 + sum_{i<=j} P_ji r_i                    P_ji = scale e^{g_{i+1} + .. + g_j} q_j . k_i
//   S_8 = e^{g_1 + .. + g_8} S_0 + sum_i e^{g_{i+1} + .. + g_8} k_i r_i^T
//
// and the state space is the same without y and M (r_i = x_i, dt_i and D folded into P and the tails). Decays are exponentials
// of sums over (i, j], never of differences, so a gate of minus infinity stays a plain reset. Everything is fp32 on the FMA
// pipe, as in the one-token kernels; with a channel gate the block's vectors are k e^{..}, q e^{..} and k e^{.. to the end}.
//
//   * block_coef: a warp per (block, head) forms the 8 x 8 products and decays (100 floats per block and head).
//   * block_scan: the columns of a state never meet, so a CTA of two warps owns (sequence, head, column tile). SPLIT adjacent
//     lanes share CPT columns, each with DK / SPLIT rows of them in registers; k and q rows are fp32 in shared memory, two
//     stages, fetched a block ahead through registers. Loads are 16 bytes per lane, the same for all columns of a warp (one
//     wavefront), and every float loaded meets CPT columns, so with CPT = 4 the FMA pipe is what is left.
//
// Compiled without fast-math.
#include "common.cuh"

namespace edl {
namespace {

constexpr int BS_C = 8;              // tokens per block
constexpr int BS_THREADS = 64;
constexpr int BS_REC = 100;          // floats per (block, head): products 64 | es 8 | tail 8 | beta 8 | eb 8 | total 1 | -
constexpr int BS_ES = 64, BS_TAIL = 72, BS_BETA = 80, BS_EB = 88, BS_TOTAL = 96;

enum BsMode { BS_DELTA = 0, BS_CHANNEL = 1, BS_SSD = 2 };

struct BsParams {
  const __nv_bfloat16 *q, *k, *v;    // [T, rows' heads, DK] x 2, [T, H, DV]
  const float* g;                    // delta: [T, H] or [T, H, DK] log decays, or null
  const __nv_bfloat16* beta;         // delta: [T, H] or null
  const __nv_bfloat16* dt;           // state space: [T, H]
  const float *A, *Dskip, *dt_bias;  // [H]
  int softplus;
  const int* cu;
  int T, B, H, G, DV;                // G: heads of q and k (H for the delta rule)
  float scale;
  float* rec;                        // [slots, H, BS_REC]
  float* state;                      // delta [B, H, DK, DV], state space [B, H, DV, DK]; or null
  __nv_bfloat16* o;                  // [T, H, DV]
};

// A block's place in the record array: unique and increasing over (sequence, block), below T / 8 + B + 1.
__device__ __forceinline__ int bs_slot(int t, int b) { return t / BS_C + b; }

__device__ __forceinline__ float bs_softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }

// ---- coefficients -----------------------------------------------------------------------------------------------------
// The 64 products of a block share one array: entry [8 j + i], i <= j, is q_j . k_i, entry [8 i + j], i < j, is k_j . k_i.
template <int MODE, int DK>
__global__ void __launch_bounds__(128) block_coef_kernel(const BsParams p, int heads_per_warp) {
  constexpr int VD = DK >= 32 ? DK / 32 : 1;
  const int lane = threadIdx.x & 31;
  const int h0 = (blockIdx.y * 4 + (threadIdx.x >> 5)) * heads_per_warp;
  if (h0 >= p.H) return;
  const int slot = blockIdx.x;
  int lo = 0, hi = p.B;                 // the last sequence whose first block is not past this slot
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (bs_slot(p.cu[mid], mid) <= slot) lo = mid;
    else hi = mid;
  }
  const int first = p.cu[lo], end = p.cu[lo + 1];
  const int t0 = first + (slot - bs_slot(first, lo)) * BS_C;
  if (t0 < first || t0 >= end) return;
  const int n = min(BS_C, end - t0);
  const int rows = h0 / (p.H / p.G);    // head of q and k
  const int d0 = lane * VD;
  float k[BS_C][VD], q[BS_C][VD];
#pragma unroll
  for (int j = 0; j < BS_C; ++j)
#pragma unroll
    for (int e = 0; e < VD; ++e) {
      const bool on = j < n && d0 + e < DK;
      const long long at = ((long long)(t0 + j) * p.G + rows) * DK + d0 + e;
      k[j][e] = on ? __bfloat162float(p.k[at]) : 0.f;
      q[j][e] = on ? __bfloat162float(p.q[at]) : 0.f;
    }
  float w[64];
#pragma unroll
  for (int i = 0; i < 64; ++i) w[i] = 0.f;
  if constexpr (MODE == BS_CHANNEL) {
    float g[BS_C][VD];
#pragma unroll
    for (int j = 0; j < BS_C; ++j)
#pragma unroll
      for (int e = 0; e < VD; ++e)
        g[j][e] = j < n && d0 + e < DK ? p.g[((long long)(t0 + j) * p.H + h0) * DK + d0 + e] : 0.f;
#pragma unroll
    for (int i = 0; i < BS_C; ++i)
#pragma unroll
      for (int e = 0; e < VD; ++e) {
        float sum = 0.f;
        w[9 * i] = fmaf(q[i][e], k[i][e], w[9 * i]);
#pragma unroll
        for (int j = i + 1; j < BS_C; ++j) {
          sum += g[j][e];
          const float ki = k[i][e] * expf(sum);
          w[8 * j + i] = fmaf(q[j][e], ki, w[8 * j + i]);
          w[8 * i + j] = fmaf(k[j][e], ki, w[8 * i + j]);
        }
      }
  } else {
#pragma unroll
    for (int i = 0; i < BS_C; ++i)
#pragma unroll
      for (int j = i; j < BS_C; ++j)
#pragma unroll
        for (int e = 0; e < VD; ++e) {
          w[8 * j + i] = fmaf(q[j][e], k[i][e], w[8 * j + i]);
          if (MODE == BS_DELTA && j > i) w[8 * i + j] = fmaf(k[j][e], k[i][e], w[8 * i + j]);
        }
  }
  // sums over the lanes, spread: lane l is left with entries 2 l and 2 l + 1
#pragma unroll
  for (int o = 16, m = 32; o > 0; o >>= 1, m >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < m; ++i) {
      const float got = __shfl_xor_sync(0xffffffffu, up ? w[i] : w[i + m], o);
      w[i] = (up ? w[i + m] : w[i]) + got;
    }
  }
  for (int h = h0; h < min(p.H, h0 + heads_per_warp); ++h) {
    float g[BS_C], a[BS_C];             // log decays; beta or dt
#pragma unroll
    for (int j = 0; j < BS_C; ++j) {
      const bool on = j < n;
      const long long at = (long long)(t0 + j) * p.H + h;
      if (MODE == BS_SSD) {
        float d = 0.f;
        if (on) {
          d = __bfloat162float(p.dt[at]) + (p.dt_bias ? p.dt_bias[h] : 0.f);
          if (p.softplus) d = bs_softplus(d);
        }
        a[j] = d;
        g[j] = d * p.A[h];
      } else {
        a[j] = !on ? 0.f : p.beta ? __bfloat162float(p.beta[at]) : 1.f;
        g[j] = MODE == BS_DELTA && on && p.g ? p.g[at] : 0.f;
      }
    }
    float* dst = p.rec + ((long long)slot * p.H + h) * BS_REC;
    float out[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int x = 2 * lane + e, r = x >> 3, c = x & 7, j = max(r, c), i = min(r, c);
      float sum = 0.f, aj = 0.f, ai = 0.f;
#pragma unroll
      for (int l = 0; l < BS_C; ++l) {
        if (l > i && l <= j) sum += g[l];
        if (l == j) aj = a[l];
        if (l == i) ai = a[l];
      }
      float f = expf(sum) * w[e];
      if (MODE == BS_SSD) {
        f *= ai;
        if (r == c && p.Dskip) f += p.Dskip[h];
      } else {
        f *= r >= c ? p.scale : aj;
      }
      out[e] = f;
    }
    *reinterpret_cast<float2*>(dst + 2 * lane) = make_float2(out[0], out[1]);
    if (lane <= BS_C) {                 // lane 8: the whole block
      float before = 0.f, after = 0.f, mine = 0.f;
#pragma unroll
      for (int l = 0; l < BS_C; ++l) {
        if (l <= lane) before += g[l];
        else after += g[l];
        if (l == lane) mine = a[l];
      }
      const float e = expf(before);
      if (lane == BS_C) {
        dst[BS_TOTAL] = e;
      } else {
        dst[BS_ES + lane] = e * p.scale;
        dst[BS_TAIL + lane] = expf(after) * (MODE == BS_SSD ? mine : 1.f);
        dst[BS_BETA + lane] = mine;
        dst[BS_EB + lane] = e * mine;
      }
    }
  }
}

// ---- scan -------------------------------------------------------------------------------------------------------------
template <int MODE, int DK, int SPLIT, int CPT>
__global__ void __launch_bounds__(BS_THREADS) block_scan_kernel(const BsParams p) {
  constexpr int RPT = DK / SPLIT, NK = RPT / 4, CT = BS_THREADS / SPLIT * CPT;
  constexpr int VEC = BS_C * DK / 8;                      // 16-byte pieces of a block's k (or q) rows
  constexpr int NV = (2 * VEC + BS_THREADS - 1) / BS_THREADS;
  constexpr int NX = (BS_C * CT + BS_THREADS - 1) / BS_THREADS;
  constexpr int CH4 = DK / 4;                             // channel gate: threads that hold four channels of all tokens
  constexpr bool CH = MODE == BS_CHANNEL;
  constexpr int KINDS = MODE == BS_SSD ? 1 : 2;
  static_assert(RPT % 4 == 0 && CPT * KINDS <= SPLIT && (!CH || 2 * CH4 <= BS_THREADS), "");
  __shared__ __align__(16) float sk[2][BS_C][DK], sq[2][BS_C][DK], sv[2][BS_C][CT], srec[2][BS_REC];
  __shared__ __align__(16) float su[CH ? 2 : 1][CH ? BS_C : 1][CH ? DK : 4], sd[CH ? 2 : 1][CH ? DK : 4];
  const int tid = threadIdx.x, lane = tid & 31;
  const int part = tid % SPLIT, grp = tid / SPLIT;
  const int h = blockIdx.y, b = blockIdx.z;
  const int col0 = blockIdx.x * CT, col = col0 + grp * CPT;
  const int t0 = p.cu[b], t1 = p.cu[b + 1];
  if (t0 >= t1) return;
  const int H = p.H, DV = p.DV, rows = h / (p.H / p.G);

  uint4 xkq[CH ? 1 : NV];
  uint2 xc[CH ? BS_C : 1];
  float4 gc[CH ? BS_C : 1];
  __nv_bfloat16 xv[NX];
  float4 xr;
  const bool c_on = CH && tid < 2 * CH4, c_is_q = tid >= CH4;
  const int c4 = (tid % CH4) * 4;
  auto fetch = [&](int tb) {
    const int n = min(BS_C, t1 - tb);
    if constexpr (CH) {
      if (c_on) {
#pragma unroll
        for (int j = 0; j < BS_C; ++j) {
          const long long at = ((long long)(tb + j) * H + h) * DK + c4;
          xc[j] = j < n ? *reinterpret_cast<const uint2*>((c_is_q ? p.q : p.k) + at) : make_uint2(0u, 0u);
          gc[j] = j < n ? *reinterpret_cast<const float4*>(p.g + at) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int x = tid + i * BS_THREADS, y = x % VEC, j = y / (DK / 8), d = (y % (DK / 8)) * 8;
        xkq[i] = make_uint4(0u, 0u, 0u, 0u);
        if (x < 2 * VEC && j < n)
          xkq[i] = *reinterpret_cast<const uint4*>((x < VEC ? p.k : p.q) + ((long long)(tb + j) * p.G + rows) * DK + d);
      }
    }
#pragma unroll
    for (int i = 0; i < NX; ++i) {
      const int x = tid + i * BS_THREADS, j = x / CT, c = col0 + x % CT;
      xv[i] = __float2bfloat16(0.f);
      if (x < BS_C * CT && j < n && c < DV) xv[i] = p.v[((long long)(tb + j) * H + h) * DV + c];
    }
    if (tid < BS_REC / 4)
      xr = *reinterpret_cast<const float4*>(p.rec + ((long long)bs_slot(tb, b) * H + h) * BS_REC + 4 * tid);
  };
  auto store = [&](int buf) {
    if constexpr (CH) {
      if (c_on) {
        float x[BS_C][4], s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < BS_C; ++j) {
          const float2 a = unpack_bf16x2(xc[j].x), c = unpack_bf16x2(xc[j].y);
          x[j][0] = a.x; x[j][1] = a.y; x[j][2] = c.x; x[j][3] = c.y;
          const float g[4] = {gc[j].x, gc[j].y, gc[j].z, gc[j].w};
          float y[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            s[e] += g[e];
            y[e] = x[j][e] * expf(s[e]);
          }
          *reinterpret_cast<float4*>(c_is_q ? &sq[buf][j][c4] : &sk[buf][j][c4]) = make_float4(y[0], y[1], y[2], y[3]);
        }
        if (!c_is_q) {
          *reinterpret_cast<float4*>(&sd[buf][c4]) = make_float4(expf(s[0]), expf(s[1]), expf(s[2]), expf(s[3]));
          s[0] = s[1] = s[2] = s[3] = 0.f;
#pragma unroll
          for (int j = BS_C - 1; j >= 0; --j) {
            *reinterpret_cast<float4*>(&su[buf][j][c4]) =
                make_float4(x[j][0] * expf(s[0]), x[j][1] * expf(s[1]), x[j][2] * expf(s[2]), x[j][3] * expf(s[3]));
            s[0] += gc[j].x; s[1] += gc[j].y; s[2] += gc[j].z; s[3] += gc[j].w;
          }
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int x = tid + i * BS_THREADS, y = x % VEC, j = y / (DK / 8), d = (y % (DK / 8)) * 8;
        if (x >= 2 * VEC) break;
        const uint4 w = xkq[i];
        const float2 a = unpack_bf16x2(w.x), c = unpack_bf16x2(w.y), e = unpack_bf16x2(w.z), f = unpack_bf16x2(w.w);
        float4* dst = reinterpret_cast<float4*>(x < VEC ? &sk[buf][j][d] : &sq[buf][j][d]);
        dst[0] = make_float4(a.x, a.y, c.x, c.y);
        dst[1] = make_float4(e.x, e.y, f.x, f.y);
      }
    }
#pragma unroll
    for (int i = 0; i < NX; ++i) {
      const int x = tid + i * BS_THREADS;
      if (x < BS_C * CT) sv[buf][x / CT][x % CT] = __bfloat162float(xv[i]);
    }
    if (tid < BS_REC / 4) *reinterpret_cast<float4*>(&srec[buf][4 * tid]) = xr;
  };

  fetch(t0);
  // rows of this thread: 4 (part + SPLIT i) + j, i < NK, j < 4; packed arithmetic takes rows j, j + 1 as a pair
  float S[NK][4][CPT];
  float* pool = p.state ? p.state + ((long long)b * H + h) * DK * DV : nullptr;
  const long long row_step = MODE == BS_SSD ? 1 : DV, col_step = MODE == BS_SSD ? DK : 1;
#pragma unroll
  for (int i = 0; i < NK; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int c = 0; c < CPT; ++c)
        S[i][j][c] = pool && col + c < DV ? pool[(4 * (part + SPLIT * i) + j) * row_step + (col + c) * col_step] : 0.f;
  // after the sums a lane holds one column (and one kind of product): which one is read off the low bits of `part`
  constexpr int KB = KINDS == 2 ? 1 : 0;                 // bits that tell the kind
  constexpr int CB = CPT == 4 ? 2 : CPT == 2 ? 1 : 0;    // bits that tell the column
  const int mine = CPT == 4 ? ((part >> KB) & 1) * 2 + ((part >> (KB + 1)) & 1) : CPT == 2 ? (part >> KB) & 1 : 0;
  const bool writes = (KINDS == 1 || (part & 1)) && (part >> (KB + CB)) == 0 && col + mine < DV;
  store(0);
  int buf = 0;
  for (int tb = t0; tb < t1; tb += BS_C, buf ^= 1) {
    __syncthreads();                    // this stage is filled, and nobody reads the other one any more
    const bool more = tb + BS_C < t1;
    if (more) fetch(tb + BS_C);
    const float* rec = srec[buf];
    float sum[KINDS][BS_C][CPT];
#pragma unroll
    for (int j = 0; j < BS_C; ++j)
#pragma unroll
      for (int kind = 0; kind < KINDS; ++kind) {
        const float* x = (kind == KINDS - 1 ? sq[buf][j] : sk[buf][j]) + 4 * part;
        float a[CPT][2];
#pragma unroll
        for (int i = 0; i < NK; ++i) {
          const float4 r = *reinterpret_cast<const float4*>(x + 4 * SPLIT * i);
#pragma unroll
          for (int c = 0; c < CPT; ++c) {
            if (i == 0) mul2(a[c][0], a[c][1], r.x, r.y, S[i][0][c], S[i][1][c]);
            else fma2(a[c][0], a[c][1], r.x, r.y, S[i][0][c], S[i][1][c], a[c][0], a[c][1]);
            fma2(a[c][0], a[c][1], r.z, r.w, S[i][2][c], S[i][3][c], a[c][0], a[c][1]);
          }
        }
#pragma unroll
        for (int c = 0; c < CPT; ++c) sum[kind][j][c] = a[c][0] + a[c][1];
      }
    // ---- sums over the lanes that share the columns; the first exchanges also spread kinds and columns over them
    if constexpr (KINDS == 2) {
      const bool up = part & 1;
#pragma unroll
      for (int j = 0; j < BS_C; ++j)
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          const float got = __shfl_xor_sync(0xffffffffu, up ? sum[0][j][c] : sum[KINDS - 1][j][c], 1);
          sum[0][j][c] = (up ? sum[KINDS - 1][j][c] : sum[0][j][c]) + got;
        }
    }
    if constexpr (CPT == 4) {
      const bool up = part & (1 << KB);
#pragma unroll
      for (int j = 0; j < BS_C; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const float got = __shfl_xor_sync(0xffffffffu, up ? sum[0][j][c] : sum[0][j][(c + 2) % CPT], 1 << KB);
          sum[0][j][c] = (up ? sum[0][j][(c + 2) % CPT] : sum[0][j][c]) + got;
        }
    }
    if constexpr (CPT >= 2) {
      constexpr int BIT = 1 << (KB + CB - 1);
      const bool up = part & BIT;
#pragma unroll
      for (int j = 0; j < BS_C; ++j) {
        const float got = __shfl_xor_sync(0xffffffffu, up ? sum[0][j][0] : sum[0][j][1 % CPT], BIT);
        sum[0][j][0] = (up ? sum[0][j][1 % CPT] : sum[0][j][0]) + got;
      }
    }
#pragma unroll
    for (int bit = 1 << (KB + CB); bit < SPLIT; bit <<= 1)
#pragma unroll
      for (int j = 0; j < BS_C; ++j) sum[0][j][0] += __shfl_xor_sync(0xffffffffu, sum[0][j][0], bit);
    // ---- r of this lane's column, then of all its columns
    float r[BS_C], all[BS_C][CPT];
    if constexpr (MODE == BS_SSD) {
#pragma unroll
      for (int j = 0; j < BS_C; ++j) {
        r[j] = sv[buf][j][grp * CPT + mine];
#pragma unroll
        for (int c = 0; c < CPT; ++c) all[j][c] = sv[buf][j][grp * CPT + c];
      }
    } else {
#pragma unroll
      for (int j = 0; j < BS_C; ++j) r[j] = rec[BS_BETA + j] * sv[buf][j][grp * CPT + mine] - rec[BS_EB + j] * sum[0][j][0];
#pragma unroll
      for (int i = 0; i < BS_C; ++i)      // r_i is final: take it out of the later ones
#pragma unroll
        for (int j = i + 1; j < BS_C; ++j) r[j] = fmaf(-rec[8 * i + j], r[i], r[j]);
#pragma unroll
      for (int j = 0; j < BS_C; ++j) {
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          const int from = CPT == 4 ? ((c >> 1) << 1) + ((c & 1) << 2) : CPT == 2 ? c << 1 : 0;
          all[j][c] = __shfl_sync(0xffffffffu, r[j], (lane & ~(SPLIT - 1)) + from);
        }
        r[j] = __shfl_sync(0xffffffffu, r[j], lane & ~1);      // a lane of outputs takes its column's r
      }
    }
    // ---- outputs
    const int n = min(BS_C, t1 - tb);
#pragma unroll
    for (int j = 0; j < BS_C; ++j) {
      float o = rec[BS_ES + j] * sum[0][j][0];
#pragma unroll
      for (int i = 0; i <= j; ++i) o = fmaf(rec[8 * j + i], r[i], o);
      if (writes && j < n) p.o[((long long)(tb + j) * H + h) * DV + col + mine] = __float2bfloat16(o);
    }
    // ---- the state behind the block
    if constexpr (!CH) {
      const float total = rec[BS_TOTAL];
#pragma unroll
      for (int i = 0; i < NK; ++i)
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          mul2(S[i][0][c], S[i][1][c], S[i][0][c], S[i][1][c], total, total);
          mul2(S[i][2][c], S[i][3][c], S[i][2][c], S[i][3][c], total, total);
        }
    } else {
#pragma unroll
      for (int i = 0; i < NK; ++i) {
        const float4 d = *reinterpret_cast<const float4*>(&sd[CH ? buf : 0][CH ? 4 * (part + SPLIT * i) : 0]);
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          mul2(S[i][0][c], S[i][1][c], S[i][0][c], S[i][1][c], d.x, d.y);
          mul2(S[i][2][c], S[i][3][c], S[i][2][c], S[i][3][c], d.z, d.w);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < BS_C; ++j) {
      const float* x = (CH ? su[CH ? buf : 0][CH ? j : 0] : sk[buf][j]) + 4 * part;
      float f[CPT];
#pragma unroll
      for (int c = 0; c < CPT; ++c) f[c] = CH ? all[j][c] : all[j][c] * rec[BS_TAIL + j];
#pragma unroll
      for (int i = 0; i < NK; ++i) {
        const float4 k4 = *reinterpret_cast<const float4*>(x + 4 * SPLIT * i);
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          fma2(S[i][0][c], S[i][1][c], k4.x, k4.y, f[c], f[c], S[i][0][c], S[i][1][c]);
          fma2(S[i][2][c], S[i][3][c], k4.z, k4.w, f[c], f[c], S[i][2][c], S[i][3][c]);
        }
      }
    }
    if (more) store(buf ^ 1);
  }
  if (pool) {
#pragma unroll
    for (int i = 0; i < NK; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int c = 0; c < CPT; ++c)
          if (col + c < DV) pool[(4 * (part + SPLIT * i) + j) * row_step + (col + c) * col_step] = S[i][j][c];
  }
}

template <int MODE, int DK, int SPLIT, int CPT>
int launch_block_scan(const BsParams& p, cudaStream_t s) {
  constexpr int CT = BS_THREADS / SPLIT * CPT;
  block_scan_kernel<MODE, DK, SPLIT, CPT><<<dim3((p.DV + CT - 1) / CT, p.H, p.B), BS_THREADS, 0, s>>>(p);
  return check_cuda(cudaGetLastError(), "block_scan launch");
}

template <int MODE, int DK>
int run_block_scan(const BsParams& p, cudaStream_t s) {
  int per = 1;                          // heads that share a block's products
  if (MODE == BS_SSD)
    while (per < 8 && (p.H / p.G) % (2 * per) == 0) per *= 2;
  const int slots = p.T / BS_C + p.B + 1;
  block_coef_kernel<MODE, DK><<<dim3(slots, (p.H / per + 3) / 4), 128, 0, s>>>(p, per);
  if (check_cuda(cudaGetLastError(), "block_coef launch")) return -1;
  // Fewer columns per lane make more warps to hide the lanes' latency behind, more columns make fewer loads and exchanges
  // per column. Measured (delta rule, 32 heads of 128 x 128, us with 1 / 2 / 4 columns): one sequence of 4096 tokens and 16
  // heads 889 / 975 / 1636 (512 warps at one column), 5328 + 2864 tokens 2652 / 1888 / 2613 (2048), four of 2048 tokens
  // 2646 / 1548 / 1327 (4096). Short sequences of a ragged step end early and count for little.
  constexpr int SPLIT = DK == 128 ? 8 : 4, MAXC = DK == 128 ? 4 : 2;
  const long long groups = (long long)min((long long)p.B, (long long)(p.T / 64 + 1)) * p.H * p.DV * SPLIT / 32;   // warps at one column
  const long long room = 4LL * sm_count();
  if constexpr (MAXC == 4) {
    if (groups > 4 * room) return launch_block_scan<MODE, DK, SPLIT, 4>(p, s);
  }
  if (groups > room) return launch_block_scan<MODE, DK, SPLIT, 2>(p, s);
  return launch_block_scan<MODE, DK, SPLIT, 1>(p, s);
}

bool bs_aligned(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

int bs_check(const char* who, const BsParams& p, int DK) {
  if (p.H < 1 || p.H > 65535 || p.B > 65535 || p.DV < 1 || p.DV > 256 || !p.rec || !bs_aligned(p.rec) || !bs_aligned(p.q) ||
      !bs_aligned(p.k) || (DK & 15)) {
    set_last_error("%s: sizes (B=%d, H=%d, DK=%d, DV=%d) or unaligned operands", who, p.B, p.H, DK, p.DV);
    return -1;
  }
  return 0;
}

}  // namespace
}  // namespace edl

using namespace edl;

// q, k [T, H, DK], v [T, H, DV], beta [T, H] or null: bf16; g fp32 [T, H], or [T, H, DK] with g_per_channel, or null;
// state fp32 [nseq, H, DK, DV] or null; o bf16 [T, H, DV]; rec: workspace of (T / 8 + nseq + 1) * H * 100 floats.
EDL_HOST_API int edl_delta_rule_blocks(const void* q, const void* k, const void* v, const float* g, const void* beta,
                                       int g_per_channel, const int* cu, int T, int nseq, int H, int DK, int DV, float scale,
                                       float* state, void* o, float* rec, void* stream) {
  if (nseq <= 0 || H <= 0 || T <= 0) return 0;
  BsParams p{};
  p.q = (const __nv_bfloat16*)q; p.k = (const __nv_bfloat16*)k; p.v = (const __nv_bfloat16*)v; p.g = g;
  p.beta = (const __nv_bfloat16*)beta; p.cu = cu; p.T = T; p.B = nseq; p.H = p.G = H; p.DV = DV; p.scale = scale; p.rec = rec;
  p.state = state; p.o = (__nv_bfloat16*)o;
  if (bs_check("edl_delta_rule_blocks", p, DK)) return -1;
  cudaStream_t s = (cudaStream_t)stream;
  if (g_per_channel) {
    if (!g || !bs_aligned(g)) {
      set_last_error("edl_delta_rule_blocks: a channel gate needs 16-byte aligned gates");
      return -1;
    }
    switch (DK) {
      case 32: return run_block_scan<BS_CHANNEL, 32>(p, s);
      case 64: return run_block_scan<BS_CHANNEL, 64>(p, s);
      case 128: return run_block_scan<BS_CHANNEL, 128>(p, s);
    }
  } else {
    switch (DK) {
      case 32: return run_block_scan<BS_DELTA, 32>(p, s);
      case 64: return run_block_scan<BS_DELTA, 64>(p, s);
      case 128: return run_block_scan<BS_DELTA, 128>(p, s);
    }
  }
  set_last_error("edl_delta_rule_blocks: key head_dim %d not in {32, 64, 128}", DK);
  return -1;
}

// x [T, H, P], dt [T, H], B, C [T, G, N]: bf16; A, D, dt_bias fp32 [H] (D, dt_bias or null); state fp32 [nseq, H, P, N] or
// null; y bf16 [T, H, P]; rec as above.
EDL_HOST_API int edl_ssd_scan_blocks(const void* x, const void* dt, const float* A, const void* B, const void* C,
                                     const float* D, const float* dt_bias, int softplus, const int* cu, int T, int nseq, int H,
                                     int P, int G, int N, float* state, void* y, float* rec, void* stream) {
  if (nseq <= 0 || H <= 0 || T <= 0) return 0;
  if (G < 1 || H % G) {
    set_last_error("edl_ssd_scan_blocks: heads %d not a multiple of groups %d", H, G);
    return -1;
  }
  BsParams p{};
  p.q = (const __nv_bfloat16*)C; p.k = (const __nv_bfloat16*)B; p.v = (const __nv_bfloat16*)x; p.dt = (const __nv_bfloat16*)dt;
  p.A = A; p.Dskip = D; p.dt_bias = dt_bias; p.softplus = softplus; p.cu = cu; p.T = T; p.B = nseq; p.H = H; p.G = G; p.DV = P;
  p.scale = 1.f; p.rec = rec; p.state = state; p.o = (__nv_bfloat16*)y;
  if (bs_check("edl_ssd_scan_blocks", p, N)) return -1;
  cudaStream_t s = (cudaStream_t)stream;
  switch (N) {
    case 16: return run_block_scan<BS_SSD, 16>(p, s);
    case 32: return run_block_scan<BS_SSD, 32>(p, s);
    case 64: return run_block_scan<BS_SSD, 64>(p, s);
    case 128: return run_block_scan<BS_SSD, 128>(p, s);
  }
  set_last_error("edl_ssd_scan_blocks: state size %d not in {16, 32, 64, 128}", N);
  return -1;
}
