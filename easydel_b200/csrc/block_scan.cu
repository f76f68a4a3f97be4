// Token scan of the delta rule with a decay per key channel (Kimi delta attention), eight tokens at a time. Per head, with a
// [DK, DV] state S in fp32,
//
//   S <- diag(e^{g_t}) S ;  r_t = beta_t (v_t - S^T k_t) ;  S <- S + k_t r_t^T ;  o_t = scale S^T q_t
//
// Walking token by token, a step costs the latency of its own chain: two products with the state, each summed over lanes, one
// behind the other. Here a block of eight tokens meets the state once:
//
//   y_j = (k_j e^{g_1 + .. + g_j}) . S_0, and the same with q_j, for all eight (independent, summed over lanes together)
//   r_j = beta_j (v_j - y_j) - sum_{i<j} M_ji r_i          M_ji = beta_j  k_j . (e^{g_{i+1} + .. + g_j} k_i)
//   o_j = scale y'_j + sum_{i<=j} P_ji r_i                 P_ji = scale   q_j . (e^{g_{i+1} + .. + g_j} k_i)
//   S_8 = diag(e^{g_1 + .. + g_8}) S_0 + sum_i (e^{g_{i+1} + .. + g_8} k_i) r_i^T
//
// Decays are exponentials of sums over (i, j], never of differences, so a gate of minus infinity stays a plain reset.
// Everything is fp32 on the FMA pipe, as in the one-token kernel.
//
//   * block_coef: a warp per (block, head) forms the 8 x 8 products.
//   * block_scan: the columns of a state never meet, so a CTA of two warps owns (sequence, head, column tile). SPLIT adjacent
//     lanes share CPT columns, each with DK / SPLIT rows of them in registers; the block's rows are fp32 in shared memory, two
//     stages, fetched a block ahead through registers. Loads are 16 bytes per lane, the same for all columns of a warp, and
//     every float loaded meets CPT columns. What bounds it is latency: a scheduler holds one to four warps.
//
// 4096 tokens, 16 heads of 128 x 128: 1.63 ms; eight sequences of 512 tokens, 32 heads: 0.82 ms (one token at a time: 17.7 ms
// and 4.6 ms).
// Compiled without fast-math.
#include "common.cuh"

namespace edl {
namespace {

constexpr int BS_C = 8;              // tokens per block
constexpr int BS_THREADS = 64;
constexpr int BS_REC = 72;           // floats per (block, head): products 64 | beta 8
constexpr int BS_BETA = 64;

struct BsParams {
  const __nv_bfloat16 *q, *k, *v;    // [T, H, DK] x 2, [T, H, DV]
  const float* g;                    // [T, H, DK] log decays
  const __nv_bfloat16* beta;         // [T, H] or null
  const int* cu;
  int T, B, H, DV;
  float scale;
  float* rec;                        // [slots, H, BS_REC]
  float* state;                      // [B, H, DK, DV] or null
  __nv_bfloat16* o;                  // [T, H, DV]
};

// A block's place in the record array: unique and increasing over (sequence, block), below T / 8 + B + 1.
__device__ __forceinline__ int bs_slot(int t, int b) { return t / BS_C + b; }

// ---- coefficients -----------------------------------------------------------------------------------------------------
// The 64 products of a block share one array: entry [8 j + i], i <= j, is q_j . k_i, entry [8 i + j], i < j, is k_j . k_i.
template <int DK>
__global__ void __launch_bounds__(128) block_coef_kernel(const BsParams p) {
  constexpr int VD = DK / 32;
  const int lane = threadIdx.x & 31, h = blockIdx.y * 4 + (threadIdx.x >> 5);
  if (h >= p.H) return;
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
  float k[BS_C][VD], q[BS_C][VD], g[BS_C][VD], w[64];
#pragma unroll
  for (int j = 0; j < BS_C; ++j)
#pragma unroll
    for (int e = 0; e < VD; ++e) {
      const long long at = ((long long)(t0 + j) * p.H + h) * DK + lane * VD + e;
      k[j][e] = j < n ? __bfloat162float(p.k[at]) : 0.f;
      q[j][e] = j < n ? __bfloat162float(p.q[at]) : 0.f;
      g[j][e] = j < n ? p.g[at] : 0.f;
    }
#pragma unroll
  for (int i = 0; i < 64; ++i) w[i] = 0.f;
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
  float* dst = p.rec + ((long long)slot * p.H + h) * BS_REC;
  auto beta = [&](int j) { return j >= n ? 0.f : p.beta ? __bfloat162float(p.beta[(long long)(t0 + j) * p.H + h]) : 1.f; };
  float out[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int x = 2 * lane + e, r = x >> 3, c = x & 7;
    out[e] = w[e] * (r >= c ? p.scale : beta(c));
  }
  *reinterpret_cast<float2*>(dst + 2 * lane) = make_float2(out[0], out[1]);
  if (lane < BS_C) dst[BS_BETA + lane] = beta(lane);
}

// ---- scan -------------------------------------------------------------------------------------------------------------
template <int DK, int SPLIT, int CPT>
__global__ void __launch_bounds__(BS_THREADS) block_scan_kernel(const BsParams p) {
  constexpr int RPT = DK / SPLIT, NK = RPT / 4, CT = BS_THREADS / SPLIT * CPT;
  constexpr int NX = (BS_C * CT + BS_THREADS - 1) / BS_THREADS;
  constexpr int CH4 = DK / 4;                             // threads that hold four channels of k (or q) of all tokens
  static_assert(RPT % 4 == 0 && 2 * CPT <= SPLIT && 2 * CH4 <= BS_THREADS, "");
  __shared__ __align__(16) float sk[2][BS_C][DK], sq[2][BS_C][DK], sv[2][BS_C][CT], srec[2][BS_REC];
  __shared__ __align__(16) float su[2][BS_C][DK], sd[2][DK];
  const int tid = threadIdx.x, lane = tid & 31;
  const int part = tid % SPLIT, grp = tid / SPLIT;
  const int h = blockIdx.y, b = blockIdx.z;
  const int col0 = blockIdx.x * CT, col = col0 + grp * CPT;
  const int t0 = p.cu[b], t1 = p.cu[b + 1];
  if (t0 >= t1) return;
  const int H = p.H, DV = p.DV;

  uint2 xc[BS_C];
  float4 gc[BS_C];
  __nv_bfloat16 xv[NX];
  float4 xr;
  const bool c_on = tid < 2 * CH4, c_is_q = tid >= CH4;
  const int c4 = (tid % CH4) * 4;
  auto fetch = [&](int tb) {
    const int n = min(BS_C, t1 - tb);
    if (c_on) {
#pragma unroll
      for (int j = 0; j < BS_C; ++j) {
        const long long at = ((long long)(tb + j) * H + h) * DK + c4;
        xc[j] = j < n ? *reinterpret_cast<const uint2*>((c_is_q ? p.q : p.k) + at) : make_uint2(0u, 0u);
        gc[j] = j < n ? *reinterpret_cast<const float4*>(p.g + at) : make_float4(0.f, 0.f, 0.f, 0.f);
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
#pragma unroll
  for (int i = 0; i < NK; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int c = 0; c < CPT; ++c)
        S[i][j][c] = pool && col + c < DV ? pool[(4 * (part + SPLIT * i) + j) * (long long)DV + col + c] : 0.f;
  // after the sums a lane holds one column (and one kind of product): which one is read off the low bits of `part`
  constexpr int CB = CPT == 4 ? 2 : CPT == 2 ? 1 : 0;    // bits that tell the column
  const int mine = CPT == 4 ? ((part >> 1) & 1) * 2 + ((part >> 2) & 1) : CPT == 2 ? (part >> 1) & 1 : 0;
  const bool writes = (part & 1) && (part >> (1 + CB)) == 0 && col + mine < DV;
  store(0);
  int buf = 0;
  for (int tb = t0; tb < t1; tb += BS_C, buf ^= 1) {
    __syncthreads();                    // this stage is filled, and nobody reads the other one any more
    const bool more = tb + BS_C < t1;
    if (more) fetch(tb + BS_C);
    const float* rec = srec[buf];
    float sum[2][BS_C][CPT];
#pragma unroll
    for (int j = 0; j < BS_C; ++j)
#pragma unroll
      for (int kind = 0; kind < 2; ++kind) {
        const float* x = (kind ? sq[buf][j] : sk[buf][j]) + 4 * part;
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
    {
      const bool up = part & 1;
#pragma unroll
      for (int j = 0; j < BS_C; ++j)
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          const float got = __shfl_xor_sync(0xffffffffu, up ? sum[0][j][c] : sum[1][j][c], 1);
          sum[0][j][c] = (up ? sum[1][j][c] : sum[0][j][c]) + got;
        }
    }
    if constexpr (CPT == 4) {
      const bool up = part & 2;
#pragma unroll
      for (int j = 0; j < BS_C; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const float got = __shfl_xor_sync(0xffffffffu, up ? sum[0][j][c] : sum[0][j][(c + 2) % CPT], 2);
          sum[0][j][c] = (up ? sum[0][j][(c + 2) % CPT] : sum[0][j][c]) + got;
        }
    }
    if constexpr (CPT >= 2) {
      constexpr int BIT = 1 << (1 + CB - 1);
      const bool up = part & BIT;
#pragma unroll
      for (int j = 0; j < BS_C; ++j) {
        const float got = __shfl_xor_sync(0xffffffffu, up ? sum[0][j][0] : sum[0][j][1 % CPT], BIT);
        sum[0][j][0] = (up ? sum[0][j][1 % CPT] : sum[0][j][0]) + got;
      }
    }
#pragma unroll
    for (int bit = 1 << (1 + CB); bit < SPLIT; bit <<= 1)
#pragma unroll
      for (int j = 0; j < BS_C; ++j) sum[0][j][0] += __shfl_xor_sync(0xffffffffu, sum[0][j][0], bit);
    // ---- r of this lane's column, then of all its columns
    float r[BS_C], all[BS_C][CPT];
#pragma unroll
    for (int j = 0; j < BS_C; ++j) r[j] = rec[BS_BETA + j] * (sv[buf][j][grp * CPT + mine] - sum[0][j][0]);
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
    // ---- outputs
    const int n = min(BS_C, t1 - tb);
#pragma unroll
    for (int j = 0; j < BS_C; ++j) {
      float o = p.scale * sum[0][j][0];
#pragma unroll
      for (int i = 0; i <= j; ++i) o = fmaf(rec[8 * j + i], r[i], o);
      if (writes && j < n) p.o[((long long)(tb + j) * H + h) * DV + col + mine] = __float2bfloat16(o);
    }
    // ---- the state behind the block
#pragma unroll
    for (int i = 0; i < NK; ++i) {
      const float4 d = *reinterpret_cast<const float4*>(&sd[buf][4 * (part + SPLIT * i)]);
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        mul2(S[i][0][c], S[i][1][c], S[i][0][c], S[i][1][c], d.x, d.y);
        mul2(S[i][2][c], S[i][3][c], S[i][2][c], S[i][3][c], d.z, d.w);
      }
    }
#pragma unroll
    for (int j = 0; j < BS_C; ++j) {
      const float* x = su[buf][j] + 4 * part;
#pragma unroll
      for (int i = 0; i < NK; ++i) {
        const float4 k4 = *reinterpret_cast<const float4*>(x + 4 * SPLIT * i);
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          fma2(S[i][0][c], S[i][1][c], k4.x, k4.y, all[j][c], all[j][c], S[i][0][c], S[i][1][c]);
          fma2(S[i][2][c], S[i][3][c], k4.z, k4.w, all[j][c], all[j][c], S[i][2][c], S[i][3][c]);
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
          if (col + c < DV) pool[(4 * (part + SPLIT * i) + j) * (long long)DV + col + c] = S[i][j][c];
  }
}

template <int DK, int SPLIT, int CPT>
int launch_block_scan(const BsParams& p, cudaStream_t s) {
  constexpr int CT = BS_THREADS / SPLIT * CPT;
  block_scan_kernel<DK, SPLIT, CPT><<<dim3((p.DV + CT - 1) / CT, p.H, p.B), BS_THREADS, 0, s>>>(p);
  return check_cuda(cudaGetLastError(), "block_scan launch");
}

template <int DK>
int run_block_scan(const BsParams& p, cudaStream_t s) {
  block_coef_kernel<DK><<<dim3(p.T / BS_C + p.B + 1, (p.H + 3) / 4), 128, 0, s>>>(p);
  if (check_cuda(cudaGetLastError(), "block_coef launch")) return -1;
  // Fewer columns per lane make more warps to hide the lanes' latency behind, more columns make fewer loads and exchanges
  // per column. Measured (us with 1 / 2 / 4 columns): one sequence of 4096 tokens and 16 heads of 128 x 128 1755 / 1806 / 2713
  // (512 warps at one column), eight of 512 tokens and 32 heads 1573 / 1136 / 839 (8192). Short sequences of a ragged step
  // end early and count for little.
  constexpr int SPLIT = DK == 128 ? 8 : 4;
  const long long groups = (long long)min((long long)p.B, (long long)(p.T / 64 + 1)) * p.H * p.DV * SPLIT / 32;   // warps at one column
  const long long room = 4LL * sm_count();
  if constexpr (DK == 128) {
    if (groups > 4 * room) return launch_block_scan<DK, SPLIT, 4>(p, s);
  }
  if (groups > room) return launch_block_scan<DK, SPLIT, 2>(p, s);
  return launch_block_scan<DK, SPLIT, 1>(p, s);
}

bool bs_aligned(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace
}  // namespace edl

using namespace edl;

// q, k [T, H, DK], v [T, H, DV], beta [T, H] or null: bf16; g fp32 [T, H, DK]; state fp32 [nseq, H, DK, DV] or null; o bf16
// [T, H, DV]; rec: workspace of (T / 8 + nseq + 1) * H * 72 floats. DK 32, 64 or 128, DV up to 256; q, k, g 16-byte aligned.
EDL_HOST_API int edl_delta_rule_blocks(const void* q, const void* k, const void* v, const float* g, const void* beta,
                                       const int* cu, int T, int nseq, int H, int DK, int DV, float scale, float* state, void* o,
                                       float* rec, void* stream) {
  if (nseq <= 0 || H <= 0 || T <= 0) return 0;
  if (H > 65535 || nseq > 65535 || DV < 1 || DV > 256 || !g || !rec || !bs_aligned(rec) || !bs_aligned(q) || !bs_aligned(k) ||
      !bs_aligned(g)) {
    set_last_error("edl_delta_rule_blocks: sizes (B=%d, H=%d, DK=%d, DV=%d) or unaligned operands", nseq, H, DK, DV);
    return -1;
  }
  const BsParams p{(const __nv_bfloat16*)q, (const __nv_bfloat16*)k, (const __nv_bfloat16*)v, g, (const __nv_bfloat16*)beta, cu, T,
                   nseq, H, DV, scale, rec, state, (__nv_bfloat16*)o};
  cudaStream_t s = (cudaStream_t)stream;
  switch (DK) {
    case 32: return run_block_scan<32>(p, s);
    case 64: return run_block_scan<64>(p, s);
    case 128: return run_block_scan<128>(p, s);
  }
  set_last_error("edl_delta_rule_blocks: key head_dim %d not in {32, 64, 128}", DK);
  return -1;
}
