// Decode attention over pages of latent rows (multi-head latent attention, absorbed form).
//
// The cache holds one row [compressed key/value (L) | rotary key (R)] per token, shared by every head. With the key
// up-projection folded into the query and the value up-projection applied afterwards, a decode step is
//     s[h, t] = scale * q[h, :L+R] . row[t, :L+R],   o[h, :L] = softmax_t(s[h, :]) . row[t, :L]
// i.e. an (L+R)-wide score product and an L-wide value sum over the SAME rows: every page byte is read once per group
// of 16 heads. A sliding window starts the walk at its first tile; a learned sink joins the denominator once. One CTA
// serves one (sequence, 16-head group, key split):
//   * thread 0 streams 32-row tiles (NB 64-column boxes, 128-byte swizzle, zeros past the row's end) through a
//     four-stage ring by TMA, two tiles ahead of the consumers;
//   * warp w computes the scores of rows 8w..8w+7 of the tile (4 NB m16n8k16 bf16 products against query fragments that
//     stay in registers), the four warps agree on the tile's row maxima through shared memory, write their
//     probabilities there, and each warp accumulates its own quarter of the output columns from the whole tile, so
//     the output needs no merge across warps;
//   * with key splits the partial outputs and log-sum-exps are merged by edl_attn_combine.
// L and R are multiples of 8 with L + R <= 64 NB and L <= 512.
// Many heads and long sequences go to the tcgen05 form further down, one CTA per 128 heads and half of the value columns; where
// the CTAs of both forms fit the GPU at once, the length of each sequence decides on the device.
//
// Role of the reference's multi-latent ragged page attention for decode steps
// (easydel/operations/kernels/multi_latent_ragged_page_attention.py:282-700).
#include "common.cuh"
#include "tmem_ops.cuh"

namespace edl {
namespace {

constexpr int ML_TK = 32;              // rows per tile
constexpr int ML_WARPS = 4;
constexpr int ML_THREADS = ML_WARPS * 32;
constexpr int ML_STAGES = 4;
constexpr int ML_AHEAD = ML_STAGES - 2;
constexpr int ML_PAGE = 128;
constexpr int ML_PPITCH = ML_TK * 2 + 16;   // one row of probabilities (32 bf16) padded against bank conflicts
constexpr float ML_LOG2E = 1.4426950408889634f;

template <int NB>
struct MlCfg {
  static constexpr int W = NB * 64;                      // row width as loaded
  static constexpr int NKS = W / 16;                     // k-steps of the score product
  static constexpr int NJ = 2 * (NB < 8 ? NB : 8);       // 8-column output blocks per warp
  static constexpr int TILE_BYTES = ML_TK * W * 2;
  static constexpr int QPITCH = W * 2 + 16;
  static constexpr int OFF_Q = ML_STAGES * TILE_BYTES;
  static constexpr int OFF_P = OFF_Q + 16 * QPITCH;                // [2][16 rows][ML_PPITCH]
  static constexpr int OFF_MAX = OFF_P + 2 * 16 * ML_PPITCH;       // [2][4 warps][16] floats
  static constexpr int OFF_SUM = OFF_MAX + 2 * ML_WARPS * 16 * 4;  // [4 warps][16] floats
  static constexpr int OFF_BAR = OFF_SUM + ML_WARPS * 16 * 4;
  static constexpr int SMEM = OFF_BAR + 64 + 1024;
};

struct MlaParams {
  const __nv_bfloat16* q;   // latent part of the query: sequence b, head h at b * q_seq + h * q_head
  long long q_seq, q_head;
  const __nv_bfloat16* qr;  // rotary part, likewise
  long long qr_seq, qr_head;
  __nv_bfloat16* o;         // [splits, B, ldo]: head h at columns h * L
  long long ldo;
  float* lse;               // [splits, H, B] or null
  const int* kv_lens;
  const int* page_table;
  const float* sinks;       // [H] or null (only without splits)
  int pt_stride, B, H, splits, L, R, window;
  float scale_log2;
  int* status;
};

__device__ __forceinline__ void ml_ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ml_ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ml_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Byte offset of (row, 16-byte chunk) in a tile stored as nine boxes of [32 rows x 128 bytes], 128-byte swizzle.
__device__ __forceinline__ uint32_t ml_tile_off(int row, int chunk) {
  const int box = chunk >> 3, c = chunk & 7;
  return box * (ML_TK * 128) + row * 128 + ((c ^ (row & 7)) << 4);
}

// The first four warps meet; the tcgen05 form's CTAs have six.
__device__ __forceinline__ void ml_sync() { asm volatile("bar.sync 1, %0;" ::"n"(ML_THREADS) : "memory"); }

template <int NB>
__device__ __forceinline__ void mla_decode_simple(const CUtensorMap& tmap, const MlaParams& p, uint8_t* smem, int id) {
  using C = MlCfg<NB>;
  const uint32_t sbase = smem_u32(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int groups = (p.H + 15) / 16;
  const int split = id % p.splits;
  const int hg = (id / p.splits) % groups;
  const int b = id / (p.splits * groups);
  const int heads = min(16, p.H - hg * 16);
  const int kv_len = p.kv_lens[b];
  const int* pt = p.page_table + (long long)b * p.pt_stride;

  const int lo = p.window > 0 ? max(0, kv_len - p.window) : 0;
  const int t_first = lo / ML_TK, t_end = (kv_len + ML_TK - 1) / ML_TK;
  const int per_split = (t_end - t_first + p.splits - 1) / p.splits;
  const int t0 = t_first + split * per_split;
  const int n_tiles = max(0, min(t_end, t0 + per_split) - t0);

  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  const uint32_t bar0 = smem_u32(bars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + C::OFF_BAR + 8 * ML_STAGES);
  if (threadIdx.x == 0) {
    for (int i = 0; i < ML_STAGES; ++i) mbar_init(bar0 + 8 * i, 1);
    *abort_flag = 0;
    fence_mbar_init();
    prefetch_tmap(&tmap);
  }
  {  // this group's query rows -> shared memory (rows past the last head and columns past L + R are zero)
    const __nv_bfloat16* ql = p.q + b * p.q_seq + (long long)hg * 16 * p.q_head;
    const __nv_bfloat16* qr = p.qr + b * p.qr_seq + (long long)hg * 16 * p.qr_head;
    for (int i = threadIdx.x; i < 16 * (C::W / 8); i += ML_THREADS) {
      const int r = i / (C::W / 8), c = (i % (C::W / 8)) * 8;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (r < heads && c < p.L) v = *reinterpret_cast<const uint4*>(ql + r * p.q_head + c);
      else if (r < heads && c < p.L + p.R) v = *reinterpret_cast<const uint4*>(qr + r * p.qr_head + c - p.L);
      *reinterpret_cast<uint4*>(smem + C::OFF_Q + r * C::QPITCH + c * 2) = v;
    }
  }
  ml_sync();

  auto issue = [&](int i) {  // thread 0 only
    const int tile = t0 + i;
    const int page = pt[tile / (ML_PAGE / ML_TK)];
    const int row = page * ML_PAGE + (tile % (ML_PAGE / ML_TK)) * ML_TK;
    const int st = i % ML_STAGES;
    const uint32_t bar = bar0 + 8 * st;
    const uint32_t dst = sbase + st * C::TILE_BYTES;
    mbar_expect_tx(bar, C::TILE_BYTES);
#pragma unroll
    for (int c = 0; c < NB; ++c) tma_load_2d(dst + c * (ML_TK * 128), &tmap, bar, c * 64, row);
  };
  if (threadIdx.x == 0)
    for (int i = 0; i < min(n_tiles, ML_AHEAD); ++i) issue(i);

  // A fragments of the 16 query rows for all 36 k-steps, kept in registers
  uint32_t qa[C::NKS][4];
  {
    const uint32_t qb = sbase + C::OFF_Q;
    const int r = (lane & 7) + ((lane >> 3) & 1) * 8;
#pragma unroll
    for (int ks = 0; ks < C::NKS; ++ks) ml_ldmatrix_x4(qb + r * C::QPITCH + (ks * 2 + (lane >> 4)) * 16, qa[ks]);
  }

  float o_acc[C::NJ][4];  // this warp's quarter of the output columns: blocks of 8
#pragma unroll
  for (int j = 0; j < C::NJ; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) o_acc[j][e] = 0.f;
  float m_run[2] = {-1e30f, -1e30f};  // rows lane / 4 and lane / 4 + 8 (identical in every warp)
  float l_run[2] = {0.f, 0.f};        // this warp's share of the row sums (its 8 rows of every tile)
  float* s_max = reinterpret_cast<float*>(smem + C::OFF_MAX);
  bool alive = true;
  const int r0 = lane >> 2;

  for (int i = 0; i < n_tiles; ++i) {
    const int st = i % ML_STAGES, par = i & 1;
    // the stage refilled here held tile i - 2, which every warp finished before the first barrier of step i - 1
    if (threadIdx.x == 0 && i + ML_AHEAD < n_tiles && alive) issue(i + ML_AHEAD);
    if (alive) alive = mbar_wait(bar0 + 8 * st, (i / ML_STAGES) & 1, abort_flag, p.status, EDL_TIMEOUT_SOFTMAX);
    const uint32_t tile = sbase + st * C::TILE_BYTES;
    // ---- scores of rows 8w .. 8w+7 of the tile
    float s[4] = {0.f, 0.f, 0.f, 0.f}, s2[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    if (alive) {                      // three independent chains of products
      const int row = warp * 8 + (lane & 7);
#pragma unroll
      for (int ks = 0; ks < C::NKS; ks += 2) {
        uint32_t kb[4];
        ml_ldmatrix_x4(tile + ml_tile_off(row, ks * 2 + (lane >> 3)), kb);
        const int chain = (ks >> 1) % 3;
        if (chain == 0) {
          ml_mma(s, qa[ks], kb[0], kb[1]);
          ml_mma(s2[0], qa[ks + 1], kb[2], kb[3]);
        } else if (chain == 1) {
          ml_mma(s2[1], qa[ks], kb[0], kb[1]);
          ml_mma(s, qa[ks + 1], kb[2], kb[3]);
        } else {
          ml_mma(s2[0], qa[ks], kb[0], kb[1]);
          ml_mma(s2[1], qa[ks + 1], kb[2], kb[3]);
        }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) s[e] += s2[0][e] + s2[1][e];
    }
    const int key0 = (t0 + i) * ML_TK + warp * 8 + (lane & 3) * 2;
    float mx[2];
#pragma unroll
    for (int e = 0; e < 4; ++e) s[e] = (alive && key0 + (e & 1) < kv_len && key0 + (e & 1) >= lo) ? s[e] * p.scale_log2 : -INFINITY;
    mx[0] = fmaxf(s[0], s[1]);
    mx[1] = fmaxf(s[2], s[3]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
      mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
    }
    if ((lane & 3) == 0) {
      s_max[(par * ML_WARPS + warp) * 16 + r0] = mx[0];
      s_max[(par * ML_WARPS + warp) * 16 + r0 + 8] = mx[1];
    }
    ml_sync();
    float alpha[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float m_new = m_run[h];
#pragma unroll
      for (int w = 0; w < ML_WARPS; ++w) m_new = fmaxf(m_new, s_max[(par * ML_WARPS + w) * 16 + r0 + h * 8]);
      alpha[h] = exp2f(m_run[h] - m_new);
      m_run[h] = m_new;
      l_run[h] *= alpha[h];
    }
    {  // probabilities of this warp's 8 rows -> columns 8w .. 8w+7 of the shared [16 x 32] block
      const float e0 = exp2f(s[0] - m_run[0]), e1 = exp2f(s[1] - m_run[0]);
      const float e2 = exp2f(s[2] - m_run[1]), e3 = exp2f(s[3] - m_run[1]);
      l_run[0] += e0 + e1;
      l_run[1] += e2 + e3;
      uint8_t* pb = smem + C::OFF_P + par * 16 * ML_PPITCH + (warp * 8 + (lane & 3) * 2) * 2;
      *reinterpret_cast<uint32_t*>(pb + r0 * ML_PPITCH) = pack_bf16x2(e0, e1);
      *reinterpret_cast<uint32_t*>(pb + (r0 + 8) * ML_PPITCH) = pack_bf16x2(e2, e3);
    }
    ml_sync();
    // ---- O[:, this warp's columns] = O * alpha + P V
#pragma unroll
    for (int j = 0; j < C::NJ; ++j) {
      o_acc[j][0] *= alpha[0];
      o_acc[j][1] *= alpha[0];
      o_acc[j][2] *= alpha[1];
      o_acc[j][3] *= alpha[1];
    }
    if (alive) {
      const uint32_t pbase = sbase + C::OFF_P + par * 16 * ML_PPITCH;
#pragma unroll
      for (int t = 0; t < ML_TK / 16; ++t) {
        uint32_t pa[4];
        ml_ldmatrix_x4(pbase + ((lane & 7) + ((lane >> 3) & 1) * 8) * ML_PPITCH + (t * 2 + (lane >> 4)) * 16, pa);
#pragma unroll
        for (int j = 0; j < C::NJ; j += 2) {
          uint32_t vb[4];
          const int row = t * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
          ml_ldmatrix_x4_trans(tile + ml_tile_off(row, warp * C::NJ + j + (lane >> 4)), vb);
          ml_mma(o_acc[j], pa, vb[0], vb[1]);
          ml_mma(o_acc[j + 1], pa, vb[2], vb[3]);
        }
      }
    }
  }

  // ---- row sums over the four warps, then every warp writes its columns
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 1);
    l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 2);
  }
  float* s_sum = reinterpret_cast<float*>(smem + C::OFF_SUM);
  if ((lane & 3) == 0) {
    s_sum[warp * 16 + r0] = l_run[0];
    s_sum[warp * 16 + r0 + 8] = l_run[1];
  }
  ml_sync();
  const long long orow = (long long)split * p.B + b;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = r0 + h * 8;
    float l = 0.f;
#pragma unroll
    for (int w = 0; w < ML_WARPS; ++w) l += s_sum[w * 16 + r];
    if (r >= heads) continue;
    if (p.sinks && p.splits == 1) l += exp2f(p.sinks[hg * 16 + r] * ML_LOG2E - m_run[h]);
    const float inv = l > 0.f ? 1.f / l : 0.f;
    __nv_bfloat16* dst = p.o + orow * p.ldo + (long long)(hg * 16 + r) * p.L;
#pragma unroll
    for (int j = 0; j < C::NJ; ++j) {
      const int c = (warp * C::NJ + j) * 8;
      if (c < p.L) *reinterpret_cast<uint32_t*>(dst + c + (lane & 3) * 2) = pack_bf16x2(o_acc[j][2 * h] * inv, o_acc[j][2 * h + 1] * inv);
    }
    if (p.lse && warp == 0 && (lane & 3) == 0)
      p.lse[((long long)split * p.H + hg * 16 + r) * p.B + b] =
          l > 0.f ? (m_run[h] + log2f(l)) * 0.6931471805599453f : -INFINITY;
  }
  if (*abort_flag) {   // a wait ran out: give copies still in flight time to land before shared memory is released
    long long t0c = clock64();
    while (clock64() - t0c < 400000) {
    }
  }
}

template <int NB>
__global__ void __launch_bounds__(ML_THREADS, NB > 4 ? 1 : 2)
mla_decode_kernel(const __grid_constant__ CUtensorMap tmap, const MlaParams p) {
  extern __shared__ uint8_t smem_raw[];
  mla_decode_simple<NB>(tmap, p, reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023)), blockIdx.x);
}

template <int NB>
int launch_mla(const void* pages, long long num_pages, const MlaParams& p, cudaStream_t stream) {
  using C = MlCfg<NB>;
  const int w = p.L + p.R;
  CUtensorMap tm;
  if (make_tmap_2d_16b(&tm, pages, (uint64_t)num_pages * ML_PAGE, w, w, ML_TK, 64)) return -1;
  auto kern = mla_decode_kernel<NB>;
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!attr_set[dev]) {
    if (check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM),
                   "cudaFuncSetAttribute(mla_decode)"))
      return -1;
    attr_set[dev] = true;
  }
  const long long blocks = (long long)p.B * ((p.H + 15) / 16) * p.splits;
  kern<<<(unsigned)blocks, ML_THREADS, C::SMEM, stream>>>(tm, p);
  return check_cuda(cudaGetLastError(), "mla_decode launch");
}

// ---------------------------------------------------------------------------------------------------------------
// tcgen05 form for many heads. With 16 heads per CTA every row was read from L2 eight times for 128 heads and multiplied
// on mma.sync, two CTA-wide meetings per 32 rows. Here up to 128 heads are the M side of the products and a tile is 64
// rows: S[heads, 64] = Q row^T (36 products for 576-wide rows), O[heads, 256] += P V (8 products). O takes 256 of the 512
// tensor-memory columns, so a CTA owns half of the (up to 512) value columns and computes the scores in full: 1.5 times the
// multiplications of one pass, on a pipe that is otherwise idle, against rows that are read twice and not eight times.
//   tensor memory: S / P (parts 32 columns apart) even [0,64)  odd [64,128)   first 256 columns of Q, bf16 [128,256)   O [256,512)
//   shared memory: the other columns of Q (up to 5 boxes of 128 x 64), three stages of the half's up to 4 value boxes (64
//   rows x 64 columns, held until PV), a ring of six boxes for the columns that only the scores need
//   warp 0 loads rows; warp 1 issues S(i + 1) before PV(i), so that the softmax of tile i (warps 2..5, one thread per
//   head) runs under the scores of tile i + 1; O is rescaled only when a maximum has grown by more than 2^8. The largest
//   probability is then no longer 1, exact in bf16, so P enters as two bf16 parts (16 bits): relative error against 64
//   bits 1.66e-3, which is the rounding of the output, against 2.06e-3 with one part (32 sequences of 600 to 2000 rows)
//   and 1.99e-3 of the mma.sync form. The second part costs 4.9 of 48 us; one part and a rescale for every new maximum
//   46.2 us, but 2.07e-3 against 2.06e-3 of the mma.sync form on 100 sequences of 60 to 200 rows.
// The keys of a sequence are cut over a cluster (1 to 4 CTAs, as many as fill the SMs). Each
// sends every other one its part of that one's columns by one bulk copy between shared memories (4-byte loads from a
// neighbour ran at 6 bytes a clock) and sums the parts in rank order.
// 32 sequences of 600 to 2000 rows, 128 heads, 512 + 64 columns: 145 -> 48 us; one of 16000: 61 -> 29 us; 128 of 450 to
// 1500: 393 -> 107 us. Bound now by the products with 64 rows (N = 64 takes as long as N = 128 would: 66 clocks).
constexpr int MT_TK = 64;
constexpr int MT_THREADS = 192;
constexpr int MT_MAX_BOXES = 9;
constexpr int MT_QT_BOXES = 4;                              // boxes of Q in tensor memory
constexpr int MT_BOX = MT_TK * 128;
constexpr int MT_OWN = 4;                                   // value boxes of a half
constexpr int MT_STAGES = 3;
constexpr int MT_RING = 6;
constexpr int MT_QBOX = 128 * 128;
constexpr int MT_OFF_V = (MT_MAX_BOXES - MT_QT_BOXES) * MT_QBOX;
constexpr int MT_OFF_RING = MT_OFF_V + MT_STAGES * MT_OWN * MT_BOX;
constexpr int MT_OFF_BAR = MT_OFF_RING + MT_RING * MT_BOX;
constexpr int MT_OFF_ML = MT_OFF_BAR + 256;                  // maxima and sums of 128 heads, then the parts' weights
constexpr int MT_SMEM = MT_OFF_ML + 1024 + 512 + 1024;
constexpr int MT_PART_BYTES = 256 * 128 * 4;                // partial outputs of a CTA
constexpr int MT_MAX_PARTS = 4;                             // its own sums and the others' share of them fill the shared memory
constexpr int MT_MIN_TILES = 3;
constexpr float MT_GROWTH = 8.f;

__device__ __forceinline__ void mt_send(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "r"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ float mt_ld_peer(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

__device__ __forceinline__ void mla_decode_tc(const CUtensorMap& tmap, const CUtensorMap& tql, const CUtensorMap& tqr,
                                              const MlaParams& p, const int parts, const int halves, const int swap_l,
                                              const int swap_r, uint8_t* smem, int id) {
  const uint32_t sbase = smem_u32(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int groups = (p.H + 127) / 128;
  const int part = id % parts;
  id /= parts;
  const int half = id % halves;
  id /= halves;
  const int split = id % p.splits;
  id /= p.splits;
  const int hg = id % groups, b = id / groups;
  const int heads = min(128, p.H - hg * 128);
  const int kv_len = p.kv_lens[b];
  const int* pt = p.page_table + (long long)b * p.pt_stride;
  // boxes of a row: the latent part's, then the rotary part's, which start at column L (columns of a latent box past L
  // meet zeros of Q)
  const int nl = (p.L + 63) / 64, nb = nl + (p.R + 63) / 64;
  const int v0 = half * MT_OWN, v1 = min(v0 + MT_OWN, nl);   // this half's value boxes
  const int n_own = v1 - v0, n_other = nb - n_own;

  const int lo = p.window > 0 ? max(0, kv_len - p.window) : 0;
  const int t_first = lo / MT_TK, t_end = (kv_len + MT_TK - 1) / MT_TK;
  const int per_split = (t_end - t_first + p.splits - 1) / p.splits;
  // A part of fewer than MT_MIN_TILES tiles costs more to bring together than it saves (every CTA of a cluster sees the same)
  int act = parts;
  while (act > 1 && per_split < act * MT_MIN_TILES) act >>= 1;
  if (part >= act) {
    if (act > 1) {
      cluster_sync_all();
      cluster_sync_all();
    }
    return;
  }
  const int s0 = t_first + split * per_split, s1 = min(t_end, s0 + per_split), per = (per_split + act - 1) / act;
  const int t0 = s0 + part * per;
  const int n = max(0, min(s1, t0 + per) - t0);

  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + MT_OFF_BAR);
  const uint32_t b_fullA = smem_u32(bars);           // [MT_RING]
  const uint32_t b_emptyA = b_fullA + 8 * MT_RING;   // [MT_RING]
  const uint32_t b_fullV = b_emptyA + 8 * MT_RING;   // [MT_STAGES]
  const uint32_t b_emptyV = b_fullV + 8 * MT_STAGES; // [MT_STAGES]
  const uint32_t b_s = b_emptyV + 8 * MT_STAGES;     // [2] scores ready
  const uint32_t b_p = b_s + 16;                     // [2] probabilities written
  const uint32_t b_pv = b_p + 16;                    // [2] PV product of an even / odd tile done
  const uint32_t b_q = b_pv + 16;
  const uint32_t b_x = b_q + 8;                      // the other CTAs' shares have arrived
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * MT_RING + 2 * MT_STAGES + 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t vring = sbase + MT_OFF_V, ring = sbase + MT_OFF_RING;

  // thread 0 only
  auto row_of = [&](int i) {
    const int tile = t0 + i;
    return i < n ? pt[tile / (ML_PAGE / MT_TK)] * ML_PAGE + (tile % (ML_PAGE / MT_TK)) * MT_TK : 0;
  };
  auto column = [&](int c) { return c < nl ? c * 64 : p.L + (c - nl) * 64; };
  auto load_own = [&](int i, int row) {
    const int st = i % MT_STAGES;
    mbar_expect_tx(b_fullV + 8 * st, n_own * MT_BOX);
    for (int c = v0; c < v1; ++c)
      tma_load_2d(vring + (st * MT_OWN + c - v0) * MT_BOX, &tmap, b_fullV + 8 * st, column(c), row);
  };
  auto load_other = [&](int i, int j, int row) {     // the j-th of tile i's boxes that only the scores need
    const int c = j < v0 ? j : j + n_own, slot = (i * n_other + j) % MT_RING;
    mbar_expect_tx(b_fullA + 8 * slot, MT_BOX);
    tma_load_2d(ring + slot * MT_BOX, &tmap, b_fullA + 8 * slot, column(c), row);
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < MT_RING; ++i) {
      mbar_init(b_fullA + 8 * i, 1);
      mbar_init(b_emptyA + 8 * i, 1);
    }
    for (int i = 0; i < MT_STAGES; ++i) {
      mbar_init(b_fullV + 8 * i, 1);
      mbar_init(b_emptyV + 8 * i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(b_s + 8 * i, 1);
      mbar_init(b_p + 8 * i, 128);
      mbar_init(b_pv + 8 * i, 1);
    }
    mbar_init(b_q, 1);
    mbar_init(b_x, 1);
    *abort_flag = 0;
    fence_mbar_init();
    // Q: the first boxes pass through value stages 1 and 2 on their way to tensor memory, the others stay in shared memory
    mbar_expect_tx(b_q, nb * MT_QBOX);
    for (int c = 0; c < nb; ++c) {
      const bool swap = c < nl ? swap_l : swap_r;
      tma_load_3d(c < MT_QT_BOXES ? vring + MT_OWN * MT_BOX + c * MT_QBOX : sbase + (c - MT_QT_BOXES) * MT_QBOX,
                  c < nl ? &tql : &tqr, b_q, (c < nl ? c : c - nl) * 64, swap ? b : hg * 128, swap ? hg * 128 : b);
    }
    if (n > 0) {
      const int row = row_of(0);
      load_own(0, row);
      for (int j = 0; j < min(n_other, MT_RING); ++j) load_other(0, j, row);   // a half can need more boxes than the ring has
    }
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tQ = tmem + 128, tO = tmem + 256;

  if (warp >= 2 && __all_sync(0xffffffffu, mbar_wait(b_q, 0, abort_flag, p.status, EDL_TIMEOUT_SOFTMAX))) {
    const int q = warp & 3, r = q * 32 + lane;
    const uint8_t* src = smem + MT_OFF_V + MT_OWN * MT_BOX + r * 128;
#pragma unroll 1
    for (int c = 0; c < min(nb, MT_QT_BOXES); ++c) {
      uint32_t x[32];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint4 v = *reinterpret_cast<const uint4*>(src + c * MT_QBOX + ((j ^ (r & 7)) << 4));
        x[4 * j] = v.x, x[4 * j + 1] = v.y, x[4 * j + 2] = v.z, x[4 * j + 3] = v.w;
      }
      tmem_st_32x32b_x32(tQ + (uint32_t(q * 32) << 16) + c * 32, x);
    }
    tc_wait_st();
    fence_proxy_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  float m_ref = -1e30f, l = 0.f;
  bool alive = true;
  if (warp == 0) {
    if (lane == 0) {
      int row = row_of(0);
      bool ok = true;
      for (int i = 0; i < n && ok; ++i) {
        const int next = row_of(i + 1);              // read a tile ahead of its use
        if (i > 0) {
          if (i >= MT_STAGES)
            ok = mbar_wait(b_emptyV + 8 * (i % MT_STAGES), (i / MT_STAGES - 1) & 1, abort_flag, p.status, EDL_TIMEOUT_PRODUCER);
          if (!ok) break;
          load_own(i, row);
        }
        for (int j = i > 0 ? 0 : MT_RING; j < n_other && ok; ++j) {
          const int u = i * n_other + j;
          if (u >= MT_RING)
            ok = mbar_wait(b_emptyA + 8 * (u % MT_RING), (u / MT_RING - 1) & 1, abort_flag, p.status, EDL_TIMEOUT_PRODUCER);
          if (ok) load_other(i, j, row);
        }
        row = next;
      }
    }
  } else if (warp == 1) {
    const bool leader = elect_one();
    const uint32_t id_s = umma_idesc_bf16(128, MT_TK, 0, 0), id_o = umma_idesc_bf16(128, n_own * 64, 0, 1);
    auto score_box = [&](int i, int c, uint32_t kb, bool first) {
      if (leader) {
        const uint32_t d = tmem + (i & 1) * 64, acc = first ? 0u : 1u;
        const uint64_t bd = umma_smem_desc_sw128(kb, 16, 1024);      // 32 bytes further: 2 in its address field
        if (c < MT_QT_BOXES) {
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_f16_ts(d, tQ + c * 32 + k * 8, bd + 2 * k, id_s, k ? 1u : acc);
        } else {
          const uint64_t ad = umma_smem_desc_sw128(sbase + (c - MT_QT_BOXES) * MT_QBOX, 16, 1024);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_f16_ss(d, ad + 2 * k, bd + 2 * k, id_s, k ? 1u : acc);
        }
      }
      __syncwarp();
    };
    auto issue_s = [&](int i) -> bool {
      for (int j = 0; j < n_other; ++j) {
        const int u = i * n_other + j, slot = u % MT_RING;
        if (!mbar_wait(b_fullA + 8 * slot, (u / MT_RING) & 1, abort_flag, p.status, EDL_TIMEOUT_MMA)) return false;
        tc_fence_after();
        score_box(i, j < v0 ? j : j + n_own, ring + slot * MT_BOX, j == 0);
        if (leader) tc_commit(b_emptyA + 8 * slot);
      }
      const int st = i % MT_STAGES;
      if (!mbar_wait(b_fullV + 8 * st, (i / MT_STAGES) & 1, abort_flag, p.status, EDL_TIMEOUT_MMA)) return false;
      tc_fence_after();
      for (int c = v0; c < v1; ++c)
        score_box(i, c, vring + (st * MT_OWN + c - v0) * MT_BOX, n_other == 0 && c == v0);
      if (leader) tc_commit(b_s + 8 * (i & 1));
      return true;
    };
    bool ok = n > 0 && issue_s(0);
    for (int i = 0; i < n && ok; ++i) {
      if (i + 1 < n && !issue_s(i + 1)) break;
      if (!mbar_wait(b_p + 8 * (i & 1), (i >> 1) & 1, abort_flag, p.status, EDL_TIMEOUT_MMA)) break;
      tc_fence_after();
      const uint32_t vb = vring + (i % MT_STAGES) * MT_OWN * MT_BOX;
#pragma unroll
      for (int k = 0; k < MT_TK / 16; ++k)
        if (leader)
#pragma unroll
          for (int part = 0; part < 2; ++part)
            umma_f16_ts(tO, tmem + (i & 1) * 64 + part * 32 + k * 8, umma_smem_desc_sw128(vb + k * 2048, MT_BOX, 1024), id_o,
                        (i | k | part) != 0 ? 1u : 0u);
      if (leader) {
        tc_commit(b_emptyV + 8 * (i % MT_STAGES));
        tc_commit(b_pv + 8 * (i & 1));
      }
    }
  } else {
    const uint32_t row_sel = uint32_t((warp & 3) * 32) << 16;
    for (int i = 0; i < n; ++i) {
      alive = mbar_wait(b_s + 8 * (i & 1), (i >> 1) & 1, abort_flag, p.status, EDL_TIMEOUT_SOFTMAX);
      alive = __all_sync(0xffffffffu, alive);
      if (!alive) break;
      tc_fence_after();
      uint32_t s[64];
      tmem_ld_32x32b_x64(tmem + (i & 1) * 64 + row_sel, s);
      tc_wait_ld();
      const int key0 = (t0 + i) * MT_TK;
      float x[64];
#pragma unroll
      for (int e = 0; e < 64; e += 2)
        mul2(x[e], x[e + 1], __uint_as_float(s[e]), __uint_as_float(s[e + 1]), p.scale_log2, p.scale_log2);
      if (key0 + MT_TK > kv_len || key0 < lo) {
#pragma unroll
        for (int e = 0; e < 64; ++e)
          if (key0 + e >= kv_len || key0 + e < lo) x[e] = -INFINITY;
      }
      float mx[4] = {x[0], x[1], x[2], x[3]};
#pragma unroll
      for (int e = 4; e < 64; ++e) mx[e & 3] = fmaxf(mx[e & 3], x[e]);
      const float m = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      if (i == 0) {
        m_ref = fmaxf(m_ref, m);
      } else if (__any_sync(0xffffffffu, m > m_ref + MT_GROWTH)) {
        // the barrier of tile i - 1 is at most one phase ahead of tile i - 3, whose product came before S(i - 1)
        alive = mbar_wait(b_pv + 8 * ((i - 1) & 1), ((i - 1) >> 1) & 1, abort_flag, p.status, EDL_TIMEOUT_SOFTMAX);
        alive = __all_sync(0xffffffffu, alive);
        if (!alive) break;
        tc_fence_after();
        const float m_new = fmaxf(m_ref, m), f = exp2f(m_ref - m_new);
        m_ref = m_new;
        l *= f;
#pragma unroll 1
        for (int c = 0; c < n_own * 64; c += 32) {
          uint32_t o[32];
          tmem_ld_32x32b_x32(tO + row_sel + c, o);
          tc_wait_ld();
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
          tmem_st_32x32b_x32(tO + row_sel + c, o);
        }
        tc_wait_st();
      }
      uint32_t pk[32], pl[32];
      float ls[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int e = 0; e < 64; e += 2) {
        const float e0 = exp2f(x[e] - m_ref), e1 = exp2f(x[e + 1] - m_ref);
        ls[e & 2] += e0;
        ls[(e & 2) + 1] += e1;
        pk[e >> 1] = pack_bf16x2(e0, e1);
        pl[e >> 1] = pack_bf16x2(e0 - __uint_as_float(pk[e >> 1] << 16), e1 - __uint_as_float(pk[e >> 1] & 0xffff0000u));
      }
      l += (ls[0] + ls[1]) + (ls[2] + ls[3]);
      tmem_st_32x32b_x32(tmem + (i & 1) * 64 + row_sel, pk);
      tmem_st_32x32b_x32(tmem + (i & 1) * 64 + 32 + row_sel, pl);
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(b_p + 8 * (i & 1));
    }
    if (alive && n > 0) {
      alive = mbar_wait(b_pv + 8 * ((n - 1) & 1), ((n - 1) >> 1) & 1, abort_flag, p.status, EDL_TIMEOUT_EPILOGUE);
      alive = __all_sync(0xffffffffu, alive);
      tc_fence_after();
    }
  }
  __syncwarp();

  // Outputs -> shared memory from its start (Q and every loaded row have been consumed), 1 KB per head with its 16-byte
  // pieces XOR-ed by the head; a CTA of a cluster finishes 128 / act heads, whose sums the others send behind its own.
  const int rows = 128 / act, row0 = part * rows;
  const int width = min(n_own * 64, p.L - v0 * 64);          // value columns of this half
  float* po = reinterpret_cast<float*>(smem);
  float* pm = reinterpret_cast<float*>(smem + MT_OFF_ML);
  if (warp >= 2 && alive) {
    const int r = (warp & 3) * 32 + lane;
    const uint32_t src = tO + (uint32_t((warp & 3) * 32) << 16);
#pragma unroll 1
    for (int c = 0; c < n_own * 64; c += 32) {
      uint32_t o[32];
      if (n > 0) {
        tmem_ld_32x32b_x32(src + c, o);
        tc_wait_ld();
      } else {
#pragma unroll
        for (int e = 0; e < 32; ++e) o[e] = 0u;
      }
#pragma unroll
      for (int e = 0; e < 8; ++e)
        *reinterpret_cast<uint4*>(po + r * 256 + (((c >> 2) + e) ^ (r & 7)) * 4) =
            make_uint4(o[4 * e], o[4 * e + 1], o[4 * e + 2], o[4 * e + 3]);
    }
    pm[r] = m_ref;
    pm[128 + r] = l;
    fence_proxy_async_smem();
  }
  tc_fence_before();
  if (act > 1) {
    if (threadIdx.x == 0) mbar_expect_tx(b_x, (act - 1) * rows * 1024);
    __syncwarp();
    cluster_sync_all();
    if (threadIdx.x == 0)
      for (int j = 1; j < act; ++j) {
        const int to = (part + j) % act;                     // slot of part s at CTA `to`: (s - to - 1) mod act
        mt_send(mapa_shared(sbase + MT_PART_BYTES + (act - j - 1) * rows * 1024, to), sbase + to * rows * 1024, rows * 1024,
                mapa_shared(b_x, to));
      }
    __syncwarp();
  } else {
    __syncthreads();
  }
  const bool fine = *abort_flag == 0;
  float* pw = reinterpret_cast<float*>(smem + MT_OFF_ML + 1024);   // [head of this CTA][part] weight over the denominator
  const long long orow = (long long)split * p.B + b;
  if (threadIdx.x < rows && fine) {
    const int r = row0 + threadIdx.x, head = hg * 128 + r;
    float w[MT_MAX_PARTS], mm = -1e30f, sum = 0.f;
    const uint32_t ml = sbase + MT_OFF_ML + r * 4;
#pragma unroll
    for (int j = 0; j < MT_MAX_PARTS; ++j)
      if (j < act) {
        w[j] = act > 1 ? mt_ld_peer(mapa_shared(ml, j)) : pm[r];
        mm = fmaxf(mm, w[j]);
      }
#pragma unroll
    for (int j = 0; j < MT_MAX_PARTS; ++j)
      if (j < act) {
        w[j] = exp2f(w[j] - mm);
        sum += w[j] * (act > 1 ? mt_ld_peer(mapa_shared(ml + 512, j)) : pm[128 + r]);
      }
    float den = sum;
    if (r < heads) {
      if (p.sinks && p.splits == 1) den += exp2f(p.sinks[head] * ML_LOG2E - mm);
      if (p.lse && half == 0)
        p.lse[((long long)split * p.H + head) * p.B + b] = sum > 0.f ? (mm + log2f(sum)) * 0.6931471805599453f : -INFINITY;
    }
    const float inv = den > 0.f ? 1.f / den : 0.f;
#pragma unroll
    for (int j = 0; j < MT_MAX_PARTS; ++j)
      if (j < act) pw[threadIdx.x * act + j] = w[j] * inv;
  }
  __syncthreads();
  if (fine && (act == 1 || mbar_wait(b_x, 0, abort_flag, p.status, EDL_TIMEOUT_EPILOGUE))) {
    const int c = lane * 8;
#pragma unroll 1
    for (int i = warp; i < rows && row0 + i < heads; i += MT_THREADS / 32) {
      const int r = row0 + i;
      const int piece = ((2 * lane) ^ (r & 7)) * 4, piece2 = ((2 * lane + 1) ^ (r & 7)) * 4;
      float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < MT_MAX_PARTS; ++j)
        if (j < act) {
          const float* src = j == part ? po + r * 256 : po + (128 + ((j - part - 1 + act) % act) * rows + i) * 256;
          const float4 x = *reinterpret_cast<const float4*>(src + piece), y = *reinterpret_cast<const float4*>(src + piece2);
          const float w = pw[i * act + j];
          v[0] = fmaf(w, x.x, v[0]), v[1] = fmaf(w, x.y, v[1]), v[2] = fmaf(w, x.z, v[2]), v[3] = fmaf(w, x.w, v[3]);
          v[4] = fmaf(w, y.x, v[4]), v[5] = fmaf(w, y.y, v[5]), v[6] = fmaf(w, y.z, v[6]), v[7] = fmaf(w, y.w, v[7]);
        }
      if (c < width)
        *reinterpret_cast<uint4*>(p.o + orow * p.ldo + (long long)(hg * 128 + r) * p.L + v0 * 64 + c) = make_uint4(
            pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
    }
  }
  __syncwarp();
  if (*abort_flag) {   // a wait ran out: give copies still in flight time to land before shared memory is released
    const long long t0c = clock64();
    while (clock64() - t0c < 400000) {
    }
  }
  tc_fence_before();
  __syncthreads();
  if (act > 1) cluster_sync_all();   // no CTA leaves while another may still read its maxima and sums
  if (warp == 1) tmem_dealloc(tmem, 512);
}

__global__ void __launch_bounds__(MT_THREADS, 1)
mla_decode_tc_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ CUtensorMap tql,
                     const __grid_constant__ CUtensorMap tqr, const MlaParams p, const int parts, const int halves,
                     const int swap_l, const int swap_r) {
  extern __shared__ uint8_t smem_raw[];
  mla_decode_tc(tmap, tql, tqr, p, parts, halves, swap_l, swap_r,
                reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023)), blockIdx.x);
}

// What either form takes for one round of its CTAs, in us: see mla_takes_tc.
__host__ __device__ inline float mla_time_simple(long long seen, int splits) {
  const long long tiles = (seen + ML_TK - 1) / ML_TK;
  return 5.f + 1.4f * ((tiles + splits - 1) / splits);
}
__host__ __device__ inline float mla_time_tc(long long seen, int splits, int parts) {
  const long long tiles = (seen + MT_TK - 1) / MT_TK, mine = (tiles + splits - 1) / splits;
  int act = parts;
  while (act > 1 && mine < act * MT_MIN_TILES) act >>= 1;
  return (act > 1 ? 12.5f : 10.f) + 2.f * ((mine + act - 1) / act);
}

// Either form, by the length of the sequence, where the CTAs of both fit the GPU at once: a page table has room for the longest
// sequence there can be, so the host does not know, and a captured step keeps its launches while the sequences grow. A sequence
// has `slots` CTAs, as many as the form that needs more of them takes; the others leave.
template <int NB>
__global__ void __launch_bounds__(MT_THREADS, 1)
mla_decode_either_kernel(const __grid_constant__ CUtensorMap tsimple, const __grid_constant__ CUtensorMap tmap,
                         const __grid_constant__ CUtensorMap tql, const __grid_constant__ CUtensorMap tqr, const MlaParams p,
                         const int parts, const int halves, const int swap_l, const int swap_r, const int slots) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int b = blockIdx.x / slots, i = blockIdx.x - b * slots;
  const int kv_len = p.kv_lens[b], seen = p.window > 0 ? min(kv_len, p.window) : kv_len;
  if (mla_time_simple(seen, p.splits) <= mla_time_tc(seen, p.splits, parts)) {
    const int mine = (p.H + 15) / 16 * p.splits;
    if (i < mine && threadIdx.x < ML_THREADS) mla_decode_simple<NB>(tsimple, p, smem, b * mine + i);
  } else {
    const int mine = (p.H + 127) / 128 * p.splits * halves * parts;
    if (i < mine) mla_decode_tc(tmap, tql, tqr, p, parts, halves, swap_l, swap_r, smem, b * mine + i);
  }
}

// CTAs of a cluster that share a (sequence, 128 heads, half, split): as many as the SMs take at once.
int mla_parts(const MlaParams& p) {
  const long long ctas = (long long)p.B * ((p.H + 127) / 128) * (p.L > 256 ? 2 : 1) * p.splits;
  int parts = 1;
  while (parts < MT_MAX_PARTS && ctas * parts * 2 <= sm_count()) parts *= 2;
  return parts;
}

// Which form is the faster one, from sizes alone (the table's width bounds the keys): a fixed cost and a time per tile of 32
// (64) rows, times the rounds the CTAs take. Fitted to both on one B200: the mma.sync form starts in 5 us and takes 1.4 us
// a tile, this one 10 (12.5 over a cluster) and 2. Where the two are close so are the measurements (16 sequences of 200 to 700
// rows, 24 heads, 4 splits: 17.2 against 17.8 us; 64 of 90 to 300, 20 heads: 19.3 against 18.1).
bool mla_tc_supports(const MlaParams& p) {
  return (p.L + 63) / 64 + (p.R + 63) / 64 <= MT_MAX_BOXES && !(p.ldo & 7) && !(reinterpret_cast<uintptr_t>(p.o) & 15);
}
bool mla_takes_tc(const MlaParams& p) {
  const long long sms = sm_count(), keys = (long long)p.pt_stride * ML_PAGE;
  const long long seen = p.window > 0 && p.window < keys ? p.window : keys;
  auto rounds = [&](long long ctas) { return (double)((ctas + sms - 1) / sms); };
  const int parts = mla_parts(p);
  const double simple = 5.0 + (mla_time_simple(seen, p.splits) - 5.0) * rounds((long long)p.B * ((p.H + 15) / 16) * p.splits);
  const double here = 10.0 + (mla_time_tc(seen, p.splits, parts) - 10.0) *
                                 rounds((long long)p.B * ((p.H + 127) / 128) * (p.L > 256 ? 2 : 1) * p.splits * parts);
  return here < simple;
}
// CTAs of a sequence in the launch that can take either form, 0 where they do not all fit the GPU at once.
int mla_either_slots(const MlaParams& p) {
  const int parts = mla_parts(p), halves = p.L > 256 ? 2 : 1;
  const long long simple = (long long)(p.H + 15) / 16 * p.splits, tc = (long long)(p.H + 127) / 128 * p.splits * halves * parts;
  const long long slots = ((simple > tc ? simple : tc) + parts - 1) / parts * parts;
  return slots * p.B <= sm_count() ? (int)slots : 0;
}

// NB: of the mma.sync form where a launch can take either, else 0.
template <int NB>
int launch_mla_tc(const void* pages, long long num_pages, const MlaParams& p, cudaStream_t stream) {
  CUtensorMap ts, tm, tql, tqr;
  const int w = p.L + p.R;
  if (make_tmap_2d_16b(&tm, pages, (uint64_t)num_pages * ML_PAGE, w, w, MT_TK, 64)) return -1;
  if (NB > 0 && make_tmap_2d_16b(&ts, pages, (uint64_t)num_pages * ML_PAGE, w, w, ML_TK, 64)) return -1;
  // queries as [sequence][head][column] or, where heads lie further apart than sequences, [head][sequence][column]
  const bool swap_l = p.B > 1 && p.q_seq < p.q_head, swap_r = p.B > 1 && p.qr_seq < p.qr_head;
  auto map_q = [&](CUtensorMap* m, const void* base, int cols, long long seq, long long head, bool swap) {
    if (p.B == 1) seq = head * p.H;
    return swap ? make_tmap_3d_16b(m, base, cols, p.B, p.H, seq, head, 64, 1, 128, 3)
                : make_tmap_3d_16b(m, base, cols, p.H, p.B, head, seq, 64, 128, 1, 3);
  };
  if (map_q(&tql, p.q, p.L, p.q_seq, p.q_head, swap_l)) return -1;
  tqr = tql;
  if (p.R > 0 && map_q(&tqr, p.qr, p.R, p.qr_seq, p.qr_head, swap_r)) return -1;
  const void* kern = reinterpret_cast<const void*>(mla_decode_tc_kernel);
  if constexpr (NB > 0) kern = reinterpret_cast<const void*>(mla_decode_either_kernel<NB>);
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!attr_set[dev]) {
    if (check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MT_SMEM),
                   "cudaFuncSetAttribute(mla_decode_tc)"))
      return -1;
    attr_set[dev] = true;
  }
  const int halves = p.L > 256 ? 2 : 1, parts = mla_parts(p);
  const long long ctas = (long long)p.B * ((p.H + 127) / 128) * halves * p.splits * parts;
  const int slots = NB > 0 ? mla_either_slots(p) : 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(NB > 0 ? (long long)slots * p.B : ctas), 1, 1);
  cfg.blockDim = dim3(MT_THREADS, 1, 1);
  cfg.dynamicSmemBytes = MT_SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = parts;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaError_t e;
  if constexpr (NB > 0)
    e = cudaLaunchKernelEx(&cfg, mla_decode_either_kernel<NB>, ts, tm, tql, tqr, p, parts, halves, (int)swap_l, (int)swap_r, slots);
  else
    e = cudaLaunchKernelEx(&cfg, mla_decode_tc_kernel, tm, tql, tqr, p, parts, halves, (int)swap_l, (int)swap_r);
  return check_cuda(e, "mla_decode_tc launch");
}

template <int NB>
int launch_mla_sized(const void* pages, long long num_pages, const MlaParams& p, cudaStream_t s) {
  static_assert(MlCfg<NB>::SMEM <= MT_SMEM, "");
  if (mla_tc_supports(p) && mla_takes_tc(p))
    return mla_either_slots(p) ? launch_mla_tc<NB>(pages, num_pages, p, s) : launch_mla_tc<0>(pages, num_pages, p, s);
  return launch_mla<NB>(pages, num_pages, p, s);
}

}  // namespace
}  // namespace edl

using namespace edl;

// q: latent part (L) of the absorbed queries, head h of sequence b at b * q_seq + h * q_head; qr: their rotated rotary
// part (R), likewise. pages: [num_pages, 128, L + R] bf16 rows (compressed key/value | rotated rotary key).
// o: [splits, B, ldo] bf16, head h at columns [h * L, (h + 1) * L): softmax-weighted sums of the rows' first L columns;
// lse: [splits, H, B] fp32 natural log-sum-exp without the sinks (required when splits > 1, may be null otherwise).
// kv_lens [B], page_table [B, pt_stride] int32; window: 0 or the number of latest keys a query sees (itself included);
// sinks [H] fp32 or null: an extra logit in every denominator (applied here with one split, by edl_attn_combine with
// more). scale multiplies the (L + R)-wide dot products.
EDL_HOST_API int edl_attn_mla_decode(const void* q, long long q_seq, long long q_head, const void* qr, long long qr_seq,
                                     long long qr_head, const void* pages, void* o, float* lse, long long ldo,
                                     const int* kv_lens, const int* page_table, int pt_stride, int B,
                                     long long num_pages, int H, int L, int R, float scale, int window,
                                     const float* sinks, int splits, int* status, void* stream) {
  if (B <= 0 || H <= 0) return 0;
  if (L < 8 || L > 512 || R < 0 || L + R > 576 || (L & 7) || (R & 7)) {
    set_last_error("edl_attn_mla_decode: rows of multiples of 8, latent up to 512 and 576 in all (L=%d, R=%d)", L, R);
    return -1;
  }
  if (splits < 1 || (splits > 1 && !lse) || ((q_seq | q_head | qr_seq | qr_head) & 7) || (ldo & 1) ||
      ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(qr)) & 15) || (reinterpret_cast<uintptr_t>(o) & 3)) {
    set_last_error("edl_attn_mla_decode: splits=%d needs lse; query pitches must be multiples of 8, 16-byte aligned",
                   splits);
    return -1;
  }
  MlaParams p{reinterpret_cast<const __nv_bfloat16*>(q), q_seq, q_head, reinterpret_cast<const __nv_bfloat16*>(qr), qr_seq,
              qr_head, reinterpret_cast<__nv_bfloat16*>(o), ldo, lse, kv_lens, page_table, sinks, pt_stride, B, H, splits,
              L, R, window, scale * ML_LOG2E, status};
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  switch ((L + R + 63) / 64) {
    case 1: return launch_mla_sized<1>(pages, num_pages, p, s);
    case 2: return launch_mla_sized<2>(pages, num_pages, p, s);
    case 3: return launch_mla_sized<3>(pages, num_pages, p, s);
    case 4: return launch_mla_sized<4>(pages, num_pages, p, s);
    case 5: return launch_mla_sized<5>(pages, num_pages, p, s);
    case 6: return launch_mla_sized<6>(pages, num_pages, p, s);
    case 7: return launch_mla_sized<7>(pages, num_pages, p, s);
    case 8: return launch_mla_sized<8>(pages, num_pages, p, s);
    default: return launch_mla_sized<9>(pages, num_pages, p, s);
  }
}
