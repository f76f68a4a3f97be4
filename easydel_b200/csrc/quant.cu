// Weight-only quantised linears: code-book dequantisation and a skinny fused dequant-GEMV.
//
// Every supported format (int8, affine 4/8-bit, nf4, mxfp4, nvfp4, mxfp8, nvfp8) is stored the same way:
//   codes  [N, K * bits / 8] uint8   (4-bit codes: two per byte, low nibble = even k)
//   scales [N, K / group] bf16       (already decoded from e8m0 / e4m3 where the format uses those)
//   zeros  [N, K / group] bf16       (affine formats only, else null)
//   lut    float[1 << bits]          (code -> value before scaling: the format's number system)
// so that  w[n, k] = lut[code[n, k]] * scales[n, k / group] (+ zeros[n, k / group]).
//
//   edl_dequant_bf16 : materialises bf16 weights (prefill / training path, followed by the tcgen05 GEMM).
//   edl_qgemv        : y[M, N] = x[M, K] * W^T for a few rows (decode steps), the weights read once as codes.
// Counterpart in the reference: ejkernel quantized_matmul reached from
// easydel/layers/linears/_linear_quantized.py:1030-1108.
#include "common.cuh"

namespace edl {
namespace {

// One thread per 8 neighbouring weights: a 16-byte store, whole lines per warp. 28672 x 4096 nf4: 800 us with one thread per
// 32 weights and 2-byte stores, 81 us now (2 bytes written and half a byte read per weight).
template <int BITS>
__global__ void dequant_kernel(const uint8_t* __restrict__ codes, const __nv_bfloat16* __restrict__ scales,
                               const __nv_bfloat16* __restrict__ zeros, const float* __restrict__ lut, int N, int K,
                               int group, __nv_bfloat16* __restrict__ out, long long ldo) {
  __shared__ float s_lut[1 << BITS];
  for (int i = threadIdx.x; i < (1 << BITS); i += blockDim.x) s_lut[i] = lut[i];
  __syncthreads();
  const int vecs = K / 8, groups = K / group;
  const bool wide = (ldo & 7) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  const bool small = (long long)N * vecs < (1LL << 32);
  const bool pairs = (reinterpret_cast<uintptr_t>(codes) & 7) == 0;      // 8-bit codes may start on 4 bytes only
  for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < (long long)N * vecs;
       v += (long long)gridDim.x * blockDim.x) {
    const long long n = small ? (uint32_t)v / (uint32_t)vecs : v / vecs;
    const int k0 = (int)(v - n * vecs) * 8;
    uint32_t w[2];
    if (BITS == 4) {
      w[0] = reinterpret_cast<const uint32_t*>(codes)[v];
    } else {
      const uint32_t* at = reinterpret_cast<const uint32_t*>(codes) + 2 * v;
      const uint2 t = pairs ? *reinterpret_cast<const uint2*>(at) : make_uint2(at[0], at[1]);
      w[0] = t.x, w[1] = t.y;
    }
    float f[8], sc = 0.f, zr = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i == 0 || (group & 7)) {                         // groups are multiples of 8, or smaller than that
        const long long g = n * groups + (k0 + i) / group;
        sc = __bfloat162float(__ldg(scales + g));
        zr = zeros ? __bfloat162float(__ldg(zeros + g)) : 0.f;
      }
      const uint32_t code = BITS == 4 ? (w[0] >> (4 * i)) & 0xF : (w[i >> 2] >> ((i & 3) * 8)) & 0xFF;
      f[i] = s_lut[code] * sc + zr;
    }
    __nv_bfloat16* o = out + n * ldo + k0;
    if (wide) {
      *reinterpret_cast<uint4*>(o) = make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]),
                                                pack_bf16x2(f[6], f[7]));
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] = __float2bfloat16(f[i]);
    }
  }
}

// y[M, N] = x[M, K] W^T for a few rows (M <= 16). The weights cross HBM once at 4 or 8 bits per value; what the time goes to
// beside that is turning codes into operands, so the kernel is built around the shared-memory reads that takes:
//  * a warp owns 16 weight rows, the m side of mma.m16n8k16; the activation rows (8 per n tile) are the other. The order of
//    k inside a product is free as long as both operands agree, so codes go straight into registers: a block is 16 bytes of
//    rows g and g + 8 per lane (g = lane / 4), three blocks in flight per warp, and two code bytes are a step's A fragments.
//    Where a scale group is smaller than the 64 bytes that the four lanes of a row cover, they trade words (a 4 x 4
//    transpose by shuffles), after which the word j of all four lies within bytes 16 j to 16 j + 15 of the block.
//  * a 4-bit code byte holds two neighbouring k of one row: one 8-byte read of a table of 256 entries (16 copies, one per
//    pair of banks) gives both values as bf16 pairs of their leading and of their remaining bits, which enter as two
//    products, so that code books of fp32 values (nf4) keep 16 bits. Code books that are exact in bf16 skip the second. The
//    error against 64 bits is that of fp32 code books on the FMA pipe to five digits (22016 x 4160, 1 row: 1.6579e-3 both,
//    the output's rounding to bf16); a third part would cost a third more time (28672 x 4096, 4 rows: 44 -> 59 us).
//    8-bit codes take one 4-byte read each for both parts.
//  * activations are staged once per CTA in the order the fragments are read in (one 16-byte read per two steps).
//  * a run (the part of a block in one group) is scaled into fp32 sums in the accumulator layout; zero points multiply the
//    run's sum of activations, which a product with ones gives in the same layout. Scales are read four blocks at a time,
//    one block's by each of a row's four lanes.
// The reduction is cut over a cluster whose sums meet in rank order; rows per CTA and parts are chosen so that the warps of
// all SMs have the same work (launch_qgemv).
// nf4 in groups of 64, 4 rows, us (before: one warp per 16 rows with codes staged by TMA, or 4 rows per warp on the FMA pipe):
// 4096 x 14336 75 -> 25, 4096 x 4096 27 -> 13, 6144 x 4096 27 -> 16.7, 28672 x 4096 48 -> 44; int8 28672 x 4096 105 -> 47.
// 16 rows, against expanding the weights first: 28672 x 4096 858 -> 83. Bound by the latency of a warp's block (1.1
// thousand clocks: table reads, then a chain of products), at 1 to 2.5 TB/s.
constexpr int QG_DEPTH = 3;
constexpr int QG_MAX_M = 16;
constexpr int QG_MAX_CLUSTER = 8;
constexpr int QG_TABLE_BYTES = 256 * 128;
constexpr int QG_SMEM_MAX = 216 * 1024;
constexpr int QG_PASS_WARPS = 8;                            // of a CTA that takes row tiles in turn
constexpr int QG_PASS_BYTES = 8 * 16 * QG_PASS_WARPS * 4;   // its sums of one pass

struct QgParams {
  const __nv_bfloat16* x;
  long long ldx;
  const uint8_t* codes;
  const __nv_bfloat16* scales;
  const __nv_bfloat16* zeros;
  const float* lut;
  __nv_bfloat16* out;
  long long ldo;
  const __nv_bfloat16* bias;
  int M, N, K, group;
};

__device__ __forceinline__ void qg_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Word j of lane t before: bytes 16 t + 4 j of the row's 64; after: bytes 16 j + 4 t.
__device__ __forceinline__ void qg_transpose(uint32_t (&w)[4], int t) {
  const bool odd = t & 1, high = t & 2;
  uint32_t a = odd ? w[0] : w[1], b = odd ? w[2] : w[3];
  a = __shfl_xor_sync(0xffffffffu, a, 1);
  b = __shfl_xor_sync(0xffffffffu, b, 1);
  if (odd) w[0] = a, w[2] = b;
  else w[1] = a, w[3] = b;
  a = high ? w[0] : w[2], b = high ? w[1] : w[3];
  a = __shfl_xor_sync(0xffffffffu, a, 2);
  b = __shfl_xor_sync(0xffffffffu, b, 2);
  if (high) w[0] = a, w[1] = b;
  else w[2] = a, w[3] = b;
}

// RUNS: groups that a block is cut into (1: it lies within one and lanes keep their own 16 bytes).
template <int BITS, int RUNS, int NT, bool LO, bool ZERO>
__device__ __forceinline__ void qg_rows(const QgParams& p, const unsigned char* tab, const uint4* s_x, int row0, int blk0,
                                        int blk1, float (&acc)[NT][4]) {
  constexpr int BLOCK_K = 512 / BITS, STEPS = BLOCK_K / 16, RUN_STEPS = STEPS / RUNS, RUN_K = BLOCK_K / RUNS;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int groups = p.K / p.group;
  const int row_bytes = (int)((long long)p.K * BITS / 8);
  const bool wide = (reinterpret_cast<uintptr_t>(p.codes) & 15) == 0;
  const int r0 = min(row0 + g, p.N - 1), r1 = min(row0 + g + 8, p.N - 1);
  const uint8_t* c0 = p.codes + (long long)r0 * row_bytes;
  const uint8_t* c1 = p.codes + (long long)r1 * row_bytes;
  const long long g0 = (long long)r0 * groups, g1 = (long long)r1 * groups;

  uint32_t cw[QG_DEPTH][2][4];
  auto fetch_row = [&](uint32_t (&w)[4], const uint8_t* row, int blk) {
    const int at = blk * 64 + t * 16;                      // rows are multiples of 16 bytes
    if (wide) {
      const uint4 v = blk < blk1 && at < row_bytes ? __ldcs(reinterpret_cast<const uint4*>(row + at)) : make_uint4(0u, 0u, 0u, 0u);
      w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        w[j] = blk < blk1 && at < row_bytes ? __ldg(reinterpret_cast<const uint32_t*>(row + at) + j) : 0u;
    }
  };
  // scales (and zero points) of block blk0 + 4 i + t, rows g and g + 8: runs as bf16 pairs
  constexpr int SW = (RUNS + 1) / 2;
  uint32_t sc[2][2][SW], zr[ZERO ? 2 : 1][2][SW];
  auto fetch_scales = [&](int slot, int blk) {
#pragma unroll
    for (int u = 0; u < RUNS; ++u) {
      const int k = (blk + t) * BLOCK_K + u * RUN_K;
      const int gi = blk + t < blk1 && k < p.K ? k / p.group : 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t v = __ldg(reinterpret_cast<const uint16_t*>(p.scales) + (h ? g1 : g0) + gi);
        sc[slot][h][u >> 1] = u & 1 ? sc[slot][h][u >> 1] | v << 16 : v;
        if (ZERO) {
          const uint32_t z = __ldg(reinterpret_cast<const uint16_t*>(p.zeros) + (h ? g1 : g0) + gi);
          zr[slot][h][u >> 1] = u & 1 ? zr[slot][h][u >> 1] | z << 16 : z;
        }
      }
    }
  };
#pragma unroll
  for (int i = 0; i < QG_DEPTH - 1; ++i) {
    fetch_row(cw[i][0], c0, blk0 + i);
    fetch_row(cw[i][1], c1, blk0 + i);
  }
  fetch_scales(0, blk0);

  // One block per turn, the register sets handed on by moves: unrolled over the sets (twelve blocks) the loop no longer fit
  // into the instruction cache and took twice the time.
#pragma unroll 1
  for (int b = blk0; b < blk1; ++b) {
    {
      constexpr int slot = 0;
      const int q = b - blk0;
      fetch_row(cw[QG_DEPTH - 1][0], c0, b + QG_DEPTH - 1);
      fetch_row(cw[QG_DEPTH - 1][1], c1, b + QG_DEPTH - 1);
      if constexpr (RUNS > 1) {
        qg_transpose(cw[slot][0], t);
        qg_transpose(cw[slot][1], t);
      }
      uint32_t f[2][SW], z[2][SW];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int u = 0; u < SW; ++u) {
          f[h][u] = __shfl_sync(0xffffffffu, sc[0][h][u], (lane & 28) + (q & 3));
          if (ZERO) z[h][u] = __shfl_sync(0xffffffffu, zr[0][h][u], (lane & 28) + (q & 3));
        }
      if ((q & 3) == 3) {                                  // the last of four: the next set has been asked for at the first
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int u = 0; u < SW; ++u) {
            sc[0][h][u] = sc[1][h][u];
            if (ZERO) zr[0][h][u] = zr[ZERO ? 1 : 0][h][u];
          }
      }
      if ((q & 3) == 0) fetch_scales(1, b + 4);
      const uint4* xb = s_x + (size_t)(b - blk0) * (STEPS / 2) * NT * 32 + lane;
      float d[NT][4], e[NT][4], ones[ZERO ? NT : 1][4];
#pragma unroll
      for (int s = 0; s < STEPS; ++s) {                    // products of 16 k
        const int u = s / RUN_STEPS;
        if (s % RUN_STEPS == 0) {
#pragma unroll
          for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              d[n][i] = 0.f;
              if (LO) e[n][i] = 0.f;
              if (ZERO) ones[n][i] = 0.f;
            }
        }
        uint32_t hi[4], lo[4];
        if constexpr (BITS == 4) {
          // bytes 2 (s % 2) and the next one of word s / 2; entry i of the table sits 128 i bytes from its start
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t word = cw[slot][i & 1][s >> 1];
            const uint32_t at = ((word >> (16 * (s & 1) + 8 * (i >> 1))) & 0xffu) << 7;
            if (LO) {
              const uint2 v = *reinterpret_cast<const uint2*>(tab + (lane & 15) * 8 + at);
              hi[i] = v.x, lo[i] = v.y;
            } else {
              hi[i] = *reinterpret_cast<const uint32_t*>(tab + lane * 4 + at);
            }
          }
        } else {                                           // one value per entry: leading and remaining bits as a pair
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t word = cw[slot][i & 1][s];
            const unsigned char* tb = tab + lane * 4;
            const uint32_t v0 = *reinterpret_cast<const uint32_t*>(tb + (((word >> (16 * (i >> 1))) & 0xffu) << 7));
            const uint32_t v1 = *reinterpret_cast<const uint32_t*>(tb + (((word >> (16 * (i >> 1) + 8)) & 0xffu) << 7));
            hi[i] = __byte_perm(v0, v1, 0x5410);
            if (LO) lo[i] = __byte_perm(v0, v1, 0x7632);
          }
        }
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          const uint4 xv = xb[((s >> 1) * NT + n) * 32];
          const uint32_t b0 = s & 1 ? xv.z : xv.x, b1 = s & 1 ? xv.w : xv.y;
          qg_mma(d[n], hi, b0, b1);
          if (LO) qg_mma(e[n], lo, b0, b1);
          if (ZERO) {
            const uint32_t one[4] = {0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u};
            qg_mma(ones[n], one, b0, b1);
          }
        }
        if (s % RUN_STEPS == RUN_STEPS - 1) {
          auto value = [&](const uint32_t (&v)[SW]) { return __uint_as_float(u & 1 ? v[u >> 1] & 0xffff0000u : v[u >> 1] << 16); };
#pragma unroll
          for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              acc[n][i] = fmaf(value(f[i >> 1]), LO ? d[n][i] + e[n][i] : d[n][i], acc[n][i]);
              if (ZERO) acc[n][i] = fmaf(value(z[i >> 1]), ones[n][i], acc[n][i]);
            }
        }
      }
#pragma unroll
      for (int i = 0; i + 1 < QG_DEPTH; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          cw[i][0][j] = cw[i + 1][0][j];
          cw[i][1][j] = cw[i + 1][1][j];
        }
    }
  }
}

// PASSES: a CTA takes several row tiles in turn, with its table and activations in place (up to 25 more registers).
template <int BITS, int RUNS, int NT, bool PASSES>
__global__ void __launch_bounds__(NT == 1 ? 512 : 256, 1) qgemv_kernel(const QgParams p, const int cluster, const int passes,
                                                                       const int x_bytes) {
  constexpr int BLOCK_K = 512 / BITS, PAIRS = BLOCK_K / 32;
  extern __shared__ __align__(128) unsigned char q_smem[];
  unsigned char* tab = q_smem;
  uint4* s_x = reinterpret_cast<uint4*>(q_smem + QG_TABLE_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows = blockDim.x / 2;                         // 16 per warp
  const int first = blockIdx.x / cluster, rank = blockIdx.x - first * cluster;
  const int blocks = (p.K + BLOCK_K - 1) / BLOCK_K;
  const int blk0 = (int)((long long)blocks * rank / cluster), blk1 = (int)((long long)blocks * (rank + 1) / cluster);

  __shared__ float s_lut[256];
  bool rest = false;                                       // some value is not exact in bf16
  for (int i = threadIdx.x; i < (1 << BITS); i += blockDim.x) {
    const float v = p.lut[i];
    s_lut[i] = v;
    rest |= v != __bfloat162float(__float2bfloat16(v));
  }
  const bool lo = __syncthreads_or(rest);
  auto part = [&](int i, bool low) {
    const float v = s_lut[i], h = __bfloat162float(__float2bfloat16(v));
    return low ? v - h : v;
  };
  for (int i = threadIdx.x; i < 256 * 32; i += blockDim.x) {
    const int e = i >> 5, l = i & 31;
    uint32_t v;
    if (BITS == 8) v = pack_bf16x2(part(e, false), part(e, true));
    else v = pack_bf16x2(part(e & 15, lo && (l & 1)), part(e >> 4, lo && (l & 1)));   // words alternate: leading, remaining
    *reinterpret_cast<uint32_t*>(tab + e * 128 + l * 4) = v;
  }
  // activations in the order of the B fragments: per lane and pair of products 8 k of one row, two runs' four k each where
  // a word is half a pair
  for (int i = threadIdx.x; i < (blk1 - blk0) * PAIRS * NT * 32; i += blockDim.x) {
    const int l = i & 31, n = (i >> 5) % NT, s2 = (i >> 5) / NT;
    const int blk = s2 / PAIRS, pr = s2 % PAIRS, m = n * 8 + (l >> 2), t = l & 3;
    const int k = (blk0 + blk) * BLOCK_K;
    const __nv_bfloat16* row = p.x + m * p.ldx;
    auto four = [&](int at) {
      return m < p.M && at < p.K ? __ldg(reinterpret_cast<const uint2*>(row + at)) : make_uint2(0u, 0u);
    };
    uint2 a, b;
    if (BITS == 8 && RUNS > 1) {
      a = four(k + 2 * pr * 16 + t * 4);
      b = four(k + (2 * pr + 1) * 16 + t * 4);
    } else {
      const int at = k + (RUNS > 1 ? pr * 32 + t * 8 : t * (BLOCK_K / 4) + pr * 8);
      a = four(at);
      b = four(at + 4);
    }
    s_x[i] = make_uint4(a.x, a.y, b.x, b.y);
  }
  __syncthreads();

  // sums -> [activation row][weight row], then over the cluster in rank order
  auto take_tile = [&](int tile, float* sums) {
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
    const int row0 = tile * rows + warp * 16;
    if (row0 < p.N) {
      if (p.zeros) {
        if (lo) qg_rows<BITS, RUNS, NT, true, true>(p, tab, s_x, row0, blk0, blk1, acc);
        else qg_rows<BITS, RUNS, NT, false, true>(p, tab, s_x, row0, blk0, blk1, acc);
      } else {
        if (lo) qg_rows<BITS, RUNS, NT, true, false>(p, tab, s_x, row0, blk0, blk1, acc);
        else qg_rows<BITS, RUNS, NT, false, false>(p, tab, s_x, row0, blk0, blk1, acc);
      }
    }
    if (!PASSES) __syncthreads();                          // the sums go over the table
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        sums[(n * 8 + (lane & 3) * 2 + (i & 1)) * rows + warp * 16 + (lane >> 2) + (i >> 1) * 8] = acc[n][i];
    if (cluster > 1) cluster_sync_all();
    else __syncthreads();
    const uint32_t base = smem_u32(sums);
    for (int v = rank * blockDim.x + threadIdx.x; v < p.M * rows; v += cluster * blockDim.x) {
      const int m = v / rows, n = tile * rows + v % rows;
      if (n >= p.N) continue;
      float a = 0.f;
      for (int r = 0; r < cluster; ++r) {
        float t;
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(t) : "r"(mapa_shared(base + v * 4, r)) : "memory");
        a += t;
      }
      if (p.bias) a += __bfloat162float(p.bias[n]);
      p.out[m * p.ldo + n] = __float2bfloat16(a);
    }
    __syncwarp();
  };
  if constexpr (PASSES) {
    // two buffers in turn behind the activations, one meeting per pass: a buffer is written again behind the next meeting,
    // which everybody reaches after reading it
    float* const buffers = reinterpret_cast<float*>(q_smem + QG_TABLE_BYTES + x_bytes);
    const int clusters = gridDim.x / cluster;
    for (int pass = 0; pass < passes; ++pass) take_tile(first + pass * clusters, buffers + (pass & 1) * (NT * 8 * rows));
  } else {
    take_tile(first, reinterpret_cast<float*>(q_smem));
  }
  if (cluster > 1) cluster_sync_all();   // no CTA leaves while another may still read its sums
}

template <int BITS, int RUNS, int NT>
int launch_qgemv(const QgParams& p, cudaStream_t stream) {
  constexpr int BLOCK_K = 512 / BITS, PAIRS = BLOCK_K / 32;
  const int blocks = (p.K + BLOCK_K - 1) / BLOCK_K, row_tiles = (p.N + 15) / 16, sms = sm_count();
  auto smem_of = [&](int c) { return QG_TABLE_BYTES + (long long)((blocks + c - 1) / c) * PAIRS * NT * 512; };
  // Warps per CTA and parts of the reduction: a warp's block takes about 1100 clocks and 70 more for every warp on its SM,
  // a CTA's start 6000, and clusters of 4 or 8 leave the SMs of a GPC that do not make up another one idle (132 and 128 of
  // 148 take part). One B200, nf4, 4 rows, us for (warps, parts): 6144 x 4096 (12, 4) 14.7, (16, 4) 16.4, (8, 2) 19.6, (8, 8)
  // 21.8, (8, 1) 32.3; 4096 x 14336 (8, 8) 25.2, (8, 4) 30.7; 28672 x 4096 (13, 1) 44.2, (13, 2) 50.2, (8, 4) 58.6.
  // Five warps put two of them on one of the four schedulers (22016 x 4096, two CTAs of five per SM 40, one of ten 36); with
  // 16 rows, whose products take longer, that shows where the registers hold one such CTA only (mxfp4 28672 x 4096 99, 64).
  int warps = 0, cluster = 0, passes = 1;
  long long best = 0, smem = 0, grid = 0;
  for (int c = 1; c <= QG_MAX_CLUSTER && c <= blocks; c *= 2) {
    if (smem_of(c) > QG_SMEM_MAX) continue;
    const int usable = c == 8 ? sms * 128 / 148 : c == 4 ? sms * 132 / 148 : c == 2 ? sms & ~1 : sms;
    for (int w = 4; w <= (NT == 1 ? 16 : 8); ++w) {
      if (w == 5 && (NT == 1 || RUNS == 4)) continue;
      const long long tiles = (row_tiles + w - 1) / w, per_sm = (tiles * c + usable - 1) / usable;
      const int by_smem = (int)(QG_SMEM_MAX / smem_of(c)), by_regs = (NT == 1 ? 16 : RUNS == 4 ? 10 : 12) / w;
      const int most = by_smem < by_regs ? by_smem : by_regs, resident = (int)(per_sm < most ? per_sm : most);
      const long long rounds = (per_sm + resident - 1) / resident;
      const long long cost = rounds * ((1100 + 70LL * resident * w) * ((blocks + c - 1) / c) + 6000);
      if (!warps || cost < best) best = cost, warps = w, cluster = c, smem = smem_of(c), grid = tiles * c, passes = (int)rounds;
    }
  }
  // Where that takes several rounds of CTAs, two CTAs of eight warps stay on every SM instead and take row tiles in turn: their
  // start is paid once, and half the reduction per tile fills the last pass better. Up to 8 rows (more need the registers);
  // us, in rounds / in passes, 1 row: nf4 55296 x 5120 88.1 / 80.0, 57344 x 8192 153.2 / 144.6, 128256 x 4096 171 / 148.
  // Two CTAs interleave better than the clocks above say, unless zero points or 8-bit codes load them more: 57344 x 8192 int8
  // 168 / 193, 4-bit with zero points 136 / 147, and those stay in rounds by this.
  const bool rounds = passes > 1;
  const int part = BITS == 4 && !p.zeros ? 9 : 10;
  passes = 1;
  for (int c = 1; NT == 1 && rounds && c <= 2 && c <= blocks; c *= 2) {
    const long long need = smem_of(c) + 2 * QG_PASS_BYTES;
    if (need > QG_SMEM_MAX) continue;
    const long long tiles = (row_tiles + QG_PASS_WARPS - 1) / QG_PASS_WARPS, here = sms / c * (2 * need <= QG_SMEM_MAX ? 2 : 1);
    const long long turns = (tiles + here - 1) / here, on_sm = 2 * need <= QG_SMEM_MAX ? 2 * QG_PASS_WARPS : QG_PASS_WARPS;
    if (turns < 2) continue;
    const long long cost = turns * ((1100 + 70 * on_sm) * part * ((blocks + c - 1) / c) / 10 + (c > 1 ? 1500 : 500)) + 6000;
    if (cost < best) best = cost, warps = QG_PASS_WARPS, cluster = c, smem = need, grid = here * c, passes = (int)turns;
  }
  if (!warps) {
    set_last_error("edl_qgemv: %d activation rows of %d do not fit into shared memory", p.M, p.K);
    return -1;
  }
  auto kern = qgemv_kernel<BITS, RUNS, NT, false>;
  if constexpr (NT == 1)
    if (passes > 1) kern = qgemv_kernel<BITS, RUNS, NT, true>;
  static bool attr_set[64][2] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!attr_set[dev][passes > 1]) {
    if (check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, QG_SMEM_MAX),
                   "cudaFuncSetAttribute(qgemv)"))
      return -1;
    attr_set[dev][passes > 1] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid, 1, 1);
  cfg.blockDim = dim3(warps * 32, 1, 1);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cluster;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return check_cuda(cudaLaunchKernelEx(&cfg, kern, p, cluster, passes, (int)(smem_of(cluster) - QG_TABLE_BYTES)), "qgemv launch");
}

template <int BITS, int RUNS>
int launch_qgemv_rows(const QgParams& p, cudaStream_t stream) {
  return p.M <= 8 ? launch_qgemv<BITS, RUNS, 1>(p, stream) : launch_qgemv<BITS, RUNS, 2>(p, stream);
}

}  // namespace
}  // namespace edl

using namespace edl;

static int check_quant_args(const char* who, int bits, int N, int K, int group) {
  const int per16 = bits == 4 ? 32 : 16;
  if ((bits != 4 && bits != 8) || N <= 0 || K <= 0 || group <= 0 || K % per16 || K % group ||
      (group % per16 && per16 % group)) {
    set_last_error("%s: bits must be 4 or 8, K a multiple of %d and of the group size (bits=%d K=%d group=%d)", who,
                   per16, bits, K, group);
    return -1;
  }
  return 0;
}

// Codes start on 4 bytes or more.
EDL_HOST_API int edl_dequant_bf16(const void* codes, const void* scales, const void* zeros, const float* lut, int bits,
                                  int N, int K, int group, void* out, long long ldo, void* stream) {
  if (check_quant_args("edl_dequant_bf16", bits, N, K, group)) return -1;
  if ((uintptr_t)codes & 3) {
    set_last_error("edl_dequant_bf16: codes must start on 4 bytes");
    return -1;
  }
  const long long total = (long long)N * (K / 8);
  long long blocks = (total + 255) / 256, cap = (long long)sm_count() * 16;
  if (blocks > cap) blocks = cap;
  auto kern = bits == 4 ? dequant_kernel<4> : dequant_kernel<8>;
  kern<<<(int)blocks, 256, 0, (cudaStream_t)stream>>>((const uint8_t*)codes, (const __nv_bfloat16*)scales,
                                                      (const __nv_bfloat16*)zeros, lut, N, K, group, (__nv_bfloat16*)out, ldo);
  return check_cuda(cudaGetLastError(), "dequant launch");
}

// x [M, K] bf16 (16-byte aligned rows of pitch ldx), M <= 16; out [M, N] bf16. The group size must be a multiple of the number
// of weights in one 16-byte code vector (32 for 4-bit, 16 for 8-bit). Codes that do not start on 16 bytes are read 4 bytes
// at a time.
EDL_HOST_API int edl_qgemv(const void* x, long long ldx, const void* codes, const void* scales, const void* zeros,
                           const float* lut, int bits, int M, int N, int K, int group, void* out, long long ldo,
                           const void* bias, void* stream) {
  if (check_quant_args("edl_qgemv", bits, N, K, group)) return -1;
  const int per16 = bits == 4 ? 32 : 16;
  if (M < 1 || M > QG_MAX_M || (ldx & 7) || ((uintptr_t)x & 15) || ((uintptr_t)codes & 3) || group % per16) {
    set_last_error("edl_qgemv: M must be in [1, %d], rows 16-byte aligned and group a multiple of %d", QG_MAX_M, per16);
    return -1;
  }
  const QgParams p{(const __nv_bfloat16*)x, ldx, (const uint8_t*)codes, (const __nv_bfloat16*)scales,
                   (const __nv_bfloat16*)zeros, lut, (__nv_bfloat16*)out, ldo, (const __nv_bfloat16*)bias, M, N, K, group};
  cudaStream_t s = (cudaStream_t)stream;
  // a block is four 16-byte vectors: one run where they always share a group, two, or one run per vector
  const int per_group = group % (4 * per16) == 0 ? 1 : group % (2 * per16) == 0 ? 2 : 4;
  if (bits == 4) {
    if (per_group == 1) return launch_qgemv_rows<4, 1>(p, s);
    return per_group == 2 ? launch_qgemv_rows<4, 2>(p, s) : launch_qgemv_rows<4, 4>(p, s);
  }
  if (per_group == 1) return launch_qgemv_rows<8, 1>(p, s);
  return per_group == 2 ? launch_qgemv_rows<8, 2>(p, s) : launch_qgemv_rows<8, 4>(p, s);
}
