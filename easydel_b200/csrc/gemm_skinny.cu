// C[M,N] = A[M,K] B[N,K]^T for a few rows (M <= 128): the linears and the head of a decode step.
//
// The weight matrix B crosses HBM once and is what the time goes to (2 N K bytes against 2 M K of activations), so the
// kernel is a weight stream: 128 weight rows are the M side of tcgen05.mma and the activation rows, padded to a multiple
// of 16, its N side. A stage holds 16 KB of weights and only as many activation rows as there are; with the activations on
// the 128-row side half of every stage was padding. Two CTAs per SM keep about 200 KB of ring per SM, so that one's
// start, drain and epilogue run under the other's stream.
// A tile's reduction is cut over the CTAs of a cluster (1 to 8), which meet in shared memory over distributed shared
// memory in rank order: no workspace, no second launch, the same sums on every run.
//
// Against the 128 x 128 kernel with split-K and its reduction launch: 28672 x 4096, 1 row 66.2 -> 41.4 us (5.7 TB/s), 48
// rows 47.6 -> 44.7; 4096 x 14336, 1 row 32.8 -> 23.9; the cut of the reduction is chosen by _skinny_plan in
// ops/kernels.py, which has the measurements.
#include "common.cuh"

namespace edl {
namespace {

constexpr int SK_THREADS = 192;
constexpr int SK_BN = 128;                      // weight rows per tile
constexpr int SK_BK = 64;
constexpr int SK_W_BYTES = SK_BN * SK_BK * 2;
constexpr int SK_RING_BYTES = 104 * 1024;       // two CTAs per SM
constexpr int SK_MAX_STAGES = 8;
constexpr int SK_BAR_BYTES = 256;
constexpr int SK_MAX_ROWS = 128;
constexpr int SK_MAX_CLUSTER = 8;

enum SkinnyFlags : int { SK_OUT_F32 = 1, SK_ACCUMULATE = 2, SK_BIAS = 4 };   // as edl_gemm_bf16

struct SkinnyParams {
  void* c;
  const __nv_bfloat16* bias;
  long long ldc;
  int M, N, num_kb, np, stages, tmem_cols, flags;
  int* status;
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr)
               : "memory");
  return v;
}

__global__ void __launch_bounds__(SK_THREADS, 2)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tma_w, const __grid_constant__ CUtensorMap tma_x,
                   const SkinnyParams p, const int cluster) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int stage_bytes = SK_W_BYTES + p.np * (SK_BK * 2);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SK_RING_BYTES);
  const uint32_t full0 = smem_u32(bars);
  const uint32_t empty0 = full0 + 8 * SK_MAX_STAGES;
  const uint32_t b_done = empty0 + 8 * SK_MAX_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * SK_MAX_STAGES + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x / cluster, rank = blockIdx.x - tile * cluster;
  const int n0 = tile * SK_BN;
  const int kb0 = (int)((long long)p.num_kb * rank / cluster), kb1 = (int)((long long)p.num_kb * (rank + 1) / cluster);

  const uint32_t sbase = smem_u32(smem);
  auto load = [&](int kb, int stage) {   // thread 0 only
    const uint32_t fb = full0 + 8 * stage, dst = sbase + stage * stage_bytes;
    mbar_expect_tx(fb, stage_bytes);
    tma_load_2d(dst, &tma_w, fb, kb * SK_BK, n0);
    tma_load_2d(dst + SK_W_BYTES, &tma_x, fb, kb * SK_BK, 0);
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    mbar_init(b_done, 1);
    *abort_flag = 0;
    fence_mbar_init();
    // the first loads wait for nothing: they leave before the CTA meets and tensor memory is there
    for (int s = 0; s < p.stages && kb0 + s < kb1; ++s) load(kb0 + s, s);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), p.tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0 + p.stages; kb < kb1; ++kb) {
        if (!mbar_wait(empty0 + 8 * stage, phase, abort_flag, p.status, EDL_TIMEOUT_PRODUCER)) break;
        load(kb, stage);
        if (++stage == p.stages) stage = 0, phase ^= 1;
      }
    }
  } else if (warp == 1) {
    const bool leader = elect_one();
    const uint32_t idesc = umma_idesc_bf16(SK_BN, p.np, 0, 0);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      ok = mbar_wait(full0 + 8 * stage, phase, abort_flag, p.status, EDL_TIMEOUT_MMA);
      if (!ok) break;
      tc_fence_after();
      const uint32_t w = sbase + stage * stage_bytes, x = w + SK_W_BYTES;
#pragma unroll
      for (int k = 0; k < SK_BK / 16; ++k)
        if (leader)
          umma_f16_ss(tmem, umma_smem_desc_sw128(w + k * 32, 16, 1024), umma_smem_desc_sw128(x + k * 32, 16, 1024), idesc,
                      (kb != kb0 || k != 0) ? 1u : 0u);
      if (leader) tc_commit(empty0 + 8 * stage);
      if (++stage == p.stages) stage = 0, phase ^= 1;
    }
    if (ok && leader) tc_commit(b_done);
  }
  __syncwarp();

  // Partial sums -> shared memory as [activation row][weight row] (the ring is drained: every product has been read)
  float* part = reinterpret_cast<float*>(smem);
  if (warp >= 2) {
    const int q = warp & 3, n = q * 32 + lane;
    if (__all_sync(0xffffffffu, mbar_wait(b_done, 0, abort_flag, p.status, EDL_TIMEOUT_EPILOGUE))) {
      tc_fence_after();
      for (int m0 = 0; m0 < p.M; m0 += 16) {
        uint32_t r[16];
        tmem_ld_32x32b_x16(tmem + (uint32_t(q * 32) << 16) + m0, r);
        tc_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) part[(m0 + j) * SK_BN + n] = __uint_as_float(r[j]);
      }
      tc_fence_before();
    }
  }
  if (cluster > 1) cluster_sync_all();
  else __syncthreads();
  tc_fence_after();

  // four neighbouring outputs of a row per thread, summed over the cluster in rank order
  if (*abort_flag == 0) {
    uint32_t peer[SK_MAX_CLUSTER];
    for (int r = 0; r < SK_MAX_CLUSTER; ++r) peer[r] = r < cluster ? mapa_shared(sbase, r) : 0u;
    const int quads = p.M * (SK_BN / 4);
    for (int v = rank * SK_THREADS + threadIdx.x; v < quads; v += cluster * SK_THREADS) {
      const int m = v / (SK_BN / 4), nl = (v % (SK_BN / 4)) * 4, n = n0 + nl;
      if (n >= p.N) continue;
      float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int r = 0; r < SK_MAX_CLUSTER; ++r)
        if (r < cluster) {
          const float4 t = ld_cluster_f4(peer[r] + (m * SK_BN + nl) * 4);
          a[0] += t.x, a[1] += t.y, a[2] += t.z, a[3] += t.w;
        }
      const int left = min(4, p.N - n);
      if (p.flags & SK_BIAS)
        for (int e = 0; e < left; ++e) a[e] += __bfloat162float(p.bias[n + e]);
      if (p.flags & SK_OUT_F32) {
        float* dst = reinterpret_cast<float*>(p.c) + m * p.ldc + n;
        if (left == 4) {       // the base and the pitch keep 16-byte alignment
          if (p.flags & SK_ACCUMULATE) {
            const float4 o = *reinterpret_cast<const float4*>(dst);
            a[0] += o.x, a[1] += o.y, a[2] += o.z, a[3] += o.w;
          }
          *reinterpret_cast<float4*>(dst) = make_float4(a[0], a[1], a[2], a[3]);
        } else {
          for (int e = 0; e < left; ++e) dst[e] = (p.flags & SK_ACCUMULATE) ? dst[e] + a[e] : a[e];
        }
      } else {
        __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.c) + m * p.ldc + n;
        if (left == 4) *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(a[0], a[1]), pack_bf16x2(a[2], a[3]));
        else
          for (int e = 0; e < left; ++e) dst[e] = __float2bfloat16(a[e]);
      }
    }
  } else {   // a wait ran out: copies still in flight get time to land before the shared memory is released
    const long long t0 = clock64();
    while (clock64() - t0 < 400000) {
    }
  }
  __syncthreads();
  if (cluster > 1) cluster_sync_all();   // no CTA leaves while another may still read its sums
  if (warp == 1) tmem_dealloc(tmem, p.tmem_cols);
}

}  // namespace
}  // namespace edl

// C[M,N] (+)= A[M,K] * B[N,K]^T (+ bias), bf16 operands, fp32 sums, M <= 128. `cluster` (1 to 8, at most ceil(K / 64)) CTAs
// share the reduction of a 128-column tile. flags as edl_gemm_bf16, accumulation into fp32 outputs only. lda and ldb
// multiples of 8, C 16-byte aligned with ldc a multiple of 8 (bf16) or 4 (fp32).
EDL_HOST_API int edl_gemm_skinny(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, long long lda,
                                 long long ldb, long long ldc, int cluster, int flags, int* status, void* stream) {
  using namespace edl;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  const int num_kb = (K + SK_BK - 1) / SK_BK;
  if (M > SK_MAX_ROWS || cluster < 1 || cluster > SK_MAX_CLUSTER || cluster > num_kb) {
    set_last_error("edl_gemm_skinny: up to %d rows and 1 <= cluster <= %d reduction parts (M=%d cluster=%d K=%d)", SK_MAX_ROWS,
                   SK_MAX_CLUSTER, M, cluster, K);
    return -1;
  }
  if ((lda & 7) || (ldb & 7) || (reinterpret_cast<uintptr_t>(C) & 15) || ((flags & SK_OUT_F32) ? (ldc & 3) : (ldc & 7)) ||
      ((flags & SK_ACCUMULATE) && !(flags & SK_OUT_F32))) {
    set_last_error("edl_gemm_skinny: 16-byte alignment of rows (lda=%lld ldb=%lld ldc=%lld), accumulation in fp32", lda, ldb,
                   ldc);
    return -1;
  }
  SkinnyParams p{C, reinterpret_cast<const __nv_bfloat16*>(bias), ldc, M, N, num_kb, (M + 15) / 16 * 16, 0, 32, flags, status};
  if (!bias) p.flags &= ~SK_BIAS;
  const int stage_bytes = SK_W_BYTES + p.np * SK_BK * 2;
  p.stages = SK_RING_BYTES / stage_bytes;
  if (p.stages > SK_MAX_STAGES) p.stages = SK_MAX_STAGES;
  while (p.tmem_cols < p.np) p.tmem_cols *= 2;
  CUtensorMap tw, tx;
  if (make_tmap_2d_16b(&tw, B, N, K, ldb, SK_BN, SK_BK) || make_tmap_2d_16b(&tx, A, M, K, lda, p.np, SK_BK)) return -1;
  constexpr int smem = SK_RING_BYTES + SK_BAR_BYTES + 1024;
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!attr_set[dev]) {
    if (check_cuda(cudaFuncSetAttribute(gemm_skinny_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                   "cudaFuncSetAttribute(gemm_skinny)"))
      return -1;
    attr_set[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(((N + SK_BN - 1) / SK_BN) * cluster), 1, 1);
  cfg.blockDim = dim3(SK_THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = reinterpret_cast<cudaStream_t>(stream);
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cluster;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return check_cuda(cudaLaunchKernelEx(&cfg, gemm_skinny_kernel, tw, tx, p, cluster), "gemm_skinny launch");
}
