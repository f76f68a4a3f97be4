// Serving-side kernels: paged KV append, token sampling (greedy / top-k / top-p / min-p /
// temperature with presence, frequency and repetition penalties), token-count bookkeeping.
//
// Counterparts in the reference: the KV page update of easydel/caching/ragged_page/utils.py:126-387
// and the sampler of easydel/inference/esurge/core/sampler.py:43-357 (penalties -> top-k -> top-p ->
// temperature -> min-p -> categorical with per-row seeds; top-p limited to the 64 best candidates).
#include <cooperative_groups.h>

#include "common.cuh"

namespace edl {
namespace cg = cooperative_groups;

namespace {

// k/v: [T, width] new rows (bf16, row strides ldk/ldv); pages: [num_slots, ld_page]; slot[t] < 0 skips.
__global__ void kv_append_kernel(const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v,
                                 __nv_bfloat16* __restrict__ k_pages, __nv_bfloat16* __restrict__ v_pages,
                                 const int* __restrict__ slots, int T, int width, long long ldk, long long ldv,
                                 long long ld_page, long long num_slots, int* status) {
  const int vecs = width / 8;
  const long long total = (long long)T * vecs;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(i / vecs);
    const int c = (int)(i - (long long)t * vecs) * 8;
    const long long s = slots[t];
    if (s < 0) continue;
    if (s >= num_slots) {
      if (status) atomicCAS(status, 0, EDL_BAD_INDEX);
      continue;
    }
    *reinterpret_cast<uint4*>(k_pages + s * ld_page + c) = *reinterpret_cast<const uint4*>(k + t * ldk + c);
    *reinterpret_cast<uint4*>(v_pages + s * ld_page + c) = *reinterpret_cast<const uint4*>(v + t * ldv + c);
  }
}

constexpr int SAMP_THREADS = 512;
constexpr int MAX_CAND = 64;

__device__ __forceinline__ float load_logit(const void* logits, int is_f32, long long idx) {
  return is_f32 ? reinterpret_cast<const float*>(logits)[idx]
                : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(logits)[idx]);
}

__device__ __forceinline__ uint32_t hash_u32(uint32_t x) {
  x ^= x >> 16;
  x *= 0x7feb352dU;
  x ^= x >> 15;
  x *= 0x846ca68bU;
  x ^= x >> 16;
  return x;
}

// Adjusted logit of token v for row r: repetition penalty (divide positive / multiply negative logits of
// seen tokens), then presence and frequency penalties from the per-row token counts.
__device__ __forceinline__ float penalised(float z, int cnt, float presence, float frequency, float repetition) {
  if (cnt > 0) {
    if (repetition != 1.f) z = z > 0.f ? z / repetition : z * repetition;
    z -= presence + frequency * (float)cnt;
  }
  return z;
}

struct ArgMax {
  float v;
  int i;
};
__device__ __forceinline__ ArgMax better(ArgMax a, ArgMax b) {
  return (b.v > a.v || (b.v == a.v && b.i < a.i)) ? b : a;
}
__device__ __forceinline__ ArgMax block_argmax(ArgMax a, ArgMax* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax b{__shfl_xor_sync(0xffffffffu, a.v, o), __shfl_xor_sync(0xffffffffu, a.i, o)};
    a = better(a, b);
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[w] = a;
  __syncthreads();
  ArgMax t = lane < (blockDim.x >> 5) ? red[lane] : ArgMax{-INFINITY, 0x7fffffff};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax b{__shfl_xor_sync(0xffffffffu, t.v, o), __shfl_xor_sync(0xffffffffu, t.i, o)};
    t = better(t, b);
  }
  return t;
}

// Cluster barrier in two halves (every thread of the cluster takes both).
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

struct SampleArgs {
  const void* logits;
  int is_f32;
  long long ld;
  int V;
  const float* temperature;
  const int* top_k;
  const float *top_p, *min_p, *presence, *frequency, *repetition;
  const int* counts;
  long long ld_counts;
  const unsigned long long* seeds;
  const int* steps;
  int* out;
  float* out_logprob;
};

constexpr int SAMP_MAX_SLICES = 8;
constexpr int SAMP_LIST = 1024;       // candidates a slice can hold before it is sorted

// Bits of a float whose unsigned order is the order of the values, and back.
__device__ __forceinline__ uint32_t ordered_bits(float v) {
  const uint32_t u = __float_as_uint(v);
  return u ^ ((u >> 31) ? 0xffffffffu : 0x80000000u);
}
__device__ __forceinline__ float from_ordered_bits(uint32_t k) {
  return __uint_as_float(k ^ ((k >> 31) ? 0x80000000u : 0xffffffffu));
}

// Values [i, i + N) of a row as the sampler sees them (penalties applied).
template <int N>
__device__ __forceinline__ void row_values(const SampleArgs& a, const char* rowp, const int* cnt, int i, float pres,
                                           float freq, float rep, float (&z)[N]) {
  if constexpr (N == 8) {
    if (a.is_f32) {
      const float4 x = *reinterpret_cast<const float4*>(rowp + 4LL * i);
      const float4 y = *reinterpret_cast<const float4*>(rowp + 4LL * i + 16);
      z[0] = x.x; z[1] = x.y; z[2] = x.z; z[3] = x.w;
      z[4] = y.x; z[5] = y.y; z[6] = y.z; z[7] = y.w;
    } else {
      const uint4 q = *reinterpret_cast<const uint4*>(rowp + 2LL * i);
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(w[j]);
        z[2 * j] = f.x;
        z[2 * j + 1] = f.y;
      }
    }
    if (cnt) {
      const int4 c0 = *reinterpret_cast<const int4*>(cnt + i), c1 = *reinterpret_cast<const int4*>(cnt + i + 4);
      const int c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) z[j] = penalised(z[j], c[j], pres, freq, rep);
    }
  } else {
    z[0] = load_logit(rowp, a.is_f32, i);
    if (cnt) z[0] = penalised(z[0], cnt[i], pres, freq, rep);
  }
}

// One row of logits per cluster of CTAs, a slice of the row per CTA. Greedy rows (temperature <= 0 or top_k == 1) take
// the arg-max of the penalised logits. Other rows take the `top_k` (<= 64) best candidates, apply temperature, top-p and
// min-p to them and draw one with a counter-based RNG keyed by (seed[row], step[row]). A row without a value above minus
// infinity gives token 0 with log-probability minus infinity.
//
// What bounds it is the latency of a few passes over a slice, so the row is read once: every thread keeps the maximum (and
// the online sum of exponentials) of its own values. The k-th largest of those maxima, found bit by bit with block-wide
// counts, is a lower bound of the k-th largest value, and only the few threads whose maximum reaches it read their values
// again to collect candidates: about k of them, which are ordered by counting. A slice hands its k best to the first CTA of
// the cluster through shared memory, and that CTA merges the sorted lists. Values that crowd around the bound (a
// row of nearly equal logits) can overflow the list: such a slice is searched by k rounds of arg-max. Slices are cut while
// the grid stays within two CTAs per SM.
// 64 sampled rows of 128256 bf16 logits with log-probabilities: 31.8 us, of which 2.5 us are the bytes at the copy rate; 2590
// us when every candidate was a pass of one CTA over the row.
template <int N>
__global__ void __launch_bounds__(SAMP_THREADS, 2) sample_kernel(const SampleArgs a, int slices) {
  __shared__ ArgMax red[32];
  __shared__ float list_v[SAMP_LIST];
  __shared__ int list_i[SAMP_LIST];
  __shared__ int s_count;
  __shared__ float s_parts[32];
  // filled by every CTA of the cluster in the first one's memory
  __shared__ float top_v[SAMP_MAX_SLICES][MAX_CAND];
  __shared__ int top_i[SAMP_MAX_SLICES][MAX_CAND];
  __shared__ int top_n[SAMP_MAX_SLICES];
  __shared__ float top_m[SAMP_MAX_SLICES], top_s[SAMP_MAX_SLICES];
  __shared__ float cand_v[MAX_CAND], prob[MAX_CAND], share[MAX_CAND];
  __shared__ int cand_i[MAX_CAND];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = slices > 1 ? (int)cluster.block_rank() : 0;
  const int row = blockIdx.x / slices, tid = threadIdx.x;
  const float temp = a.temperature ? a.temperature[row] : 0.f;
  int k = a.top_k ? a.top_k[row] : 0;
  const float pres = a.presence ? a.presence[row] : 0.f, freq = a.frequency ? a.frequency[row] : 0.f;
  const float rep = a.repetition ? a.repetition[row] : 1.f;
  const bool pen = a.counts && (pres != 0.f || freq != 0.f || rep != 1.f);
  const int* cnt = pen ? a.counts + (long long)row * a.ld_counts : nullptr;
  const bool greedy = temp <= 0.f || k == 1;
  if (k <= 0 || k > MAX_CAND) k = MAX_CAND;
  if (greedy) k = 1;
  const float inv_t = greedy ? 1.f : 1.f / temp;
  const char* rowp = reinterpret_cast<const char*>(a.logits) + row * a.ld * (a.is_f32 ? 4 : 2);
  const int units = (a.V + N - 1) / N, per = (units + slices - 1) / slices;     // N divides V in the wide form
  const int u0 = min(units, rank * per), u1 = min(units, u0 + per);
  if (tid == 0) s_count = 0;
  if (slices > 1) cluster_arrive();     // the first CTA's memory may be written once every CTA runs

  // ---- the pass over the slice
  ArgMax best{-INFINITY, 0x7fffffff};
  float m = -INFINITY, ssum = 0.f;
#pragma unroll 4
  for (int u = u0 + tid; u < u1; u += SAMP_THREADS) {
    float z[N];
    row_values<N>(a, rowp, cnt, u * N, pres, freq, rep, z);
    float cm = z[0];
#pragma unroll
    for (int j = 1; j < N; ++j) cm = fmaxf(cm, z[j]);
    if (greedy) {
#pragma unroll
      for (int j = 0; j < N; ++j)
        if (z[j] > best.v || (z[j] == best.v && u * N + j < best.i)) best = ArgMax{z[j], u * N + j};
    } else {
      best.v = fmaxf(best.v, cm);
    }
    if (a.out_logprob) {
      const float nm = fmaxf(m, cm);
      if (nm > -INFINITY) {
        float add = 0.f;
#pragma unroll
        for (int j = 0; j < N; ++j) add += __expf((z[j] - nm) * inv_t);
        ssum = ssum * __expf((m - nm) * inv_t) + add;
        m = nm;
      } else {
#pragma unroll
        for (int j = 0; j < N; ++j) ssum += z[j] == z[j] ? 0.f : z[j];     // not a number: nor is the sum
      }
    }
  }
  if (a.out_logprob) {
    const float bm = block_max(m, s_parts);
    const float part = bm > -INFINITY ? ssum * __expf((m - bm) * inv_t) : ssum;
    const float tot = block_sum(part, s_parts);
    m = bm;
    ssum = tot;
  }

  // ---- the slice's k best, in order (value down, index up)
  float* dst_v = slices > 1 ? cluster.map_shared_rank(&top_v[rank][0], 0) : top_v[0];
  int* dst_i = slices > 1 ? cluster.map_shared_rank(&top_i[rank][0], 0) : top_i[0];
  int found = 1;
  if (greedy) {
    best = block_argmax(best, red);
    if (slices > 1) cluster_wait();
    if (tid == 0) {
      dst_v[0] = best.v;
      dst_i[0] = best.i;
    }
  } else {
    const uint32_t key = ordered_bits(best.v);
    uint32_t bound = 0;      // the low 12 bits stay zero: a slightly lower bound
    for (int bit = 31; bit >= 12; --bit) {
      const uint32_t trial = bound | (1u << bit);
      if (__syncthreads_count(key >= trial) >= k) bound = trial;
    }
    const float low = bound <= 0x007fffffu ? -INFINITY : from_ordered_bits(bound);
    if (best.v >= low && best.v > -INFINITY) {
      for (int u = u0 + tid; u < u1; u += SAMP_THREADS) {
        float z[N];
        row_values<N>(a, rowp, cnt, u * N, pres, freq, rep, z);
#pragma unroll
        for (int j = 0; j < N; ++j)
          if (z[j] >= low && z[j] > -INFINITY) {
            const int at = atomicAdd(&s_count, 1);
            if (at < SAMP_LIST) {
              list_v[at] = z[j];
              list_i[at] = u * N + j;
            }
          }
      }
    }
    __syncthreads();
    const int c = s_count;
    if (slices > 1) cluster_wait();
    found = min(c, k);
    if (c <= SAMP_LIST) {
      for (int t = tid; t < c; t += SAMP_THREADS) {
        const float v = list_v[t];
        const int i = list_i[t];
        int at = 0;
        for (int j = 0; j < c; ++j) at += list_v[j] > v || (list_v[j] == v && list_i[j] < i);
        if (at < k) {
          dst_v[at] = v;
          dst_i[at] = i;
        }
      }
    } else {
      float bound_v = INFINITY;  // candidates in strictly decreasing (value, -index) order
      int bound_i = -1;
      for (int rd = 0; rd < k; ++rd) {
        ArgMax top{-INFINITY, 0x7fffffff};
        for (int u = u0 + tid; u < u1; u += SAMP_THREADS) {
          float z[N];
          row_values<N>(a, rowp, cnt, u * N, pres, freq, rep, z);
#pragma unroll
          for (int j = 0; j < N; ++j) {
            const bool after = z[j] < bound_v || (z[j] == bound_v && u * N + j > bound_i);
            if (after) top = better(top, ArgMax{z[j], u * N + j});
          }
        }
        top = block_argmax(top, red);
        if (tid == 0) {
          dst_v[rd] = top.v;
          dst_i[rd] = top.i;
        }
        bound_v = top.v;
        bound_i = top.i;
        __syncthreads();
      }
    }
  }
  if (tid == 0) {
    *(slices > 1 ? cluster.map_shared_rank(&top_n[rank], 0) : &top_n[0]) = found;
    *(slices > 1 ? cluster.map_shared_rank(&top_m[rank], 0) : &top_m[0]) = m;
    *(slices > 1 ? cluster.map_shared_rank(&top_s[rank], 0) : &top_s[0]) = ssum;
  }
  if (slices > 1) {
    cluster_arrive();
    cluster_wait();
    if (rank != 0) return;
  } else {
    __syncthreads();
  }

  // ---- the first CTA merges the slices' lists: a candidate's place is its own plus what beats it in the others
  int total = 0;
  for (int l = 0; l < slices; ++l) total += top_n[l];
  const int n_all = min(total, k);
  for (int t = tid; t < slices * MAX_CAND; t += SAMP_THREADS) {
    const int own = t / MAX_CAND, pos = t % MAX_CAND;
    if (pos >= top_n[own]) continue;
    const ArgMax mine{top_v[own][pos], top_i[own][pos]};
    int at = pos;
    for (int l = 0; l < slices; ++l) {
      if (l == own) continue;
      int lo = 0, hi = top_n[l];
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (top_v[l][mid] > mine.v || (top_v[l][mid] == mine.v && top_i[l][mid] < mine.i)) lo = mid + 1;
        else hi = mid;
      }
      at += lo;
    }
    if (at < k) {
      cand_v[at] = mine.v;
      cand_i[at] = mine.i;
    }
  }
  __syncthreads();
  float lse = 0.f;
  if (a.out_logprob) {
    float gm = top_m[0], sum = 0.f;
    for (int l = 1; l < slices; ++l) gm = fmaxf(gm, top_m[l]);
    for (int l = 0; l < slices; ++l) sum += gm > -INFINITY ? top_s[l] * __expf((top_m[l] - gm) * inv_t) : top_s[l];
    lse = gm * inv_t + __logf(sum);
  }
  if (greedy) {
    if (tid == 0) {
      const bool none = cand_v[0] == -INFINITY;      // nothing above minus infinity in the row, as for sampled rows below
      a.out[row] = none ? 0 : cand_i[0];
      if (a.out_logprob) a.out_logprob[row] = none ? -INFINITY : cand_v[0] - lse;
    }
    return;
  }
  // candidates sorted descending; temperature, then top-p, then min-p on the renormalised top-k set. The sums run in one
  // thread, in order; what they add is formed by all.
  if (tid < n_all) prob[tid] = __expf(fmaf(cand_v[tid], inv_t, -__fmul_rn(cand_v[0], inv_t)));
  __syncthreads();
  float tot = 0.f;
  for (int j = 0; j < n_all; ++j) tot += prob[j];
  if (tid < n_all) share[tid] = prob[tid] / tot;
  __syncthreads();
  if (tid != 0) return;
  const float tp = a.top_p ? a.top_p[row] : 1.f;
  const float mp = a.min_p ? a.min_p[row] : 0.f;
  float cum = 0.f, keep_tot = 0.f;
  int kept = 0;
  for (int j = 0; j < n_all; ++j) {
    if (cand_v[j] == -INFINITY) break;
    if (j > 0 && (cum >= tp || prob[j] < mp * prob[0])) break;
    cum += share[j];
    keep_tot += prob[j];
    ++kept;
  }
  const unsigned long long sd = a.seeds ? a.seeds[row] : 0ULL;
  const uint32_t st = a.steps ? (uint32_t)a.steps[row] : 0u;
  uint32_t hsh = hash_u32((uint32_t)sd ^ hash_u32((uint32_t)(sd >> 32) + 0x9e3779b9U * (st + 1u)) ^ hash_u32(row));
  const float u = ((hsh >> 8) + 0.5f) * (1.0f / 16777216.0f) * keep_tot;
  float acc = 0.f;
  int pick = kept - 1;
  for (int j = 0; j < kept; ++j) {
    acc += prob[j];
    if (u <= acc) {
      pick = j;
      break;
    }
  }
  if (pick < 0) {      // no candidate above minus infinity
    a.out[row] = 0;
    if (a.out_logprob) a.out_logprob[row] = -INFINITY;
    return;
  }
  a.out[row] = cand_i[pick];
  if (a.out_logprob) a.out_logprob[row] = cand_v[pick] * inv_t - lse;
}

// counts[row, token[row]] += 1 for rows whose token is valid
__global__ void count_update_kernel(int* counts, long long ld_counts, const int* tokens, const int* row_slots, int R,
                                    int V) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= R) return;
  const int t = tokens[r];
  const int slot = row_slots ? row_slots[r] : r;
  if (t >= 0 && t < V && slot >= 0) atomicAdd(counts + (long long)slot * ld_counts + t, 1);
}

// out[r, :] = src[idx[r], :] (bf16 rows; used to pick each sequence's last hidden state)
__global__ void gather_rows_kernel(const __nv_bfloat16* __restrict__ src, const int* __restrict__ idx,
                                   __nv_bfloat16* __restrict__ out, int R, int width, long long ld_src) {
  const int vecs = width / 8;
  const long long total = (long long)R * vecs;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(i / vecs);
    const int c = (int)(i - (long long)r * vecs) * 8;
    *reinterpret_cast<uint4*>(out + (long long)r * width + c) =
        *reinterpret_cast<const uint4*>(src + (long long)idx[r] * ld_src + c);
  }
}

}  // namespace
}  // namespace edl

using namespace edl;

EDL_HOST_API int edl_paged_kv_append(const void* k, const void* v, void* k_pages, void* v_pages, const int* slots,
                                     int T, int width, long long ldk, long long ldv, long long ld_page,
                                     long long num_slots, int* status, void* stream) {
  if (T <= 0) return 0;
  if (width % 8 || ldk % 8 || ldv % 8 || ld_page % 8) {
    set_last_error("edl_paged_kv_append: widths and strides must be multiples of 8 elements");
    return -1;
  }
  long long work = (long long)T * (width / 8);
  long long blocks = (work + 255) / 256, cap = (long long)sm_count() * 8;
  kv_append_kernel<<<(int)(blocks > cap ? cap : blocks), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)k, (const __nv_bfloat16*)v, (__nv_bfloat16*)k_pages, (__nv_bfloat16*)v_pages, slots, T,
      width, ldk, ldv, ld_page, num_slots, status);
  return check_cuda(cudaGetLastError(), "kv_append launch");
}

// logits: [R, V] (bf16 or fp32, row stride ld). Per-row parameter arrays may be null (greedy, no penalties).
// counts: [*, ld_counts] int32 token occurrence table (row r of the batch uses row r), may be null.
EDL_HOST_API int edl_sample(const void* logits, int is_f32, long long ld, int R, int V, const float* temperature,
                            const int* top_k, const float* top_p, const float* min_p, const float* presence,
                            const float* frequency, const float* repetition, const int* counts, long long ld_counts,
                            const unsigned long long* seeds, const int* steps, int* out, float* out_logprob,
                            void* stream) {
  if (R <= 0) return 0;
  const SampleArgs a{logits, is_f32, ld, V, temperature, top_k, top_p, min_p, presence, frequency, repetition, counts,
                     ld_counts, seeds, steps, out, out_logprob};
  auto odd = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
  const bool wide = (V & 7) == 0 && (ld & 7) == 0 && !odd(logits) && (!counts || (!(ld_counts & 3) && !odd(counts)));
  // a row is cut into slices while the grid stays within two CTAs per SM and a slice is worth a CTA
  int slices = 1;
  while (slices < SAMP_MAX_SLICES && 2LL * slices * R <= 2LL * sm_count() && V >= 2 * slices * 4096) slices *= 2;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)R * slices);
  cfg.blockDim = dim3(SAMP_THREADS);
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = slices;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (check_cuda(wide ? cudaLaunchKernelEx(&cfg, sample_kernel<8>, a, slices) : cudaLaunchKernelEx(&cfg, sample_kernel<1>, a, slices),
                 "sample launch"))
    return -1;
  return check_cuda(cudaGetLastError(), "sample launch");
}

EDL_HOST_API int edl_count_update(int* counts, long long ld_counts, const int* tokens, const int* row_slots, int R,
                                  int V, void* stream) {
  if (R <= 0) return 0;
  count_update_kernel<<<(R + 127) / 128, 128, 0, (cudaStream_t)stream>>>(counts, ld_counts, tokens, row_slots, R, V);
  return check_cuda(cudaGetLastError(), "count_update launch");
}

EDL_HOST_API int edl_gather_rows(const void* src, const int* idx, void* out, int R, int width, long long ld_src,
                                 void* stream) {
  if (R <= 0) return 0;
  if (width % 8 || ld_src % 8) {
    set_last_error("edl_gather_rows: width and stride must be multiples of 8");
    return -1;
  }
  long long work = (long long)R * (width / 8);
  long long blocks = (work + 255) / 256, cap = (long long)sm_count() * 8;
  gather_rows_kernel<<<(int)(blocks > cap ? cap : blocks), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)src, idx, (__nv_bfloat16*)out, R, width, ld_src);
  return check_cuda(cudaGetLastError(), "gather_rows launch");
}
