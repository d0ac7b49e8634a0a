// Mixture-of-experts routing and data movement kernels.
//
//   topk_softmax     softmax over E expert logits, top-k, optional renormalisation  (Qwen3-MoE, Mixtral)
//   grouped_topk     sigmoid (or softmax) scores + correction bias, experts arranged in groups, the
//                    topk_group best groups (by the sum of their two best biased scores) stay, top-k
//                    inside them, weights from the unbiased scores, renormalised and scaled (DeepSeek-V3)
//   moe_align        counting sort of the T*k (token, slot) pairs by expert: per-expert row ranges padded
//                    to 128 rows, the source pair of every sorted row, and the expert of every 128-row block
//   moe_gather       A_sorted[row] = x[token of row]   (zero rows for padding)
//   moe_combine      out[t] = sum_k w[t,k] * y[row of (t,k)]   (+ optional shared-expert output)
//
// One warp per token for the routers (E <= 512); one CTA does the sort (T*k up to a few 100k pairs).
// Reference behaviour: lightllm/common/basemodel/triton_kernel/fused_moe/{topk_select,grouped_topk,
// softmax_topk,grouped_fused_moe (moe_align*), moe_sum_reduce}.py.
#include "common.cuh"

using namespace llb;
LLB_DEBUG_BOUNDS_STORAGE(moe)


namespace {

constexpr int MAX_E_PER_LANE = 16;  // E <= 512

// Picks the top-k of per-lane candidate arrays (value v[j] belongs to expert lane + 32*j) by k rounds of
// warp arg-max; ties go to the lower expert id.  `sel` (optional) receives a copy of the selected scores.
template <typename F>
__device__ __forceinline__ void warp_topk(float* v, int n_per_lane, int k, F emit) {
  const int lane = threadIdx.x & 31;
  for (int r = 0; r < k; ++r) {
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int j = 0; j < n_per_lane; ++j) {
      if (v[j] > best) {
        best = v[j];
        bi = lane + 32 * j;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      float ob = __shfl_xor_sync(0xffffffffu, best, o);
      int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) {
        best = ob;
        bi = oi;
      }
    }
    emit(r, bi, best);
    if ((bi & 31) == lane && bi != 0x7fffffff) v[bi >> 5] = -INFINITY;
  }
}

template <typename T>
__device__ __forceinline__ float ld_f(const T* p, int64_t i);
template <>
__device__ __forceinline__ float ld_f<float>(const float* p, int64_t i) {
  return p[i];
}
template <>
__device__ __forceinline__ float ld_f<bf16>(const bf16* p, int64_t i) {
  return __bfloat162float(p[i]);
}

template <typename T>
__global__ void __launch_bounds__(128) topk_softmax_kernel(const T* __restrict__ logits, int64_t stride, int Tn, int E,
                                                           int k, int renorm, float scale, int* __restrict__ ids,
                                                           float* __restrict__ weights) {
  const int t = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (t >= Tn) return;
  const int lane = threadIdx.x & 31;
  const int npl = (E + 31) >> 5;
  float v[MAX_E_PER_LANE];
  float mx = -INFINITY;
  for (int j = 0; j < npl; ++j) {
    int e = lane + 32 * j;
    v[j] = e < E ? ld_f(logits, (int64_t)t * stride + e) : -INFINITY;
    mx = fmaxf(mx, v[j]);
  }
  mx = warp_max(mx);
  float z = 0.f;
  for (int j = 0; j < npl; ++j) {
    v[j] = (lane + 32 * j) < E ? __expf(v[j] - mx) : -INFINITY;
    if (lane + 32 * j < E) z += v[j];
  }
  z = warp_sum(z);
  float sel_sum = 0.f;
  float my_w = 0.f;
  int my_id = 0;
  warp_topk(v, npl, k, [&](int r, int e, float val) {
    sel_sum += val;
    if (r == lane) {
      my_w = val;
      my_id = e;
    }
  });
  // k <= 32: lane r holds the r-th choice
  if (lane < k) {
    float w = my_w / (renorm ? sel_sum : z);
    ids[(int64_t)t * k + lane] = my_id;
    weights[(int64_t)t * k + lane] = w * scale;
  }
}

template <typename T>
__global__ void __launch_bounds__(128)
grouped_topk_kernel(const T* __restrict__ logits, int64_t stride, const float* __restrict__ bias, int Tn, int E, int k,
                    int n_group, int topk_group, int use_sigmoid, int renorm, float scale, int* __restrict__ ids,
                    float* __restrict__ weights) {
  const int t = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (t >= Tn) return;
  const int lane = threadIdx.x & 31;
  const int npl = (E + 31) >> 5;
  const int gsz = E / n_group;
  __shared__ float s_score[4][512];   // unbiased scores
  __shared__ float s_biased[4][512];  // scores + correction bias (selection only)
  __shared__ float s_group[4][32];
  float* sc = s_score[threadIdx.x >> 5];
  float* sb = s_biased[threadIdx.x >> 5];
  float* sg = s_group[threadIdx.x >> 5];
  float mx = -INFINITY;
  for (int j = 0; j < npl; ++j) {
    int e = lane + 32 * j;
    if (e < E) mx = fmaxf(mx, ld_f(logits, (int64_t)t * stride + e));
  }
  mx = warp_max(mx);
  float z = 0.f;
  for (int j = 0; j < npl; ++j) {
    int e = lane + 32 * j;
    if (e < E) {
      float x = ld_f(logits, (int64_t)t * stride + e);
      float s = use_sigmoid ? 1.f / (1.f + __expf(-x)) : __expf(x - mx);
      sc[e] = s;
      z += s;
    }
  }
  z = warp_sum(z);
  for (int j = 0; j < npl; ++j) {
    int e = lane + 32 * j;
    if (e < E) {
      if (!use_sigmoid) sc[e] /= z;
      sb[e] = sc[e] + (bias ? bias[e] : 0.f);
    }
  }
  __syncwarp();
  // group score: sum of the two best biased scores of the group (with a bias) or the best one (without)
  if (lane < n_group) {
    float b1 = -INFINITY, b2 = -INFINITY;
    for (int i = 0; i < gsz; ++i) {
      float x = sb[lane * gsz + i];
      if (x > b1) {
        b2 = b1;
        b1 = x;
      } else if (x > b2) {
        b2 = x;
      }
    }
    sg[lane] = bias ? (b1 + b2) : b1;
  }
  __syncwarp();
  // keep the topk_group best groups
  float gv[1] = {lane < n_group ? sg[lane] : -INFINITY};
  unsigned keep_mask = 0;
  warp_topk(gv, 1, topk_group, [&](int r, int g, float val) { keep_mask |= 1u << g; });
  float v[MAX_E_PER_LANE];
  for (int j = 0; j < npl; ++j) {
    int e = lane + 32 * j;
    v[j] = (e < E && ((keep_mask >> (e / gsz)) & 1u)) ? sb[e] : -INFINITY;
  }
  float sel_sum = 0.f, my_w = 0.f;
  int my_id = 0;
  warp_topk(v, npl, k, [&](int r, int e, float val) {
    float w = (e != 0x7fffffff) ? sc[e] : 0.f;
    sel_sum += w;
    if (r == lane) {
      my_w = w;
      my_id = e == 0x7fffffff ? 0 : e;
    }
  });
  if (lane < k) {
    float w = renorm ? my_w / (sel_sum + 1e-20f) : my_w;
    ids[(int64_t)t * k + lane] = my_id;
    weights[(int64_t)t * k + lane] = w * scale;
  }
}

// ---- alignment (counting sort by expert) ----
// pairs: p = t*k + slot, expert ids[p] (ids outside [e0, e0+E_local) are dropped: expert parallel ranks)
// outputs: sorted_pair[M_pad] (pair index of each sorted row, -1 for padding), pair_row[T*k] (row of each pair,
// -1 if dropped), mblock_expert[M_pad/128] (local expert id or -1), expert_rows[E_local+1] (padded offsets),
// total_rows[1]
// `id_of(p)`: expert of pair p (negative: none).
template <typename IdOf>
__device__ __forceinline__ void align_pairs(IdOf id_of, int n_pairs, int e0, int E_local, int m_pad,
                                            int* __restrict__ sorted_pair, int* __restrict__ pair_row,
                                            int* __restrict__ mblock_expert, int* __restrict__ expert_off,
                                            int* __restrict__ total_rows) {
  extern __shared__ int sm[];
  int* cnt = sm;                 // [E_local]
  int* off = sm + E_local;       // [E_local + 1]
  int* cur = sm + 2 * E_local + 1;  // [E_local]
  for (int i = threadIdx.x; i < E_local; i += blockDim.x) cnt[i] = 0;
  __syncthreads();
  // eight look-ups in flight per thread: they are latency-bound
  constexpr int U = 8;
  for (int p0 = threadIdx.x; p0 < n_pairs; p0 += U * blockDim.x) {
    int e[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int p = p0 + u * blockDim.x;
      e[u] = p < n_pairs ? id_of(p) - e0 : -1;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (e[u] >= 0 && e[u] < E_local) atomicAdd(&cnt[e[u]], 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int e = 0; e < E_local; ++e) {
      off[e] = acc;
      acc += ((cnt[e] + 127) / 128) * 128;
    }
    off[E_local] = acc;
    total_rows[0] = acc;
  }
  __syncthreads();
  for (int i = threadIdx.x; i <= E_local; i += blockDim.x) expert_off[i] = off[i];
  for (int i = threadIdx.x; i < E_local; i += blockDim.x) cur[i] = 0;
  for (int r = threadIdx.x; r < m_pad; r += blockDim.x) sorted_pair[r] = -1;
  for (int b = threadIdx.x; b < m_pad / 128; b += blockDim.x) {
    // expert of block b: the one whose padded range contains row b*128
    int row = b * 128, e = -1;
    if (row < off[E_local]) {
      int lo = 0, hi = E_local - 1;
      while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= row) lo = mid; else hi = mid - 1;
      }
      e = lo;
      // skip experts with zero rows that share the same offset
      while (e + 1 < E_local && off[e + 1] <= row) ++e;
    }
    mblock_expert[b] = e;
  }
  __syncthreads();
  for (int p0 = threadIdx.x; p0 < n_pairs; p0 += U * blockDim.x) {
    int e[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int p = p0 + u * blockDim.x;
      e[u] = p < n_pairs ? id_of(p) - e0 : -1;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int p = p0 + u * blockDim.x;
      if (p >= n_pairs) break;
      int r = -1;
      if (e[u] >= 0 && e[u] < E_local) {
        r = off[e[u]] + atomicAdd(&cur[e[u]], 1);
        sorted_pair[r] = p;
      }
      pair_row[p] = r;
    }
  }
}

__global__ void __launch_bounds__(1024)
moe_align_kernel(const int* __restrict__ ids, int n_pairs, int e0, int E_local, int m_pad, int* __restrict__ sorted_pair,
                 int* __restrict__ pair_row, int* __restrict__ mblock_expert, int* __restrict__ expert_off,
                 int* __restrict__ total_rows) {
  align_pairs([&](int p) { return ids[p] < 0 ? ids[p] : LLB_CHECK_EXPERT(ids[p]); }, n_pairs, e0, E_local, m_pad,
              sorted_pair, pair_row, mblock_expert, expert_off, total_rows);
}

// Table routing: the experts of a token are a row of the layer's table [vocab, k], looked up by token id, so the
// expert-sorted layouts of ALL layers are known before the first one runs.  One CTA per layer; its slab of `stride`
// ints holds sorted_pair [m_pad], pair_row [T * k], mblock_expert [m_pad / 128], expert_off [E_local + 1],
// total_rows [1], with m_pad = T * k + min(E_local, T * k) * 127 rounded up to 128.
struct TableRoute {
  const int* table;
  int k, e0, E_local, pad;
};
__global__ void __launch_bounds__(1024)
moe_table_align_kernel(const TableRoute* __restrict__ routes, const int64_t* __restrict__ token_ids, int64_t vocab, int T,
                       int* __restrict__ out, int64_t stride) {
  const TableRoute r = routes[blockIdx.x];
  const int n = T * r.k;
  const int m_pad = ((n + min(r.E_local, n) * 127 + 127) / 128) * 128;
  int* sorted_pair = out + (int64_t)blockIdx.x * stride;
  int* pair_row = sorted_pair + m_pad;
  int* mblock = pair_row + n;
  int* off = mblock + m_pad / 128;
  align_pairs(
      [&](int p) {
        const int64_t tok = token_ids[p / r.k];
        return tok >= 0 && tok < vocab ? r.table[tok * r.k + p % r.k] : -1;
      },
      n, r.e0, r.E_local, m_pad, sorted_pair, pair_row, mblock, off, off + r.E_local + 1);
}

// The same layout from a cluster of 8 CTAs for the many pairs of a prompt pass (one CTA took 60 us for 65536): every CTA counts its
// part of the pairs, the counts are read through distributed shared memory, and a CTA's rows of an expert follow those of the CTAs
// before it.
constexpr int kAlignCtas = 8;
__device__ __forceinline__ int peer_int(const int* local, int rank) {
  uint32_t a;
  int v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(local)), "r"(rank));
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void align_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__global__ void __cluster_dims__(kAlignCtas, 1, 1) __launch_bounds__(1024)
moe_align_cluster_kernel(const int* __restrict__ ids, int n_pairs, int e0, int E_local, int m_pad,
                         int* __restrict__ sorted_pair, int* __restrict__ pair_row, int* __restrict__ mblock_expert,
                         int* __restrict__ expert_off, int* __restrict__ total_rows) {
  extern __shared__ int sm[];
  int* cnt = sm;                    // [E_local] my pairs
  int* off = sm + E_local;          // [E_local + 1] first row of an expert
  int* cur = sm + 2 * E_local + 1;  // [E_local] next row of mine
  const int rank = blockIdx.x;
  const int each = (n_pairs + kAlignCtas - 1) / kAlignCtas, p0 = min(n_pairs, rank * each), p1 = min(n_pairs, p0 + each);
  auto expert = [&](int p) {
    const int e = ids[p] < 0 ? -1 : LLB_CHECK_EXPERT(ids[p]) - e0;
    return e >= 0 && e < E_local ? e : -1;
  };
  for (int i = threadIdx.x; i < E_local; i += blockDim.x) cnt[i] = 0;
  for (int r = rank * blockDim.x + threadIdx.x; r < m_pad; r += kAlignCtas * blockDim.x) sorted_pair[r] = -1;
  __syncthreads();
  for (int p = p0 + threadIdx.x; p < p1; p += blockDim.x) {
    const int e = expert(p);
    if (e >= 0) atomicAdd(&cnt[e], 1);
  }
  align_barrier();  // the counts of all CTAs are there, and sorted_pair is cleared
  for (int e = threadIdx.x; e < E_local; e += blockDim.x) {
    int before = 0, all = 0;
    for (int r = 0; r < kAlignCtas; ++r) {
      const int c = peer_int(cnt + e, r);
      if (r < rank) before += c;
      all += c;
    }
    cur[e] = before;
    off[e] = (all + 127) / 128 * 128;
  }
  __syncthreads();
  if (threadIdx.x < 32) {  // exclusive prefix sum over the experts
    int acc = 0;
    for (int e = threadIdx.x; e < (E_local + 31) / 32 * 32; e += 32) {
      const int v = e < E_local ? off[e] : 0;
      int upto = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, upto, o);
        if ((int)threadIdx.x >= o) upto += u;
      }
      if (e < E_local) off[e] = acc + upto - v;
      acc += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (threadIdx.x == 0) off[E_local] = acc;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E_local; e += blockDim.x) cur[e] += off[e];
  if (rank == 0) {
    for (int i = threadIdx.x; i <= E_local; i += blockDim.x) expert_off[i] = off[i];
    if (threadIdx.x == 0) total_rows[0] = off[E_local];
  }
  for (int b = rank * blockDim.x + threadIdx.x; b < m_pad / 128; b += kAlignCtas * blockDim.x) {
    const int row = b * 128;
    int e = -1;
    if (row < off[E_local]) {  // the last expert that starts at or before the row
      int lo = 0, hi = E_local - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= row) lo = mid; else hi = mid - 1;
      }
      e = lo;
    }
    mblock_expert[b] = e;
  }
  __syncthreads();
  for (int p = p0 + threadIdx.x; p < p1; p += blockDim.x) {
    const int e = expert(p);
    int r = -1;
    if (e >= 0) {
      r = atomicAdd(&cur[e], 1);
      sorted_pair[r] = p;
    }
    pair_row[p] = r;
  }
  align_barrier();  // nobody leaves while a peer may still read its counts
}

// A_sorted[row] = x[sorted_pair[row] / k]; padding rows are zeroed, or left as they are (zero_pad 0).  A warp per row, eight 16-byte
// loads in flight per lane.
__global__ void __launch_bounds__(256)
moe_gather_kernel(bf16* __restrict__ a_sorted, const bf16* __restrict__ x, const int* __restrict__ sorted_pair,
                  const int* __restrict__ total_rows, int k, int H_vec, int64_t x_stride_vec, int zero_pad) {
  const int rows = total_rows[0], lane = threadIdx.x & 31;
  constexpr int U = 8;
  for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += gridDim.x * 8) {
    const int p = sorted_pair[r];
    if (p < 0 && !zero_pad) continue;
    uint4* dst = reinterpret_cast<uint4*>(a_sorted) + (int64_t)r * H_vec;
    const uint4* src = reinterpret_cast<const uint4*>(x) + (int64_t)(p < 0 ? 0 : p / k) * x_stride_vec;
    for (int v0 = lane; v0 < H_vec; v0 += 32 * U) {
      uint4 w[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        w[u] = make_uint4(0, 0, 0, 0);
        if (p >= 0 && v0 + 32 * u < H_vec) w[u] = src[v0 + 32 * u];
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (v0 + 32 * u < H_vec) dst[v0 + 32 * u] = w[u];
    }
  }
}

// out[t] = (accumulate ? out[t] : 0) + sum_k w[t,k] * y[pair_row[t*k + s]]
__global__ void __launch_bounds__(256)
moe_combine_kernel(bf16* __restrict__ out, const bf16* __restrict__ y, const int* __restrict__ pair_row,
                   const float* __restrict__ weights, int k, int H_vec, int accumulate) {
  const int t = blockIdx.x;
  for (int v = threadIdx.x; v < H_vec; v += blockDim.x) {
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
    if (accumulate) unpack8(reinterpret_cast<const bf16x8*>(out)[(int64_t)t * H_vec + v], acc);
    for (int s = 0; s < k; ++s) {
      const int r = pair_row[t * k + s];
      if (r < 0) continue;
      const float w = weights[t * k + s];
      float f[8];
      unpack8(reinterpret_cast<const bf16x8*>(y)[(int64_t)r * H_vec + v], f);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += w * f[i];
    }
    reinterpret_cast<bf16x8*>(out)[(int64_t)t * H_vec + v] = pack8(acc);
  }
}

}  // namespace

// dtype: 0 = fp32 logits, 1 = bf16 logits
LLB_EXPORT int llb_topk_softmax(const void* logits, int dtype, int64_t stride, int T, int E, int k, int renorm,
                                float scale, int* ids, float* weights, cudaStream_t st) {
  if (T <= 0) return LLB_OK;
  if (E > 512 || k > 32 || k > E) return LLB_ERR_UNSUPPORTED;
  if (dtype == 0)
    topk_softmax_kernel<float><<<cdiv(T, 4), 128, 0, st>>>((const float*)logits, stride, T, E, k, renorm, scale, ids, weights);
  else
    topk_softmax_kernel<bf16><<<cdiv(T, 4), 128, 0, st>>>((const bf16*)logits, stride, T, E, k, renorm, scale, ids, weights);
  LLB_LAUNCH_CHECK();
  return LLB_OK;
}

// routes: device array of L {table pointer, k, first local expert, number of local experts, 0}.
LLB_EXPORT int llb_moe_table_align(const void* routes, int L, int max_experts, const int64_t* token_ids, int64_t vocab,
                                   int T, int* out, int64_t stride, cudaStream_t st) {
  if (T <= 0 || L <= 0) return LLB_OK;
  const size_t smem = (3 * (size_t)max_experts + 1) * sizeof(int);
  if (smem > 48 * 1024) return LLB_ERR_UNSUPPORTED;
  moe_table_align_kernel<<<L, 1024, smem, st>>>((const TableRoute*)routes, token_ids, vocab, T, out, stride);
  LLB_LAUNCH_CHECK();
  return LLB_OK;
}

LLB_EXPORT int llb_grouped_topk(const void* logits, int dtype, int64_t stride, const float* bias, int T, int E, int k,
                                int n_group, int topk_group, int use_sigmoid, int renorm, float scale, int* ids,
                                float* weights, cudaStream_t st) {
  if (T <= 0) return LLB_OK;
  if (E > 512 || k > 32 || n_group > 32 || E % n_group != 0 || topk_group > n_group) return LLB_ERR_UNSUPPORTED;
  if (dtype == 0)
    grouped_topk_kernel<float><<<cdiv(T, 4), 128, 0, st>>>((const float*)logits, stride, bias, T, E, k, n_group,
                                                            topk_group, use_sigmoid, renorm, scale, ids, weights);
  else
    grouped_topk_kernel<bf16><<<cdiv(T, 4), 128, 0, st>>>((const bf16*)logits, stride, bias, T, E, k, n_group,
                                                           topk_group, use_sigmoid, renorm, scale, ids, weights);
  LLB_LAUNCH_CHECK();
  return LLB_OK;
}

// Redundant experts under expert parallelism: counts how often every expert is chosen (the statistic the placement
// of redundant experts is taken from) and rewrites the router's expert ids into the "physical" id space
// rank x (experts per rank + redundant per rank) through this rank's table, in which an expert this rank holds a
// copy of points at the copy.
__global__ void moe_count_remap_kernel(const int* __restrict__ ids, int n_pairs, const int* __restrict__ table, int E,
                                       int* __restrict__ counter, int* __restrict__ out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_pairs; i += gridDim.x * blockDim.x) {
    int e = ids[i];
    if (e < 0 || e >= E) {
      out[i] = -1;
      continue;
    }
    if (counter != nullptr) atomicAdd(counter + e, 1);
    out[i] = table[e];
  }
}

// Routed-expert capture: buf[slot[t], layer, :] = ids[t, :] as 8- or 16-bit integers (buf is [slots, layers, k]).
template <typename OUT>
__global__ void route_capture_kernel(const int* __restrict__ ids, const int* __restrict__ slot, int n_pairs, int k,
                                     OUT* __restrict__ buf, int n_slots, int n_layers, int layer) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_pairs; i += gridDim.x * blockDim.x) {
    int t = i / k, j = i - t * k;
    int s = slot[t];
    if (s < 0 || s >= n_slots) continue;
    buf[((int64_t)s * n_layers + layer) * k + j] = (OUT)ids[i];
  }
}

LLB_EXPORT int llb_route_capture(const int* ids, const int* slot, int T, int k, void* buf, int n_slots, int n_layers,
                                 int layer, int elem_bytes, cudaStream_t st) {
  if (T <= 0) return LLB_OK;
  if (elem_bytes != 1 && elem_bytes != 2) return LLB_ERR_UNSUPPORTED;
  int n = T * k, blocks = cdiv(n, 256);
  if (blocks > 296) blocks = 296;
  if (elem_bytes == 1)
    route_capture_kernel<uint8_t><<<blocks, 256, 0, st>>>(ids, slot, n, k, (uint8_t*)buf, n_slots, n_layers, layer);
  else
    route_capture_kernel<int16_t><<<blocks, 256, 0, st>>>(ids, slot, n, k, (int16_t*)buf, n_slots, n_layers, layer);
  LLB_LAUNCH_CHECK();
  return LLB_OK;
}

LLB_EXPORT int llb_moe_count_remap(const int* ids, int n_pairs, const int* table, int E, int* counter, int* out,
                                   cudaStream_t st) {
  if (n_pairs <= 0) return LLB_OK;
  int blocks = cdiv(n_pairs, 256);
  moe_count_remap_kernel<<<blocks < 296 ? blocks : 296, 256, 0, st>>>(ids, n_pairs, table, E, counter, out);
  LLB_LAUNCH_CHECK();
  return LLB_OK;
}

LLB_EXPORT int llb_moe_align(const int* ids, int n_pairs, int e0, int E_local, int m_pad, int* sorted_pair,
                             int* pair_row, int* mblock_expert, int* expert_off, int* total_rows, cudaStream_t st) {
  if (E_local > 2048 || m_pad % 128 != 0) return LLB_ERR_UNSUPPORTED;
  int smem = (3 * E_local + 1) * sizeof(int);
  // B200, us, one CTA / cluster: 4096 pairs of 8 experts 5.6 / 4.6, of 128 11.3 / 5.4, of 256 16.1 / 5.6; 65536 of 128 58.9 / 12.3.  Fewer
  // pairs, decode steps, were not timed on the cluster.
  if (n_pairs >= 4096)
    moe_align_cluster_kernel<<<kAlignCtas, 1024, smem, st>>>(ids, n_pairs, e0, E_local, m_pad, sorted_pair, pair_row, mblock_expert,
                                                             expert_off, total_rows);
  else
    moe_align_kernel<<<1, 1024, smem, st>>>(ids, n_pairs, e0, E_local, m_pad, sorted_pair, pair_row, mblock_expert,
                                            expert_off, total_rows);
  LLB_LAUNCH_CHECK();
  return LLB_OK;
}

LLB_EXPORT int llb_moe_gather_rows(void* a_sorted, const void* x, const int* sorted_pair, const int* total_rows, int k,
                                   int H, int64_t x_stride, int max_rows, int zero_pad, cudaStream_t st) {
  if (max_rows <= 0) return LLB_OK;
  if (H % 8 || x_stride % 8) return LLB_ERR_UNSUPPORTED;
  const int blocks = cdiv(max_rows, 8) < 148 * 8 ? cdiv(max_rows, 8) : 148 * 8;
  moe_gather_kernel<<<blocks, 256, 0, st>>>((bf16*)a_sorted, (const bf16*)x, sorted_pair, total_rows, k, H / 8,
                                            x_stride / 8, zero_pad);
  LLB_LAUNCH_CHECK();
  return LLB_OK;
}

LLB_EXPORT int llb_moe_combine(void* out, const void* y, const int* pair_row, const float* weights, int T, int k, int H,
                               int accumulate, cudaStream_t st) {
  if (T <= 0) return LLB_OK;
  if (H % 8) return LLB_ERR_UNSUPPORTED;
  moe_combine_kernel<<<T, 256, 0, st>>>((bf16*)out, (const bf16*)y, pair_row, weights, k, H / 8, accumulate);
  LLB_LAUNCH_CHECK();
  return LLB_OK;
}

// ---------------------------------------------------------------------------------------
// Experts with biases (GPT-OSS): the grouped GEMMs run with the plain store epilogue and these two kernels add
// the per-expert bias rows.  Rows live in 128-row blocks of one expert each (mblock_expert, -1 = padding block).
//   moe_bias_act: h [M_pad, 2I] with gate / up interleaved in 32-column blocks -> out [M_pad, I]
//     kind 0 / 1: SiLU / GELU(tanh) gate;  kind 2: clamped "swiglu_oai":
//       g = min(g, limit); u = clamp(u, -limit, limit); out = (u + 1) * g * sigmoid(alpha * g)
//   moe_add_bias: y [M_pad, H] += b2[expert of the row's block]
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) moe_bias_act_kernel(const bf16* __restrict__ h, const bf16* __restrict__ b13,
                                                           const int* __restrict__ mblock_expert,
                                                           bf16* __restrict__ out, int I, int kind, float alpha,
                                                           float limit) {
  const int row = blockIdx.x;
  const int e = mblock_expert[row >> 7];
  if (e < 0) return;
  const bf16* hr = h + (int64_t)row * 2 * I;
  const bf16* br = b13 ? b13 + (int64_t)e * 2 * I : nullptr;
  for (int i = threadIdx.x; i < I; i += blockDim.x) {
    const int blk = i >> 5, j = i & 31;
    const int gi = blk * 64 + j, ui = gi + 32;
    float g = __bfloat162float(hr[gi]), u = __bfloat162float(hr[ui]);
    if (br) {
      g += __bfloat162float(br[gi]);
      u += __bfloat162float(br[ui]);
    }
    float o;
    if (kind == 2) {
      g = fminf(g, limit);
      u = fminf(fmaxf(u, -limit), limit);
      o = (u + 1.f) * g / (1.f + __expf(-alpha * g));
    } else if (kind == 1) {
      const float k0 = 0.7978845608028654f, k1 = 0.044715f;
      o = 0.5f * g * (1.f + tanhf(k0 * (g + k1 * g * g * g))) * u;
    } else {
      o = g / (1.f + __expf(-g)) * u;
    }
    out[(int64_t)row * I + i] = __float2bfloat16(o);
  }
}

__global__ void __launch_bounds__(256) moe_add_bias_kernel(bf16* __restrict__ y, const bf16* __restrict__ b2,
                                                           const int* __restrict__ mblock_expert, int H) {
  const int row = blockIdx.x;
  const int e = mblock_expert[row >> 7];
  if (e < 0) return;
  for (int i = threadIdx.x; i < H; i += blockDim.x)
    y[(int64_t)row * H + i] = __float2bfloat16(__bfloat162float(y[(int64_t)row * H + i]) +
                                                __bfloat162float(b2[(int64_t)e * H + i]));
}

LLB_EXPORT int llb_moe_bias_act(const void* h, const void* b13, const int* mblock_expert, void* out, int M_pad, int I,
                                int kind, float alpha, float limit, cudaStream_t st) {
  if (M_pad <= 0) return LLB_OK;
  if ((I % 32) || kind < 0 || kind > 2) return LLB_ERR_UNSUPPORTED;
  moe_bias_act_kernel<<<M_pad, 256, 0, st>>>((const bf16*)h, (const bf16*)b13, mblock_expert, (bf16*)out, I, kind, alpha,
                                             limit);
  LLB_LAUNCH_CHECK();
  return LLB_OK;
}

LLB_EXPORT int llb_moe_add_bias(void* y, const void* b2, const int* mblock_expert, int M_pad, int H, cudaStream_t st) {
  if (M_pad <= 0) return LLB_OK;
  moe_add_bias_kernel<<<M_pad, 256, 0, st>>>((bf16*)y, (const bf16*)b2, mblock_expert, H);
  LLB_LAUNCH_CHECK();
  return LLB_OK;
}
