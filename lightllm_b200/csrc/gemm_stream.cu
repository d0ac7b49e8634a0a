// bf16 GEMM for few tokens (decode):  C[M, N] = A[M, K] . W[N, K]^T  (+ epilogue),  M <= 128.
//
// Bound by the one pass over W.  The other kernels (gemm_tcgen05.cu) put the tokens into the 128-row M side of the MMA: a
// stage then holds 16 KB of mostly empty token rows per 8 to 32 KB of weights, one CTA fills an SM, and nothing of W moves
// before the previous kernel has drained.  Here the weights are the M side and the tokens the N side:
//   * a CTA owns 128 weight rows and a share of K; a stage is 16 KB of W and NT x 128 bytes of tokens.  Two CTAs fit an SM
//     (about 100 KB each), so tiles x splits up to 2 x 148 CTAs run at once and share the bandwidth: a grid that is no
//     multiple of 148 leaves no last wave, and the start and the end of one CTA hide behind the other
//   * the K shares of a tile are a cluster; their fp32 partial tiles meet through distributed shared memory (no workspace,
//     no counters, a fixed order of the sum)
//   * w_ready: W was not written by the kernel queued just before, so the first stages of W are fetched before the
//     programmatic wait.  (A kernel of this library starts after the last but one kernel has completed: each lets its
//     successor start only after its own wait.)  On 148 SMs that is up to 28 MB of W that move while the predecessor ends
// Measured on B200 (decode steps with captured graphs, both sides in turn): see plan_splits.
#include "sm100_ptx.cuh"

using namespace llb;
using namespace llb::sm100;

namespace {

constexpr int TN = 128;  // weight rows of a CTA
constexpr int BK = 64;   // 64 bf16 = 128 bytes = one swizzle row
constexpr int THREADS = 192;
constexpr int W_BYTES = TN * BK * 2;
constexpr int MAX_SPLITS = 8;  // portable cluster size

enum Epi { EPI_STORE = 0, EPI_RESIDUAL = 1, EPI_GATED_SILU = 2, EPI_F32 = 3, EPI_GATED_GELU = 4, EPI_RELU2 = 5 };
__host__ __device__ constexpr bool epi_gated(int epi) { return epi == EPI_GATED_SILU || epi == EPI_GATED_GELU; }

struct Params {
  void* C;
  const bf16* residual;  // [M, ldc]
  const bf16* bias;      // [N] or null
  int* status;
  int M, N, K;
  int64_t ldc;  // elements
  float out_scale, softcap;
  int w_ready;
};

template <int NT>
constexpr int stage_bytes() { return W_BYTES + NT * BK * 2; }
template <int NT>
constexpr int stages() { return NT <= 16 ? 6 : NT <= 32 ? 5 : NT <= 64 ? 4 : 3; }
template <int NT>
constexpr int smem_bytes() { return stages<NT>() * stage_bytes<NT>() + 1024 /*align slack*/ + 256 /*barriers*/; }
static_assert(2 * (smem_bytes<16>() + 1024) <= 227 * 1024 && 2 * (smem_bytes<32>() + 1024) <= 227 * 1024 &&
                  2 * (smem_bytes<64>() + 1024) <= 227 * 1024 && 2 * (smem_bytes<128>() + 1024) <= 227 * 1024,
              "two CTAs per SM");

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ float silu_f(float v) { return v / (1.f + __expf(-v)); }
__device__ __forceinline__ float gelu_tanh_f(float v) {
  return 0.5f * v * (1.f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)));
}

template <int NT, int EPI>
__global__ void __launch_bounds__(THREADS, 2)
gemm_stream_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const Params p) {
  constexpr int STAGES = stages<NT>();
  constexpr int STAGE_BYTES = stage_bytes<NT>();
  constexpr uint32_t TMEM_COLS = NT < 32 ? 32 : NT;
  constexpr uint32_t IDESC = umma_idesc(TN, NT, 1);
  static_assert(STAGES * STAGE_BYTES >= NT * TN * 4, "partial tile fits the drained stages");

  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  float* part = reinterpret_cast<float*>(smem_raw + (smem_base - smem_u32(smem_raw)));  // [token][128], after the K loop
  const uint32_t bar_base = smem_base + STAGES * STAGE_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8 * s; };
  auto empty_bar = [&](int s) { return bar_base + 8 * (STAGES + s); };
  const uint32_t tfull_bar = bar_base + 8 * (2 * STAGES);
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int splits = gridDim.x, split = blockIdx.x;  // the cluster is one row of the grid: its rank is the share of K
  const int n0 = blockIdx.y * TN;
  const int kb_total = (p.K + BK - 1) / BK;
  const int kb0 = (int)((int64_t)split * kb_total / splits);
  const int nk = (int)((int64_t)(split + 1) * kb_total / splits) - kb0;  // >= 1: splits <= kb_total

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(tfull_bar, 1);
    fence_barrier_init();
    if (p.w_ready) {  // the barriers are this thread's own: the first stages of W need no one else
      const int pre = nk < STAGES ? nk : STAGES;
      for (int i = 0; i < pre; ++i) {
        mbar_expect_tx(full_bar(i), STAGE_BYTES);
        tma_load_2d(smem_base + i * STAGE_BYTES, &tmW, full_bar(i), (kb0 + i) * BK, n0);
      }
    }
  }
  __syncwarp();
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_base_slot), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  const uint32_t tmem_base = tmem_base_slot;

  if (warp == 0) {
    if (lane == 0) {  // ---- TMA producer ----
      int stage = 0;
      uint32_t phase = 0;
      for (int i = 0; i < nk; ++i) {
        mbar_wait(empty_bar(stage), phase ^ 1, &abort_flag, p.status, 61);
        const uint32_t sa = smem_base + stage * STAGE_BYTES;
        if (i >= STAGES || !p.w_ready) {
          mbar_expect_tx(full_bar(stage), STAGE_BYTES);
          tma_load_2d(sa, &tmW, full_bar(stage), (kb0 + i) * BK, n0);
        }
        tma_load_2d(sa + W_BYTES, &tmX, full_bar(stage), (kb0 + i) * BK, 0);
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {  // ---- MMA issuer ----
      int stage = 0;
      uint32_t phase = 0;
      for (int i = 0; i < nk; ++i) {
        mbar_wait(full_bar(stage), phase, &abort_flag, p.status, 62);
        tc_fence_after();
        const uint32_t sa = smem_base + stage * STAGE_BYTES;
        const uint64_t dw = umma_smem_desc_sw128(sa), dx = umma_smem_desc_sw128(sa + W_BYTES);
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) umma_bf16(tmem_base, dw + 2 * k, dx + 2 * k, IDESC, (i | k) != 0);
        umma_commit(empty_bar(stage));
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
      umma_commit(tfull_bar);
    }
    __syncwarp();
  } else {
    // ---- accumulator -> shared memory: a thread has one weight row, a warp stores 32 of them per token ----
    const int lane_grp = warp & 3;
    mbar_wait(tfull_bar, 0, &abort_flag, p.status, 63);
    tc_fence_after();
    const uint32_t t_row = tmem_base + ((uint32_t)(lane_grp * 32) << 16);
#pragma unroll
    for (int c = 0; c < NT; c += 32) {
      uint32_t r[32];
      tmem_ld_32x32(t_row + c, r);
      tmem_wait_ld();
#pragma unroll
      for (int j = 0; j < (NT < 32 ? NT : 32); ++j) part[(c + j) * TN + lane_grp * 32 + lane] = __uint_as_float(r[j]);
    }
    tc_fence_before();
  }
  __syncthreads();
  cluster_sync_all();  // every share of the tile is in its CTA's shared memory

  // ---- sum over the shares + epilogue: this CTA's part of the (token, 4 columns) items ----
  const uint32_t rows = (uint32_t)(p.M < NT ? p.M : NT);
  const uint32_t groups = epi_gated(EPI) ? TN / 8 : TN / 4;  // outputs of a token in groups of 4
  const uint32_t total = rows * groups;
  const uint32_t i0 = total * (uint32_t)split / (uint32_t)splits, i1 = total * (uint32_t)(split + 1) / (uint32_t)splits;
  auto summed = [&](uint32_t off) {
    float4 v[MAX_SPLITS];
#pragma unroll
    for (int s = 0; s < MAX_SPLITS; ++s)
      if (s < splits) v[s] = ld_cluster_f4(map_to_cta(smem_base, (uint32_t)s) + off);
    float4 a = v[0];
#pragma unroll
    for (int s = 1; s < MAX_SPLITS; ++s)
      if (s < splits) a.x += v[s].x, a.y += v[s].y, a.z += v[s].z, a.w += v[s].w;
    return a;
  };
  for (uint32_t i = i0 + threadIdx.x; i < i1; i += THREADS) {
    const uint32_t row = i / groups, g = i % groups;
    if (epi_gated(EPI)) {  // columns come as [32 gate | 32 up] pairs
      const uint32_t c = (g >> 3) * 64 + (g & 7) * 4;
      if (n0 + (int)c >= p.N) continue;
      const float4 a = summed((row * TN + c) * 4), u = summed((row * TN + c + 32) * 4);
      auto f = [](float x, float y) { return (EPI == EPI_GATED_SILU ? silu_f(x) : gelu_tanh_f(x)) * y; };
      *reinterpret_cast<uint2*>((bf16*)p.C + row * p.ldc + n0 / 2 + g * 4) =
          make_uint2(pack_bf16x2(f(a.x, u.x), f(a.y, u.y)), pack_bf16x2(f(a.z, u.z), f(a.w, u.w)));
      continue;
    }
    const int col = n0 + (int)g * 4;
    if (col >= p.N) continue;
    const float4 a = summed((row * TN + g * 4) * 4);
    float v[4] = {a.x, a.y, a.z, a.w};
    const int n = p.N - col < 4 ? p.N - col : 4;
    const int64_t off = row * p.ldc + col;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (e >= n) continue;
      if (p.bias != nullptr) v[e] += __bfloat162float(p.bias[col + e]);
      if (EPI == EPI_RELU2) v[e] = v[e] > 0.f ? v[e] * v[e] : 0.f;
      if (EPI == EPI_F32) {
        v[e] *= p.out_scale;
        // c tanh(v / c) = c - 2 c / (1 + e^(2 v / c)), as in gemm_tcgen05.cu
        if (p.softcap > 0.f) v[e] = p.softcap - __fdividef(2.f * p.softcap, 1.f + __expf(v[e] * __fdividef(2.f, p.softcap)));
      }
    }
    if (EPI == EPI_F32) {
      float* c = (float*)p.C + off;
      if (n == 4) {
        *reinterpret_cast<float4*>(c) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
        for (int e = 0; e < n; ++e) c[e] = v[e];
      }
    } else {
      bf16* c = (bf16*)p.C + off;
      if (n == 4) {
        if (EPI == EPI_RESIDUAL) {
          const uint2 r = *reinterpret_cast<const uint2*>(p.residual + off);
          v[0] += __uint_as_float(r.x << 16), v[1] += __uint_as_float(r.x & 0xffff0000u);
          v[2] += __uint_as_float(r.y << 16), v[3] += __uint_as_float(r.y & 0xffff0000u);
        }
        *reinterpret_cast<uint2*>(c) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
      } else {
        for (int e = 0; e < n; ++e)
          c[e] = __float2bfloat16(v[e] + (EPI == EPI_RESIDUAL ? __bfloat162float(p.residual[off + e]) : 0.f));
      }
    }
  }
  cluster_sync_all();  // nobody leaves while a peer may still read its share
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// Clusters of `splits` CTAs that run at once on this device (asked once per kernel and cluster size).
template <int NT, int EPI>
int resident_clusters(int splits) {
  static int known[DeviceOnce::kMaxDevices][MAX_SPLITS + 1] = {};
  const int dev = DeviceOnce::current();
  if (dev < 0) return 0;
  if (known[dev][splits] == 0) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(splits, 1, 1);
    cfg.blockDim = dim3(THREADS, 1, 1);
    cfg.dynamicSmemBytes = smem_bytes<NT>();
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = splits;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_stream_kernel<NT, EPI>, &cfg) != cudaSuccess) n = 0;
    (void)cudaGetLastError();
    known[dev][splits] = n > 0 ? n : -1;
  }
  return known[dev][splits];
}

// Shares of K: as many as let every tile's cluster run at once (a second wave of clusters costs more than the shares give:
// [6144, 4096] at 1 token took 13 us with 3 or 4 shares and 17 us with 6, whose 48 clusters do not all fit), at least 4 k-blocks
// each.  Per weight, in a chain of norm + GEMM: [6144, 4096] 26.7 -> 13.0 us, [4096, 4096] 24.9 -> 10.8, [28672, 4096] 76 -> 42 (floor
// 36), [4096, 14336] 49 -> 28 at 1 token; 18 -> 16, 15.5 -> 13.3, 61 -> 47, 34 -> 32 at 64.
template <int NT, int EPI>
int plan_splits(int tiles, int kb) {
  for (int s = MAX_SPLITS; s > 1; --s)
    if (s * 4 <= kb && s * tiles <= 2 * sm_count() && tiles <= resident_clusters<NT, EPI>(s)) return s;
  return 1;
}

template <int NT, int EPI>
int launch_stream(const CUtensorMap& tx, const CUtensorMap& tw, const Params& p, int splits, cudaStream_t st) {
  static DeviceOnce configured;
  if (!configured.done()) {
    cudaError_t e = cudaFuncSetAttribute(gemm_stream_kernel<NT, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         smem_bytes<NT>());
    if (e != cudaSuccess) return (int)e;
    configured.set();
  }
  if (splits == 0) splits = plan_splits<NT, EPI>(cdiv(p.N, TN), cdiv(p.K, BK));
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(splits, cdiv(p.N, TN), 1);
  cfg.blockDim = dim3(THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem_bytes<NT>();
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = splits;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_stream_kernel<NT, EPI>, tx, tw, p);
  return e == cudaSuccess ? LLB_OK : (int)e;
}

template <int NT>
int dispatch_epi(int epi, const CUtensorMap& tx, const CUtensorMap& tw, const Params& p, int splits, cudaStream_t st) {
  switch (epi) {
    case EPI_STORE: return launch_stream<NT, EPI_STORE>(tx, tw, p, splits, st);
    case EPI_RESIDUAL: return launch_stream<NT, EPI_RESIDUAL>(tx, tw, p, splits, st);
    case EPI_GATED_SILU: return launch_stream<NT, EPI_GATED_SILU>(tx, tw, p, splits, st);
    case EPI_F32: return launch_stream<NT, EPI_F32>(tx, tw, p, splits, st);
    case EPI_GATED_GELU: return launch_stream<NT, EPI_GATED_GELU>(tx, tw, p, splits, st);
    case EPI_RELU2: return launch_stream<NT, EPI_RELU2>(tx, tw, p, splits, st);
  }
  return LLB_ERR_UNSUPPORTED;
}

}  // namespace

// Epilogue codes, bias, residual, out_scale and softcap as in llb_gemm_bf16 / llb_gemm_bf16_fused.  splits: shares of K (0:
// plan_splits).  w_ready: see the top of the file.
LLB_EXPORT int llb_gemm_stream(const void* A, int64_t lda, const void* W, int64_t ldw, void* C, int64_t ldc,
                               const void* residual, const void* bias, int M, int N, int K, int epi, int splits,
                               float out_scale, float softcap, int w_ready, int* status, cudaStream_t st) {
  if (M <= 0 || N <= 0) return LLB_OK;
  if (K <= 0 || (K % 8) != 0 || M > 128 || splits < 0) return LLB_ERR_UNSUPPORTED;
  if (epi_gated(epi) && ((N % 64) != 0 || bias != nullptr)) return LLB_ERR_UNSUPPORTED;
  if (((uintptr_t)C & 15) || (ldc % (epi == EPI_F32 ? 4 : 8))) return LLB_ERR_BAD_ARG;
  if (epi == EPI_RESIDUAL && (residual == nullptr || ((uintptr_t)residual & 15))) return LLB_ERR_BAD_ARG;
  const int tiles = cdiv(N, TN), kb = cdiv(K, BK);
  if (tiles > 65535) return LLB_ERR_UNSUPPORTED;
  if (splits > MAX_SPLITS || splits > kb) return LLB_ERR_UNSUPPORTED;
  const int nt = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128;
  CUtensorMap tx, tw;
  int rc = make_tmap_2d(&tx, A, 2, (uint64_t)M, (uint64_t)K, (uint64_t)lda, (uint32_t)nt, BK);
  if (rc) return rc;
  rc = make_tmap_2d(&tw, W, 2, (uint64_t)N, (uint64_t)K, (uint64_t)ldw, TN, BK);
  if (rc) return rc;
  const Params p{C, (const bf16*)residual, (const bf16*)bias, status, M, N, K, ldc, out_scale, softcap, w_ready};
  switch (nt) {
    case 16: return dispatch_epi<16>(epi, tx, tw, p, splits, st);
    case 32: return dispatch_epi<32>(epi, tx, tw, p, splits, st);
    case 64: return dispatch_epi<64>(epi, tx, tw, p, splits, st);
  }
  return dispatch_epi<128>(epi, tx, tw, p, splits, st);
}
