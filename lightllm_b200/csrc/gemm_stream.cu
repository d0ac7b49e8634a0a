// bf16 GEMM for few tokens (decode):  C[M, N] = A[M, K] . W[N, K]^T  (+ epilogue),  M <= 128.
//
// Bound by the one pass over W.  The other kernels (gemm_tcgen05.cu) put the tokens into the 128-row M side of the MMA: a
// stage then holds 16 KB of mostly empty token rows per 8 to 32 KB of weights, one CTA fills an SM, and nothing of W moves
// before the previous kernel has drained.  Here the weights are the M side and the tokens the N side:
//   * a CTA owns 128 weight rows and a share of K; a stage is 16 KB of W and up to NT x 128 bytes of tokens.  Two CTAs fit an SM
//     (about 100 KB each), so tiles x splits up to 2 x 148 CTAs run at once and share the bandwidth: a grid that is no
//     multiple of 148 leaves no last wave, and the start and the end of one CTA hide behind the other
//   * the K shares of a tile are a cluster; their fp32 partial tiles meet through distributed shared memory (no workspace,
//     no counters, a fixed order of the sum)
//   * w_ready: W was not written by the kernel queued just before, so the first stages of W are fetched before the
//     programmatic wait.  (A kernel of this library starts after the last but one kernel has completed: each lets its
//     successor start only after its own wait.)  On 148 SMs that is up to 28 MB of W that move while the predecessor ends
// fp8 (e4m3 with block scales, as in gemm_fp8.cu): a stage is one 128-wide group of K; its products go to one of two tensor-memory
// buffers and are added, scaled, into fp32 registers, two threads per weight row, while the tensor core works on the next group.  The
// chain tensor memory -> sums -> buffer free is what a group waits for, so its reads are issued together.
// Experts: a CTA has 128 rows of one expert's weights and that expert's tokens, of which a decode step brings a few: only 16-row groups
// that hold tokens are fetched and multiplied.  (The 128-row kernels multiply and store a whole padded block per expert.)
// Measured on B200 (decode steps with captured graphs, both sides in turn): see plan_splits.
#include "sm100_ptx.cuh"
#include <atomic>

using namespace llb;
using namespace llb::sm100;

namespace {

constexpr int TN = 128;  // weight rows of a CTA
constexpr int ROW = 128;  // bytes of K per stage and row: 64 bf16 or 128 e4m3 (one scale group) = one swizzle row
// warps: TMA, MMA, then 4 that drain the accumulator, or 8 where every K group has to be drained (fp8)
template <bool FP8>
constexpr int threads() { return FP8 ? 320 : 192; }
constexpr int W_BYTES = TN * ROW;
constexpr int MAX_SPLITS = 8;  // portable cluster size

enum Epi { EPI_STORE = 0, EPI_RESIDUAL = 1, EPI_GATED_SILU = 2, EPI_F32 = 3, EPI_GATED_GELU = 4, EPI_RELU2 = 5 };
__host__ __device__ constexpr bool epi_gated(int epi) { return epi == EPI_GATED_SILU || epi == EPI_GATED_GELU; }

// Where the token rows come from: DENSE rows 0 .. M-1; SORTED rows of the expert-sorted matrix [M_pad, K] (128-row blocks, see
// gemm_grouped); GATHER rows of the unsorted matrix [T, K], picked through the sorted order by TMA gathers
enum Mode { DENSE = 0, SORTED = 1, GATHER = 2 };

struct Params {
  void* C;
  const bf16* residual;  // [M, ldc]
  const bf16* bias;      // [N] or null
  int* status;
  int M, N, K;
  int64_t ldc;  // elements
  float out_scale, softcap;
  int w_ready;
  // fp8: scales of the tokens [K / 128][a_scale_ld] and of blocks of ws_rows x 128 weights
  const float *a_scale, *w_scale;
  int64_t a_scale_ld;
  int ws_rows, ws_total_rows;
  // experts: expert of each 128-row block (-1: none), (token * topk + choice) of each sorted row (-1: padding)
  const int *mblock_expert, *sorted_pair;
  int topk, halves, T;
};

template <int NT>
constexpr int stage_bytes() { return W_BYTES + NT * ROW; }
template <int NT>
constexpr int stages() { return NT <= 16 ? 6 : NT <= 32 ? 5 : NT <= 64 ? 4 : 3; }
constexpr int SCALE_GROUPS = 32;  // groups of K whose token scales are held at a time (fp8)
template <int NT, bool FP8>
constexpr int smem_bytes() {
  return stages<NT>() * stage_bytes<NT>() + 1024 /*align slack*/ + 256 /*barriers*/ + (FP8 ? SCALE_GROUPS * NT * 4 : 0);
}
static_assert(2 * (smem_bytes<16, true>() + 2048) <= 227 * 1024 && 2 * (smem_bytes<32, true>() + 2048) <= 227 * 1024 &&
                  2 * (smem_bytes<64, true>() + 2048) <= 227 * 1024 && 2 * (smem_bytes<128, false>() + 2048) <= 227 * 1024,
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

template <int NT, int EPI, bool FP8, int MODE>
__global__ void __launch_bounds__(threads<FP8>(), 2)
gemm_stream_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const Params p) {
  constexpr int STAGES = stages<NT>();
  constexpr int STAGE_BYTES = stage_bytes<NT>();
  constexpr int BK = FP8 ? ROW : ROW / 2;  // elements of K per stage
  constexpr uint32_t TMEM_COLS = FP8 ? 2 * NT : (NT < 32 ? 32 : NT);
  static_assert(STAGES * STAGE_BYTES >= NT * TN * 4, "partial tile fits the drained stages");
  static_assert(!FP8 || NT <= 64, "a thread holds NT / 2 scaled sums");
  constexpr int THREADS = threads<FP8>();
  constexpr int HC = FP8 ? (NT >= 32 ? NT / 2 : NT) : 1;    // fp8: tokens of a draining thread
  constexpr int DRAIN = FP8 && NT >= 32 ? 8 : 4;            // draining warps

  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  float* part = reinterpret_cast<float*>(smem_gen);  // [token][128], after the K loop
  const uint32_t bar_base = smem_base + STAGES * STAGE_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8 * s; };
  auto empty_bar = [&](int s) { return bar_base + 8 * (STAGES + s); };
  auto tfull_bar = [&](int b) { return bar_base + 8 * (2 * STAGES + b); };
  auto tempty_bar = [&](int b) { return bar_base + 8 * (2 * STAGES + 2 + b); };
  float* scales = reinterpret_cast<float*>(smem_gen + STAGES * STAGE_BYTES + 256);  // fp8: [SCALE_GROUPS][NT]
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;
  __shared__ int tokens[MODE == GATHER ? NT : 1];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int splits = gridDim.x, split = blockIdx.x;  // the cluster is one row of the grid: its rank is the share of K
  const int n0 = blockIdx.y * TN;
  const int kb_total = (p.K + BK - 1) / BK;
  const int kb0 = (int)((int64_t)split * kb_total / splits);
  const int nk = (int)((int64_t)(split + 1) * kb_total / splits) - kb0;  // >= 1: splits <= kb_total
  int row0 = blockIdx.z * NT, rows = min(NT, p.M - row0), w_row0 = n0;
  if (MODE != DENSE) {  // the layout comes from a kernel shortly before this one
    pdl_wait();
    const int mb = blockIdx.z / p.halves;
    row0 = mb * 128 + (blockIdx.z - mb * p.halves) * NT;
    const int e = p.mblock_expert[mb];
    if (e < 0) return;  // the whole cluster: nothing allocated yet
    int pair = -1;
    if (threadIdx.x < NT) {
      pair = p.sorted_pair[row0 + threadIdx.x];
      if (MODE == GATHER) tokens[threadIdx.x] = pair >= 0 ? pair / p.topk : p.T;  // row T: out of range, reads zeros
    }
    rows = __syncthreads_count(pair >= 0);  // an expert's tokens come first in its block
    if (rows == 0) return;
    w_row0 += e * p.N;
  }
  const int groups16 = (rows + 15) >> 4;
  const uint32_t idesc = umma_idesc(TN, 0, FP8 ? 0 : 1) | ((uint32_t)(groups16 * 2) << 17);  // N = 16 groups16
  const uint32_t tx_bytes = W_BYTES + (MODE == DENSE ? NT : groups16 * 16) * ROW;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(tfull_bar(b), 1);
      mbar_init(tempty_bar(b), DRAIN);
    }
    fence_barrier_init();
    if (MODE == DENSE && p.w_ready) {  // the barriers are this thread's own: the first stages of W need no one else
      const int pre = nk < STAGES ? nk : STAGES;
      for (int i = 0; i < pre; ++i) {
        mbar_expect_tx(full_bar(i), tx_bytes);
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
  if (MODE == DENSE) pdl_wait();
  const uint32_t tmem_base = tmem_base_slot;

  if (warp == 0) {
    // ---- TMA producer: lane 0, and with gathered rows one lane per 4 tokens ----
    const bool ahead = MODE == DENSE && p.w_ready;
    int r4[4] = {0, 0, 0, 0};
    if (MODE == GATHER && lane < groups16 * 4) {
#pragma unroll
      for (int e = 0; e < 4; ++e) r4[e] = tokens[lane * 4 + e];
    }
    int stage = 0;
    uint32_t phase = 0;
    const bool issuer = elect_one();
    for (int i = 0; i < nk; ++i) {
      const uint32_t sa = smem_base + stage * STAGE_BYTES;
      const int k = (kb0 + i) * BK;
      const bool free = !issuer || mbar_wait(empty_bar(stage), phase ^ 1, &abort_flag, p.status, 61);
      if (MODE == GATHER ? !__all_sync(0xffffffffu, free) : !free) break;
      if (issuer) {
        if (i >= STAGES || !ahead) {
          mbar_expect_tx(full_bar(stage), tx_bytes);
          tma_load_2d(sa, &tmW, full_bar(stage), k, w_row0);
        }
        if (MODE == DENSE) tma_load_2d(sa + W_BYTES, &tmX, full_bar(stage), k, row0);  // one box: two cost 1.5 us a call at 24 tokens
        if (MODE == SORTED)
          for (int g = 0; g < groups16; ++g) tma_load_2d(sa + W_BYTES + g * 16 * ROW, &tmX, full_bar(stage), k, row0 + g * 16);
      }
      if (MODE == GATHER) {
        __syncwarp();  // the expected bytes before the copies
        if (lane < groups16 * 4)
          tma_gather4(sa + W_BYTES + lane * 4 * ROW, &tmX, full_bar(stage), k, r4[0], r4[1], r4[2], r4[3]);
      }
      if (++stage == STAGES) {
        stage = 0;
        phase ^= 1;
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {  // ---- MMA issuer ----
      int stage = 0;
      uint32_t phase = 0;
      for (int i = 0; i < nk; ++i) {
        const int buf = FP8 ? i & 1 : 0;
        if (FP8 && !mbar_wait(tempty_bar(buf), (((uint32_t)i >> 1) & 1u) ^ 1u, &abort_flag, p.status, 64)) break;
        if (!mbar_wait(full_bar(stage), phase, &abort_flag, p.status, 62)) break;
        tc_fence_after();
        const uint32_t sa = smem_base + stage * STAGE_BYTES;
        const uint64_t dw = umma_smem_desc_sw128(sa), dx = umma_smem_desc_sw128(sa + W_BYTES);
#pragma unroll
        for (int k = 0; k < 4; ++k) {  // 32 bytes of K per instruction
          if (FP8)
            umma_fp8(tmem_base + buf * NT, dw + 2 * k, dx + 2 * k, idesc, k != 0);
          else
            umma_bf16(tmem_base, dw + 2 * k, dx + 2 * k, idesc, (i | k) != 0);
        }
        umma_commit(empty_bar(stage));
        if (FP8) umma_commit(tfull_bar(buf));
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (!FP8) umma_commit(tfull_bar(0));  // also after a wait that ran out: the drain ends, and stores nothing
    }
    __syncwarp();
  } else if (warp < 2 + DRAIN) {
    // ---- accumulator -> shared memory: a thread has one weight row, a warp stores 32 of them per token ----
    const int lane_grp = warp & 3, et = threadIdx.x - 64;
    const uint32_t t_row = tmem_base + ((uint32_t)(lane_grp * 32) << 16);
    if (FP8) {
      const int c0 = ((warp - 2) >> 2) * HC;
      auto drain_sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(DRAIN * 32) : "memory"); };
      float acc[HC];
#pragma unroll
      for (int j = 0; j < HC; ++j) acc[j] = 0.f;
      const float* ws = p.w_scale + (int64_t)min((w_row0 + lane_grp * 32) / p.ws_rows, p.ws_total_rows - 1) * kb_total + kb0;
      float sw_next = __ldg(ws);
      for (int i = 0; i < nk; ++i) {
        if (i % SCALE_GROUPS == 0) {  // token scales of the next groups (all draining warps have finished with the last ones)
          if (i > 0) drain_sync();
          const int n = min(SCALE_GROUPS, nk - i) * NT;
          const int c = et & (NT - 1);
          const float* as = p.a_scale + (MODE == GATHER ? tokens[MODE == GATHER ? (c < rows ? c : 0) : 0] : row0 + (c < rows ? c : 0));
#pragma unroll 8
          for (int j = et; j < n; j += DRAIN * 32) scales[j] = as[(int64_t)(kb0 + i + j / NT) * p.a_scale_ld];
          drain_sync();
        }
        const float sw = sw_next;
        if (i + 1 < nk) sw_next = __ldg(ws + i + 1);
        const float* sc = scales + (i % SCALE_GROUPS) * NT + c0;
        const int buf = i & 1;
        mbar_wait(tfull_bar(buf), ((uint32_t)i >> 1) & 1u, &abort_flag, p.status, 63);
        tc_fence_after();
        uint32_t r[HC < 16 ? 16 : HC];
#pragma unroll
        for (int c = 0; c < HC; c += 16)
          if (c0 + c < rows) tmem_ld_32x16(t_row + buf * NT + c0 + c, r + c);
#pragma unroll
        for (int c = 0; c < HC; c += 16) {
          if (c0 + c < rows) {
            tmem_wait_ld_of(r + c);
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
              const float4 s4 = *reinterpret_cast<const float4*>(sc + c + j);
              const float sv[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (c + j + e < HC) acc[c + j + e] = fmaf(__uint_as_float(r[c + j + e]), sw * sv[e], acc[c + j + e]);
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty_bar(buf));
      }
      drain_sync();  // every group has been read: the stages are drained for all these warps
#pragma unroll
      for (int j = 0; j < HC; ++j)
        if (c0 + j < rows) part[(c0 + j) * TN + lane_grp * 32 + lane] = acc[j];
    } else {
      mbar_wait(tfull_bar(0), 0, &abort_flag, p.status, 63);
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < NT; c += 16) {
        if (c < rows) {
          uint32_t r[16];
          tmem_ld_32x16(t_row + c, r);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) part[(c + j) * TN + lane_grp * 32 + lane] = __uint_as_float(r[j]);
        }
      }
      tc_fence_before();
    }
  }
  __syncthreads();
  cluster_sync_all();  // every share of the tile is in its CTA's shared memory

  // ---- sum over the shares + epilogue: this CTA's part of the (token, 4 columns) items ----
  const uint32_t groups = epi_gated(EPI) ? TN / 8 : TN / 4;  // outputs of a token in groups of 4
  const uint32_t total = (uint32_t)rows * groups;
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
  const bool aborted = *(volatile int*)&abort_flag != 0;
  for (uint32_t i = i0 + threadIdx.x; i < i1 && !aborted; i += THREADS) {
    const uint32_t row = i / groups, g = i % groups;
    if (epi_gated(EPI)) {  // columns come as [32 gate | 32 up] pairs
      const uint32_t c = (g >> 3) * 64 + (g & 7) * 4;
      if (n0 + (int)c >= p.N) continue;
      const float4 a = summed((row * TN + c) * 4), u = summed((row * TN + c + 32) * 4);
      auto f = [](float x, float y) { return (EPI == EPI_GATED_SILU ? silu_f(x) : gelu_tanh_f(x)) * y; };
      *reinterpret_cast<uint2*>((bf16*)p.C + (row0 + row) * p.ldc + n0 / 2 + g * 4) =
          make_uint2(pack_bf16x2(f(a.x, u.x), f(a.y, u.y)), pack_bf16x2(f(a.z, u.z), f(a.w, u.w)));
      continue;
    }
    const int col = n0 + (int)g * 4;
    if (col >= p.N) continue;
    const float4 a = summed((row * TN + g * 4) * 4);
    float v[4] = {a.x, a.y, a.z, a.w};
    const int n = p.N - col < 4 ? p.N - col : 4;
    const int64_t off = (row0 + row) * p.ldc + col;
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
  if (aborted) settle_after_abort();
  cluster_sync_all();  // nobody leaves while a peer may still read its share
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// Clusters of `splits` CTAs that run at once on this device.  All instances run two CTAs per SM, so one of them is asked, once per
// device and cluster size (a millisecond each).
std::atomic<int> g_resident[DeviceOnce::kMaxDevices][MAX_SPLITS + 1];
template <int NT, int EPI, bool FP8, int MODE>
int resident_clusters(int splits) {
  const int dev = DeviceOnce::current();
  if (dev < 0) return 0;
  int n = g_resident[dev][splits].load();
  if (n == 0) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(splits, 1, 1);
    cfg.blockDim = dim3(threads<FP8>(), 1, 1);
    cfg.dynamicSmemBytes = smem_bytes<NT, FP8>();
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = splits;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_stream_kernel<NT, EPI, FP8, MODE>, &cfg) != cudaSuccess) n = 0;
    (void)cudaGetLastError();
    if (n <= 0) n = -1;
    g_resident[dev][splits].store(n);
  }
  return n;
}

// Shares of K: as many as let every tile's cluster run at once (a second wave of clusters costs more than the shares give:
// [6144, 4096] at 1 token took 13 us with 3 or 4 shares and 17 us with 6, whose 48 clusters do not all fit), at least 4 k-blocks
// each.  Per weight, in a chain of norm + GEMM: [6144, 4096] 26.7 -> 13.0 us, [4096, 4096] 24.9 -> 10.8, [28672, 4096] 76 -> 42 (floor
// 36), [4096, 14336] 49 -> 28 at 1 token; 18 -> 16, 15.5 -> 13.3, 61 -> 47, 34 -> 32 at 64.
template <int NT, int EPI, bool FP8, int MODE>
int plan_splits(int tiles, int kb) {
  for (int s = MAX_SPLITS; s > 1; --s)
    if (s * 4 <= kb && s * tiles <= 2 * sm_count() && tiles <= resident_clusters<NT, EPI, FP8, MODE>(s)) return s;
  return 1;
}

template <int NT, int EPI, bool FP8, int MODE>
int launch_stream(const CUtensorMap& tx, const CUtensorMap& tw, const Params& p, int blocks, int splits, cudaStream_t st) {
  static DeviceOnce configured;
  if (!configured.done()) {
    cudaError_t e = cudaFuncSetAttribute(gemm_stream_kernel<NT, EPI, FP8, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         smem_bytes<NT, FP8>());
    if (e != cudaSuccess) return (int)e;
    configured.set();
  }
  if (splits == 0) splits = plan_splits<NT, EPI, FP8, MODE>(cdiv(p.N, TN) * blocks, cdiv(p.K, FP8 ? ROW : ROW / 2));
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(splits, cdiv(p.N, TN), blocks);
  cfg.blockDim = dim3(threads<FP8>(), 1, 1);
  cfg.dynamicSmemBytes = smem_bytes<NT, FP8>();
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
  cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_stream_kernel<NT, EPI, FP8, MODE>, tx, tw, p);
  return e == cudaSuccess ? LLB_OK : (int)e;
}

template <int NT>
int dispatch_dense(int epi, const CUtensorMap& tx, const CUtensorMap& tw, const Params& p, int splits, cudaStream_t st) {
  switch (epi) {
    case EPI_STORE: return launch_stream<NT, EPI_STORE, false, DENSE>(tx, tw, p, 1, splits, st);
    case EPI_RESIDUAL: return launch_stream<NT, EPI_RESIDUAL, false, DENSE>(tx, tw, p, 1, splits, st);
    case EPI_GATED_SILU: return launch_stream<NT, EPI_GATED_SILU, false, DENSE>(tx, tw, p, 1, splits, st);
    case EPI_F32: return launch_stream<NT, EPI_F32, false, DENSE>(tx, tw, p, 1, splits, st);
    case EPI_GATED_GELU: return launch_stream<NT, EPI_GATED_GELU, false, DENSE>(tx, tw, p, 1, splits, st);
    case EPI_RELU2: return launch_stream<NT, EPI_RELU2, false, DENSE>(tx, tw, p, 1, splits, st);
  }
  return LLB_ERR_UNSUPPORTED;
}
template <int NT>
int dispatch_fp8(int epi, const CUtensorMap& tx, const CUtensorMap& tw, const Params& p, int blocks, cudaStream_t st) {
  switch (epi) {
    case EPI_STORE: return launch_stream<NT, EPI_STORE, true, DENSE>(tx, tw, p, blocks, 0, st);
    case EPI_RESIDUAL: return launch_stream<NT, EPI_RESIDUAL, true, DENSE>(tx, tw, p, blocks, 0, st);
    case EPI_GATED_SILU: return launch_stream<NT, EPI_GATED_SILU, true, DENSE>(tx, tw, p, blocks, 0, st);
  }
  return LLB_ERR_UNSUPPORTED;
}
template <int NT, bool FP8>
int dispatch_experts(int epi, bool gather, const CUtensorMap& tx, const CUtensorMap& tw, const Params& p, int blocks,
                     cudaStream_t st) {
  if (epi == EPI_STORE && !gather) return launch_stream<NT, EPI_STORE, FP8, SORTED>(tx, tw, p, blocks, 0, st);
  if (epi == EPI_GATED_SILU && gather) return launch_stream<NT, EPI_GATED_SILU, FP8, GATHER>(tx, tw, p, blocks, 0, st);
  if (epi == EPI_GATED_GELU && gather && !FP8) return launch_stream<NT, EPI_GATED_GELU, false, GATHER>(tx, tw, p, blocks, 0, st);
  return LLB_ERR_UNSUPPORTED;
}
int token_tile(int M) { return M <= 16 ? 16 : M <= 32 ? 32 : 64; }

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
  if (cdiv(N, TN) > 65535) return LLB_ERR_UNSUPPORTED;
  if (splits > MAX_SPLITS || splits > cdiv(K, ROW / 2)) return LLB_ERR_UNSUPPORTED;
  CUtensorMap tx, tw;
  int rc = make_tmap_2d(&tx, A, 2, (uint64_t)M, (uint64_t)K, (uint64_t)lda, M > 64 ? 128 : token_tile(M), ROW / 2);
  if (rc) return rc;
  rc = make_tmap_2d(&tw, W, 2, (uint64_t)N, (uint64_t)K, (uint64_t)ldw, TN, ROW / 2);
  if (rc) return rc;
  Params p;
  memset(&p, 0, sizeof(p));
  p.C = C, p.residual = (const bf16*)residual, p.bias = (const bf16*)bias, p.status = status;
  p.M = M, p.N = N, p.K = K, p.ldc = ldc, p.out_scale = out_scale, p.softcap = softcap, p.w_ready = w_ready;
  if (M > 64) return dispatch_dense<128>(epi, tx, tw, p, splits, st);
  switch (token_tile(M)) {
    case 16: return dispatch_dense<16>(epi, tx, tw, p, splits, st);
    case 32: return dispatch_dense<32>(epi, tx, tw, p, splits, st);
  }
  return dispatch_dense<64>(epi, tx, tw, p, splits, st);
}

// The arguments of llb_gemm_fp8_block without experts, M <= 128 (two blocks of 64 tokens above 64: they read a weight tile one after
// the other, the second time from L2).
LLB_EXPORT int llb_gemm_stream_fp8(const void* A, int64_t lda, const float* a_scale, int64_t a_scale_ld, const void* W, int64_t ldw,
                                   const float* w_scale, int ws_rows, int w_rows_total, void* C, int64_t ldc,
                                   const void* residual, int M, int N, int K, int epi, int w_ready, int* status, cudaStream_t st) {
  if (M <= 0 || N <= 0) return LLB_OK;
  if (K <= 0 || (K % 16) || (lda % 16) || (ldw % 16) || (ldc % 8) || ((uintptr_t)C & 15)) return LLB_ERR_BAD_ARG;
  if (ws_rows != 128 && ws_rows != 32) return LLB_ERR_BAD_ARG;
  if (M > 128 || cdiv(N, TN) > 65535 || (epi == EPI_GATED_SILU && (N % 64))) return LLB_ERR_UNSUPPORTED;
  if (epi == EPI_RESIDUAL && (residual == nullptr || ((uintptr_t)residual & 15))) return LLB_ERR_BAD_ARG;
  CUtensorMap tx, tw;
  int rc = make_tmap_2d(&tx, A, 1, (uint64_t)M, (uint64_t)K, (uint64_t)lda, token_tile(M), ROW);
  if (rc) return rc;
  rc = make_tmap_2d(&tw, W, 1, (uint64_t)w_rows_total, (uint64_t)K, (uint64_t)ldw, TN, ROW);
  if (rc) return rc;
  Params p;
  memset(&p, 0, sizeof(p));
  p.C = C, p.residual = (const bf16*)residual, p.status = status, p.M = M, p.N = N, p.K = K, p.ldc = ldc, p.w_ready = w_ready;
  p.out_scale = 1.f, p.a_scale = a_scale, p.a_scale_ld = a_scale_ld, p.w_scale = w_scale, p.ws_rows = ws_rows;
  p.ws_total_rows = cdiv(w_rows_total, ws_rows);
  switch (token_tile(M)) {
    case 16: return dispatch_fp8<16>(epi, tx, tw, p, 1, st);
    case 32: return dispatch_fp8<32>(epi, tx, tw, p, 1, st);
  }
  return dispatch_fp8<64>(epi, tx, tw, p, cdiv(M, 64), st);
}

// Grouped GEMM of a decode step: T <= 128 tokens with topk choices each, sorted by expert into 128-row blocks (M_pad rows,
// mblock_expert, sorted_pair as from llb_moe_align; with at most 128 tokens every expert has one block).  gather: A [T, K] holds the
// tokens (a_scale [K / 128][a_scale_ld >= T] theirs) and C [M_pad, N / 2] comes out sorted (gated epilogues); else A [M_pad, K] and C
// [M_pad, N] are sorted (store).  a_scale null: bf16 operands.  Rows of C without a token are not written.
LLB_EXPORT int llb_gemm_stream_experts(const void* A, int64_t lda, int gather, const float* a_scale, int64_t a_scale_ld, const void* W,
                                       int64_t ldw, const float* w_scale, int ws_rows, int w_rows_total, void* C, int64_t ldc,
                                       const int* mblock_expert, const int* sorted_pair, int T, int topk, int M_pad, int N, int K,
                                       int epi, int* status, cudaStream_t st) {
  if (T <= 0 || M_pad <= 0 || N <= 0) return LLB_OK;
  const bool fp8 = a_scale != nullptr;
  const int elem = fp8 ? 1 : 2;
  if (K <= 0 || ((K * elem) % 16) || (ldc % 8) || ((uintptr_t)C & 15)) return LLB_ERR_BAD_ARG;
  if (fp8 && ((ws_rows != 128 && ws_rows != 32) || (N % ws_rows))) return LLB_ERR_BAD_ARG;
  if (T > 128 || topk <= 0 || (M_pad % 128) || cdiv(N, TN) > 65535 || (N % 8) || (epi_gated(epi) && (N % 64))) return LLB_ERR_UNSUPPORTED;
  CUtensorMap tx, tw;
  int rc = make_tmap_2d(&tx, A, elem, (uint64_t)(gather ? T : M_pad), (uint64_t)K, (uint64_t)lda, gather ? 1 : 16, ROW / elem);
  if (rc) return rc;
  rc = make_tmap_2d(&tw, W, elem, (uint64_t)w_rows_total, (uint64_t)K, (uint64_t)ldw, TN, ROW / elem);
  if (rc) return rc;
  Params p;
  memset(&p, 0, sizeof(p));
  p.C = C, p.status = status, p.M = M_pad, p.N = N, p.K = K, p.ldc = ldc, p.out_scale = 1.f;
  p.a_scale = a_scale, p.a_scale_ld = a_scale_ld, p.w_scale = w_scale, p.ws_rows = ws_rows;
  p.ws_total_rows = fp8 ? cdiv(w_rows_total, ws_rows) : 0;
  p.mblock_expert = mblock_expert, p.sorted_pair = sorted_pair, p.topk = topk, p.T = T, p.halves = T > 64 ? 2 : 1;
  const int blocks = M_pad / 128 * p.halves;
  if (blocks > 65535) return LLB_ERR_UNSUPPORTED;
  switch (token_tile(T)) {
    case 16: return fp8 ? dispatch_experts<16, true>(epi, gather, tx, tw, p, blocks, st) : dispatch_experts<16, false>(epi, gather, tx, tw, p, blocks, st);
    case 32: return fp8 ? dispatch_experts<32, true>(epi, gather, tx, tw, p, blocks, st) : dispatch_experts<32, false>(epi, gather, tx, tw, p, blocks, st);
  }
  return fp8 ? dispatch_experts<64, true>(epi, gather, tx, tw, p, blocks, st) : dispatch_experts<64, false>(epi, gather, tx, tw, p, blocks, st);
}
