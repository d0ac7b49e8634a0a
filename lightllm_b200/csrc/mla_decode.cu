// Decode attention of the latent cache (absorbed form) on tcgen05: scores q_lat . c_kv + q_pe . k_pe over rows of 576 values, output the
// weighted sum of their first 512.  One new token per request, up to 128 heads per CTA.
//
// The heads are the 128-row M side, so a row of the pool is read once per CTA for all heads; mla.cu reads it once per 16 heads and
// multiplies with mma.sync (55 TFLOP/s).  A CTA has one half of the value columns of one request (and share of its keys): the fp32
// output takes 256 of the 512 tensor-memory columns, and the scores are computed twice.
//   S  = Q . K^T   64 keys at a time.  Q's first 256 columns are in tensor memory, the other 320 in shared memory: with all of Q in
//                  shared memory (147 KB) only one 72 KB tile of keys would fit beside it
//   P  = exp2(S - m), one thread per head, written as bf16 over the scores
//   O += P . V     V is the CTA's half of the key tile itself, read as an MN-major operand
// The scores of the next tile are issued before the weights of the current one are waited for.  Tiles of 64 pool rows come by TMA
// gathers through the slot table, two in flight.  The output is rescaled whenever a head's maximum grows, as in attention_fa.cu.
//
// What bounds it: 1152 cycles of MMA for the scores of a tile (64 keys: as many as the 16 KB of Q per 16 columns take to read) and 512
// for P . V, against 72 KB per tile from L2.  B200, us, mla.cu / here: 96 requests of 1025 to 2048 positions, 128 heads 747 / 176, 64
// 435 / 173, 32 285 / 173, 16 182 / 169, 8 181 / 166.
#include "sm100_ptx.cuh"

using namespace llb;
using namespace llb::sm100;
LLB_DEBUG_BOUNDS_STORAGE(mla_decode)

namespace {

constexpr int LAT = 512, ROPE = 64, ROW = LAT + ROPE;
constexpr int BN = 64, BLOCK = BN * 128;               // keys of a tile; bytes of 64 columns of it
constexpr int KBLOCKS = ROW / 64, STAGE = KBLOCKS * BLOCK;
constexpr int Q_TMEM = 256, QBLOCKS = (ROW - Q_TMEM) / 64, QBLOCK = 128 * 128;
constexpr int OFF_K = QBLOCKS * QBLOCK, OFF_BAR = OFF_K + 2 * STAGE, SMEM = OFF_BAR + 256;
static_assert(SMEM <= 227 * 1024, "shared memory");
constexpr int S_COL = 0, Q_COL = 128, O_COL = 256;     // tensor memory: S0 | S1 | Q | O
constexpr int LOADERS = 8;                             // a gather costs its warp about 70 cycles to issue, and a tile has 144
constexpr int THREADS = (5 + LOADERS) * 32;            // warp 0 and 6 ..: loads, warp 1: MMA, warps 2..5: softmax
constexpr float kLog2e = 1.4426950408889634f;

struct Params {
  const bf16* q_lat;  // [T, H, 512]
  const int *req_to_token, *b_req_idx, *cu_q, *b_ready_len;
  int64_t r2t_stride;
  bf16* out;          // [T, H, 512]
  float *part_o, *part_lse;  // splits > 1: [T, H, splits, 512], [T, H, splits]
  int* status;
  int H, n_slots, splits;
  float scale_log2;
};

__device__ __forceinline__ float ex2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__global__ void __launch_bounds__(THREADS, 1)
mla_decode_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmPe,
                  const __grid_constant__ CUtensorMap tmKV, const Params p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t bar = smem_base + OFF_BAR;
  auto full = [&](int s) { return bar + 8 * s; };
  auto empty = [&](int s) { return bar + 8 * (2 + s); };
  auto s_full = [&](int s) { return bar + 8 * (4 + s); };
  // one per score buffer: the scores of a tile may be there before all warps have finished with the tile before it, and a warp that runs
  // ahead (another one may be rescaling) must not be counted for it
  auto p_full = [&](int s) { return bar + 8 * (6 + s); };
  const uint32_t o_full = bar + 8 * 8, q_full = bar + 8 * 9, qt_full = bar + 8 * 10, done = bar + 8 * 11;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + OFF_BAR + 128);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + OFF_BAR + 132);

  const int half = blockIdx.x & 1, split = blockIdx.x >> 1, b = blockIdx.y, head0 = blockIdx.z * 128;
  const int rows = min(128, p.H - head0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < 2; ++s) mbar_init(full(s), 1), mbar_init(empty(s), 1), mbar_init(s_full(s), 1), mbar_init(p_full(s), 4);
    mbar_init(o_full, 1);
    mbar_init(done, 1);
    mbar_init(q_full, 1);
    mbar_init(qt_full, 4);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();

  const int kv_len = p.b_ready_len[b] + (b - p.cu_q[b]) + 1;
  const int tiles = (kv_len + BN - 1) / BN, per = (tiles + p.splits - 1) / p.splits;
  const int t0 = split * per, n = max(0, min(tiles, t0 + per) - t0);
  const int64_t qrow = (int64_t)b * p.H + head0;

  if (n == 0) {  // a share without keys: nothing to merge
    if (p.splits > 1 && half == 0 && threadIdx.x < rows) p.part_lse[(qrow + threadIdx.x) * p.splits + split] = -INFINITY;
  } else if (warp == 0 || warp >= 6) {
    // ---- loads: the gathers of a tile are shared out over the warps ----
    const int w = warp == 0 ? 0 : warp - 5;
    if (w == 0 && elect_one()) {
      mbar_expect_tx(q_full, QBLOCKS * QBLOCK);
#pragma unroll
      for (int c = 0; c < QBLOCKS; ++c) {
        const bool pe = Q_TMEM + c * 64 >= LAT;
        tma_load_2d(smem_base + c * QBLOCK, pe ? &tmPe : &tmQ, q_full, pe ? 0 : Q_TMEM + c * 64, (int)qrow);
      }
    }
    __syncwarp();
    const int* table = p.req_to_token + (int64_t)LLB_CHECK_REQ(p.b_req_idx[b]) * p.r2t_stride;
    // quad q of four keys of block c: item c * 16 + q goes to warp item % LOADERS, lane item / LOADERS
    constexpr int ITEMS = KBLOCKS * (BN / 4);
    static_assert(ITEMS <= 32 * LOADERS && BN / 4 == 16, "one gather per lane and tile");
    const int item = lane * LOADERS + w, quad = item & 15, c = item >> 4;
    const bool active = item < ITEMS;
    int next[4];
    auto fetch = [&](int j) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int pos = (t0 + j) * BN + quad * 4 + e;
        next[e] = active && pos < kv_len ? LLB_CHECK_SLOT(table[pos]) : p.n_slots;  // out of range: reads zeros
      }
    };
    fetch(0);
    for (int j = 0; j < n; ++j) {
      const int s = j & 1;
      const int r0 = next[0], r1 = next[1], r2 = next[2], r3 = next[3];
      if (j + 1 < n) fetch(j + 1);
      if (!__all_sync(0xffffffffu, mbar_wait(empty(s), ((j >> 1) & 1) ^ 1, abort_flag, p.status, 81))) break;
      if (w == 0 && lane == 0) mbar_expect_tx(full(s), STAGE);
      if (active) tma_gather4(smem_base + OFF_K + s * STAGE + c * BLOCK + quad * 512, &tmKV, full(s), c * 64, r0, r1, r2, r3);
      __syncwarp();
    }
  } else if (warp == 1) {
    if (elect_one()) {
      // ---- MMA issuer (MMAs of one thread run in the order they are issued) ----
      constexpr uint32_t IDESC_S = umma_idesc(128, BN, 1);
      constexpr uint32_t IDESC_PV = umma_idesc(128, 64, 1) | (1u << 16);  // B operand MN-major
      auto scores = [&](int j) {
        const uint32_t k = smem_base + OFF_K + (j & 1) * STAGE;
        if (!mbar_wait(full(j & 1), (j >> 1) & 1, abort_flag, p.status, 82)) return false;
        tc_fence_after();
        const uint32_t d = tmem_base + S_COL + (j & 1) * BN;
        const uint64_t dk = umma_smem_desc_sw128(k), dq = umma_smem_desc_sw128(smem_base);  // offsets count 16-byte units
#pragma unroll
        for (int i = 0; i < ROW / 16; ++i) {
          const uint64_t kd = dk + ((i >> 2) * (BLOCK / 16) + (i & 3) * 2);
          if (i * 16 < Q_TMEM)
            umma_bf16_ts(d, tmem_base + Q_COL + i * 8, kd, IDESC_S, i != 0);
          else
            umma_bf16(d, dq + (((i - Q_TMEM / 16) >> 2) * (QBLOCK / 16) + (i & 3) * 2), kd, IDESC_S, 1);
        }
        umma_commit(s_full(j & 1));
        return true;
      };
      const bool ready = mbar_wait(q_full, 0, abort_flag, p.status, 83) && mbar_wait(qt_full, 0, abort_flag, p.status, 84);
      tc_fence_after();
      const bool first = ready && scores(0);
      for (int j = 0; j < n && first; ++j) {  // a wait that ran out: nothing more is issued
        if (j + 1 < n && !scores(j + 1)) break;
        if (!mbar_wait(p_full(j & 1), (j >> 1) & 1, abort_flag, p.status, 85)) break;
        tc_fence_after();
        const uint32_t v = smem_base + OFF_K + (j & 1) * STAGE + half * 4 * BLOCK;
        const uint64_t dv = umma_smem_desc_sw128_mn(v);
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < BN / 16; ++i)
            umma_bf16_ts(tmem_base + O_COL + c * 64, tmem_base + S_COL + (j & 1) * BN + i * 8, dv + (c * (BLOCK / 16) + i * 128),
                         IDESC_PV, (j | i) != 0);
        umma_commit(o_full);
        umma_commit(empty(j & 1));
      }
      umma_commit(done);
    }
    __syncwarp();
  } else {
    // ---- softmax: one thread per head ----
    const int lane_grp = warp & 3, row = lane_grp * 32 + lane;
    const uint32_t t_lane = tmem_base + ((uint32_t)(lane_grp * 32) << 16);
    {
      const uint4* src = reinterpret_cast<const uint4*>(p.q_lat + (qrow + row) * LAT);
#pragma unroll
      for (int c = 0; c < Q_TMEM / 64; ++c) {
        uint32_t w[32];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const uint4 v = row < rows ? src[c * 8 + e] : make_uint4(0u, 0u, 0u, 0u);
          w[4 * e] = v.x, w[4 * e + 1] = v.y, w[4 * e + 2] = v.z, w[4 * e + 3] = v.w;
        }
        tmem_st_32x32(t_lane + Q_COL + c * 32, w);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(qt_full);
    }
    float m = -INFINITY, l = 0.f;
    for (int j = 0; j < n; ++j) {
      const uint32_t t_s = t_lane + S_COL + (j & 1) * BN;
      if (!__all_sync(0xffffffffu, mbar_wait(s_full(j & 1), (j >> 1) & 1, abort_flag, p.status, 86))) break;
      tc_fence_after();
      uint32_t s[BN];
      tmem_ld_32x32(t_s, s);
      tmem_ld_32x32(t_s + 32, s + 32);
#pragma unroll
      for (int c = 0; c < BN; c += 16) tmem_wait_ld_of(s + c);
      const int lim = kv_len - (t0 + j) * BN;  // keys of this tile
      if (lim < BN) {
#pragma unroll
        for (int c = 0; c < BN; ++c)
          if (c >= lim) s[c] = 0xff800000u;
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < BN; ++c) mx[c & 3] = fmaxf(mx[c & 3], __uint_as_float(s[c]));
      const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale_log2;
      const bool moved = top > m || m == -INFINITY;
      if (__any_sync(0xffffffffu, moved)) {
        const float m_new = moved ? fmaxf(m, top) : m;
        if (j > 0) {  // O holds the tiles before this one
          const float alpha = m_new == m ? 1.f : ex2_fast(m - m_new);
          l *= alpha;
          mbar_wait(o_full, (j - 1) & 1, abort_flag, p.status, 87);  // s_full of tile j came after P . V of tile j - 2: one phase behind
          tc_fence_after();
          tmem_scale<256>(t_lane + O_COL, alpha);
        }
        m = m_new;
      }
      const float base = m == -INFINITY ? 0.f : m;
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t w[32];
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        const float x = ex2_fast(fmaf(__uint_as_float(s[2 * c]), p.scale_log2, -base));
        const float y = ex2_fast(fmaf(__uint_as_float(s[2 * c + 1]), p.scale_log2, -base));
        sum[(2 * c) & 3] += x;
        sum[(2 * c + 1) & 3] += y;
        w[c] = pack_bf16x2(x, y);
      }
      tmem_st_32x32(t_s, w);
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full(j & 1));
    }
    // not o_full: the scores of the last tile were issued ahead of the last but one P . V, so o_full may be two phases behind here
    const int valid = __all_sync(0xffffffffu, mbar_wait(done, 0, abort_flag, p.status, 88)) && !*abort_flag ? rows : 0;  // rows to store
    tc_fence_after();
    // output through the (now idle) query blocks: a warp parks 32 rows x 64 columns and writes whole lines
    const float inv = l > 0.f ? 1.f / l : 0.f;
    float* stg = reinterpret_cast<float*>(smem + lane_grp * (32 * 260));  // 32 rows x 65 floats
    if (p.splits > 1 && half == 0 && row < valid)
      p.part_lse[(qrow + row) * p.splits + split] = l > 0.f ? (m + log2f(l)) / kLog2e : -INFINITY;
#pragma unroll 1
    for (int c = 0; c < 256; c += 64) {
#pragma unroll
      for (int u = 0; u < 64; u += 32) {
        uint32_t r[32];
        tmem_ld_32x32(t_lane + O_COL + c + u, r);
        tmem_wait_ld_of(r);
        tmem_wait_ld_of(r + 16);
#pragma unroll
        for (int e = 0; e < 32; ++e) stg[lane * 65 + u + e] = __uint_as_float(r[e]) * inv;
      }
      __syncwarp();
      const int col = half * 256 + c + lane * 2;
      for (int r = 0; r < 32; ++r) {
        const int hr = lane_grp * 32 + r;
        if (hr >= valid) break;
        const float x = stg[r * 65 + lane * 2], y = stg[r * 65 + lane * 2 + 1];
        if (p.splits == 1)
          *reinterpret_cast<uint32_t*>(p.out + (qrow + hr) * LAT + col) = pack_bf16x2(x, y);
        else
          *reinterpret_cast<float2*>(p.part_o + ((qrow + hr) * p.splits + split) * LAT + col) = make_float2(x, y);
      }
      __syncwarp();
    }
    tc_fence_before();
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) settle_after_abort();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// out[row] = sum of the shares' outputs, weighted by exp(lse - max)
__global__ void __launch_bounds__(128)
mla_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_lse, bf16* __restrict__ out, int splits) {
  pdl_wait();
  const int64_t row = blockIdx.x;
  const int d = threadIdx.x * 4;
  const float* lse = part_lse + row * splits;
  float M = -INFINITY;
  for (int s = 0; s < splits; ++s) M = fmaxf(M, lse[s]);
  float4 num = make_float4(0.f, 0.f, 0.f, 0.f);
  float den = 0.f;
  for (int s = 0; s < splits; ++s) {
    if (lse[s] == -INFINITY) continue;  // its partial row was never written
    const float w = __expf(lse[s] - M);
    const float4 v = *reinterpret_cast<const float4*>(part_o + (row * splits + s) * LAT + d);
    num.x += w * v.x, num.y += w * v.y, num.z += w * v.z, num.w += w * v.w;
    den += w;
  }
  const float inv = den > 0.f ? 1.f / den : 0.f;
  *reinterpret_cast<uint2*>(out + row * LAT + d) =
      make_uint2(pack_bf16x2(num.x * inv, num.y * inv), pack_bf16x2(num.z * inv, num.w * inv));
}

}  // namespace

// q_lat [T, H, 512] contiguous, q_pe [T, H, 64] with qpe_st = H * qpe_sh, pool rows [n_slots, 576]; token t belongs to request t, which
// sees b_ready_len[t] + (t - cu_q[t]) + 1 positions.  splits: shares of a request's keys (1: no scratch).
LLB_EXPORT int llb_mla_decode(const void* q_lat, const void* q_pe, int64_t qpe_st, int64_t qpe_sh, const void* kv_layer, int n_slots,
                              const int* req_to_token, int64_t r2t_stride, const int* b_req_idx, const int* cu_q,
                              const int* b_ready_len, void* out, float* part_o, float* part_lse, int T, int H, int splits,
                              float scale, int* status, cudaStream_t st) {
  if (T <= 0) return LLB_OK;
  if (H <= 0 || T > 65535 || splits < 1 || splits > 64 || qpe_st != (int64_t)H * qpe_sh || !(scale > 0.f)) return LLB_ERR_UNSUPPORTED;
  if (splits > 1 && (part_o == nullptr || part_lse == nullptr)) return LLB_ERR_BAD_ARG;
  if (((uintptr_t)q_lat & 15) || ((uintptr_t)out & 15) || n_slots <= 0) return LLB_ERR_BAD_ARG;
  CUtensorMap tq, tp, tkv;
  int rc = make_tmap_2d(&tq, q_lat, 2, (uint64_t)T * H, LAT, LAT, 128, 64);
  if (rc) return rc;
  rc = make_tmap_2d(&tp, q_pe, 2, (uint64_t)T * H, ROPE, (uint64_t)qpe_sh, 128, 64);
  if (rc) return rc;
  rc = make_tmap_2d(&tkv, kv_layer, 2, (uint64_t)n_slots, ROW, ROW, 1, 64);
  if (rc) return rc;
  static DeviceOnce configured;
  if (!configured.done()) {
    cudaError_t e = cudaFuncSetAttribute(mla_decode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
    configured.set();
  }
  const Params p{(const bf16*)q_lat, req_to_token, b_req_idx, cu_q, b_ready_len, r2t_stride, (bf16*)out, part_o, part_lse, status,
                 H, n_slots, splits, scale * kLog2e};
  cudaError_t e = launch_pdl(mla_decode_kernel, dim3(2 * splits, T, cdiv(H, 128)), dim3(THREADS), SMEM, st, tq, tp, tkv, p);
  if (e != cudaSuccess) return (int)e;
  if (splits > 1) {
    e = launch_pdl(mla_merge_kernel, dim3((unsigned)(T * H)), dim3(128), 0, st, (const float*)part_o, (const float*)part_lse, (bf16*)out,
                   splits);
    if (e != cudaSuccess) return (int)e;
  }
  return LLB_OK;
}
